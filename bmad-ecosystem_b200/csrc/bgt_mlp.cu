// bgt_mlp.cu -- survival classifier for pruning dynamic-aperture scans:
// feature extraction from tracked particles, a 64-256-256-256-1 MLP whose
// hidden layers are tcgen05 tensor-core GEMMs (BF16 operands, FP32
// accumulators in tensor memory), the output layer / loss / Adam on CUDA
// cores.  C ABI in include/bgt_mlp.h.  No counterpart in the reference.
//
// Inference is one kernel for all layers (forward_kernel, below).  Training
// runs a launch per layer and weight gradient of the GEMM kernel, with the
// output layer, the column sums and one pass over the parameters beside them
// (train_batch).
//
// GEMM kernel (gemm_kernel<NT, EPI, BRES>): C = A[M][K] . B[NT][K]^T with
// both operands K-major (row-major, K contiguous), in 128 x NT output tiles
// (NT = 256, or 64 for the first layer's weight gradient), optionally split
// over K (weight gradients over the batch: each split writes its own FP32
// partial tile).  Persistent: min(tiles, SMs) CTAs walk the tiles in a
// static round robin.  BRES (one split, K <= 256: the forward and
// backward-data layers, where B is the layer's weights): B is loaded into
// shared memory once per CTA and only A streams through the ring.  Ten
// warps, each with one job:
//   warp 0     TMA producer: one lane issues cp.async.bulk.tensor loads of
//              the 128 x 64 block of A and the NT x 64 block of B into a
//              ring of shared-memory stages (128-byte swizzle, the canonical
//              K-major layout the MMA reads), completing on the stage's
//              "full" mbarrier;
//   warp 1     MMA issuer: owns the tensor memory; one lane waits for a full
//              stage, issues four tcgen05.mma (M=128, N=NT, K=16) into the
//              tile's accumulator and commits them to the stage's "empty"
//              mbarrier (the producer refills it when they complete); after
//              the tile's last block it commits to the accumulator's "full"
//              mbarrier;
//   warps 2-9  epilogue: each warp owns the 32 tensor-memory lanes (tile
//              rows) of its warp index mod 4 and half of the columns; it
//              reads 64 FP32 columns at a time with tcgen05.ld, applies the
//              layer's epilogue (bias from shared memory; the ReLU mask
//              requested before the tensor-memory load), writes each 32 x 32
//              block into its swizzled shared-memory staging buffer and
//              stores it with a TMA tensor store.
// The accumulator is double-buffered in tensor memory (2 x NT columns), so
// the epilogue of one tile runs while the MMAs of the next tile do.
// Epilogues:
//   EPI_FWD  bias + ReLU -> bf16 row-major and (optionally) a transposed copy
//   EPI_BWD  ReLU mask of the previous activation -> bf16 row-major / transposed
//   EPI_F32  FP32 tile (the test GEMM; split-K partials of weight gradients)
// Every TMA load is a plain per-CTA load of this GPU's own memory: each CTA
// loads its own tiles, none is shared across a cluster.
// Every mbarrier wait is bounded (%globaltimer, 2 s by default).  A role
// whose wait runs out sets the error flag and leaves its loop; the roles
// waiting on it then run out too.  Before the tensor memory is freed the MMA
// lane waits (bounded) for its own MMAs and the producer for its own loads,
// so nothing is in flight when the CTA exits.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/bgt.h"
#include "../../include/bgt_mlp.h"

namespace bgt {
namespace mlp {

typedef __nv_bfloat16 bf16;

constexpr int BM = 128;
constexpr int BK = 64;
#ifndef BGT_GEMM_EPI_WARPS
#define BGT_GEMM_EPI_WARPS 8
#endif
constexpr int EPI_WARPS = BGT_GEMM_EPI_WARPS;  // 4 or 8: one or two warps per tensor-memory lane quarter
constexpr int THREADS = 64 + 32 * EPI_WARPS;   // producer warp, MMA warp, epilogue warps
constexpr int H = BGT_MLP_HIDDEN;
constexpr int IN = BGT_MLP_IN;
constexpr int KSPLIT = 128;  // fewest samples per split-K chunk of a weight gradient

// flat parameter layout
constexpr int64_t OFF_W1 = 0;
constexpr int64_t OFF_B1 = OFF_W1 + (int64_t)H * IN;
constexpr int64_t OFF_W2 = OFF_B1 + H;
constexpr int64_t OFF_B2 = OFF_W2 + (int64_t)H * H;
constexpr int64_t OFF_W3 = OFF_B2 + H;
constexpr int64_t OFF_B3 = OFF_W3 + (int64_t)H * H;
constexpr int64_t OFF_W4 = OFF_B3 + H;
constexpr int64_t OFF_B4 = OFF_W4 + H;
constexpr int64_t N_PARAMS = OFF_B4 + 1;
static_assert(N_PARAMS == BGT_MLP_N_PARAMS, "parameter layout");

enum { EPI_FWD = 0, EPI_BWD = 1, EPI_F32 = 2 };

// ---------------------------------------------------------------------------
// PTX wrappers

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}
// Wait for the phase of `parity` to complete; false after limit_ns.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, uint64_t limit_ns) {
  if (mbar_try_wait(bar, parity)) return true;
  const uint64_t t0 = global_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (global_ns() - t0 > limit_ns) return false;
  }
  return true;
}

// TMA: 2-D tile load into this CTA's shared memory, completing on an
// mbarrier, and 2-D tile store from shared memory in a bulk group
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int32_t x, int32_t y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(
          dst),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int32_t x, int32_t y, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];\n" ::"l"(
                   reinterpret_cast<uint64_t>(map)),
               "r"(x), "r"(y), "r"(src)
               : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// at most N of this thread's store groups still reading shared memory
template <int N>
__device__ __forceinline__ void bulk_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory");
}
// all of this thread's store groups complete
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void prefetch_map(const CUtensorMap* map) {
  asm volatile("prefetch.tensormap [%0];\n" ::"l"(reinterpret_cast<uint64_t>(map)) : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(dst_smem), "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// D[tmem] (+)= A[smem desc] . B[smem desc]^T, kind::f16 (bf16 in, f32 accumulate)
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// arrive (once) on `bar` when every MMA this thread issued so far has completed
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar)
               : "memory");
}
// 32 consecutive FP32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// 64 consecutive FP32 columns of this thread's tensor-memory lane
__device__ __forceinline__ void tmem_ld64(uint32_t taddr, uint32_t (&r)[64]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x64.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, "
      "%32, %33, %34, %35, %36, %37, %38, %39, %40, %41, %42, %43, %44, %45, %46, %47, "
      "%48, %49, %50, %51, %52, %53, %54, %55, %56, %57, %58, %59, %60, %61, %62, %63}, [%64];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31]),
        "=r"(r[32]), "=r"(r[33]), "=r"(r[34]), "=r"(r[35]), "=r"(r[36]), "=r"(r[37]), "=r"(r[38]), "=r"(r[39]),
        "=r"(r[40]), "=r"(r[41]), "=r"(r[42]), "=r"(r[43]), "=r"(r[44]), "=r"(r[45]), "=r"(r[46]), "=r"(r[47]),
        "=r"(r[48]), "=r"(r[49]), "=r"(r[50]), "=r"(r[51]), "=r"(r[52]), "=r"(r[53]), "=r"(r[54]), "=r"(r[55]),
        "=r"(r[56]), "=r"(r[57]), "=r"(r[58]), "=r"(r[59]), "=r"(r[60]), "=r"(r[61]), "=r"(r[62]), "=r"(r[63])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: start address
// (>> 4), leading byte offset 1 (unused for swizzled K-major), stride byte
// offset 1024 B between 8-row atoms, descriptor version 1, layout type 2.
// The TMA's 128-byte swizzle writes exactly this layout: row r of a block
// at r * 128 bytes, its 16-byte chunk c at chunk c ^ (r % 8).
__device__ __forceinline__ uint64_t sw128_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// The same with a 64-byte swizzle: rows of 64 bytes, atoms of 8 rows 512 B
// apart, layout type 4.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// Instruction descriptor, kind::f16: FP32 accumulator (bits 4-5 = 1), A and
// B BF16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

// ---------------------------------------------------------------------------
// GEMM

struct Epi {
  const float* bias;   // EPI_FWD: [N]
  bf16* out_t;         // optional transposed copy [N][ldt] (EPI_FWD / EPI_BWD)
  int64_t ldt;
  const bf16* mask;    // EPI_BWD: previous activation, row-major [M][ldm]
  int64_t ldm;
};

// Shared memory of one CTA: [stationary B: K <= 256, one split only]
// [ring of STAGES stages: A block, and the B block when B is not stationary]
// [one 32 x 32 output staging buffer per epilogue warp] + alignment slack.
template <int NT, bool BRES>
struct GemmCfg {
  static constexpr uint32_t A_BYTES = BM * BK * 2;
  static constexpr uint32_t B_BYTES = NT * BK * 2;
  static constexpr int BRES_BLOCKS = 4;  // K blocks of a stationary B (K <= 256)
  static constexpr uint32_t BRES_BYTES = BRES ? BRES_BLOCKS * B_BYTES : 0;
  static constexpr uint32_t STAGE_BYTES = BRES ? A_BYTES : A_BYTES + B_BYTES;
  static constexpr uint32_t EPI_BUF = 4096;  // 32 x 32 FP32 (or bf16) output block
  static constexpr uint32_t EPI_BYTES = EPI_WARPS * EPI_BUF;
  static constexpr uint32_t TMEM_COLS = 2 * NT;
  static constexpr int COLS_PER_WARP = NT / (EPI_WARPS / 4);  // accumulator columns one epilogue warp drains
  // as many stages as fit (at most 6), leaving 2 KB for the static shared
  // memory and 1 KB of alignment slack
  static constexpr int STAGES_FIT = (int)((232448u - 2048u - EPI_BYTES - BRES_BYTES) / STAGE_BYTES);
  static constexpr int STAGES = STAGES_FIT < 6 ? STAGES_FIT : 6;
  static constexpr int SMEM = BRES_BYTES + STAGES * STAGE_BYTES + EPI_BYTES + 1024;
};
static_assert(EPI_WARPS == 4 || EPI_WARPS == 8, "epilogue warps");
static_assert(GemmCfg<256, false>::STAGES >= 4 && GemmCfg<256, true>::STAGES >= 4 &&
                  GemmCfg<64, false>::COLS_PER_WARP >= 32,
              "GEMM configuration");
static_assert(GemmCfg<256, false>::SMEM <= 230400 && GemmCfg<256, true>::SMEM <= 230400, "shared memory per CTA");

__device__ int g_gemm_error;

// Tile t of a (m_tiles x splits) grid: rows mt * 128, K blocks [kb0, kb1)
// of split sp.  Every split has at least one K block (host check).
struct TileIdx {
  int mt, sp, kb0, kb1;
};
__device__ __forceinline__ TileIdx tile_of(int t, int m_tiles, int splits, int kb_total) {
  TileIdx r;
  r.mt = t % m_tiles;
  r.sp = t / m_tiles;
  r.kb0 = (int)((int64_t)r.sp * kb_total / splits);
  r.kb1 = (int)((int64_t)(r.sp + 1) * kb_total / splits);
  return r;
}

// BRES: B (the layer's weights in the forward and backward-data GEMMs) is
// loaded into shared memory once per CTA and stays there for all its tiles;
// only A streams through the ring.  Needs one split and K <= 256.
template <int NT, int EPI, bool BRES>
__global__ void __launch_bounds__(THREADS, 1)
    gemm_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                const __grid_constant__ CUtensorMap tmC, int m_tiles, int splits, int kb_total, Epi ep, int* err,
                uint64_t wait_ns, int skip_mma) {
  using C = GemmCfg<NT, BRES>;
  constexpr int S = C::STAGES;
  constexpr uint32_t IDESC = idesc_bf16(BM, NT);
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[S], empty_bar[S], acc_full[2], acc_empty[2], done_bar, bres_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float bias_s[EPI == EPI_FWD ? NT : 1];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t ring = base + C::BRES_BYTES;  // stage s at ring + s * STAGE_BYTES
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_tiles = m_tiles * splits;

  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), C::TMEM_COLS);
    tmem_relinquish();
  }
  // Launched as a programmatic dependent of the previous kernel on the
  // stream: everything above runs while that kernel drains; no global
  // memory is touched before the previous grid has completed and its writes
  // are visible.  Then this grid lets the next one begin its own launch.
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  if (EPI == EPI_FWD) {
    for (int j = tid; j < NT; j += THREADS) bias_s[j] = ep.bias[j];
  }
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(smem_u32(&acc_full[b]), 1);
      mbar_init(smem_u32(&acc_empty[b]), EPI_WARPS);  // one arrival per epilogue warp
    }
    mbar_init(smem_u32(&done_bar), 1);
    mbar_init(smem_u32(&bres_bar), 1);
    fence_mbar_init();
    prefetch_map(&tmA);
    prefetch_map(&tmB);
    prefetch_map(&tmC);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  bool ok = true;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      if (BRES) {
        // the stationary B: all its K blocks on one barrier
        mbar_arrive_expect_tx(smem_u32(&bres_bar), (uint32_t)kb_total * C::B_BYTES);
        for (int kb = 0; kb < kb_total; kb++)
          tma_load_2d(base + (uint32_t)kb * C::B_BYTES, &tmB, kb * BK, 0, smem_u32(&bres_bar));
      }
      int it = 0;  // ring loads issued
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        const TileIdx ti = tile_of(t, m_tiles, splits, kb_total);
        for (int kb = ti.kb0; kb < ti.kb1; kb++) {
          const int s = it % S;
          const uint32_t ph = (uint32_t)(it / S) & 1u;
          // the stage's previous MMAs are done (the first pass waits on the
          // phase before the barrier's first, which counts as complete)
          if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1u, wait_ns)) {
            ok = false;
            break;
          }
          const uint32_t sa = ring + (uint32_t)s * C::STAGE_BYTES;
          const uint32_t fb = smem_u32(&full_bar[s]);
          mbar_arrive_expect_tx(fb, C::STAGE_BYTES);
          tma_load_2d(sa, &tmA, kb * BK, ti.mt * BM, fb);
          if (!BRES) tma_load_2d(sa + C::A_BYTES, &tmB, kb * BK, 0, fb);
          it++;
        }
      }
      // every load issued has landed before the CTA can exit (bounded)
      for (int s = 0; s < S && s < it; s++) {
        const int last = it - 1 - ((it - 1 - s) % S);  // the last load into stage s
        mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(last / S) & 1u, wait_ns);
      }
      if (BRES) mbar_wait(smem_u32(&bres_bar), 0u, wait_ns);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int it = 0, tc = 0;
      bool issued = false;
      if (BRES && !mbar_wait(smem_u32(&bres_bar), 0u, wait_ns)) ok = false;
      for (int t = blockIdx.x; t < n_tiles && ok; t += gridDim.x, tc++) {
        const TileIdx ti = tile_of(t, m_tiles, splits, kb_total);
        const int b = tc & 1;
        const uint32_t tph = (uint32_t)(tc >> 1) & 1u;
        // the epilogue has drained this accumulator buffer
        if (!mbar_wait(smem_u32(&acc_empty[b]), tph ^ 1u, wait_ns)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t d = tmem + (uint32_t)(b * NT);
        for (int kb = ti.kb0; kb < ti.kb1; kb++, it++) {
          const int s = it % S;
          if (!mbar_wait(smem_u32(&full_bar[s]), (uint32_t)(it / S) & 1u, wait_ns)) {
            ok = false;
            break;
          }
          tc_fence_after();
          // skip_mma (tests only): no MMA and no commit are issued, so the
          // other roles' waits run out with nothing outstanding
          if (!skip_mma) {
            const uint32_t sa = ring + (uint32_t)s * C::STAGE_BYTES;
            const uint32_t sb = BRES ? base + (uint32_t)kb * C::B_BYTES : sa + C::A_BYTES;
#pragma unroll
            for (int k = 0; k < BK / 16; k++) {
              // K step of 16 bf16 = 32 bytes inside the 128-byte swizzle atom
              mma_bf16(d, sw128_desc(sa + k * 32), sw128_desc(sb + k * 32), IDESC,
                       (kb > ti.kb0 || k > 0) ? 1u : 0u);
            }
            mma_commit(smem_u32(&empty_bar[s]));
            issued = true;
          }
        }
        if (!ok) break;
        if (!skip_mma) mma_commit(smem_u32(&acc_full[b]));
      }
      // every MMA issued has completed before tensor memory is freed (bounded)
      if (issued) {
        mma_commit(smem_u32(&done_bar));
        mbar_wait(smem_u32(&done_bar), 0u, wait_ns);
      }
    }
  } else {
    // ---------------- epilogue ----------------
    const int q = warp & 3;  // tensor-memory lanes 32q .. 32q + 31 = tile rows
    const int col0 = ((warp - 2) >> 2) * C::COLS_PER_WARP;  // this warp's accumulator columns
    constexpr int GROUP = C::COLS_PER_WARP >= 64 ? 64 : 32;  // columns per tensor-memory load
    const uint32_t buf = ring + (uint32_t)S * C::STAGE_BYTES + (uint32_t)(warp - 2) * C::EPI_BUF;
    uint8_t* buf_ptr = base_ptr + (buf - base);
    int tc = 0;
    for (int t = blockIdx.x; t < n_tiles; t += gridDim.x, tc++) {
      const TileIdx ti = tile_of(t, m_tiles, splits, kb_total);
      const int b = tc & 1;
      const int64_t row = (int64_t)ti.mt * BM + q * 32 + lane;  // this lane's output row
      const bool w = mbar_wait(smem_u32(&acc_full[b]), (uint32_t)(tc >> 1) & 1u, wait_ns);
      if (!__all_sync(0xffffffffu, w)) {
        ok = false;
        break;
      }
      tc_fence_after();
      // row of the 32 x 32 store box in the output map
      const int32_t ybox = (EPI == EPI_F32 ? ti.sp * m_tiles * BM : 0) + ti.mt * BM + q * 32;
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * NT);
#pragma unroll 1
      for (int g0 = col0; g0 < col0 + C::COLS_PER_WARP; g0 += GROUP) {
        // EPI_BWD: the ReLU mask of this group's columns, requested before
        // the tensor-memory load so the two latencies overlap
        uint4 mk[GROUP / 8];
        if (EPI == EPI_BWD) {
          const uint4* mp = reinterpret_cast<const uint4*>(ep.mask + row * ep.ldm + g0);
#pragma unroll
          for (int c = 0; c < GROUP / 8; c++) mk[c] = mp[c];
        }
        uint32_t r[64];
        if (GROUP == 64) {
          tmem_ld64(taddr + g0, r);
        } else {
          tmem_ld32(taddr + g0, *reinterpret_cast<uint32_t(*)[32]>(r));
        }
        if (g0 + GROUP == col0 + C::COLS_PER_WARP) {
          // this warp's part of the accumulator buffer is read: the next
          // tile's MMAs may overwrite it
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&acc_empty[b]));
        }
#pragma unroll
        for (int h = 0; h < GROUP / 32; h++) {
          const int c0 = g0 + 32 * h;
          float v[32];
#pragma unroll
          for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[32 * h + j]);
          // the staging buffer's previous store has finished reading it
          if (lane == 0) bulk_wait_read<0>();
          __syncwarp();
          if (EPI == EPI_F32) {
            // 32 rows x 128 bytes, 128-byte swizzle: chunk c of row r at c ^ (r % 8)
#pragma unroll
            for (int c = 0; c < 8; c++)
              *reinterpret_cast<float4*>(buf_ptr + lane * 128 + ((c ^ (lane & 7)) << 4)) =
                  make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
          } else {
            if (EPI == EPI_FWD) {
#pragma unroll
              for (int c = 0; c < 8; c++) {
                const float4 bb = *reinterpret_cast<const float4*>(&bias_s[c0 + 4 * c]);
                v[4 * c] = fmaxf(v[4 * c] + bb.x, 0.0f);
                v[4 * c + 1] = fmaxf(v[4 * c + 1] + bb.y, 0.0f);
                v[4 * c + 2] = fmaxf(v[4 * c + 2] + bb.z, 0.0f);
                v[4 * c + 3] = fmaxf(v[4 * c + 3] + bb.w, 0.0f);
              }
            } else {
#pragma unroll
              for (int c = 0; c < 4; c++) {
                const bf16* hh = reinterpret_cast<const bf16*>(&mk[4 * h + c]);
#pragma unroll
                for (int j = 0; j < 8; j++)
                  if (!(__bfloat162float(hh[j]) > 0.0f)) v[8 * c + j] = 0.0f;
              }
            }
            uint4 pk[4];
            bf16* ph = reinterpret_cast<bf16*>(pk);
#pragma unroll
            for (int j = 0; j < 32; j++) ph[j] = __float2bfloat16_rn(v[j]);
            // 32 rows x 64 bytes, 64-byte swizzle: chunk c of row r at c ^ ((r / 2) % 4)
#pragma unroll
            for (int c = 0; c < 4; c++)
              *reinterpret_cast<uint4*>(buf_ptr + lane * 64 + ((c ^ ((lane >> 1) & 3)) << 4)) = pk[c];
            if (ep.out_t) {
#pragma unroll
              for (int j = 0; j < 32; j++) ep.out_t[(int64_t)(c0 + j) * ep.ldt + row] = ph[j];
            }
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) {
            tma_store_2d(&tmC, c0, ybox, buf);
            bulk_commit();
          }
        }
      }
    }
    if (lane == 0) bulk_wait_all();
  }
  if (!ok) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, C::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------------
// Tensor maps (driver entry point, resolved once through the runtime)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = []() -> EncodeTiledFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      return nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// 2-D map of a row-major matrix: `rows` rows of `cols` elements, `ld`
// elements apart; boxes of box_rows x box_cols
static bool make_map(CUtensorMap* map, CUtensorMapDataType dt, size_t esize, const void* ptr, uint64_t cols,
                     uint64_t rows, uint64_t ld, uint32_t box_cols, uint32_t box_rows, CUtensorMapSwizzle sw) {
  EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {ld * esize};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(map, dt, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, sw,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

static int sm_count() {
  int dev = 0, n = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 148;
}

template <int NT, int EPI, bool BRES>
static cudaError_t launch_gemm_kernel(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc, int m_tiles,
                                      int splits, int kb_total, const Epi& ep, int* err, cudaStream_t st,
                                      uint64_t wait_ns, int skip_mma) {
  using C = GemmCfg<NT, BRES>;
  static bool attr_set[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63]) {
    cudaError_t e =
        cudaFuncSetAttribute(gemm_kernel<NT, EPI, BRES>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63] = true;
  }
  const int grid = std::min(m_tiles * splits, sm_count());
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = C::SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, gemm_kernel<NT, EPI, BRES>, ma, mb, mc, m_tiles, splits, kb_total, ep, err,
                            wait_ns, skip_mma);
}

// C = A . B^T over K = k: A [a_rows][lda] bf16 (a_rows a multiple of 128),
// B [NT][ldb] bf16, k a multiple of 64 split into `splits` chunks of whole
// 64-blocks.  Output: EPI_F32 -> out FP32 [splits][a_rows][NT];
// EPI_FWD / EPI_BWD -> out bf16 [a_rows][ldo] (columns 0..NT-1).  With one
// split and K <= 256 the kernel keeps B stationary in shared memory.
template <int NT, int EPI>
static cudaError_t launch_gemm(const bf16* A, int64_t lda, int64_t a_rows, const bf16* B, int64_t ldb, int64_t k,
                               int splits, void* out, int64_t ldo, const Epi& ep, int* err, cudaStream_t st,
                               uint64_t wait_ns = 2000000000ull, int skip_mma = 0) {
  const int m_tiles = (int)(a_rows / BM);
  const int kb_total = (int)(k / BK);
  if (m_tiles <= 0 || kb_total <= 0 || splits <= 0 || splits > kb_total || a_rows % BM || k % BK)
    return cudaErrorInvalidValue;
  CUtensorMap ma, mb, mc;
  bool good = make_map(&ma, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, A, (uint64_t)k, (uint64_t)a_rows, (uint64_t)lda,
                       BK, BM, CU_TENSOR_MAP_SWIZZLE_128B) &&
              make_map(&mb, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, B, (uint64_t)k, (uint64_t)NT, (uint64_t)ldb, BK, NT,
                       CU_TENSOR_MAP_SWIZZLE_128B);
  if (EPI == EPI_F32)
    good = good && make_map(&mc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, out, (uint64_t)NT,
                            (uint64_t)splits * (uint64_t)a_rows, (uint64_t)ldo, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    good = good && make_map(&mc, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, out, (uint64_t)NT, (uint64_t)a_rows,
                            (uint64_t)ldo, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B);
  if (!good) return cudaErrorInvalidValue;
  if (splits == 1 && kb_total <= GemmCfg<NT, true>::BRES_BLOCKS)
    return launch_gemm_kernel<NT, EPI, true>(ma, mb, mc, m_tiles, splits, kb_total, ep, err, st, wait_ns, skip_mma);
  return launch_gemm_kernel<NT, EPI, false>(ma, mb, mc, m_tiles, splits, kb_total, ep, err, st, wait_ns, skip_mma);
}

// ---------------------------------------------------------------------------
// Inference: the three hidden layers and the output layer of 128 rows in one
// CTA, no activation leaving the SM.
//
// As three GEMMs and a head kernel the activations made six trips through L2
// and HBM (134 MB a layer at 262,144 rows), and each launch had its ramp and
// tail.  Here a tile's activations stay in shared memory (a 128 x 256 bf16
// buffer in the MMA's K-major 128-byte-swizzled layout: the input rows first,
// then rewritten by each layer's epilogue) and only the weights stream, 288 KB
// a tile from L2 through a ring of five 16 KB stages (a layer's outputs x 32
// columns, 64-byte swizzle; all three layers do not fit beside the activations).
//
// One tile is a chain MMA -> epilogue -> MMA, 4,600 cycles of it MMA; so a CTA
// holds two tiles, each with its activation buffer and half of tensor memory,
// and the MMA of one can run under the epilogue of the other.  On B200 262,144
// rows take 93 us (three GEMMs and a head 247), 1,152 rows 10.8 (22.5): 12,800
// cycles a tile, against 14,000 with one tile in flight, so little of the chain
// is hidden yet.  Tensor pipe 42 % busy, L2 reads 288 KB a tile (a quarter of
// its rate), DRAM 5 %.
//
// Roles (18 warps): 0 TMA producer, 1 MMA issuer, 2-9 hidden epilogues (two
// per tensor-memory lane quarter, half of the columns each), 10-17 output
// layer (half a row per thread; by four warps, a row per thread, it alone took
// 109 us).  The sums are those of the separate kernels: K blocks in the same
// order, the output layer's 32 partial sums of 8 columns in the order of
// head_kernel's lanes and shuffles.
constexpr int FWD_HIDDEN_WARPS = 8;
constexpr int FWD_COLS = H / (FWD_HIDDEN_WARPS / 4);  // columns a hidden-epilogue warp handles
constexpr int FWD_HEAD = 2 + FWD_HIDDEN_WARPS;         // first output-layer warp
constexpr int FWD_THREADS = 32 * (FWD_HEAD + 8);
constexpr int FWD_STAGES = 5;
constexpr int FWD_WK = BK / 2;                 // columns of a weight stage
constexpr uint32_t FWD_W_BYTES = H * FWD_WK * 2;
constexpr uint32_t FWD_A_BLOCK = BM * BK * 2;  // 64 columns of a tile's activations
constexpr uint32_t FWD_A_BYTES = 4 * FWD_A_BLOCK;
constexpr int FWD_SMEM = FWD_STAGES * FWD_W_BYTES + 2 * FWD_A_BYTES + 1024;

// two ReLU outputs as bf16, the first in the low half
__device__ __forceinline__ uint32_t relu_bf16x2(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(fmaxf(a, 0.0f), fmaxf(b, 0.0f));
  return *reinterpret_cast<const uint32_t*>(&v);
}
// bf16 (a ReLU output) rounded as the stored activation
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__global__ void __launch_bounds__(FWD_THREADS, 1)
    forward_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW1,
                   const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmW3, int n_tiles,
                   const float* __restrict__ params, float* __restrict__ prob, int* err, uint64_t wait_ns) {
  constexpr int S = FWD_STAGES;
  constexpr uint32_t IDESC = idesc_bf16(BM, H);
  extern __shared__ uint8_t smem_raw[];
  // per slot p (tile in flight): x_full input rows landed, a_free its buffer
  // may be loaded again, a_full block of activations written (two phases a
  // tile), acc_full a layer's accumulators complete, acc_empty drained; per
  // lane quarter, head_full / head_empty the hand-over of partial sums
  __shared__ __align__(8) uint64_t w_full[S], w_empty[S], x_full[2], a_free[2], a_full[2], acc_full[2][3],
      acc_empty[2], head_full[4], head_empty[4], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ __align__(16) float bias_s[3][H], w4_s[H];
  __shared__ float head_s[8][BM];  // partial sums handed from one half of an output row to the other
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* base_ptr = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t a_off = S * FWD_W_BYTES;  // slot p's activations at a_off + p * FWD_A_BYTES
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 1) {
    tmem_alloc(smem_u32(&tmem_slot), 2 * H);
    tmem_relinquish();
  }
  // launched as a programmatic dependent, as gemm_kernel
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  for (int j = tid; j < H; j += FWD_THREADS) {
    bias_s[0][j] = params[OFF_B1 + j];
    bias_s[1][j] = params[OFF_B2 + j];
    bias_s[2][j] = params[OFF_B3 + j];
    w4_s[j] = round_bf16(params[OFF_W4 + j]);
  }
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(smem_u32(&w_full[s]), 1);
      mbar_init(smem_u32(&w_empty[s]), 1);
    }
    for (int p = 0; p < 2; p++) {
      mbar_init(smem_u32(&x_full[p]), 1);
      mbar_init(smem_u32(&a_free[p]), 1);
      mbar_init(smem_u32(&a_full[p]), FWD_HIDDEN_WARPS);
      for (int k = 0; k < 3; k++) mbar_init(smem_u32(&acc_full[p][k]), 1);
      mbar_init(smem_u32(&acc_empty[p]), FWD_HIDDEN_WARPS);
    }
    for (int k = 0; k < 4; k++) {
      mbar_init(smem_u32(&head_full[k]), 1);
      mbar_init(smem_u32(&head_empty[k]), 1);
    }
    mbar_init(smem_u32(&done_bar), 1);
    fence_mbar_init();
    prefetch_map(&tmX);
    prefetch_map(&tmW1);
    prefetch_map(&tmW2);
    prefetch_map(&tmW3);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  bool ok = true;
  // round i: slot 0 holds tile t0 + 2 i grid, slot 1 the one grid further (if any)
  const int t0 = blockIdx.x, step = gridDim.x;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      int it = 0;            // weight blocks issued
      int nx[2] = {0, 0};    // input tiles issued
      auto load_w = [&](const CUtensorMap* map, int kb) {
        for (int k0 = kb * BK; k0 < (kb + 1) * BK; k0 += FWD_WK, it++) {
          const int s = it % S;
          if (!mbar_wait(smem_u32(&w_empty[s]), ((uint32_t)(it / S) & 1u) ^ 1u, wait_ns)) return false;
          mbar_arrive_expect_tx(smem_u32(&w_full[s]), FWD_W_BYTES);
          tma_load_2d(base + (uint32_t)s * FWD_W_BYTES, map, k0, 0, smem_u32(&w_full[s]));
        }
        return true;
      };
      // slot p's next input rows, once the last layer of its tile has read the buffer
      auto load_x = [&](int p, int t) {
        if (t >= n_tiles) return true;
        if (!mbar_wait(smem_u32(&a_free[p]), ((uint32_t)nx[p] & 1u) ^ 1u, wait_ns)) return false;
        mbar_arrive_expect_tx(smem_u32(&x_full[p]), FWD_A_BLOCK);
        tma_load_2d(base + a_off + (uint32_t)p * FWD_A_BYTES, &tmX, 0, t * BM, smem_u32(&x_full[p]));
        nx[p]++;
        return true;
      };
      for (int t = t0; t < n_tiles && ok; t += 2 * step) {
        const int slots = t + step < n_tiles ? 2 : 1;
        // (the first weights are on their way before a buffer is waited for)
        for (int p = 0; p < slots && ok; p++) ok = load_w(&tmW1, 0) && load_x(p, t + p * step);
        for (int l = 0; l < 2 && ok; l++)
          for (int p = 0; p < slots && ok; p++)
            for (int kb = 0; kb < 4 && ok; kb++) ok = load_w(l == 0 ? &tmW2 : &tmW3, kb);
      }
      // every load issued has landed before the CTA can exit (bounded)
      for (int s = 0; s < S && s < it; s++) {
        const int last = it - 1 - ((it - 1 - s) % S);
        mbar_wait(smem_u32(&w_full[s]), (uint32_t)(last / S) & 1u, wait_ns);
      }
      for (int p = 0; p < 2; p++)
        if (nx[p] > 0) mbar_wait(smem_u32(&x_full[p]), (uint32_t)(nx[p] - 1) & 1u, wait_ns);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer ----------------
    if (lane == 0) {
      int it = 0, i = 0;  // weight blocks and rounds so far
      bool issued = false;
      for (int t = t0; t < n_tiles && ok; t += 2 * step, i++) {
        const int slots = t + step < n_tiles ? 2 : 1;
        for (int layer = 0; layer < 3 && ok; layer++) {
          for (int p = 0; p < slots && ok; p++) {
            // the slot's accumulators are drained (its use 3 i + layer)
            if (!mbar_wait(smem_u32(&acc_empty[p]), ((uint32_t)(3 * i + layer) & 1u) ^ 1u, wait_ns)) ok = false;
            const uint32_t d = tmem + (uint32_t)(p * H);
            // its input rows or activations are in place
            if (ok && !(layer == 0 ? mbar_wait(smem_u32(&x_full[p]), (uint32_t)i & 1u, wait_ns)
                                   : mbar_wait(smem_u32(&a_full[p]), (uint32_t)(layer - 1) & 1u, wait_ns)))
              ok = false;
            for (int kb = 0; kb < (layer == 0 ? 1 : 4) && ok; kb++) {
              const uint32_t sa = base + a_off + (uint32_t)p * FWD_A_BYTES + (uint32_t)kb * FWD_A_BLOCK;
              for (int k0 = 0; k0 < BK && ok; k0 += FWD_WK, it++) {
                const int s = it % S;
                if (!mbar_wait(smem_u32(&w_full[s]), (uint32_t)(it / S) & 1u, wait_ns)) {
                  ok = false;
                  break;
                }
                tc_fence_after();
                const uint32_t sb = base + (uint32_t)s * FWD_W_BYTES;
#pragma unroll
                for (int k = 0; k < FWD_WK / 16; k++)
                  mma_bf16(d, sw128_desc(sa + 2 * k0 + k * 32), sw64_desc(sb + k * 32), IDESC,
                           (kb > 0 || k0 > 0 || k > 0) ? 1u : 0u);
                mma_commit(smem_u32(&w_empty[s]));
                issued = true;
              }
            }
            if (ok) mma_commit(smem_u32(&acc_full[p][layer]));
            if (ok && layer == 2) mma_commit(smem_u32(&a_free[p]));
          }
        }
      }
      // every MMA issued has completed before tensor memory is freed (bounded)
      if (issued) {
        mma_commit(smem_u32(&done_bar));
        mbar_wait(smem_u32(&done_bar), 0u, wait_ns);
      }
    }
  } else {
    const int q = warp & 3;  // tensor-memory lanes 32q .. 32q + 31 = tile rows
    const int row = q * 32 + lane;
    const bool head = warp >= FWD_HEAD;
    const int col0 = head ? 0 : ((warp - 2) >> 2) * FWD_COLS;  // a hidden-epilogue warp's first column
    int i = 0, n_head = 0;  // rounds, hand-overs
    for (int t = t0; t < n_tiles && ok; t += 2 * step, i++) {
      const int slots = t + step < n_tiles ? 2 : 1;
      for (int layer = head ? 2 : 0; layer < (head ? 3 : 2) && ok; layer++) {
        for (int p = 0; p < slots && ok; p++) {
          if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&acc_full[p][layer]), (uint32_t)i & 1u, wait_ns))) {
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(p * H);
          if (!head) {
            // ---------------- hidden epilogue: bias, ReLU, bf16 into the activation buffer
#pragma unroll 1
            for (int c0 = col0; c0 < col0 + FWD_COLS; c0 += 32) {
              uint32_t r[32];
              tmem_ld32(taddr + c0, r);
              uint8_t* dst = base_ptr + a_off + p * FWD_A_BYTES + (c0 / BK) * FWD_A_BLOCK + row * 128;
              const int chunk = (c0 % BK) / 8;
#pragma unroll
              for (int c = 0; c < 4; c++) {
                uint32_t pk[4];
#pragma unroll
                for (int j = 0; j < 8; j += 4) {
                  const float4 bb = *reinterpret_cast<const float4*>(&bias_s[layer][c0 + 8 * c + j]);
                  const uint32_t* v = &r[8 * c + j];
                  pk[j / 2] = relu_bf16x2(__uint_as_float(v[0]) + bb.x, __uint_as_float(v[1]) + bb.y);
                  pk[j / 2 + 1] = relu_bf16x2(__uint_as_float(v[2]) + bb.z, __uint_as_float(v[3]) + bb.w);
                }
                *reinterpret_cast<uint4*>(dst + (((chunk + c) ^ (row & 7)) << 4)) =
                    make_uint4(pk[0], pk[1], pk[2], pk[3]);
              }
            }
            // one fence for all of the warp's stores
            fence_proxy_async();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
              mbar_arrive(smem_u32(&acc_empty[p]));
              mbar_arrive(smem_u32(&a_full[p]));
            }
          } else {
            // ---------------- output layer: half of a row's partial sums
            // (of 8 columns each), l = 8 hb + 0..7 and 16 more
            const int hb = (warp - FWD_HEAD) >> 2;
            float part[16];
#pragma unroll
            for (int k = 0; k < 4; k++) {
              const int c0 = 64 * hb + 32 * (k & 1) + 128 * (k >> 1);
              uint32_t r[32];
              tmem_ld32(taddr + c0, r);
#pragma unroll
              for (int l = 0; l < 4; l++) {
                float acc = 0.0f;
#pragma unroll
                for (int j = 0; j < 8; j += 4) {
                  const int c = c0 + 8 * l + j;
                  const float4 bb = *reinterpret_cast<const float4*>(&bias_s[2][c]);
                  const float4 w = *reinterpret_cast<const float4*>(&w4_s[c]);
                  const uint32_t* v = &r[8 * l + j];
                  const uint32_t a01 = relu_bf16x2(__uint_as_float(v[0]) + bb.x, __uint_as_float(v[1]) + bb.y);
                  const uint32_t a23 = relu_bf16x2(__uint_as_float(v[2]) + bb.z, __uint_as_float(v[3]) + bb.w);
                  acc += __uint_as_float(a01 << 16) * w.x;
                  acc += __uint_as_float(a01 & 0xffff0000u) * w.y;
                  acc += __uint_as_float(a23 << 16) * w.z;
                  acc += __uint_as_float(a23 & 0xffff0000u) * w.w;
                }
                part[4 * k + l] = acc;
              }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&acc_empty[p]));
#pragma unroll
            for (int l = 0; l < 8; l++) part[l] += part[l + 8];
            const uint32_t hand = (uint32_t)n_head++ & 1u;
            if (hb == 1) {
              if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&head_empty[q]), hand ^ 1u, wait_ns))) {
                ok = false;
                break;
              }
#pragma unroll
              for (int l = 0; l < 8; l++) head_s[l][row] = part[l];
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&head_full[q]));
            } else {
              if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&head_full[q]), hand, wait_ns))) {
                ok = false;
                break;
              }
#pragma unroll
              for (int l = 0; l < 8; l++) part[l] += head_s[l][row];
              __syncwarp();
              if (lane == 0) mbar_arrive(smem_u32(&head_empty[q]));
#pragma unroll
              for (int o = 4; o > 0; o >>= 1)
#pragma unroll
                for (int l = 0; l < o; l++) part[l] += part[l + o];
              const float z = part[0] + params[OFF_B4];
              prob[(int64_t)(t + p * step) * BM + row] = 1.0f / (1.0f + expf(-z));
            }
          }
        }
      }
    }
  }
  if (!ok) atomicExch(err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem, 2 * H);
  }
}

// p(lost) of n rows (n % 128 == 0) from X bf16 [n][64]
static cudaError_t launch_forward(const bf16* X, int64_t n, const bf16* w1, const bf16* w2, const bf16* w3,
                                  const float* params, float* prob, int* err, cudaStream_t st) {
  CUtensorMap mx, m1, m2, m3;
  auto weights = [](CUtensorMap* m, const bf16* w, uint64_t k) {
    return make_map(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w, k, H, k, FWD_WK, H, CU_TENSOR_MAP_SWIZZLE_64B);
  };
  if (!(make_map(&mx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, IN, (uint64_t)n, IN, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B) &&
        weights(&m1, w1, IN) && weights(&m2, w2, H) && weights(&m3, w3, H)))
    return cudaErrorInvalidValue;
  static std::atomic<bool> attr_set[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (!attr_set[dev & 63].load(std::memory_order_acquire)) {
    cudaError_t e = cudaFuncSetAttribute(forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM);
    if (e != cudaSuccess) return e;
    attr_set[dev & 63].store(true, std::memory_order_release);
  }
  const int n_tiles = (int)(n / BM);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min(n_tiles, sm_count()));
  cfg.blockDim = dim3(FWD_THREADS);
  cfg.dynamicSmemBytes = FWD_SMEM;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, forward_kernel, mx, m1, m2, m3, n_tiles, params, prob, err, 2000000000ull);
}

// ---------------------------------------------------------------------------
// CUDA-core kernels

// Output layer, loss and its gradient dZ3, row-major and transposed, of 64
// samples per block (the first n / 64 blocks), and the transposed input Xt[k][s]
// = X[s][k] of 64 samples (the next n / 64).  A warp takes eight samples; the
// transposed copies pass through shared memory and leave in 16-byte stores, 64
// samples of a column at a time (2-byte stores by the sample's own warp, and a
// transpose launch of its own, took 39 us of a 8,192-sample step; 7 us now).
constexpr int HEAD_ROWS = 64;
__global__ void __launch_bounds__(256)
    head_kernel(const bf16* __restrict__ A3, int64_t n, const float* __restrict__ w4, const float* __restrict__ b4,
                const float* __restrict__ label, float inv_batch, float* __restrict__ dlogit, bf16* __restrict__ dz3,
                bf16* __restrict__ dz3_t, const bf16* __restrict__ X, bf16* __restrict__ xt, int64_t ldt,
                float* __restrict__ loss_acc) {
  __shared__ __align__(16) bf16 tile[HEAD_ROWS][H];
  __shared__ float loss_s[8];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n_head = n / HEAD_ROWS;
  if (blockIdx.x >= n_head) {
    bf16(*xs)[IN + 2] = reinterpret_cast<bf16(*)[IN + 2]>(tile);
    const int64_t s0 = (blockIdx.x - n_head) * HEAD_ROWS;
    for (int q = tid; q < HEAD_ROWS * IN / 8; q += 256) {
      const uint4 u = reinterpret_cast<const uint4*>(X + s0 * IN)[q];
      const bf16* h = reinterpret_cast<const bf16*>(&u);
#pragma unroll
      for (int j = 0; j < 8; j++) xs[q / (IN / 8)][q % (IN / 8) * 8 + j] = h[j];
    }
    __syncthreads();
    const int k = tid >> 2, r0 = (tid & 3) * 16;
#pragma unroll
    for (int r = r0; r < r0 + 16; r += 8) {
      uint4 u;
      bf16* h = reinterpret_cast<bf16*>(&u);
#pragma unroll
      for (int j = 0; j < 8; j++) h[j] = xs[r + j][k];
      *reinterpret_cast<uint4*>(xt + (int64_t)k * ldt + s0 + r) = u;
    }
    return;
  }
  const int64_t s0 = blockIdx.x * (int64_t)HEAD_ROWS;
  float w[8], loss = 0.0f;
#pragma unroll
  for (int j = 0; j < 8; j++) w[j] = round_bf16(w4[lane * 8 + j]);
  uint4 u[8];
#pragma unroll
  for (int k = 0; k < 8; k++) u[k] = *reinterpret_cast<const uint4*>(A3 + (s0 + warp * 8 + k) * H + lane * 8);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int r = warp * 8 + k;
    const bf16* a = reinterpret_cast<const bf16*>(&u[k]);
    float av[8], acc = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      av[j] = __bfloat162float(a[j]);
      acc += av[j] * w[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    const float z = acc + b4[0];
    const float p = 1.0f / (1.0f + expf(-z));
    const float y = label[s0 + r];
    const float g = (p - y) * inv_batch;
    if (lane == 0) {
      dlogit[s0 + r] = g;
      // binary cross-entropy in the softplus form
      loss += (fmaxf(z, 0.0f) - z * y + log1pf(expf(-fabsf(z)))) * inv_batch;
    }
    uint4 out;
    bf16* o = reinterpret_cast<bf16*>(&out);
#pragma unroll
    for (int j = 0; j < 8; j++) o[j] = __float2bfloat16_rn(av[j] > 0.0f ? g * w[j] : 0.0f);
    *reinterpret_cast<uint4*>(dz3 + (s0 + r) * H + lane * 8) = out;
    *reinterpret_cast<uint4*>(&tile[r][lane * 8]) = out;
  }
  if (lane == 0) loss_s[warp] = loss;
  __syncthreads();
  if (tid == 0) {
    for (int k = 1; k < 8; k++) loss += loss_s[k];
    atomicAdd(loss_acc, loss);
  }
  bf16* dst = dz3_t + (int64_t)tid * ldt + s0;
#pragma unroll
  for (int r = 0; r < HEAD_ROWS; r += 8) {
    uint4 v;
    bf16* h = reinterpret_cast<bf16*>(&v);
#pragma unroll
    for (int j = 0; j < 8; j++) h[j] = tile[r + j][tid];
    *reinterpret_cast<uint4*>(dst + r) = v;
  }
}

// Column sums over 128 rows (blockIdx.x) of dZ1, dZ2, dZ3 and of A3 weighted by
// dlogit (blockIdx.y): partial[y][x][j], rows added in order.  16 rows' loads
// are in flight at a time (one at a time, in four launches: 78 us of a
// 8,192-sample step).
__global__ void __launch_bounds__(H / 2)
    colsum_kernel(const bf16* __restrict__ dz1, const bf16* __restrict__ dz2, const bf16* __restrict__ dz3,
                  const bf16* __restrict__ a3, const float* __restrict__ dlogit, float* __restrict__ partial) {
  const int y = blockIdx.y, j = threadIdx.x;
  const int64_t s0 = blockIdx.x * (int64_t)128;
  const bf16* M = (y == 0 ? dz1 : y == 1 ? dz2 : y == 2 ? dz3 : a3) + s0 * H + 2 * j;
  float acc0 = 0.0f, acc1 = 0.0f;
  for (int s = 0; s < 128; s += 16) {
    __nv_bfloat162 v[16];
    float w[16];
#pragma unroll
    for (int k = 0; k < 16; k++) {
      v[k] = *reinterpret_cast<const __nv_bfloat162*>(M + (int64_t)(s + k) * H);
      w[k] = y == 3 ? dlogit[s0 + s + k] : 1.0f;
    }
#pragma unroll
    for (int k = 0; k < 16; k++) {
      acc0 += w[k] * __bfloat162float(v[k].x);
      acc1 += w[k] * __bfloat162float(v[k].y);
    }
  }
  float* out = partial + ((int64_t)y * gridDim.x + blockIdx.x) * H + 2 * j;
  out[0] = acc0;
  out[1] = acc1;
}

// Adam's constants of a step; lr = 0 with train = 0: gradients only
struct AdamStep {
  int train;
  float lr, bc1, bc2;
};

// The gradients from their partial sums, and with train the Adam update and
// the bf16 weights (W row-major [out][in] and, for the hidden layers, W^T) for
// the next step: one pass over the parameters, one block per 256 of them
// (every parameter array starts on a multiple of 256), and a last block for
// b4 = sum dlogit.  As seven reductions, Adam and packing they were launches
// that each waited for the one before: 66 us of a 8,192-sample step.
// Partial sums are added in order, so the gradients are deterministic.
__global__ void __launch_bounds__(256)
    finish_kernel(const float* __restrict__ p1, const float* __restrict__ p2, const float* __restrict__ p3, int splits,
                  const float* __restrict__ pc, int chunks, const float* __restrict__ dlogit, int64_t batch,
                  float* __restrict__ grads, float* __restrict__ params, float* __restrict__ adam_m,
                  float* __restrict__ adam_v, bf16* __restrict__ w1, bf16* __restrict__ w2, bf16* __restrict__ w2t,
                  bf16* __restrict__ w3, bf16* __restrict__ w3t, AdamStep step) {
  __shared__ float sh[256];
  const int64_t i0 = blockIdx.x * (int64_t)256;
  const int tid = threadIdx.x;
  int64_t i = i0 + tid;
  float g = 0.0f;
  if (i0 == OFF_B4) {
    for (int64_t k = tid; k < batch; k += 256) g += dlogit[k];
    sh[tid] = g;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (tid < o) sh[tid] += sh[tid + o];
      __syncthreads();
    }
    if (tid != 0) return;
    g = sh[0];
  } else {
    const float* src;
    int64_t stride;
    int count;
    const auto weights = [&](const float* p, int64_t off, int64_t size) {
      src = p + (i - off);
      stride = size;
      count = splits;
    };
    const auto columns = [&](int y, int64_t off) {
      src = pc + (int64_t)y * chunks * H + (i - off);
      stride = H;
      count = chunks;
    };
    if (i0 < OFF_B1) weights(p1, OFF_W1, (int64_t)H * IN);
    else if (i0 < OFF_W2) columns(0, OFF_B1);
    else if (i0 < OFF_B2) weights(p2, OFF_W2, (int64_t)H * H);
    else if (i0 < OFF_W3) columns(1, OFF_B2);
    else if (i0 < OFF_B3) weights(p3, OFF_W3, (int64_t)H * H);
    else if (i0 < OFF_W4) columns(2, OFF_B3);
    else columns(3, OFF_W4);
    int c = 0;
    for (; c + 16 <= count; c += 16) {
      float v[16];
#pragma unroll
      for (int k = 0; k < 16; k++) v[k] = src[(c + k) * stride];
#pragma unroll
      for (int k = 0; k < 16; k++) g += v[k];
    }
    for (; c < count; c++) g += src[c * stride];
  }
  grads[i] = g;
  if (!step.train) return;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float mi = b1 * adam_m[i] + (1.0f - b1) * g;
  const float vi = b2 * adam_v[i] + (1.0f - b2) * g * g;
  adam_m[i] = mi;
  adam_v[i] = vi;
  const float pi = params[i] - step.lr * (mi / step.bc1) / (sqrtf(vi / step.bc2) + eps);
  params[i] = pi;
  const bf16 h = __float2bfloat16_rn(pi);
  if (i0 < OFF_B1) {
    w1[i] = h;
  } else if (i0 >= OFF_W2 && i0 < OFF_B2) {
    i -= OFF_W2;
    w2[i] = h;
    w2t[(i % H) * H + i / H] = h;
  } else if (i0 >= OFF_W3 && i0 < OFF_B3) {
    i -= OFF_W3;
    w3[i] = h;
    w3t[(i % H) * H + i / H] = h;
  }
}
static_assert(OFF_B1 % 256 == 0 && OFF_W2 % 256 == 0 && OFF_B2 % 256 == 0 && OFF_W3 % 256 == 0 && OFF_B3 % 256 == 0 &&
                  OFF_W4 % 256 == 0 && OFF_B4 % 256 == 0,
              "a block of finish_kernel lies in one parameter array");

// bf16 weights for the GEMMs from the master parameters
__global__ void pack_kernel(const float* __restrict__ p, bf16* __restrict__ w1, bf16* __restrict__ w2,
                            bf16* __restrict__ w2t, bf16* __restrict__ w3, bf16* __restrict__ w3t) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < (int64_t)H * IN) w1[i] = __float2bfloat16_rn(p[OFF_W1 + i]);
  if (i < (int64_t)H * H) {
    const int64_t o = i / H, k = i % H;
    const bf16 a = __float2bfloat16_rn(p[OFF_W2 + i]), b = __float2bfloat16_rn(p[OFF_W3 + i]);
    w2[i] = a;
    w3[i] = b;
    w2t[k * H + o] = a;
    w3t[k * H + o] = b;
  }
}

// Classifier inputs of n particles, one thread each.  Memory-bound: 100 B in,
// 128 B (x) and 120 B (raw) out per particle.  A thread's row is written to
// shared memory and the block's rows, which are contiguous, leave it in
// 16-byte stores by consecutive threads; stored by the thread that owns the
// row, every store instruction touched 32 lines.  Chunk c of row r sits at c ^
// (r % 8), free of bank conflicts both ways; raw rows are 31 floats apart.
// 500,001 particles through the Python call: 60 us (with a zero fill of all of
// x) -> 31.5 us, 3.6 TB/s.
constexpr int FEAT_BLOCK = 128;
__global__ void __launch_bounds__(FEAT_BLOCK)
    features_kernel(const double* __restrict__ vec0, const double* __restrict__ vec, int64_t n, int64_t stride,
                    const int32_t* __restrict__ var, const double* __restrict__ table,
                    const float* __restrict__ mean, const float* __restrict__ inv_std, float* __restrict__ raw,
                    bf16* __restrict__ x) {
  extern __shared__ __align__(16) uint8_t feat_smem[];
  __shared__ float norm_s[2][BGT_MLP_FEATURES];
  const int tid = threadIdx.x;
  const int64_t i0 = blockIdx.x * (int64_t)FEAT_BLOCK, i = i0 + tid;
  const int rows = (int)min((int64_t)FEAT_BLOCK, n - i0);
  if (x && tid < BGT_MLP_FEATURES) {
    norm_s[0][tid] = mean[tid];
    norm_s[1][tid] = inv_std[tid];
  }
  uint4* xs = reinterpret_cast<uint4*>(feat_smem);
  float* rs = reinterpret_cast<float*>(feat_smem + (x ? FEAT_BLOCK * IN * sizeof(bf16) : 0));
  float f[BGT_MLP_FEATURES];
  if (i < n) {
    const double* T = table + (int64_t)(var ? var[i] : 0) * BGT_MLP_VARIANT_COLS;
    double v[6];
#pragma unroll
    for (int k = 0; k < 6; k++) {
      f[k] = (float)(vec0[k * stride + i] - T[k]);
      v[k] = vec[k * stride + i] - T[k];
      f[22 + k] = (float)v[k];
    }
#pragma unroll
    for (int k = 0; k < 16; k++) f[6 + k] = (float)T[14 + k];
    const double dp = v[5];
    const double xb = v[0] - T[6] * dp, pxb = v[1] - T[7] * dp;
    const double yb = v[2] - T[8] * dp, pyb = v[3] - T[9] * dp;
    const double ba = T[10], aa = T[11], bb = T[12], ab = T[13];
    const double ja = 0.5 * ((1 + aa * aa) / ba * xb * xb + 2 * aa * xb * pxb + ba * pxb * pxb);
    const double jb = 0.5 * ((1 + ab * ab) / bb * yb * yb + 2 * ab * yb * pyb + bb * pyb * pyb);
    f[28] = (float)sqrt(fmax(ja, 0.0));
    f[29] = (float)sqrt(fmax(jb, 0.0));
  }
  __syncthreads();  // norm_s
  if (i < n) {
    if (raw) {
#pragma unroll
      for (int k = 0; k < BGT_MLP_FEATURES; k++) rs[tid * (BGT_MLP_FEATURES + 1) + k] = f[k];
    }
    if (x) {
#pragma unroll
      for (int c = 0; c < IN / 8; c++) {
        uint4 pk;
        bf16* h = reinterpret_cast<bf16*>(&pk);
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int k = 8 * c + j, kk = k < BGT_MLP_FEATURES ? k : 0;
          h[j] = __float2bfloat16_rn(k < BGT_MLP_FEATURES ? (f[kk] - norm_s[0][kk]) * norm_s[1][kk] : 0.0f);
        }
        xs[tid * (IN / 8) + (c ^ (tid & 7))] = pk;
      }
    }
  }
  __syncthreads();
  if (x) {
    uint4* dst = reinterpret_cast<uint4*>(x + i0 * IN);
    for (int q = tid; q < rows * (IN / 8); q += FEAT_BLOCK) {
      const int r = q / (IN / 8), c = q % (IN / 8);
      dst[q] = xs[r * (IN / 8) + (c ^ (r & 7))];
    }
  }
  if (raw) {
    float* dst = raw + i0 * BGT_MLP_FEATURES;
    for (int q = tid; q < rows * BGT_MLP_FEATURES; q += FEAT_BLOCK)
      dst[q] = rs[(q / BGT_MLP_FEATURES) * (BGT_MLP_FEATURES + 1) + q % BGT_MLP_FEATURES];
  }
}

}  // namespace mlp
}  // namespace bgt

using namespace bgt::mlp;

struct bgt_mlp {
  int device = 0;
  int32_t max_batch = 0;
  std::string err;
  int64_t launches = 0;
  int64_t step = 0;
  float* params = nullptr;   // FP32 master
  float* grads = nullptr;
  float* adam_m = nullptr;
  float* adam_v = nullptr;
  float* partial = nullptr;  // split-K / column-sum partials
  float* scalars = nullptr;  // [0] loss
  int* d_err = nullptr;
  bf16 *w1 = nullptr, *w2 = nullptr, *w2t = nullptr, *w3 = nullptr, *w3t = nullptr;
  bf16 *xt = nullptr, *a1 = nullptr, *a1t = nullptr, *a2 = nullptr, *a2t = nullptr, *a3 = nullptr;
  bf16 *dz1 = nullptr, *dz1t = nullptr, *dz2 = nullptr, *dz2t = nullptr, *dz3 = nullptr, *dz3t = nullptr;
  float* dlogit = nullptr;
  std::vector<void*> allocs;
};

static int mlp_err(bgt_mlp* m, int code, const std::string& msg) {
  if (m) m->err = msg;
  return code;
}

#define MCU(m, call)                                                                          \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return mlp_err((m), BGT_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_));     \
  } while (0)

template <class T>
static cudaError_t mlp_alloc(bgt_mlp* m, T** p, size_t count) {
  cudaError_t e = cudaMalloc((void**)p, count * sizeof(T));
  if (e == cudaSuccess) m->allocs.push_back((void*)*p);
  return e;
}

// splits of a weight gradient over a batch: one chunk per CTA of a full wave,
// at least KSPLIT samples each
static int64_t max_splits(int64_t batch) {
  return std::max<int64_t>(1, std::min<int64_t>(batch / KSPLIT, sm_count() / (H / BM)));
}

static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

// splitmix64 -> uniform in [-1, 1)
static double mix_uniform(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  return (double)(z >> 11) * (1.0 / 4503599627370496.0) - 1.0;
}

static int pack_weights(bgt_mlp* m, cudaStream_t st) {
  pack_kernel<<<(H * H + 255) / 256, 256, 0, st>>>(m->params, m->w1, m->w2, m->w2t, m->w3, m->w3t);
  m->launches++;
  MCU(m, cudaGetLastError());
  return 0;
}

extern "C" {

int bgt_mlp_create(bgt_mlp** out, int32_t max_batch, uint64_t seed, int32_t device) {
  if (!out || max_batch <= 0 || max_batch % 128) return BGT_EINVAL;
  *out = nullptr;
  bgt_mlp* m = new bgt_mlp();
  m->device = device;
  m->max_batch = max_batch;
  cudaError_t e = cudaSetDevice(device);
  const int64_t B = max_batch;
  // partial sums of a step: the three weight gradients' splits, four column sums
  const int64_t partial = max_splits(B) * ((int64_t)H * IN + 2 * (int64_t)H * H) + (B / 128) * 4 * H;
  if (e == cudaSuccess) e = mlp_alloc(m, &m->params, N_PARAMS);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->grads, N_PARAMS);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->adam_m, N_PARAMS);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->adam_v, N_PARAMS);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->partial, partial);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->scalars, 8);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->d_err, 1);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->w1, (size_t)H * IN);
  bf16** hh[] = {&m->w2, &m->w2t, &m->w3, &m->w3t};
  for (auto p : hh)
    if (e == cudaSuccess) e = mlp_alloc(m, p, (size_t)H * H);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->xt, (size_t)IN * B);
  bf16** acts[] = {&m->a1, &m->a1t, &m->a2, &m->a2t, &m->a3, &m->dz1, &m->dz1t, &m->dz2, &m->dz2t, &m->dz3, &m->dz3t};
  for (auto p : acts)
    if (e == cudaSuccess) e = mlp_alloc(m, p, (size_t)H * B);
  if (e == cudaSuccess) e = mlp_alloc(m, &m->dlogit, B);
  if (e == cudaSuccess) e = cudaMemset(m->d_err, 0, sizeof(int));
  if (e != cudaSuccess) {
    fprintf(stderr, "bgt_mlp_create: %s\n", cudaGetErrorString(e));
    bgt_mlp_destroy(m);
    return BGT_ENOMEM;
  }
  // He-uniform weights, zero biases; the padded input columns stay zero
  std::vector<float> p(N_PARAMS, 0.0f);
  uint64_t s = seed;
  const double lim1 = std::sqrt(6.0 / BGT_MLP_FEATURES), limh = std::sqrt(6.0 / H);
  for (int o = 0; o < H; o++)
    for (int k = 0; k < BGT_MLP_FEATURES; k++) p[OFF_W1 + o * IN + k] = (float)(lim1 * mix_uniform(s));
  for (int64_t i = 0; i < (int64_t)H * H; i++) p[OFF_W2 + i] = (float)(limh * mix_uniform(s));
  for (int64_t i = 0; i < (int64_t)H * H; i++) p[OFF_W3 + i] = (float)(limh * mix_uniform(s));
  for (int i = 0; i < H; i++) p[OFF_W4 + i] = (float)(std::sqrt(3.0 / H) * mix_uniform(s));
  *out = m;
  return bgt_mlp_set_params(m, p.data());
}

int bgt_mlp_destroy(bgt_mlp* m) {
  if (!m) return 0;
  for (void* p : m->allocs) cudaFree(p);
  delete m;
  return 0;
}

const char* bgt_mlp_last_error(const bgt_mlp* m) { return m ? m->err.c_str() : "null handle"; }
int64_t bgt_mlp_launch_count(const bgt_mlp* m) { return m ? m->launches : 0; }

int bgt_mlp_get_params(bgt_mlp* m, float* params) {
  if (!m || !params) return BGT_EINVAL;
  MCU(m, cudaSetDevice(m->device));
  MCU(m, cudaDeviceSynchronize());
  MCU(m, cudaMemcpy(params, m->params, N_PARAMS * sizeof(float), cudaMemcpyDeviceToHost));
  return 0;
}

int bgt_mlp_set_params(bgt_mlp* m, const float* params) {
  if (!m || !params) return BGT_EINVAL;
  MCU(m, cudaSetDevice(m->device));
  MCU(m, cudaMemcpy(m->params, params, N_PARAMS * sizeof(float), cudaMemcpyHostToDevice));
  MCU(m, cudaMemset(m->adam_m, 0, N_PARAMS * sizeof(float)));
  MCU(m, cudaMemset(m->adam_v, 0, N_PARAMS * sizeof(float)));
  m->step = 0;
  int rc = pack_weights(m, 0);
  if (rc) return rc;
  MCU(m, cudaDeviceSynchronize());
  return 0;
}

}  // extern "C"

static int check_error_flag(bgt_mlp* m) {
  int flag = 0;
  MCU(m, cudaMemcpy(&flag, m->d_err, sizeof(int), cudaMemcpyDeviceToHost));
  if (flag) return mlp_err(m, BGT_ETIMEOUT, "tensor-core GEMM: mbarrier wait timed out");
  return 0;
}

// Gradients of the mean loss over one batch into `grads`; with step.train the
// Adam update and the packed weights as well.
static int train_batch(bgt_mlp* m, const bf16* X, const float* label, int32_t batch, float* grads, AdamStep step,
                       cudaStream_t st) {
  const int64_t B = batch, ldt = m->max_batch;
  MCU(m, cudaMemsetAsync(m->scalars, 0, sizeof(float), st));
  // forward, with transposed copies of the activations for the weight gradients
  Epi e{};
  e.bias = m->params + OFF_B1;
  e.out_t = m->a1t;
  e.ldt = ldt;
  MCU(m, (launch_gemm<256, EPI_FWD>(X, IN, B, m->w1, IN, IN, 1, m->a1, H, e, m->d_err, st)));
  e.bias = m->params + OFF_B2;
  e.out_t = m->a2t;
  MCU(m, (launch_gemm<256, EPI_FWD>(m->a1, H, B, m->w2, H, H, 1, m->a2, H, e, m->d_err, st)));
  e.bias = m->params + OFF_B3;
  e.out_t = nullptr;
  MCU(m, (launch_gemm<256, EPI_FWD>(m->a2, H, B, m->w3, H, H, 1, m->a3, H, e, m->d_err, st)));
  head_kernel<<<(unsigned)(2 * (B / HEAD_ROWS)), 256, 0, st>>>(
      m->a3, B, m->params + OFF_W4, m->params + OFF_B4, label, 1.0f / (float)B, m->dlogit, m->dz3, m->dz3t, X, m->xt,
      ldt, m->scalars);
  MCU(m, cudaGetLastError());
  // dZ2 = (dZ3 . W3) * relu'(A2), dZ1 = (dZ2 . W2) * relu'(A1)
  e = Epi{};
  e.ldt = ldt;
  e.ldm = H;
  e.out_t = m->dz2t;
  e.mask = m->a2;
  MCU(m, (launch_gemm<256, EPI_BWD>(m->dz3, H, B, m->w3t, H, H, 1, m->dz2, H, e, m->d_err, st)));
  e.out_t = m->dz1t;
  e.mask = m->a1;
  MCU(m, (launch_gemm<256, EPI_BWD>(m->dz2, H, B, m->w2t, H, H, 1, m->dz1, H, e, m->d_err, st)));
  // weight gradients dW = dZ^T . A_prev over the batch as FP32 partial sums
  const int splits = (int)max_splits(B);
  const int chunks = (int)(B / 128);
  float* p3 = m->partial;
  float* p2 = p3 + (int64_t)splits * H * H;
  float* p1 = p2 + (int64_t)splits * H * H;
  float* pc = p1 + (int64_t)splits * H * IN;
  const Epi f{};
  MCU(m, (launch_gemm<256, EPI_F32>(m->dz3t, ldt, H, m->a2t, ldt, B, splits, p3, 256, f, m->d_err, st)));
  MCU(m, (launch_gemm<256, EPI_F32>(m->dz2t, ldt, H, m->a1t, ldt, B, splits, p2, 256, f, m->d_err, st)));
  MCU(m, (launch_gemm<64, EPI_F32>(m->dz1t, ldt, H, m->xt, ldt, B, splits, p1, 64, f, m->d_err, st)));
  // bias gradients (column sums of dZ), w4's = sum dlogit * A3
  colsum_kernel<<<dim3((unsigned)chunks, 4), H / 2, 0, st>>>(m->dz1, m->dz2, m->dz3, m->a3, m->dlogit, pc);
  finish_kernel<<<(unsigned)(OFF_B4 / 256 + 1), 256, 0, st>>>(p1, p2, p3, splits, pc, chunks, m->dlogit, B, grads,
                                                             m->params, m->adam_m, m->adam_v, m->w1, m->w2, m->w2t,
                                                             m->w3, m->w3t, step);
  m->launches += 11;
  MCU(m, cudaGetLastError());
  return 0;
}

// whether p is a float array in the memory of the handle's device
static bool own_floats(const bgt_mlp* m, const float* p) {
  cudaPointerAttributes a{};
  if ((uintptr_t)p % sizeof(float) != 0) return false;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice && a.device == m->device;
}

static int check_batch(bgt_mlp* m, const uint16_t* d_x, const float* d_label, int32_t batch) {
  if (!m || !d_x || !d_label) return BGT_EINVAL;
  if (batch <= 0 || batch % 128 || batch > m->max_batch)
    return mlp_err(m, BGT_EINVAL, "batch must be a positive multiple of 128 and <= max_batch");
  if (!aligned16(d_x)) return mlp_err(m, BGT_EINVAL, "d_x must be 16-byte aligned");
  return 0;
}

extern "C" {

int bgt_mlp_forward(bgt_mlp* m, const uint16_t* d_x, int64_t n, float* d_prob, void* stream) {
  if (!m || !d_x || !d_prob || n < 0) return BGT_EINVAL;
  if (n % 128) return mlp_err(m, BGT_EINVAL, "n must be a multiple of 128 (pad the input rows)");
  if (!aligned16(d_x)) return mlp_err(m, BGT_EINVAL, "d_x must be 16-byte aligned");
  MCU(m, cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  const bf16* X = reinterpret_cast<const bf16*>(d_x);
  if (n == 0) return 0;
  MCU(m, launch_forward(X, n, m->w1, m->w2, m->w3, m->params, d_prob, m->d_err, st));
  m->launches++;
  return 0;
}

int bgt_mlp_gradients(bgt_mlp* m, const uint16_t* d_x, const float* d_label, int32_t batch, float* d_grad,
                      float* loss, void* stream) {
  int rc = check_batch(m, d_x, d_label, batch);
  if (rc) return rc;
  MCU(m, cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  // the kernel writes a caller's array on the handle's device itself; any
  // other (not a float's alignment, another device's, host memory) is copied to
  const bool direct = d_grad && own_floats(m, d_grad);
  rc = train_batch(m, reinterpret_cast<const bf16*>(d_x), d_label, batch, direct ? d_grad : m->grads, AdamStep{}, st);
  if (rc) return rc;
  if (d_grad && !direct)
    MCU(m, cudaMemcpyAsync(d_grad, m->grads, N_PARAMS * sizeof(float), cudaMemcpyDeviceToDevice, st));
  if (loss) {
    MCU(m, cudaMemcpyAsync(loss, m->scalars, sizeof(float), cudaMemcpyDeviceToHost, st));
    MCU(m, cudaStreamSynchronize(st));
    return check_error_flag(m);
  }
  return 0;
}

int bgt_mlp_train_step(bgt_mlp* m, const uint16_t* d_x, const float* d_label, int32_t batch, float lr, float* loss,
                       void* stream) {
  int rc = check_batch(m, d_x, d_label, batch);
  if (rc) return rc;
  MCU(m, cudaSetDevice(m->device));
  cudaStream_t st = (cudaStream_t)stream;
  m->step++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = 1.0f - (float)std::pow((double)b1, (double)m->step);
  const float bc2 = 1.0f - (float)std::pow((double)b2, (double)m->step);
  rc = train_batch(m, reinterpret_cast<const bf16*>(d_x), d_label, batch, m->grads, AdamStep{1, lr, bc1, bc2}, st);
  if (rc) {
    m->step--;
    return rc;
  }
  if (loss) {
    MCU(m, cudaMemcpyAsync(loss, m->scalars, sizeof(float), cudaMemcpyDeviceToHost, st));
    MCU(m, cudaStreamSynchronize(st));
    return check_error_flag(m);
  }
  return 0;
}

int bgt_mlp_features(const double* d_vec0, const double* d_vec, int64_t n, int64_t stride, const int32_t* d_variant,
                     const double* d_table, int32_t n_variants, const float* d_mean, const float* d_inv_std,
                     float* d_raw, uint16_t* d_x, void* stream) {
  if (!d_vec0 || !d_vec || !d_table || n < 0 || stride < n || n_variants <= 0) return BGT_EINVAL;
  if (d_x && (!d_mean || !d_inv_std || !aligned16(d_x))) return BGT_EINVAL;
  if (n == 0) return 0;
  const size_t smem = (d_x ? FEAT_BLOCK * IN * sizeof(bf16) : 0) +
                      (d_raw ? FEAT_BLOCK * (BGT_MLP_FEATURES + 1) * sizeof(float) : 0);
  features_kernel<<<(unsigned)((n + FEAT_BLOCK - 1) / FEAT_BLOCK), FEAT_BLOCK, smem, (cudaStream_t)stream>>>(
      d_vec0, d_vec, n, stride, d_variant, d_table, d_mean, d_inv_std, d_raw, reinterpret_cast<bf16*>(d_x));
  return cudaGetLastError() == cudaSuccess ? 0 : BGT_ECUDA;
}

static int gemm_bf16(const uint16_t* d_a, int64_t lda, const uint16_t* d_b, int64_t ldb, int32_t m, int32_t n,
                     int32_t k, float* d_c, void* stream, uint64_t wait_ns, int skip_mma) {
  if (!d_a || !d_b || !d_c || m <= 0 || m % BM || (n != 64 && n != 256) || k <= 0 || k % BK) return BGT_EINVAL;
  if (lda < k || ldb < k || lda % 8 || ldb % 8 || !aligned16(d_a) || !aligned16(d_b) || !aligned16(d_c))
    return BGT_EINVAL;
  cudaStream_t st = (cudaStream_t)stream;
  int* d_err = nullptr;
  if (cudaGetSymbolAddress((void**)&d_err, g_gemm_error) != cudaSuccess) return BGT_ECUDA;
  if (cudaMemsetAsync(d_err, 0, sizeof(int), st) != cudaSuccess) return BGT_ECUDA;
  Epi e{};
  const bf16* A = reinterpret_cast<const bf16*>(d_a);
  const bf16* B = reinterpret_cast<const bf16*>(d_b);
  cudaError_t ce = (n == 256)
                       ? launch_gemm<256, EPI_F32>(A, lda, m, B, ldb, k, 1, d_c, n, e, d_err, st, wait_ns, skip_mma)
                       : launch_gemm<64, EPI_F32>(A, lda, m, B, ldb, k, 1, d_c, n, e, d_err, st, wait_ns, skip_mma);
  if (ce != cudaSuccess) return BGT_ECUDA;
  if (cudaStreamSynchronize(st) != cudaSuccess) return BGT_ECUDA;
  int flag = 0;
  if (cudaMemcpy(&flag, d_err, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return BGT_ECUDA;
  return flag ? BGT_ETIMEOUT : 0;
}

int bgt_mlp_gemm_bf16(const uint16_t* d_a, int64_t lda, const uint16_t* d_b, int64_t ldb, int32_t m, int32_t n,
                      int32_t k, float* d_c, void* stream) {
  return gemm_bf16(d_a, lda, d_b, ldb, m, n, k, d_c, stream, 2000000000ull, 0);
}

int bgt_mlp_gemm_bf16_wait_test(const uint16_t* d_a, int64_t lda, const uint16_t* d_b, int64_t ldb, int32_t m,
                                int32_t n, int32_t k, float* d_c, uint32_t wait_limit_us, void* stream) {
  if (wait_limit_us == 0) return BGT_EINVAL;
  return gemm_bf16(d_a, lda, d_b, ldb, m, n, k, d_c, stream, (uint64_t)wait_limit_us * 1000ull, 1);
}

}  // extern "C"
