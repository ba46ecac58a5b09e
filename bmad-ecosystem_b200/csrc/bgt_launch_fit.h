// bgt_launch_fit.h -- the launch shape and table placement of a tracking call,
// fitted to the call.  Plain host arithmetic (bgt_track.cu; the tests build it
// on its own).
#pragma once
#include <stdint.h>

#include <algorithm>

#include "../../include/bgt.h"

namespace bgt {

// Fits a tuning whose table_mode is 0; the other modes name a placement, and
// with them the shape is launched as given.
//
// * A staged table must leave every CTA resident that the launch can use; the
//   150 KB table of an error ring leaves one.  Staged against global on B200,
//   128 x 4, one turn on four error rings: 16,000 particles (1 CTA per SM
//   wanted) 1.33 / 1.62 ms, 20,000 (2) 2.55 / 1.80, 38,000 (3) 3.78 / 2.15,
//   60,000 (4) 5.04 / 2.82.
// * 256-thread tiles become 128-thread ones of the same register cap while all
//   of them are resident at once: a CTA's warps share an SM, so few large tiles
//   leave SMs idle or uneven.  256 x 2 against 128 x 4: four turns of the FODO
//   ring, 10,000 particles 1.75 / 1.58 ms, 40,000 2.26 / 1.94, 75,000 2.45 /
//   2.42; one turn of 8,064 on four error rings 1.62 / 1.33, both staged, and
//   of 40,000 2.66 / 2.17, both global.  With a global table the 256-thread
//   tiles win once every SM is full (60,000 on one error ring 2.62 / 2.72), so
//   there the 128-thread ones must leave room for one more per SM.
// * Between the two, a table that fits beside 256-thread tiles but not beside
//   128-thread ones stays staged: 24,000 on four error rings, 256 x 2 staged
//   1.63 ms, 128 x 4 global 1.82.
//
//   n_tiles(block)              tiles of `block` particles that the call makes
//   staged_bytes(block)         dynamic shared memory of a CTA with the table
//                               staged, at most smem_limit
//   has(block, per_sm, tmode)   whether the kernel has this instance (tmode as
//                               the kernel's TMODE)
template <class NTiles, class StagedBytes, class Has>
bgt_tuning fit_tuning(bgt_tuning t, int num_sms, size_t smem_limit, const NTiles& n_tiles,
                      const StagedBytes& staged_bytes, const Has& has) {
  if (t.table_mode != 0) return t;
  // whether a staged table leaves every CTA resident that the launch can use
  // (228 KB of shared memory per SM, 1 KB of it per CTA reserved)
  auto staged_fits = [&](int block, int per_sm) {
    const size_t smem = staged_bytes(block);
    const int64_t wanted = std::min<int64_t>(per_sm, (n_tiles(block) + num_sms - 1) / num_sms);
    return smem <= smem_limit && (int64_t)((228 * 1024) / (smem + 1024)) >= wanted;
  };
  const bool fits = staged_fits(t.threads_per_block, t.blocks_per_sm);
  const int half = 2 * t.blocks_per_sm;  // the CTAs per SM of 128-thread tiles
  const bool halve = t.threads_per_block == 256 && n_tiles(256) < (int64_t)t.blocks_per_sm * num_sms;
  if (halve && has(128, half, 0) && staged_fits(128, half)) {
    t.threads_per_block = 128;
    t.blocks_per_sm = half;
  } else if (!fits) {
    if (halve && n_tiles(128) <= (int64_t)(half - 1) * num_sms && has(128, half, 1)) {
      t.threads_per_block = 128;
      t.blocks_per_sm = half;
      t.table_mode = 2;
    } else if (has(t.threads_per_block, t.blocks_per_sm, 1)) {
      t.table_mode = 2;
    }
  }
  return t;
}

}  // namespace bgt
