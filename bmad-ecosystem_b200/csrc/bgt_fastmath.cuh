// bgt_fastmath.cuh -- branch-free quotients and square roots on the operand
// ranges of the near-axis element maps, with the IEEE result bit for bit.
//
// The general '/' and sqrt carry range checks and a slow path: ~8 FP64
// instructions, a table look-up and 6-8 integer, select and branch
// instructions each, and the branches keep the compiler from overlapping
// neighbouring chains.  On the ranges here no scaling is needed, so Newton's
// iteration and Markstein's final correction (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res.
// Dev. 34(1), 1990) are straight-line code.
#pragma once
#ifdef __CUDACC__
#include <cuda_runtime.h>
#endif
#include <math.h>
#include <stdint.h>
#include <string.h>

namespace bgt {

#ifdef __CUDACC__
__device__ __forceinline__ int32_t hi_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ uint32_t lo_word(double x) { return (uint32_t)__double2loint(x); }
#else
inline int32_t hi_word(double x) {
  uint64_t b;
  memcpy(&b, &x, 8);
  return (int32_t)(b >> 32);
}
inline uint32_t lo_word(double x) {
  uint64_t b;
  memcpy(&b, &x, 8);
  return (uint32_t)b;
}
#endif
// high word of |x|: ordered like |x| (a NaN or infinity is above every finite value)
__device__ __forceinline__ int32_t abs_hi(double x) { return hi_word(x) & 0x7fffffff; }

// a / b correctly rounded from r = RN(1 / b), as div_by (bgt_device.cuh)
// argues it, without its select: a quotient -0 comes out as +0.  In the maps
// that use it a zero quotient is then added to something; the sum differs at
// most in the sign of a zero.
__device__ __forceinline__ double div_rn(double a, double b, double r) {
  const double q = a * r;
  return fma(fma(-q, b, a), r, q);
}

// Near-axis drift: v = 1 - pxy2 with d = 1 - v <= 2^-12.6 (|px|, |py| <
// NEAR_P, |pz| < NEAR_PZ).  ps = RN(sqrt(v)), r_ps = RN(1 / ps), r_ps1 =
// RN(1 / RN(ps + 1)).  The seeds are the Taylor series of 1 / sqrt(1 - d)
// and 1 / (1 + sqrt(1 - d)) to d^3 (within 2 ulp, truncation < 2^-50), each
// one ulp high (and its slope a few ulp low, which keeps the sum from the
// next tie) so that Markstein's correction also rounds the reciprocals of
// an all-ones significand; one Newton correction with the exact residual
// follows.  All three were compared with the IEEE sqrt and quotients for
// every v of the range on a B200: 1.49e12 values, no difference.
// The coefficients sit in constant memory, which an FP64 instruction reads as
// an operand; as literals each costs two moves into a register pair.
#ifdef __CUDACC__
#define BGT_FM_TABLE static __constant__ double
#else
#define BGT_FM_TABLE static const double
#endif
BGT_FM_TABLE FM_R0[4] = {0.3125, 0.375, 0.5 - 0x1p-52, 1.0 + 0x1p-52};
BGT_FM_TABLE FM_RB[4] = {0x1.4p-5, 0.0625, 0.125 - 0x1p-52, 0.5 + 0x1p-53};
// sqrt_test's and the rounding tests' factors, rsqrt_near's 3/8
BGT_FM_TABLE FM_T[8] = {0.5 - 0x1p-47, 0.5 + 0x1p-47, -0x1p-50, 0x1p-50, -0x1p-71, 0x1p-71, 0x1p-70, 0.375};
constexpr int32_t NEAR_P_HI = 0x3f800000;   // 2^-7: |px|, |py| of the near-axis maps
constexpr int32_t NEAR_PZ_HI = 0x3fc00000;  // 2^-3: |pz|
struct PsTerms {
  double ps, r_ps, r_ps1;
};
__device__ __forceinline__ PsTerms ps_terms(double v) {
  const double d = 1.0 - v;  // exact (v in [1/2, 1])
  const double r0 = fma(fma(fma(FM_R0[0], d, FM_R0[1]), d, FM_R0[2]), d, FM_R0[3]);
  const double s0 = v * r0;
  PsTerms T;
  T.ps = fma(fma(-s0, s0, v), 0.5 * r0, s0);
  T.r_ps = fma(fma(-T.ps, r0, 1.0), r0, r0);
  const double b = T.ps + 1.0;
  const double rb = fma(fma(fma(FM_RB[0], d, FM_RB[1]), d, FM_RB[2]), d, FM_RB[3]);
  T.r_ps1 = fma(fma(-b, rb, 1.0), rb, rb);
  return T;
}

// ---------------------------------------------------------------------------
// Quotients, square roots and transcendentals of a near-axis bend step.
//
// Each value comes with a rounding test: the result is formed from the lower
// and the upper end of its error interval, and `bad` collects the bits in
// which the two low words differ.  bad == 0 at the end of the map proves
// every one of them correctly rounded (rounding is monotonic, and
// neighbouring doubles always differ in the low word); otherwise the map is
// evaluated again by the general functions.  One test for a whole element in
// place of one branch per function keeps its ~250 FP64 instructions in one
// basic block.  u = 2^-53 below.

// seeds good to ~20 bits (the PTX approximations; single precision on the host)
__device__ __forceinline__ double rcp_seed(double x) {
#ifdef __CUDACC__
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#else
  return (double)(1.0f / (float)x);
#endif
}
__device__ __forceinline__ double rsqrt_seed(double x) {
#ifdef __CUDACC__
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
#else
  return (double)(1.0f / sqrtf((float)x));
#endif
}

// a faithful 1 / b: a cubic Newton step from the seed (error 2^-57 before
// its rounding)
__device__ __forceinline__ double rcp_faithful(double b) {
  const double r0 = rcp_seed(b);
  const double e = fma(-b, r0, 1.0);
  return fma(r0, fma(e, e, e), r0);
}
// RN(a / b), b > 0 in [2^-100, 2^100], |a| in [2^-900, 2^900] or 0: r = RN(1 / b) by Markstein's
// correction unless b's significand is all ones (then bad), the quotient as
// div_by
__device__ __forceinline__ double div_test(double a, double b, uint32_t& bad) {
  const double r1 = rcp_faithful(b);
  const double r = fma(fma(-b, r1, 1.0), r1, r1);
  bad |= lo_word(b) == 0xffffffffu;
  return div_rn(a, b, r);
}

// y ~ 1 / sqrt(v) to < 2^-51: y0 (1 - e)^(-1/2) to e^2, e = 1 - v y0^2
__device__ __forceinline__ double rsqrt_near(double v) {
  const double y0 = rsqrt_seed(v);
  const double e = fma(-(v * y0), y0, 1.0);
  return fma(y0 * e, fma(FM_T[7], e, 0.5), y0);
}
// RN(sqrt(v)), v in [2^-100, 2^100]: s0 = v y is within 2^-50, and sqrt(v) =
// s0 + (v - s0^2) y / 2 (1 + theta), |theta| < 2^-49 (y, the residual's
// rounding and the second-order term); the test spans 2^-46.
__device__ __forceinline__ double sqrt_test(double v, double y, uint32_t& bad) {
  const double s0 = v * y;
  const double d = fma(-s0, s0, v);
  const double s = fma(d, y * FM_T[0], s0);
  const double t = fma(d, y * FM_T[1], s0);
  bad |= lo_word(s) ^ lo_word(t);
  return s;
}

// x + c for a correction c of relative error < 7u (the test spans 8u)
__device__ __forceinline__ double add_test(double x, double c, uint32_t& bad) {
  const double a = x + fma(c, FM_T[2], c);
  const double b = x + fma(c, FM_T[3], c);
  bad |= lo_word(a) ^ lo_word(b);
  return a;
}
// sin (C = SIN_C) for |x| < 2^-6, asin (C = ASIN_C) for |x| < 2^-6.8:
// x + x y P(y), y = x^2, four terms in plain double.  Relative error of the
// correction: y, x y, the product (u each), P (< 2.1u), and the first
// omitted term (asin 0.134 y^4 < 0.05u, sin below that): < 5.5u.
template <typename T>
__device__ __forceinline__ double odd_small(double x, const T& C, uint32_t& bad) {
  const double y = x * x;
  const double p = fma(fma(C[4][0], y, C[3][0]), y * y, fma(C[2][0], y, C[1][0]));
  return add_test(x, (x * y) * p, bad);
}

// An odd series x + C1 x Y + x Y^2 Q, Y = x^2 exactly (yh + yl), with the
// leading correction in two words, so that the error is that of the y^2 term:
//   t1 + w = C1 Y + Y^2 Q,   x + x t1 exactly as hi + lo + pl,   the rest z.
// |x| < 2^-4 for sin (Q below 1/120: error < 2^-73 |x|), |x| < 2^-5 for atan
// (Q below 1/5, y < 2^-10: < 2^-72 |x|); the test spans 2^-71 |x|, 2^-17 of
// half an ulp.  A plain-double correction fails its test 0.3-0.5 % of the
// time at the 25-50 mrad of a bend, in one of eight warps.  extra: a term to
// add, its error within the same bound.
__device__ __forceinline__ double odd_two_word(double x, double yh, double yl, double y2q, double c1h, double c1l,
                                               double extra, uint32_t& bad) {
  const double t1 = yh * c1h;
  const double w = y2q + fma(yh, c1l, fma(yl, c1h, fma(yh, c1h, -t1)));
  const double p = x * t1;
  const double z = fma(x, w, fma(x, t1, -p)) + extra;
  const double hi = x + p;
  const double v = (p - (hi - x)) + z;
  const double a = hi + fma(x, FM_T[4], v);
  const double b = hi + fma(x, FM_T[5], v);
  bad |= lo_word(a) ^ lo_word(b);
  return a;
}
// sin(x), |x| < 2^-4; y2 = yh^2.  Terms to x^11 (omitted: 2^-80 |x|).
template <typename T>
__device__ __forceinline__ double sin_light(double x, double yh, double yl, double y2, const T& C, uint32_t& bad) {
  const double q = fma(fma(C[5][0], yh, C[4][0]), y2, fma(C[3][0], yh, C[2][0]));
  return odd_two_word(x, yh, yl, y2 * q, C[1][0], C[1][1], 0.0, bad);
}
// cos(x), |x| < 2^-4: 1 - Y / 2 + Y^2 Q, the first two terms exact in two
// words; error that of Y^2 Q < 2^-20.5: < 2^-70.5, the test spans 2^-70.
template <typename T>
__device__ __forceinline__ double cos_light(double yh, double yl, double y2, const T& C, uint32_t& bad) {
  const double q = fma(fma(C[5][0], yh, C[4][0]), y2, fma(C[3][0], yh, C[2][0]));
  const double w = fma(yl, -0.5, y2 * q);
  const double h = -0.5 * yh;
  const double hi = 1.0 + h;
  const double v = (h - (hi - 1.0)) + w;
  const double a = hi + (v - FM_T[6]);
  const double b = hi + (v + FM_T[6]);
  bad |= lo_word(a) ^ lo_word(b);
  return a;
}
// atan2(y, x) for x in [2^-30, 2^30], |y / x| < 2^-5 (else bad): the quotient
// qh + ql as in cr::atan2, atan(qh) by the two-word series (terms to q^15,
// omitted: 2^-84 |q|) plus ql (1 - qh^2) (dropped ql qh^4: 2^-73 |q|).
template <typename T>
__device__ __forceinline__ double atan2_light(double y, double x, const T& C, uint32_t& bad) {
  const double rx = rcp_faithful(x);
  const double q0 = y * rx;
  const double qh = fma(fma(-q0, x, y), rx, q0);
  const double ql = fma(-qh, x, y) * rx;
  bad |= abs_hi(qh) >= 0x3fa00000;
  const double yh = qh * qh, yl = fma(qh, qh, -yh), y2 = yh * yh;
  const double q = fma(fma(fma(C[7][0], yh, C[6][0]), y2, fma(C[5][0], yh, C[4][0])), y2, fma(C[3][0], yh, C[2][0]));
  return odd_two_word(qh, yh, yl, y2 * q, C[1][0], C[1][1], fma(-ql, yh, ql), bad);
}

}  // namespace bgt
