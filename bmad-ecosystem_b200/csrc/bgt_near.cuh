// bgt_near.cuh -- near-axis forms of the common element maps.
//
// In a ring nearly every particle passes nearly every element well inside
// every limit, with small angles and momentum deviation.  For those the maps
// of bgt_kernel.cuh need none of their range checks, lost-particle branches
// and general quotients, and each element becomes one or a few basic blocks
// inside the element loop; the general maps, which also decide every loss,
// have a loop of their own.  All values are the general maps': the same operations
// in the same order, quotients, square roots and transcendentals the IEEE
// (correctly rounded) ones by bgt_fastmath.cuh.
//
// What bounds the tracker is FP64 latency and the FP64 pipe at 16 warps per
// SM.  Through the general maps alone a warp takes 319,000 instructions per
// turn of the 770-element ring, 140,000 of them FP64, at 44 % FP64 pipe: 17.7
// ns per particle and turn (1M particles, 256 x 2).  With the near-axis
// forms: 153,000, 75,000 FP64, 7.6 ns; one warp alone on its scheduler
// (10,000 particles) 0.41 ms per turn instead of 1.13.
#pragma once

namespace bgt {

// |x|, |y| below max_aperture_limit and |px|, |py| < 2^-7: with |pz| < 2^-3
// orbit_too_large finds nothing (bgt_device.cuh)
__device__ __forceinline__ bool inside_limits(double x, double px, double y, double py, double mal) {
  return ((hi_word(x) | hi_word(y)) & 0x7fffffff) < hi_word(mal) && abs_hi(px) < NEAR_P_HI &&
         abs_hi(py) < NEAR_P_HI;
}

// Whether the particle surely passes the aperture (ap: AP block).  Ellipse:
// the products instead of the quotients, each within 6 roundings, against 1 -
// 2^-40; a particle closer to the limit goes to the general check.
__device__ __forceinline__ bool inside_aperture(const Part& c, const double* ap, int32_t fl) {
  if (fl & F_AP_ELLIPTICAL) {
    const double xw = ap[AP_XW], yw = ap[AP_YW];
    const double a = (c.x - ap[AP_XC]) * yw, b = (c.y - ap[AP_YC]) * xw, w = xw * yw;
    return fma(a, a, b * b) < w * w * (1.0 - 0x1p-40);
  }
  const double x1 = ap[AP_X1], x2 = ap[AP_X2], y1 = ap[AP_Y1], y2 = ap[AP_Y2];
  return !(x1 != 0 && c.x < x1) && !(x2 != 0 && c.x > x2) && !(y1 != 0 && c.y < y1) && !(y2 != 0 && c.y > y2);
}

// track_a_drift for |px|, |py| < 2^-7, |pz| < 2^-3, beta > 0: about 45 FP64
// instructions and no branch in place of 85 and four range-checked quotients
// and square roots.  a and r_pc: the memo of pz.  Returns ps_rel.
__device__ __forceinline__ double drift_near(Part& c, double length, double rel_pc, double a, double r_pc) {
  const double px_rel = div_rn(c.px, rel_pc, r_pc);
  const double py_rel = div_rn(c.py, rel_pc, r_pc);
  const double pxy2 = px_rel * px_rel + py_rel * py_rel;
  const PsTerms T = ps_terms(1 - pxy2);
  c.x = c.x + div_rn(length * px_rel, T.ps, T.r_ps);
  c.y = c.y + div_rn(length * py_rel, T.ps, T.r_ps);
  c.z = c.z + length * (a + div_rn(div_rn(-pxy2, T.ps + 1.0, T.r_ps1), T.ps, T.r_ps));
  return T.ps;
}

// Coordinates put aside in memory while a map works on them in place, for the
// case that it has to be given up.  Kept in registers instead (a copy that
// lives through the map), they make the compiler move the particle's whole
// state between registers at every element: 55 moves each.
struct Saved {
  double v[5];
  __device__ __forceinline__ explicit Saved(const Part& p) : v{p.x, p.px, p.y, p.py, p.z} { hide(); }
  __device__ __forceinline__ void restore(Part& p) {
    hide();
    p.x = v[0];
    p.px = v[1];
    p.y = v[2];
    p.py = v[3];
    p.z = v[4];
  }

 private:
  // the stores and loads stay: the values are not forwarded in registers
  __device__ __forceinline__ void hide() {
#ifdef __CUDACC__
    asm volatile("" ::"l"(v) : "memory");
#endif
  }
};

// ---------------------------------------------------------------------------
// Magnetic multipole kicks up to order 7 (ab_multipole_kicks).  The factors
// c_multi(n, m) are signed binomials, here constants of the code (no
// multiplication by the ones, no look-up).  Sums start from their first
// term: kx_tot and ky_tot start from +0, which absorbs the sign of a zero
// sum.
__device__ __forceinline__ constexpr double binomial(int n, int m) {
  int b = 1;
  for (int i = 1; i <= m; i++) b = b * (n - m + i) / i;
  return b;
}

// x^k and y^k in mexp's order of products (powi_table7), up to k = TOP
template <int TOP>
__device__ __forceinline__ void powers(double x, double (&p)[8]) {
  p[0] = 1.0;
  p[1] = x;
  if (TOP >= 2) p[2] = x * x;
  if (TOP >= 3) p[3] = x * p[2];
  if (TOP >= 4) p[4] = p[2] * p[2];
  if (TOP >= 5) p[5] = x * p[4];
  if (TOP >= 6) p[6] = p[2] * p[4];
  if (TOP >= 7) p[7] = p[3] * p[4];
}

template <int N>
__device__ __forceinline__ void kick_order(const double (&xp)[8], const double (&yp)[8], double a2, double b2,
                                           double& kx_tot, double& ky_tot) {
  double kx = 0, ky = 0;
#pragma unroll
  for (int k = 0; k <= N; k++) {
    // even m first, then odd m
    const int m = 2 * k <= N ? 2 * k : 2 * (k - N / 2) - 1;
    const double c = (m % 4 == 0 || m % 4 == 3) ? -binomial(N, m) : binomial(N, m);
    const double f = m == 0 ? c * xp[N] : m == N ? c * yp[N] : c * xp[N - m] * yp[m];
    if (m % 2 == 0) {
      kx = k == 0 ? b2 * f : kx + b2 * f;
      ky = k == 0 ? -(a2 * f) : ky - a2 * f;
    } else {
      kx = kx + a2 * f;
      ky = ky + b2 * f;
    }
  }
  kx_tot = kx_tot + kx;
  ky_tot = ky_tot + ky;
}

// Orders LO .. HI, all present: one basic block, so that the chains of sums
// of the orders (N + 1 dependent additions each, 8 cycles apart) overlap: a
// quadrupole of 16 steps with orders 3 to 6 takes a warp alone on its
// scheduler 12,900 cycles instead of the 20,500 with a block per order.
template <int LO, int HI>
struct DenseKicks {
  __device__ __forceinline__ static void apply(Part& c, const double* an, const double* bn, int32_t, double scale) {
    double xp[8], yp[8], kx = 0, ky = 0;
    powers<HI>(c.x, xp);
    powers<HI>(c.y, yp);
    sum(xp, yp, an, bn, scale, kx, ky);
    c.px = c.px + kx;
    c.py = c.py + ky;
  }
  template <int N = LO>
  __device__ __forceinline__ static void sum(const double (&xp)[8], const double (&yp)[8], const double* an,
                                             const double* bn, double scale, double& kx, double& ky) {
    kick_order<N>(xp, yp, scale * an[N], scale * bn[N], kx, ky);
    if constexpr (N < HI) sum<N + 1>(xp, yp, an, bn, scale, kx, ky);
  }
};
// Any orders up to 7: one block per order that is present (bit n of poles)
struct SparseKicks {
  __device__ __forceinline__ static void apply(Part& c, const double* an, const double* bn, int32_t poles,
                                               double scale) {
    double xp[8], yp[8], kx = 0, ky = 0;
    powers<7>(c.x, xp);
    powers<7>(c.y, yp);
    if (poles & 1) kick_order<0>(xp, yp, scale * an[0], scale * bn[0], kx, ky);
    if (poles & 2) kick_order<1>(xp, yp, scale * an[1], scale * bn[1], kx, ky);
    if (poles & 4) kick_order<2>(xp, yp, scale * an[2], scale * bn[2], kx, ky);
    if (poles & 8) kick_order<3>(xp, yp, scale * an[3], scale * bn[3], kx, ky);
    if (poles & 16) kick_order<4>(xp, yp, scale * an[4], scale * bn[4], kx, ky);
    if (poles & 32) kick_order<5>(xp, yp, scale * an[5], scale * bn[5], kx, ky);
    if (poles & 64) kick_order<6>(xp, yp, scale * an[6], scale * bn[6], kx, ky);
    if (poles & 128) kick_order<7>(xp, yp, scale * an[7], scale * bn[7], kx, ky);
    c.px = c.px + kx;
    c.py = c.py + ky;
  }
};
// Orders 0 or 2 alone, or none: kickers, plain sextupoles, and what has no field
struct PlainKicks {
  __device__ __forceinline__ static bool holds(int32_t poles) { return (poles & ~4) == 0 || poles == 1; }
  __device__ __forceinline__ static void apply(Part& c, const double* an, const double* bn, int32_t poles,
                                               double scale) {
    if (poles == 4)
      DenseKicks<2, 2>::apply(c, an, bn, poles, scale);
    else if (poles == 1)
      DenseKicks<0, 0>::apply(c, an, bn, poles, scale);
  }
};
struct NoKicks {
  __device__ __forceinline__ static void apply(Part&, const double*, const double*, int32_t, double) {}
};

// f(kicks) for the orders of `poles`: dense from the sextupole or the octupole
// up, else sparse
template <class F>
__device__ __forceinline__ bool with_kicks(int32_t poles, const F& f) {
  switch (poles) {
    case 0x04: return f(DenseKicks<2, 2>{});
    case 0x0c: return f(DenseKicks<2, 3>{});
    case 0x1c: return f(DenseKicks<2, 4>{});
    case 0x3c: return f(DenseKicks<2, 5>{});
    case 0x7c: return f(DenseKicks<2, 6>{});
    case 0xfc: return f(DenseKicks<2, 7>{});
    case 0x08: return f(DenseKicks<3, 3>{});
    case 0x18: return f(DenseKicks<3, 4>{});
    case 0x38: return f(DenseKicks<3, 5>{});
    case 0x78: return f(DenseKicks<3, 6>{});
    case 0xf8: return f(DenseKicks<3, 7>{});
    default: return f(SparseKicks{});
  }
}

// offset_particle without pitch or a drift to the edge (F_NEAR records): the
// transverse offset and the roll
__device__ __forceinline__ void offset_near(Part& c, const double* mis, int32_t fl, bool set) {
  auto roll = [&](double co, double si) {
    const double x = c.x, y = c.y, px = c.px, py = c.py;
    c.x = co * x + si * y;
    c.y = -si * x + co * y;
    c.px = co * px + si * py;
    c.py = -si * px + co * py;
  };
  if (set) {
    if (fl & F_OFFSET) {
      c.x = c.x - mis[MIS_XOFF];
      c.y = c.y - mis[MIS_YOFF];
    }
    if (fl & F_TILT) roll(mis[MIS_COS], mis[MIS_SIN]);
  } else {
    if (fl & F_TILT) roll(mis[MIS_COSU], mis[MIS_SINU]);
    if (fl & F_OFFSET) {
      c.x = c.x + mis[MIS_XOFF];
      c.y = c.y + mis[MIS_YOFF];
    }
  }
}

// ---------------------------------------------------------------------------
// Quadrupole

// the two quad_mat2_calc results of a body step
struct QuadMats {
  QMat x, y;
};

// The body steps with their kicks
template <class KICKS>
__device__ __forceinline__ void quad_steps(Part& c, const QuadMats& M, double dz_low, const RecHdr* h,
                                           const double* q) {
  const int n_step = h->n_step;
  const int32_t poles = h->poles;
  const double* an = q + Q_N;
  const double* bn = an + (h->ix_mag_max + 1);
  const double r_half = q[Q_RHALF], r_step = q[Q_RSTEP];
#pragma unroll 1
  for (int i = 0;; i++) {
    KICKS::apply(c, an, bn, poles, i == 0 || i == n_step ? r_half : r_step);
    if (i >= n_step) break;
    const double x = c.x, px = c.px, y = c.y, py = c.py;
    c.z = c.z + (M.x.z0 * (x * x) + M.x.z1 * x * px + M.x.z2 * (px * px) + M.y.z0 * (y * y) + M.y.z1 * y * py +
                 M.y.z2 * (py * py));
    c.x = M.x.cx * x + M.x.m01 * px;
    c.px = M.x.m10 * x + M.x.cx * px;
    c.y = M.y.cx * y + M.y.m01 * py;
    c.py = M.y.m10 * y + M.y.cx * py;
    c.z = c.z + dz_low;
  }
}

// low_energy_z_correction of a step: it depends on pz and the element only,
// so one value serves all steps.  false where it takes its exact form.
__device__ __forceinline__ bool quad_low_energy(double pz, const double* q, double& dz_low) {
  const double* lez = q + Q_LEZ;
  const double beta0 = lez[LEZ_BETA0];
  if (!(lez[LEZ_MASS] * ((beta0 * pz) * (beta0 * pz)) < lez[LEZ_3E7])) return false;
  dz_low = q[Q_STEP] * pz * (1 - 3 * (pz * (beta0 * beta0)) / 2 + (pz * pz) * lez[LEZ_F]) * lez[LEZ_ME2];
  return true;
}

// The step matrices from the memo of the element's class; false where it has
// none for this momentum
__device__ __forceinline__ bool quad_memo(double rel_p, int cls, QMemo qm, QuadMats& M) {
  const int s = qm.stride;
  const double* k = qm.q + (cls * 13) * s;
  if (!(cls >= 0 && k[12 * s] == rel_p)) return false;
  M.x = {k[0], k[s], k[2 * s], k[3 * s], k[4 * s], k[5 * s]};
  M.y = {k[6 * s], k[7 * s], k[8 * s], k[9 * s], k[10 * s], k[11 * s]};
  return true;
}
__device__ __forceinline__ void quad_memo_fill(double rel_p, int cls, QMemo qm, const double* q, QuadMats& M) {
  const double k1 = q[Q_B1] / (q[Q_LEN] * rel_p);
  M = {quad_mat2_calc(-k1, q[Q_STEP], rel_p), quad_mat2_calc(k1, q[Q_STEP], rel_p)};
  if (cls < 0) return;
  double* k = qm.q + (cls * 13) * qm.stride;
  const double v[13] = {M.x.cx, M.x.m01, M.x.m10, M.x.z0, M.x.z1, M.x.z2, M.y.cx,
                        M.y.m01, M.y.m10, M.y.z0, M.y.z1, M.y.z2, rel_p};
#pragma unroll
  for (int j = 0; j < 13; j++) k[j * qm.stride] = v[j];
}

// ---------------------------------------------------------------------------
// Thick multipole: kick, drift, ..., kick; false when a kick leaves the
// near-axis region before a drift
template <class KICKS>
__device__ __forceinline__ bool thick_steps(Part& c, const RecHdr* h, const double* q, double mal, double a,
                                            double r_pc) {
  const int n_step = h->n_step;
  const int32_t poles = h->poles;
  const double* an = q + TM_N;
  const double* bn = an + (h->ix_mag_max + 1);
  const double step = q[TM_STEP], rel_pc = 1 + c.pz;
  const double r_half = q[TM_RHALF], r_step = q[TM_RSTEP];
#pragma unroll 1
  for (int i = 0;; i++) {
    KICKS::apply(c, an, bn, poles, i == 0 || i == n_step ? r_half : r_step);
    if (i >= n_step) break;
    if (!inside_limits(c.x, c.px, c.y, c.py, mal)) return false;
    if (step != 0) drift_near(c, step, rel_pc, a, r_pc);
  }
  return true;
}

// ---------------------------------------------------------------------------
// The body of a F_NEAR quadrupole or thick multipole with a sextupole or
// higher order, misaligned or not: between the near-axis loop and the general
// one (track_warp_turn), so that the near-axis loop holds the registers and
// the code of the plain elements only (within it, they raised every drift's
// spills from 6 loads to 13).  The change of place costs ~150 issue slots,
// which a body with only orders 0 and 1 does not win back (606,208 particles x
// 16 such magnets 0.33 ms, by the general maps 0.18): those go to the general
// maps.  false, p unchanged, for the general maps too: the exact low-energy
// correction, or a particle that leaves the near-axis region on the way
// (offset_particle then leaves its position as it is).
//
// The kicks stand at one place in each of the loops over the steps, which are
// not unrolled: a first half kick of its own before the loop doubles the code
// (a kernel instance compiles in 55 s instead of 24), and a peeled first step
// costs registers in the near-axis loop (10,000 particles x 16 turns of the
// ring 6.5 -> 6.4 ms without).
__device__ __forceinline__ bool body_near(Part& p, const RecHdr* h, const double* mis, const double* q, double mal,
                                          double a, double r_pc, QMemo qm) {
  const int32_t fl = h->flags;
  double dz_low;
  if (h->kind == K_QUAD && !quad_low_energy(p.pz, q, dz_low)) return false;
  Saved start(p);
  if (fl & F_MISALIGN) offset_near(p, mis, fl, true);
  if (h->kind == K_QUAD) {
    QuadMats M;
    if (!quad_memo(1 + p.pz, h->aux0, qm, M)) quad_memo_fill(1 + p.pz, h->aux0, qm, q, M);
    with_kicks(h->poles, [&](auto kicks) {
      quad_steps<decltype(kicks)>(p, M, dz_low, h, q);
      return true;
    });
  } else {
    if (!with_kicks(h->poles, [&](auto kicks) { return thick_steps<decltype(kicks)>(p, h, q, mal, a, r_pc); })) {
      start.restore(p);
      return false;
    }
  }
  if (fl & F_MISALIGN) {
    if (!(abs_hi(p.px) < NEAR_P_HI && abs_hi(p.py) < NEAR_P_HI)) {
      start.restore(p);
      return false;
    }
    offset_near(p, mis, fl, false);
  }
  return true;
}

// ---------------------------------------------------------------------------
// Bend

// The Hwang edge where its constants other than gs2 (and g + gt2) vanish: a
// pole face normal to the orbit without a fringe integral or k1.  The terms
// left are the general form's, in its order; the others are zeros added to
// them.  e = 1 / (1 + pz).
template <bool ENTERING>
__device__ __forceinline__ void hwang_edge_normal(double& x, double px, double y, double& py, double& z, double e,
                                                  const double* E) {
  const double gs2 = E[EDGE_GS2], gpg = E[EDGE_GPG];
  const double y2 = y * y;
  const double dx = gs2 * y2 * e / 2;
  const double dpy = gpg * px * y * e;
  const double dz = (e * e) * 0.5 * (px * y2 * gs2);
  if (ENTERING) {
    x = x + dx;
    py = py - dpy;
    z = z - dz;
  } else {
    x = x - dx;
    py = py + dpy;
    z = z + dz;
  }
}

// The exact sector body with edges normal to the orbit (F_NEAR bends,
// bend_is_plain in bgt_compile.h):
// the arithmetic of body_bend's exact step, every rounded value the same, in
// one basic block.  false where body_bend has to decide: a rounding test
// that failed, an argument outside the light ranges, the near-axis
// semi-linear map, or a particle that may be past a limit on the way.
//
// Bends take 40 % of a turn of the FODO ring.  The general body is a chain
// of 11 quotients and square roots and six correctly rounded functions, each
// with its own range checks and fallbacks: ~1000 instructions of which 590
// FP64, in ~60 basic blocks, waiting on FP64 latency most of the time.  Here
// ~250 FP64 instructions are left and the compiler interleaves the chains.
__device__ __forceinline__ bool bend_near(Part& p, const double* q, int32_t fl, const Glob& G, const DriftMemo& m) {
  uint32_t bad = 0;
  Saved start(p);
  double x = p.x, px = p.px, y = p.y, py = p.py, z = p.z;
  const double pz = p.pz;
  const double e = m.r_pc;
  if (fl & F_EDGE_IN) hwang_edge_normal<true>(x, px, y, py, z, e, q + B_EDGE);
  bad |= !inside_limits(x, px, y, py, G.mal);
  // the semi-linear map needs |px|, |py|, |pz| < 1e-9 (high word 0x3e112e0b)
  if (fl & F_SEMI_LINEAR_OK)
    bad |= abs_hi(px) <= 0x3e112e0b && abs_hi(py) <= 0x3e112e0b && abs_hi(pz) <= 0x3e112e0b;
  const double g = q[B_G], g_tot = q[B_GTOT], angle = q[B_ANGLE], sinc_a = q[B_SINCA], step_len = q[B_STEP];
  const double rel_p = 1 + pz;
  const double pt2 = rel_p * rel_p - py * py;
  const double y_pt = rsqrt_near(pt2);
  const double pt = sqrt_test(pt2, y_pt, bad);
  const double r_pt = fma(fma(-pt, y_pt, 1.0), y_pt, y_pt);
  bad |= lo_word(pt) == 0xffffffffu;
  const double g_p = div_rn(g_tot, pt, r_pt);
  const double phi_1 = odd_small(div_rn(px, pt, r_pt), cr::ASIN_C, bad);
  const double a1 = angle + phi_1;
  bad |= abs_hi(a1) >= 0x3fb00000;
  const double ah = a1 * a1, al = fma(a1, a1, -ah), a4 = ah * ah;
  const double sin_plus = sin_light(a1, ah, al, a4, cr::SIN_C, bad), cos_plus = cos_light(ah, al, a4, cr::COS_C, bad);
  const double gx1 = 1 + g * x;
  const double t1 = gx1 * step_len * sinc_a;
  const double alpha = 2 * gx1 * sin_plus * step_len * sinc_a - g_p * (t1 * t1);
  const double r = cos_plus * cos_plus + g_p * alpha;
  bad |= (uint32_t)(hi_word(r) - 0x3fe00000) >= 0x00200000u;  // r in [1/2, 2)
  const double rad = sqrt_test(r, rsqrt_near(r), bad);
  const double xi = div_test(alpha, rad + cos_plus, bad);
  const double x1 = x * q[B_COSA] - q[B_LL2GCOSC] + xi;
  const double l_v = q[B_LLSINC] + x * q[B_SINA];  // -L_v
  bad |= (uint32_t)(hi_word(l_v) - 0x3e100000) >= 0x03e00000u;  // l_v in [2^-30, 2^32)
  const double lc2 = l_v * l_v + xi * xi;
  const double L_c = sqrt_test(lc2, rsqrt_near(lc2), bad);
  const double h = a1 - atan2_light(xi, l_v, cr::ATAN_C, bad);  // angle_p / 2
  const double ha = fabs(h);
  bad |= (uint32_t)(hi_word(ha) - 0x3e500000) >= 0x01600000u;  // |h| in [2^-26, 2^-4): above sinc's 1e-8
  const double hh = ha * ha, hl = fma(ha, ha, -hh);
  const double L_p = div_test(L_c, div_test(sin_light(ha, hh, hl, hh * hh, cr::SIN_C, bad), ha, bad), bad);
  const double arg = a1 - 2 * h;
  bad |= abs_hi(arg) >= 0x3f900000;  // 2^-6
  const double px1 = pt * odd_small(arg, cr::SIN_C, bad);
  double y1 = y + div_rn(py * L_p, pt, r_pt);
  double z1 = z + div_rn(p.beta * step_len, q[B_BETAREF], q[B_RBETAREF]) - div_rn(rel_p * L_p, pt, r_pt);
  bad |= !inside_limits(x1, px1, y1, py, G.mal);
  double x2 = x1;
  if (fl & F_EDGE_OUT) hwang_edge_normal<false>(x2, px1, y1, py, z1, e, q + B_EDGE + EDGE_N);
  p.x = x2;
  p.px = px1;
  p.y = y1;
  p.py = py;
  p.z = z1;
  if (bad) start.restore(p);
  return bad == 0;
}

// ---------------------------------------------------------------------------
// track1 through a record by its near-axis form.  What is left to do
// (track1_finish): TODO_NOTHING; TODO_EXIT, the checks after the body, where
// the particle may be past a limit or an aperture; TODO_BODY, the body and
// those checks; TODO_ALL, the whole element by the general maps.  With the
// last two p is as it was.  fl: the header's flags.  TIME: the instance
// carries the particle time.
// With then (the record has F_THEN_DRIFT) its drift record follows in the same
// call, without the loads, tests and the vote of an element of its own (1M
// particles x 2 turns 18.1 -> 16.9 ms, 10,000 x 16 turns 8.45 -> 7.35);
// TODO_DRIFT_EXIT: the checks after that drift are left.
enum NearTodo : int { TODO_NOTHING = 0, TODO_EXIT = 1, TODO_BODY = 2, TODO_ALL = 3, TODO_DRIFT_EXIT = 4 };

// a drift record (the doubles before its length are the header) for a particle
// in the near-axis region
template <bool TIME>
__device__ __forceinline__ void drift_record_near(Part& p, const double* rec, const Glob& G, double a, double r_pc) {
  const double length = rec[HDR_DW + DR_L];
  if (length == 0) return;
  const double ps = drift_near(p, length, 1 + p.pz, a, r_pc);
  if (TIME && G.track_time) add_time(p, length / (p.beta * ps * C_LIGHT));
}

template <bool TIME>
__device__ __forceinline__ int track1_near(Part& p, const double* rec, int32_t fl, const double* then,
                                           const Glob& G, DriftMemo& m, QMemo qm) {
  const RecHdr* h = reinterpret_cast<const RecHdr*>(rec);
  const int32_t kind = h->kind;
  if (!(fl & F_NEAR)) return TODO_ALL;
  drift_memo(p, G, m);
  if (!(abs_hi(p.px) < m.near_p && abs_hi(p.py) < m.near_p)) return TODO_ALL;
  const double* q = rec + HDR_DW;
  if (fl & F_MISALIGN) q += MIS_N;
  const double* ap = q;
  if (fl & (F_AP_ENTRANCE | F_AP_EXIT)) q += AP_N;
  if ((fl & F_AP_ENTRANCE) && G.ap_on && !inside_aperture(p, ap, fl)) return TODO_ALL;
  if (kind == K_DRIFT) {
    drift_record_near<TIME>(p, q - HDR_DW, G, m.a, m.r_pc);
  } else if (kind != K_MARKER) {
    const qp::Q t0 = time_of(p);
    const double z0 = p.z;
    double dt_ref;
    if (kind == K_BEND) {
      if (!bend_near(p, q, fl, G, m)) return TODO_ALL;
      dt_ref = q[B_DTREF];
    } else if (kind == K_QUAD) {
      QuadMats M;
      double dz_low;
      if ((fl & F_MISALIGN) || h->poles != 0 || !quad_memo(1 + p.pz, h->aux0, qm, M)) return TODO_BODY;
      if (!quad_low_energy(p.pz, q, dz_low)) return TODO_ALL;
      quad_steps<NoKicks>(p, M, dz_low, h, q);
      dt_ref = q[Q_DTREF];
    } else {
      if ((fl & F_MISALIGN) || !PlainKicks::holds(h->poles)) return TODO_BODY;
      Saved start(p);
      if (!thick_steps<PlainKicks>(p, h, q, G.mal, m.a, m.r_pc)) {
        start.restore(p);
        return TODO_ALL;
      }
      dt_ref = q[TM_DTREF];
    }
    if (TIME) element_exit_time(p, t0, z0, dt_ref, G);
  }
  if (!inside_limits(p.x, p.px, p.y, p.py, G.mal)) return TODO_EXIT;
  if ((fl & F_AP_EXIT) && G.ap_on && !inside_aperture(p, ap, fl)) return TODO_EXIT;
  if (then) {
    drift_record_near<TIME>(p, then, G, m.a, m.r_pc);
    if (!inside_limits(p.x, p.px, p.y, p.py, G.mal)) return TODO_DRIFT_EXIT;
  }
  return TODO_NOTHING;
}

}  // namespace bgt
