// bgt_near.cuh -- near-axis forms of the common element maps.
//
// In a ring nearly every particle passes nearly every element well inside
// every limit, with small angles and momentum deviation.  For those the maps
// of bgt_kernel.cuh need none of their range checks, lost-particle branches
// and general quotients, and each element becomes one or a few basic blocks
// inside the element loop; the general maps, which also decide every loss,
// stay out of line.  All values are the general maps': the same operations
// in the same order, quotients, square roots and transcendentals the IEEE
// (correctly rounded) ones by bgt_fastmath.cuh.
//
// What bounds the tracker is FP64 latency and the FP64 pipe at 16 warps per
// SM.  Through the general maps alone a warp takes 319,000 instructions per
// turn of the 770-element ring, 140,000 of them FP64, at 44 % FP64 pipe: 17.7
// ns per particle and turn (1M particles, 256 x 2).  With the near-axis
// forms: 170,000, 77,000 FP64, 9.2 ns; one warp alone on its scheduler
// (10,000 particles) 0.54 ms per turn instead of 1.13.
#pragma once

namespace bgt {

// |x|, |y| below max_aperture_limit and |px|, |py| < 2^-7: with |pz| < 2^-3
// orbit_too_large finds nothing (bgt_device.cuh)
__device__ __forceinline__ bool inside_limits(double x, double px, double y, double py, const Glob& G) {
  return ((hi_word(x) | hi_word(y)) & 0x7fffffff) < hi_word(G.mal) && abs_hi(px) < NEAR_P_HI &&
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
// and square roots.  Returns ps_rel.
__device__ __forceinline__ double drift_near(Part& c, double length, double rel_pc, const DriftMemo& m) {
  const double px_rel = div_rn(c.px, rel_pc, m.r_pc);
  const double py_rel = div_rn(c.py, rel_pc, m.r_pc);
  const double pxy2 = px_rel * px_rel + py_rel * py_rel;
  const PsTerms T = ps_terms(1 - pxy2);
  c.x = c.x + div_rn(length * px_rel, T.ps, T.r_ps);
  c.y = c.y + div_rn(length * py_rel, T.ps, T.r_ps);
  c.z = c.z + length * (m.a + div_rn(div_rn(-pxy2, T.ps + 1.0, T.r_ps1), T.ps, T.r_ps));
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
// multiplication by the ones, no look-up); `poles` has bit n set for the
// orders with a coefficient, so an empty order costs one uniform branch, and
// a sextupole computes x^2 and y^2 only.  Sums start from their first term:
// kx_tot and ky_tot start from +0, which absorbs the sign of a zero sum.
__device__ __forceinline__ constexpr double binomial(int n, int m) {
  int b = 1;
  for (int i = 1; i <= m; i++) b = b * (n - m + i) / i;
  return b;
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

__device__ __forceinline__ void kicks_near(Part& c, const double* an, const double* bn, int32_t poles, double scale) {
  double kx = 0, ky = 0;
  double xp[8], yp[8];
  xp[0] = yp[0] = 1.0;
  xp[1] = c.x;
  yp[1] = c.y;
  xp[2] = xp[1] * xp[1];
  yp[2] = yp[1] * yp[1];
  if (poles & 1) kick_order<0>(xp, yp, scale * an[0], scale * bn[0], kx, ky);
  if (poles & 2) kick_order<1>(xp, yp, scale * an[1], scale * bn[1], kx, ky);
  if (poles & 4) kick_order<2>(xp, yp, scale * an[2], scale * bn[2], kx, ky);
  if (poles >= 8) {
    // the powers in mexp's order of products (powi_table7)
    xp[3] = xp[1] * xp[2];
    yp[3] = yp[1] * yp[2];
    xp[4] = xp[2] * xp[2];
    yp[4] = yp[2] * yp[2];
    xp[5] = xp[1] * xp[4];
    yp[5] = yp[1] * yp[4];
    xp[6] = xp[2] * xp[4];
    yp[6] = yp[2] * yp[4];
    if (poles & 8) kick_order<3>(xp, yp, scale * an[3], scale * bn[3], kx, ky);
    if (poles & 16) kick_order<4>(xp, yp, scale * an[4], scale * bn[4], kx, ky);
    if (poles & 32) kick_order<5>(xp, yp, scale * an[5], scale * bn[5], kx, ky);
    if (poles & 64) kick_order<6>(xp, yp, scale * an[6], scale * bn[6], kx, ky);
    if (poles & 128) {
      xp[7] = xp[3] * xp[4];
      yp[7] = yp[3] * yp[4];
      kick_order<7>(xp, yp, scale * an[7], scale * bn[7], kx, ky);
    }
  }
  c.px = c.px + kx;
  c.py = c.py + ky;
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

// The two quad_mat2_calc results of a body step (once a turn per memo class,
// or per quadrupole without one): out of line, so that its sine, hyperbolic
// and quotient code stays out of the element loop.
struct QuadMats {
  QMat x, y;
};
BGT_DEV_NOINLINE QuadMats quad_mats(double b1, double length, double step, double rel_p) {
  const double k1 = b1 / (length * rel_p);
  return {quad_mat2_calc(-k1, step, rel_p), quad_mat2_calc(k1, step, rel_p)};
}

// body_quad; false, with c unchanged, where low_energy_z_correction takes its
// exact form, or where a misaligned quadrupole's body leaves the near-axis
// region.  The correction of a step depends on pz and the element
// only, so it is evaluated once for all steps.
__device__ __forceinline__ bool quad_near(Part& c, const RecHdr* h, const double* mis, const double* q, QMemo qm) {
  const double pz = c.pz;
  const double* lez = q + Q_LEZ;
  const double beta0 = lez[LEZ_BETA0];
  if (!(lez[LEZ_MASS] * ((beta0 * pz) * (beta0 * pz)) < lez[LEZ_3E7])) return false;
  const double step = q[Q_STEP];
  const double dz_low = step * pz * (1 - 3 * (pz * (beta0 * beta0)) / 2 + (pz * pz) * lez[LEZ_F]) * lez[LEZ_ME2];
  const double rel_p = 1 + pz;
  const int cls = h->aux0, n_step = h->n_step;
  double* k = qm.q + (cls * 13) * qm.stride;
  QuadMats M;
  if (cls >= 0 && k[12 * qm.stride] == rel_p) {
    const int s = qm.stride;
    M.x = {k[0], k[s], k[2 * s], k[3 * s], k[4 * s], k[5 * s]};
    M.y = {k[6 * s], k[7 * s], k[8 * s], k[9 * s], k[10 * s], k[11 * s]};
  } else {
    M = quad_mats(q[Q_B1], q[Q_LEN], step, rel_p);
    if (cls >= 0) {
      const double v[13] = {M.x.cx, M.x.m01, M.x.m10, M.x.z0, M.x.z1, M.x.z2, M.y.cx,
                            M.y.m01, M.y.m10, M.y.z0, M.y.z1, M.y.z2, rel_p};
#pragma unroll
      for (int j = 0; j < 13; j++) k[j * qm.stride] = v[j];
    }
  }
  const int ix = h->ix_mag_max;
  const int32_t poles = h->poles;
  const double* an = q + Q_N;
  const double* bn = an + (ix + 1);
  Saved start(c);
  if (h->flags & F_MISALIGN) offset_near(c, mis, h->flags, true);
  if (ix > -1) kicks_near(c, an, bn, poles, q[Q_RHALF]);
  for (int i = 1; i <= n_step; i++) {
    const double x = c.x, px = c.px, y = c.y, py = c.py;
    c.z = c.z + (M.x.z0 * (x * x) + M.x.z1 * x * px + M.x.z2 * (px * px) + M.y.z0 * (y * y) + M.y.z1 * y * py +
                 M.y.z2 * (py * py));
    c.x = M.x.cx * x + M.x.m01 * px;
    c.px = M.x.m10 * x + M.x.cx * px;
    c.y = M.y.cx * y + M.y.m01 * py;
    c.py = M.y.m10 * y + M.y.cx * py;
    c.z = c.z + dz_low;
    if (ix > -1) kicks_near(c, an, bn, poles, (i == n_step) ? q[Q_RHALF] : q[Q_RSTEP]);
  }
  if (h->flags & F_MISALIGN) {
    // (offset_particle leaves the position of a particle past the momentum
    // limit as it is)
    if (!(abs_hi(c.px) < NEAR_P_HI && abs_hi(c.py) < NEAR_P_HI)) {
      start.restore(c);
      return false;
    }
    offset_near(c, mis, h->flags, false);
  }
  return true;
}

// body_thick: kick, drift, ..., kick; false, with c unchanged, when a kick
// leaves the near-axis region before a drift or the exit offset
__device__ __forceinline__ bool thick_near(Part& c, const RecHdr* h, const double* mis, const double* q,
                                           const Glob& G, const DriftMemo& m) {
  const int32_t fl = h->flags, poles = h->poles;
  const int ix = h->ix_mag_max, n_step = h->n_step;
  const double* an = q + TM_N;
  const double* bn = an + (ix + 1);
  const double step = q[TM_STEP], rel_pc = 1 + c.pz;
  Saved start(c);
  if (fl & F_MISALIGN) offset_near(c, mis, fl, true);
  if (ix > -1) kicks_near(c, an, bn, poles, q[TM_RHALF]);
  for (int i = 1; i <= n_step; i++) {
    if (!inside_limits(c.x, c.px, c.y, c.py, G)) {
      start.restore(c);
      return false;
    }
    if (step != 0) drift_near(c, step, rel_pc, m);
    if (ix > -1) kicks_near(c, an, bn, poles, (i == n_step) ? q[TM_RHALF] : q[TM_RSTEP]);
  }
  if (fl & F_MISALIGN) {
    if (!(abs_hi(c.px) < NEAR_P_HI && abs_hi(c.py) < NEAR_P_HI)) {
      start.restore(c);
      return false;
    }
    offset_near(c, mis, fl, false);
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

// The exact sector body with edges normal to the orbit (BEND_PLAIN records):
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
  bad |= !inside_limits(x, px, y, py, G);
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
  bad |= !inside_limits(x1, px1, y1, py, G);
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
// track1 through a record by its near-axis form.  What is left to the general
// maps: TODO_NOTHING; TODO_EXIT, the checks after the body, where the particle
// may be past a limit or an aperture; TODO_ALL, the whole element, p as it
// was.  TIME: the instance carries the particle time.
enum NearTodo : int { TODO_NOTHING = 0, TODO_EXIT = 1, TODO_ALL = 2 };

template <bool TIME>
__device__ __forceinline__ int track1_near(Part& p, const double* rec, const Glob& G, DriftMemo& m, QMemo qm) {
  const RecHdr* h = reinterpret_cast<const RecHdr*>(rec);
  const int32_t fl = h->flags;
  if (!(fl & F_NEAR)) return TODO_ALL;
  drift_memo(p, G, m);
  if (!(abs_hi(p.px) < m.near_p && abs_hi(p.py) < m.near_p)) return TODO_ALL;
  const double* q = rec + HDR_DW;
  const double* mis = q;
  if (fl & F_MISALIGN) q += MIS_N;
  const double* ap = q;
  if (fl & (F_AP_ENTRANCE | F_AP_EXIT)) q += AP_N;
  if ((fl & F_AP_ENTRANCE) && G.ap_on && !inside_aperture(p, ap, fl)) return TODO_ALL;
  const int32_t kind = h->kind;
  if (kind == K_DRIFT) {
    const double length = q[DR_L];
    if (length != 0) {
      const double ps = drift_near(p, length, 1 + p.pz, m);
      if (TIME && G.track_time) add_time(p, length / (p.beta * ps * C_LIGHT));
    }
  } else {
    const qp::Q t0 = time_of(p);
    const double z0 = p.z;
    double dt_ref;
    if (kind == K_BEND) {
      if (!bend_near(p, q, fl, G, m)) return TODO_ALL;
      dt_ref = q[B_DTREF];
    } else if (kind == K_QUAD) {
      if (!quad_near(p, h, mis, q, qm)) return TODO_ALL;
      dt_ref = q[Q_DTREF];
    } else {
      if (!thick_near(p, h, mis, q, G, m)) return TODO_ALL;
      dt_ref = q[TM_DTREF];
    }
    if (TIME) element_exit_time(p, t0, z0, dt_ref, G);
  }
  if (!inside_limits(p.x, p.px, p.y, p.py, G)) return TODO_EXIT;
  if ((fl & F_AP_EXIT) && G.ap_on && !inside_aperture(p, ap, fl)) return TODO_EXIT;
  return TODO_NOTHING;
}

}  // namespace bgt
