// The near-axis element maps and the arithmetic under them (test
// infrastructure), built for the host like device_maps_host.cpp.
//
//   near_maps_check math N SEED    bgt_fastmath.cuh against IEEE sqrt and
//                                  division, and against libquadmath rounded
//                                  to double wherever the rounding test holds
//   near_maps_check maps N SEED    track1_near against track1_general for
//                                  every record form that has a near-axis
//                                  form, inside, at and outside its region
//
// Prints "name mismatches passed total" lines; "passed" counts the values
// whose rounding test held, or the particles the near-axis form took.
#define __device__
#define __host__
#define __forceinline__ inline
#define __constant__

#include <math.h>
#include <quadmath.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <random>
#include <string>
#include <vector>

#include "../bmad-ecosystem_b200/csrc/bgt_compile.h"
#include "../bmad-ecosystem_b200/csrc/bgt_kernel.cuh"

using namespace bgt;

static std::mt19937_64 rng;
static double uni(double a, double b) { return a + (b - a) * (rng() >> 11) * 0x1p-53; }
static double logu(double a, double b) { return exp(uni(log(a), log(b))); }
static double sign() { return (rng() & 1) ? 1.0 : -1.0; }

struct Count {
  std::string name;
  long bad = 0, passed = 0, total = 0;
  void add(bool test_held, bool equal) {
    total++;
    if (!test_held) return;
    passed++;
    if (!equal) bad++;
  }
  ~Count() { printf("%s %ld %ld %ld\n", name.c_str(), bad, passed, total); }
};

static void math_checks(long n) {
  {
    Count c{"ps_terms"};
    auto one = [&](double v) {
      const PsTerms t = ps_terms(v);
      const double s = sqrt(v);
      c.add(true, t.ps == s && t.r_ps == 1.0 / s && t.r_ps1 == 1.0 / (s + 1.0));
    };
    const int64_t top = (int64_t)ldexp(1.0, 53) * 2 * pow(0x1p-7 / 0.875, 2);
    for (int64_t k = 0; k < 4096; k++) one(1.0 - k * 0x1p-53);
    for (int64_t k = 0; k < 4096; k++) one(1.0 - (top - k) * 0x1p-53);
    for (long i = 0; i < n; i++) one(1.0 - floor(logu(1, top)) * 0x1p-53);
  }
  {
    Count c{"div_rn"}, d{"div_test"};
    for (long i = 0; i < n; i++) {
      double b = logu(0.01, 100), a = sign() * logu(1e-30, 100);
      if (i % 4 == 0) {  // quotients next to a midpoint
        const double q = logu(0.01, 100);
        a = (double)((__float128)b * ((__float128)q + (__float128)nextafter(q, 1e9)) / 2);
      }
      c.add(true, div_rn(a, b, 1.0 / b) == a / b);
      uint32_t bad = 0;
      const double q = div_test(a, b, bad);
      d.add(!bad, q == a / b);
    }
  }
  {
    Count c{"sqrt_test"};
    for (long i = 0; i < n; i++) {
      double v = logu(0.1, 10);
      if (i % 4 == 0) {  // roots next to a midpoint
        const double s = logu(0.3, 3);
        const __float128 m = ((__float128)s + (__float128)nextafter(s, 1e9)) / 2;
        v = (double)(m * m);
      }
      uint32_t bad = 0;
      const double s = sqrt_test(v, rsqrt_near(v), bad);
      c.add(!bad, s == sqrt(v));
    }
  }
  {
    Count s{"sin_small"}, a{"asin_small"}, sl{"sin_light"}, cl{"cos_light"}, at{"atan2_light"};
    for (long i = 0; i < n; i++) {
      uint32_t bad = 0;
      double x = sign() * (i % 16 == 0 ? logu(1e-300, 0x1p-6) : logu(1e-9, 0x1p-6));
      double f = odd_small(x, cr::SIN_C, bad);
      s.add(!bad, f == (double)sinq(x));
      x = sign() * (i % 16 == 0 ? logu(1e-300, 0x1p-6 * 0.57) : logu(1e-9, 0x1p-6 * 0.57));
      bad = 0;
      f = odd_small(x, cr::ASIN_C, bad);
      a.add(!bad, f == (double)asinq(x));
      x = sign() * (i % 2 ? logu(1e-9, 0x1p-4) : uni(0.01, 0x1p-4));
      const double yh = x * x, yl = fma(x, x, -yh);
      bad = 0;
      f = sin_light(x, yh, yl, yh * yh, cr::SIN_C, bad);
      sl.add(!bad, f == (double)sinq(x));
      bad = 0;
      f = cos_light(yh, yl, yh * yh, cr::COS_C, bad);
      cl.add(!bad, f == (double)cosq(x));
      const double q = sign() * (i % 2 ? logu(1e-12, 0x1p-5) : uni(0.005, 0x1p-5)), r = logu(1e-3, 1e3);
      bad = 0;
      f = atan2_light(q * r, r, cr::ATAN_C, bad);
      at.add(!bad, f == (double)atan2q((__float128)(q * r), (__float128)r));
    }
  }
}

// ---------------------------------------------------------------------------

static const double MASS = 0.51099895069e6, P0C = 4999999973.888007, E_TOT = 5e9;

static bgt_element element(int key, double l) {
  bgt_element e;
  memset(&e, 0, sizeof(e));
  e.key = key;
  e.ix_ele = 1;
  e.is_on = 1;
  e.num_steps = 1;
  e.fringe_type = BGT_FRINGE_NONE;
  e.fringe_at = BGT_BOTH_ENDS;
  e.aperture_at = BGT_EXIT_END;
  e.l = l;
  e.ds_step = l != 0 ? fabs(l) : 0.2;
  e.p0c = P0C;
  e.e_tot = E_TOT;
  return e;
}

static bool same(double a, double b) { return a == b || (a != a && b != b); }

// One record form alone (then = false), and with the drift that follows it
// taken along (then = true), against the general maps one record at a time.
static void one_form(const std::string& name, bgt_element e, long n, bool then) {
  bgt_species sp;
  memset(&sp, 0, sizeof(sp));
  sp.mass = MASS;
  sp.charge = -1;
  sp.aperture_limit_on = 1;
  sp.max_aperture_limit = 1e3;
  std::vector<double> all;
  std::vector<int64_t> off;
  int32_t dw = 0;
  bool rare = false;
  std::string msg;
  Count c{name + (then ? "+drift" : "")};
  const bgt_element eles[2] = {e, element(BGT_DRIFT, 0.3)};
  if (host::compile_tables(eles, then ? 2 : 1, 1, sp, QMEMO_CLASSES, all, off, dw, rare, msg) || rare) {
    c.bad = -1;
    return;
  }
  const double* tab = all.data() + off[0];
  const int32_t* seq = reinterpret_cast<const int32_t*>(tab);
  const double *rec = tab + seq[0], *next = then ? tab + seq[2] : nullptr;
  const int32_t fl = reinterpret_cast<const RecHdr*>(rec)->flags;
  if (then != ((fl & F_THEN_DRIFT) != 0)) c.bad = -1;
  Glob G{};
  G.mc2 = MASS;
  G.mc2sq = MASS * MASS;
  G.p0c = P0C;
  G.mal = sp.max_aperture_limit;
  G.ap_on = 1;
  G.charge = -1;
  double qa[QMEMO_CLASSES * 13], qb[QMEMO_CLASSES * 13];
  for (double& q : qa) q = NAN;
  for (double& q : qb) q = NAN;
  for (long i = 0; i < n; i++) {
    // beam-like, on axis in one plane or both, around the region's edges, far outside
    const int kind = i % 8;
    const double s = kind < 4 ? 1 : kind < 6 ? 30 : 300;
    Part p{};
    p.x = kind == 1 ? 0.0 : s * uni(-1e-3, 1e-3);
    p.y = kind == 2 ? 0.0 : s * uni(-1e-3, 1e-3);
    p.px = kind == 1 ? 0.0 : s * uni(-2e-4, 2e-4);
    p.py = kind == 2 ? 0.0 : s * uni(-2e-4, 2e-4);
    p.z = uni(-1e-2, 1e-2);
    p.pz = kind == 3 ? uni(-2e-9, 2e-9) : kind == 6 ? uni(-0.2, 0.2) : uni(-1e-2, 1e-2);
    if (kind == 5) p.px = sign() * uni(0.99, 1.01) * 0x1p-7;
    if (kind == 3 && i % 3 == 0) p.x = p.px = p.y = p.py = 0;
    const double pc = (1 + p.pz) * P0C;
    p.beta = pc / sqrt(pc * pc + MASS * MASS);
    p.state = ALIVE;
    Part a = p;
    DriftMemo m;
    m.pz = NAN;
    const int todo = track1_near<false>(a, rec, fl, next, G, m, QMemo{qa, 1});
    bool a_drift = next && todo == TODO_NOTHING;  // the particle is past the element
    if (todo != TODO_NOTHING) {  // as track_warp_turn
      const bool in_drift = todo == TODO_DRIFT_EXIT;
      a_drift = track1_rest<false>(a, in_drift ? next : rec, in_drift ? nullptr : next, G, m, QMemo{qa, 1},
                                   in_drift ? (int)TODO_EXIT : todo) ||
                in_drift;
    }
    GeneralCall io = {p, &G, 0, 0, nullptr};
    track1_general<false>(&io, rec, QMemo{qb, 1}, TODO_ALL);
    const bool b_drift = next && io.p.state == ALIVE;
    if (b_drift) track1_general<false>(&io, next, QMemo{qb, 1}, TODO_ALL);
    const Part& b = io.p;
    const bool equal = same(a.x, b.x) && same(a.px, b.px) && same(a.y, b.y) && same(a.py, b.py) && same(a.z, b.z) &&
                       a.pz == b.pz && a.beta == b.beta && a.state == b.state && a_drift == b_drift;
    c.total++;
    if (todo == TODO_NOTHING || todo == TODO_BODY) c.passed++;
    if (!equal) c.bad++;
  }
}
static void one_form(const std::string& name, bgt_element e, long n) {
  one_form(name, e, n, false);
  if (e.key != BGT_DRIFT) one_form(name, e, n, true);
}

static void map_checks(long n) {
  host::c_multi_tables(c_cm, c_cm0);
  bgt_element d = element(BGT_DRIFT, 0.3);
  one_form("drift", d, n);
  d.l = -0.3;
  one_form("drift_back", d, n);
  d.l = 0;
  one_form("drift_zero", d, n);
  d = element(BGT_DRIFT, 0.3);
  d.aperture_type = BGT_APERTURE_RECTANGULAR;
  d.aperture_at = BGT_BOTH_ENDS;
  d.x1_limit = d.x2_limit = 8e-3;
  d.y1_limit = d.y2_limit = 6e-3;
  one_form("drift_rect", d, n);
  for (int sgn = -1; sgn <= 1; sgn += 2) {
    bgt_element q = element(BGT_QUADRUPOLE, 0.4);
    q.bn[1] = sgn * 0.32;
    one_form("quad", q, n);
    q.aperture_type = BGT_APERTURE_ELLIPTICAL;
    q.x1_limit = q.x2_limit = 0.01;
    q.y1_limit = 4e-3;
    q.y2_limit = 6e-3;
    one_form("quad_ellipse", q, n);
    q.x_offset = 5e-5;
    q.y_offset = -3e-5;
    q.tilt = 1e-3;
    q.has_misalign = 1;
    q.ds_step = 0.1;
    for (int k = 0; k <= 7; k++) {
      for (int j = 0; j <= 7; j++) q.an[j] = q.bn[j] = 0;
      q.bn[1] = sgn * 0.32;
      q.an[k] += pow(100.0, k - 1) * 1e-4;
      if (k != 1) q.bn[k] = -pow(100.0, k - 1) * 2e-4;
      if (k > 3) q.bn[k - 2] += pow(100.0, k - 3) * 1e-4;
      one_form("quad_errors_" + std::to_string(k), q, n);
    }
  }
  bgt_element s = element(BGT_SEXTUPOLE, 0.2);
  s.bn[2] = 0.35;
  one_form("sext", s, n);
  s.ds_step = 0.05;
  s.an[7] = 1e10;
  s.bn[5] = 1e6;
  s.tilt = 0.5;
  s.has_misalign = 1;
  one_form("sext_errors", s, n);
  bgt_element k = element(BGT_HKICKER, 0);
  k.bn[0] = 1e-4;
  one_form("kicker_zero_length", k, n);
  k = element(BGT_KICKER, 0.1);
  k.an[0] = -1e-3;
  one_form("kicker", k, n);
  for (double angle : {0.049, -0.049, 0.0124, 0.0624, 1e-3}) {
    bgt_element b = element(BGT_SBEND, 2.0);
    b.g = angle / 2.0;
    one_form("bend_no_edge", b, n);
    b.fringe_type = BGT_FRINGE_BASIC_BEND;
    one_form("bend", b, n);
    b.fringe_at = BGT_EXIT_END;
    b.aperture_type = BGT_APERTURE_ELLIPTICAL;
    b.x1_limit = b.x2_limit = b.y1_limit = b.y2_limit = 0.01;
    one_form("bend_exit_edge", b, n);
  }
}

int main(int argc, char** argv) {
  const long n = argc > 2 ? atol(argv[2]) : 100000;
  rng.seed(argc > 3 ? atol(argv[3]) : 1);
  if (argc > 1 && !strcmp(argv[1], "maps"))
    map_checks(n);
  else
    math_checks(n);
  return 0;
}
