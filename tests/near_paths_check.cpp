// Which way a particle takes through a record, and that each way gives the
// general maps' values (test infrastructure), built for the host.
//
//   near_paths_check N SEED   prints "name kernel wrong inline body total"
//
// kernel: "plain", or "time" for the instances that carry the particle time,
// which is compared too.  inline: the particles that track1_near took through
// the whole record; body: those that body_near took through it.  Every
// particle goes through its record twice from the same start, the second time
// with the quadrupole matrices of its momentum in the memo, and only the
// second pass is counted; both are compared.
#define __device__
#define __host__
#define __forceinline__ inline
#define __constant__

#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <functional>
#include <random>
#include <string>
#include <vector>

#include "../bmad-ecosystem_b200/csrc/bgt_compile.h"
#include "../bmad-ecosystem_b200/csrc/bgt_kernel.cuh"

using namespace bgt;

static std::mt19937_64 rng;
static double uni(double a, double b) { return a + (b - a) * (rng() >> 11) * 0x1p-53; }
static double sign() { return (rng() & 1) ? 1.0 : -1.0; }

static const double MASS = 0.51099895069e6, P0C = 4999999973.888007, E_TOT = 5e9, C = 299792458.0;

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
  e.delta_ref_time = l / (P0C / E_TOT * C);
  return e;
}

static bool same(double a, double b) { return a == b || (a != a && b != b); }

// A particle of one of these kinds; the first four are well inside the
// near-axis region and every aperture of the forms below
enum Kind { BEAM, ON_AXIS, OFF_MOMENTUM, TINY, APERTURE, EDGE_P, EDGE_PZ, EDGE_X, WIDE, KINDS };
static Part particle(int kind, double mal) {
  Part p{};
  p.x = uni(-1e-3, 1e-3);
  p.y = uni(-1e-3, 1e-3);
  p.px = uni(-2e-4, 2e-4);
  p.py = uni(-2e-4, 2e-4);
  p.z = uni(-1e-2, 1e-2);
  p.pz = uni(-1e-2, 1e-2);
  switch (kind) {
    case ON_AXIS:
      if (rng() & 1) p.x = p.px = 0;
      else p.y = p.py = 0;
      break;
    case OFF_MOMENTUM:
      p.pz = sign() * uni(0.02, 0.12);
      break;
    case TINY:
      p.x = sign() * exp(uni(-744, -10));
      p.px = sign() * exp(uni(-744, -10));
      p.y = sign() * exp(uni(-744, -10));
      p.py = sign() * exp(uni(-744, -10));
      p.z = 0;
      break;
    case APERTURE:
      p.x = uni(-1.2e-2, 1.2e-2);
      p.y = uni(-8e-3, 8e-3);
      break;
    case EDGE_P:
      (rng() & 1 ? p.px : p.py) = sign() * (0x1p-7 + (int)(rng() % 9 - 4) * 0x1p-29);
      break;
    case EDGE_PZ:
      p.pz = sign() * (0x1p-3 + (int)(rng() % 9 - 4) * 0x1p-25);
      break;
    case EDGE_X:
      (rng() & 1 ? p.x : p.y) = sign() * mal * (1 + (int)(rng() % 9 - 4) * 0x1p-22);
      break;
    case WIDE:
      p.px = sign() * uni(0.008, 0.1);
      p.pz = uni(-0.3, 0.3);
      break;
  }
  const double pc = (1 + p.pz) * P0C;
  p.beta = pc / sqrt(pc * pc + MASS * MASS);
  p.state = ALIVE;
  const qp::Q t = qp::from_double(uni(-1e-6, 1e-6));
  p.t_lo = t.lo;
  p.t_hi = t.hi;
  return p;
}

template <bool TIME>
static void one_form(const std::string& name, const bgt_element& e, double then_length, bool then, long n) {
  bgt_species sp;
  memset(&sp, 0, sizeof(sp));
  sp.mass = MASS;
  sp.charge = -1;
  sp.aperture_limit_on = 1;
  sp.max_aperture_limit = 2.0;
  std::vector<double> all;
  std::vector<int64_t> off;
  int32_t dw = 0;
  bool rare = false;
  std::string msg;
  const bgt_element eles[2] = {e, element(BGT_DRIFT, then_length)};
  if (host::compile_tables(eles, then ? 2 : 1, 1, sp, QMEMO_CLASSES, all, off, dw, rare, msg) || rare) {
    printf("%s refused 1 0 0 0\n", name.c_str());
    return;
  }
  const double* tab = all.data() + off[0];
  const int32_t* seq = reinterpret_cast<const int32_t*>(tab);
  const double *rec = tab + seq[0], *next = then ? tab + seq[2] : nullptr;
  const int32_t fl = reinterpret_cast<const RecHdr*>(rec)->flags;
  long wrong = then != ((fl & F_THEN_DRIFT) != 0), in_line = 0, body = 0, total = 0;
  Glob G{};
  G.mc2 = MASS;
  G.mc2sq = MASS * MASS;
  G.p0c = P0C;
  G.mal = sp.max_aperture_limit;
  G.ap_on = 1;
  G.charge = -1;
  G.track_time = TIME;
  double qa[QMEMO_CLASSES * 13], qb[QMEMO_CLASSES * 13];
  for (double& q : qa) q = NAN;
  for (double& q : qb) q = NAN;
  for (long i = 0; i < n; i++) {
    const int kind = i % KINDS;
    const Part p = particle(kind, G.mal);
    GeneralCall io = {p, &G, 0, 0, nullptr};
    track1_general<TIME>(&io, rec, QMemo{qb, 1}, TODO_ALL);
    const bool b_drift = next && io.p.state == ALIVE;
    if (b_drift) track1_general<TIME>(&io, next, QMemo{qb, 1}, TODO_ALL);
    const Part& b = io.p;
    for (int pass = 0; pass < 2; pass++) {
      Part a = p;
      DriftMemo m;
      m.pz = NAN;
      const int todo = track1_near<TIME>(a, rec, fl, next, G, m, QMemo{qa, 1});
      Part f = a;  // what the near-axis forms alone make of it
      const int done = todo == TODO_NOTHING ? 2 : track1_finish<TIME>(f, rec, next, G, m, QMemo{qa, 1}, todo);
      bool a_drift = next && todo == TODO_NOTHING;
      if (todo != TODO_NOTHING) a_drift = track1_rest<TIME>(a, rec, next, G, m, QMemo{qa, 1}, todo);
      if (pass == 1 && kind <= TINY) {
        total++;
        if (todo == TODO_NOTHING || todo == TODO_EXIT || todo == TODO_DRIFT_EXIT) in_line++;
        if (todo == TODO_BODY && (done > 0 || f.state != ALIVE)) body++;
      }
      if (!(same(a.x, b.x) && same(a.px, b.px) && same(a.y, b.y) && same(a.py, b.py) && same(a.z, b.z) &&
            a.pz == b.pz && a.beta == b.beta && a.state == b.state && a_drift == b_drift && a.t_lo == b.t_lo &&
            a.t_hi == b.t_hi))
        wrong++;
    }
  }
  printf("%s %s %ld %ld %ld %ld\n", name.c_str(), TIME ? "time" : "plain", wrong, in_line, body, total);
}

static void form(const std::string& name, const bgt_element& e, long n) {
  one_form<false>(name, e, 0, false, n);
  one_form<true>(name, e, 0, false, n);
  if (e.key == BGT_DRIFT) return;
  const double lengths[] = {0.3, 0.0, -0.2, 11.0};
  for (int k = 0; k < 4; k++) {
    one_form<false>(name + "+drift" + std::to_string(k), e, lengths[k], true, n);
    one_form<true>(name + "+drift" + std::to_string(k), e, lengths[k], true, n);
  }
}

int main(int argc, char** argv) {
  const long n = argc > 1 ? atol(argv[1]) : 10000;
  rng.seed(argc > 2 ? atol(argv[2]) : 1);
  host::c_multi_tables(c_cm, c_cm0);
  auto limits = [](bgt_element& e, int type, int at) {
    e.aperture_type = type;
    e.aperture_at = at;
    e.x1_limit = e.x2_limit = 8e-3;
    e.y1_limit = 5e-3;
    e.y2_limit = 6e-3;
  };
  form("drift", element(BGT_DRIFT, 0.3), n);
  bgt_element e = element(BGT_MARKER, 0);
  form("marker", e, n);
  limits(e, BGT_APERTURE_RECTANGULAR, BGT_BOTH_ENDS);
  form("marker_rect", e, n);
  e = element(BGT_MONITOR, 0.1);
  form("monitor", e, n);
  e = element(BGT_HKICKER, 0.1);
  e.bn[0] = 1e-4;
  form("kicker", e, n);
  e.l = 0;
  e.delta_ref_time = 0;
  form("kicker_zero_length", e, n);
  for (int s = -1; s <= 1; s += 2) {
    e = element(BGT_QUADRUPOLE, 0.4);
    e.bn[1] = s * 0.32;
    form(s < 0 ? "quad_d" : "quad_f", e, n);
  }
  limits(e, BGT_APERTURE_ELLIPTICAL, BGT_BOTH_ENDS);
  form("quad_ellipse", e, n);
  e = element(BGT_SEXTUPOLE, 0.2);
  e.bn[2] = 0.35;
  form("sext", e, n);
  e.ds_step = 0.05;
  limits(e, BGT_APERTURE_RECTANGULAR, BGT_ENTRANCE_END);
  form("sext_rect", e, n);
  for (int hi = 2; hi <= 7; hi++) {
    for (int lo = 2; lo <= 4; lo++) {
      if (lo > hi) continue;
      bgt_element q = element(BGT_QUADRUPOLE, 0.4), s = element(BGT_SEXTUPOLE, 0.2);
      q.bn[1] = 0.32;
      q.ds_step = 0.1;
      s.ds_step = 0.05;
      for (int k = lo; k <= hi; k++) {
        q.an[k] = s.an[k] = pow(100.0, k - 1) * 1e-5 * (k % 2 ? 1 : -1);
        q.bn[k] = s.bn[k] = pow(100.0, k - 1) * 2e-5;
      }
      const std::string orders = std::to_string(lo) + std::to_string(hi);
      form("quad_poles" + orders, q, n);
      form("sext_poles" + orders, s, n);
      q.x_offset = s.x_offset = 5e-5;
      q.tilt = s.tilt = 1e-3;
      q.has_misalign = s.has_misalign = 1;
      form("quad_mis" + orders, q, n);
      form("sext_mis" + orders, s, n);
    }
  }
  e = element(BGT_QUADRUPOLE, 0.4);
  e.bn[1] = 0.32;
  e.y_offset = 1e-4;
  e.has_misalign = 1;
  form("quad_offset", e, n);
  for (double angle : {0.049, -0.0124}) {
    e = element(BGT_SBEND, 2.0);
    e.g = angle / 2.0;
    e.fringe_type = BGT_FRINGE_BASIC_BEND;
    form(angle > 0 ? "bend" : "bend_inverse", e, n);
  }
  return 0;
}
