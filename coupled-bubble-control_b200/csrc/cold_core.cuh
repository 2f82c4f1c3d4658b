// cold_core.cuh -- what the Richardson forms outside ckm1d_core.cuh share
// (solo_core.cuh, wide_core.cuh, duo_core.cuh): a system's scalars in shared
// memory, the right-hand side's parts as functions, the controller.
//
// Same operations in the same order as ckm1d_core.cuh.
#pragma once

#include "ckm1d_core.cuh"

namespace cbc {

// Scalars of a system that an attempt touches once or not at all: kept in
// shared memory, so that they take no registers inside the right-hand side.
// One record per system: written when the system is loaded, then read by all its
// lanes, and the counters by its first lane alone.
struct Cold {
  double sp0, sp3;             // 3 gamma, c
  double t_end, t_begin;
  double ddt;                  // spacing of the dense samples
  long long boff, step_base;   // batched form: first bubble row; steps accumulated before this load
  double fast_until;           // range of the interleaved functions
  int rejected, conv_ok, conv_fail;
  long long lin_iters;
};
static_assert(sizeof(Cold) % 16 == 8, "odd multiple of 8 bytes: neighbouring records on different banks");
// The ones that every lane of a system updates for itself.
struct LaneCold {
  double dnext;                // next dense sample time
  int idx;                     // dense samples stored
  int steps;
};

// Per-lane copy of a system's scalars.
struct ScalarState {
  double t, h, g_old;
  Cold* c;
  LaneCold* o;
  int status;
  bool active;
  bool lead;                   // first lane of its system
};

// Integrator state of a lane that holds one bubble.
struct BubbleState : ScalarState {
  double y[4];                 // R, X, U, V
};

// Coupling terms of a partner bubble j, from its state (recomputed by every
// lane that needs them exactly as the owning lane computes them: cheaper than
// exchanging seven terms).
struct PartnerTerms {
  double x1, j02, j03, h0, h1, h2, h3, h4;
};

__device__ __forceinline__ PartnerTerms partner_terms(double2 xa, double2 xb) {
  const double xj0 = xa.x, xj2 = xb.x, xj3 = xb.y;
  PartnerTerms q;
  q.x1 = xa.y;
  q.j02 = xj0 * xj0;
  q.j03 = q.j02 * xj0;
  q.h0 = xj0 * (xj2 * xj2);
  q.h1 = q.j02 * xj2;
  q.h2 = q.h1 * xj3;
  q.h3 = q.j03 * xj3;
  q.h4 = q.h3 * xj3;
  return q;
}

// Distance |x_i - x_j| (at least 1e-30) and sign of x_i - x_j.
__device__ __forceinline__ void pair_distance(double xi, double xj, double& ad, double& sg) {
  const double delta = xi - xj;
  sg = (double)((delta > 0.0) - (delta < 0.0));
  ad = fabs(delta);
  ad = ad > 1e-30 ? ad : 1e-30;
}

// The three sums a partner q at inverse distance rd contributes to, before
// the coupling coefficients, and its entries of the implicit matrix.
struct PairTerms {
  double t0, t1, t2, a, b, c, d;
};

__device__ __forceinline__ PairTerms pair_terms(const PartnerTerms& q, double rd, double sg, double m0, double m1) {
  PairTerms p;
  const double rd2 = rd * rd;
  const double srd2 = rd2 * sg;
  const double rd3 = rd2 * rd;
  p.t0 = fma(2.0 * rd, q.h0, fma(2.5 * srd2, q.h2, rd3 * q.h4));
  p.t1 = fma(srd2, q.h1, rd3 * q.h3);
  p.t2 = fma(2.0 * srd2, q.h0, (5.0 * rd3) * q.h2);
  p.a = (m0 * rd) * q.j02;
  p.b = ((0.5 * m0) * srd2) * q.j03;
  p.c = -((m1 * srd2) * q.j02);
  p.d = -((m1 * rd3) * q.j03);
  return p;
}

// Elementary functions of several arguments, interleaved (FAST) or one after the
// other with the general ones.  Same values.
template <bool FAST, int N>
__device__ __forceinline__ void f_rcp(const double (&x)[N], double (&y)[N]) {
  if constexpr (FAST) {
    cbcd::rcp(x, y);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) y[i] = 1.0 / x[i];
  }
}
template <bool FAST, int N>
__device__ __forceinline__ void f_sincos(const double (&x)[N], double (&s)[N], double (&c)[N]) {
  if constexpr (FAST) {
    cbcd::sincos(x, s, c);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) cbcm::sincos(x[i], &s[i], &c[i]);
  }
}
template <bool FAST, int N>
__device__ __forceinline__ void f_pow(const double (&x)[N], double y, double (&out)[N]) {
  if constexpr (FAST) {
    double yy[N];
#pragma unroll
    for (int i = 0; i < N; ++i) yy[i] = y;
    cbcd::pow_pos(x, yy, out);
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = cbcm::pow_pos(x[i], y);
  }
}
// Sums of the explicit coupling over the partners of one bubble.
struct PairSums {
  double g0, g1, tn, tg2, tg3;
};

// The part of a bubble's right-hand side that no partner enters: field,
// Keller--Miksis and translation (acoustic_field_1d ckm1d_def.py:79-114,
// ode_fun :418-447).
struct OwnTerms {
  double rx0, rD;                // 1 / R and 1 / denominator
  double pa, pt, px, ux;         // field at the bubble
  double p;                      // (1/R)^(3 gamma)
};

template <class Hc>
__device__ __forceinline__ void add_field(OwnTerms& o, const Hc& hc, int ac, int k, double st, double ct, double sx,
                                          double cx) {
  const double a = hc(k, 3), aw = hc(k, 4);
  if (ac == 0) {  // CONST
    o.pa = fma(a, st, o.pa);
    o.pt = fma(aw, ct, o.pt);
    return;
  }
  const double awv = hc(k, 5), au = hc(k, 6);
  if (ac == 1) {  // SW_N
    o.pa = fma(a * sx, st, o.pa);
    o.pt = fma(aw * sx, ct, o.pt);
    o.px = fma(awv * cx, st, o.px);
    o.ux = fma(au * cx, ct, o.ux);
  } else {  // SW_A
    o.pa = fma(a * cx, st, o.pa);
    o.pt = fma(aw * cx, ct, o.pt);
    o.px = fma(-(awv * sx), st, o.px);
    o.ux = fma(-(au * sx), ct, o.ux);
  }
}

// hc(k, c): harmonic constants of the system; D: the denominator.  NKC
// harmonics and field type ACC known at compile time, or (0, -1) both read
// from P.  split: the group has a lane per harmonic (group base `base`, lane
// li), so each computes one of the harmonics in time and they are shuffled;
// else every lane computes all of them.
template <int NKC, int ACC, bool FAST, bool SPLIT, class Hc>
__device__ __forceinline__ OwnTerms own_terms(const Params& P, const Hc& hc, double sp0, double t, double x0, double x1,
                                              double D, int base, int li) {
  OwnTerms o{0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int ac = ACC >= 0 ? ACC : P.ac;
  double rc[2];
  f_rcp<FAST, 2>({x0, D}, rc);
  o.rx0 = rc[0];
  o.rD = rc[1];
  if constexpr (NKC > 0) {
    // one batch: the harmonics at the bubble, then in time
    constexpr int NT = SPLIT ? 1 : NKC;
    double ph[NKC + NT], sn[NKC + NT], cn[NKC + NT];
#pragma unroll
    for (int k = 0; k < NKC; ++k) ph[k] = fma(hc(k, 2), x1, hc(k, 1));
#pragma unroll
    for (int k = 0; k < NT; ++k) {
      const int kk = SPLIT ? (li < NKC ? li : 0) : k;
      ph[NKC + k] = fma(hc(kk, 0), t, hc(kk, 1));
    }
    f_sincos<FAST>(ph, sn, cn);
#pragma unroll
    for (int k = 0; k < NKC; ++k) {
      const double st = SPLIT ? shfl(sn[NKC], base + k) : sn[NKC + (SPLIT ? 0 : k)];
      const double ct = SPLIT ? shfl(cn[NKC], base + k) : cn[NKC + (SPLIT ? 0 : k)];
      add_field(o, hc, ac, k, st, ct, sn[k], cn[k]);
    }
  } else {
#pragma unroll 1
    for (int k = 0; k < P.nk; ++k) {
      double sn[2], cn[2];
      f_sincos<FAST, 2>({fma(hc(k, 2), x1, hc(k, 1)), fma(hc(k, 0), t, hc(k, 1))}, sn, cn);
      add_field(o, hc, ac, k, sn[1], cn[1], sn[0], cn[0]);
    }
  }
  double pw[1];
  f_pow<FAST, 1>({o.rx0}, sp0, pw);
  o.p = pw[0];
  return o;
}

// Right-hand sides b0, b1 of the implicit system of a bubble; up(p): its
// constants.
template <class Up>
__device__ __forceinline__ void implicit_rhs(const OwnTerms& o, const PairSums& s, const Up& up, double sp3, double x0,
                                             double x2, double x3, double& b0, double& b1) {
  const double u7 = up(7);
  const double q = fma(u7, x2, 1.0);
  double N = fma(up(1), x2, up(0)) * o.p;
  N = fma(-up(2), q, N);
  N = fma(-up(3), o.rx0, N);
  N = fma(-(up(4) * x2), o.rx0, N);
  const double w = fma(-(u7 * (1.0 / 3.0)), x2, 1.0);
  N = fma((-1.5 * w) * x2, x2, N);
  N = fma(-(q * up(5)), o.pa, N);
  N = fma(-(up(6) * o.pt), x0, N);
  N = fma(up(8) * x3, x3, N);
  const double x02 = x0 * x0;
  const double x03 = x02 * x0;
  const double Fb1 = -(up(10) * x03) * o.px;
  const double Fd = -(up(11) * x0) * fma(x3, sp3, -o.ux);
  const double rx03 = (o.rx0 * o.rx0) * o.rx0;
  const double n0 = N * o.rD;
  const double n1 = fma((3.0 * (Fb1 + Fd)) * up(9), rx03, -(((3.0 * x2) * o.rx0) * x3));
  const double cpf1 = x3 * o.rD, cpf2 = x2 * o.rx0, cpf3 = o.rx0 * o.rx0;
  b0 = fma(s.g0, o.rD, fma(s.g1, cpf1, n0));
  b1 = n1 + fma(s.tg2, cpf2, fma(s.tg3, cpf3, s.tn));
}

// Exact sample time k of the grid dense mode.
__device__ __forceinline__ double grid_time(const ScalarState& S, int k, int ndo) {
  if (k >= ndo - 1 && ndo > 1) return S.c->t_end;
  return fma((double)k, S.c->ddt, S.c->t_begin);
}

// Sets up the dense schedule and the status at (re)load time.  Mirrors the
// kernel prologue (stepper.py:179-214) with the launch-transparent dense
// schedule.  `prev_time` is the time of the last stored sample (idx > 0).
// A stored failure status (-2, -3, -4) keeps the system stopped, so a failed
// system does not retry at every relaunch; -1 (budget spent) resumes.
__device__ __forceinline__ void prologue(ScalarState& S, const Params& P, double t_end, double t_begin, double g_store,
                                         double prev_time, int status_in) {
  S.status = (S.t >= t_end) ? ST_SUCCESS : ST_ACTIVE;
  if (fabs(g_store) < P.etol) S.status = ST_EVENT;
  if (status_in <= ST_STEP_LIMIT) S.status = status_in;
  S.active = (S.status == ST_ACTIVE);
  S.g_old = g_store;
  const double ddt = (P.ndo == 1) ? (t_end - t_begin) : (P.ndo > 1 ? (t_end - t_begin) / (double)(P.ndo - 1) : 0.0);
  if (P.dense_mode == 0) {
    if (S.o->idx == 0) S.o->dnext = S.t;
    else {
      const double nx = prev_time + ddt;
      S.o->dnext = nx < t_end ? nx : t_end;
    }
  }
  S.o->steps = 0;
  if (S.lead) {
    S.c->t_end = t_end;
    S.c->t_begin = t_begin;
    S.c->ddt = ddt;
    S.c->rejected = S.c->conv_ok = S.c->conv_fail = 0;
    S.c->lin_iters = 0;
  }
}

// Whether a system just loaded stores a dense sample before its first step.
__device__ __forceinline__ bool first_sample(const ScalarState& S, const Params& P) {
  if (!S.active || S.o->idx >= P.ndo) return false;
  return P.dense_mode == 0 ? S.o->dnext <= S.t : S.t >= grid_time(S, S.o->idx, P.ndo);
}

// Advances the dense schedule after that sample.
__device__ __forceinline__ void first_stored(ScalarState& S, const Params& P) {
  S.o->idx += 1;
  if (P.dense_mode == 0) {
    const double nx = S.t + S.c->ddt;
    S.o->dnext = nx < S.c->t_end ? nx : S.c->t_end;
  }
}

// State at Cash-Karp stage ST: y + h * sum_{m < ST} b[ST][m] k_m, the sum
// accumulated in increasing m (coefficients and loop fully compile-time).
template <int ST>
__device__ __forceinline__ void stage_state(const double* ks, int stride, double h, const double y[4], double ys[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    double acc = kStageB[ST][0] * ks[c * stride];
#pragma unroll
    for (int m = 1; m < ST; ++m) acc = fma(kStageB[ST][m], ks[(m * 4 + c) * stride], acc);
    ys[c] = fma(h, acc, y[c]);
  }
}

__device__ __forceinline__ void stage_state(int st, const double* ks, int stride, double h, const double y[4],
                                            double ys[4]) {
  switch (st) {
    case 0:
#pragma unroll
      for (int c = 0; c < 4; ++c) ys[c] = y[c];
      break;
    case 1: stage_state<1>(ks, stride, h, y, ys); break;
    case 2: stage_state<2>(ks, stride, h, y, ys); break;
    case 3: stage_state<3>(ks, stride, h, y, ys); break;
    case 4: stage_state<4>(ks, stride, h, y, ys); break;
    default: stage_state<5>(ks, stride, h, y, ys); break;
  }
}

// Step length of this attempt: h clamped to [min_step, max_step], to the rest
// of the span and (grid dense mode) to the next sample time.
__device__ __forceinline__ double attempt_step(const ScalarState& S, const Params& P, bool& landing, double& t_land) {
  double h = S.h;
  if (h < P.min_step) h = P.min_step;
  if (h > P.max_step) h = P.max_step;
  const double rem = S.c->t_end - S.t;
  if (h > rem) h = rem;
  landing = false;
  t_land = 0.0;
  if (P.dense_mode == 1 && S.o->idx < P.ndo) {
    t_land = grid_time(S, S.o->idx, P.ndo);
    const double remk = t_land - S.t;
    if (h >= remk) {
      h = remk;
      landing = true;
    }
  }
  return h;
}

// Controller, acceptance and dense-output decision after an attempt
// (stepper.py:520-645).  accepted: the candidate becomes the state (the caller
// copies it).  Returns true (per lane) if a dense sample must be stored then;
// the caller writes it.
__device__ __forceinline__ bool finish_step(ScalarState& S, const Params& P, double h, bool landing, double t_land,
                                            bool finite, bool okerr, double ratio, double g_new, int conv_fail_here,
                                            bool& accepted) {
  const bool crossing = (S.g_old * g_new < 0.0);
  bool ok;
  double h_next;
  accepted = false;
  if (crossing) {
    const double abs_old = fabs(S.g_old);
    const double denom = abs_old + fabs(g_new);
    h_next = h * ((abs_old / (denom + 1e-15)) * 0.99);
    ok = false;
  } else if (!finite) {
    S.status = ST_NONFINITE;
    S.active = false;
    if (S.lead) S.c->rejected += 1;
    S.h = h;
    return false;
  } else {
    ok = okerr;
    // 0.9 ratio^(1/5) in [0.2, 5] after an accepted step, 0.9 ratio^(1/4) in
    // [0.1, 0.5] after a rejected one: one power with a selected exponent
    const double ex = ok ? 0.2 : 0.25;
    double pw[1];
    f_pow<true, 1>({ratio}, ex, pw);
    if (!cbcd::exp_in<-400, 400>(ratio)) pw[0] = cbcm::pow_pos(ratio, ex);
    const double f = 0.9 * pw[0];
    const double lo = ok ? 0.2 : 0.1, hi = ok ? 5.0 : 0.5;
    const double fl = f > lo ? f : lo;
    h_next = h * (fl < hi ? fl : hi);
  }
  if (ok) {
    accepted = true;
    S.t = landing ? t_land : S.t + h;
    S.g_old = g_new;
  } else {
    if (S.lead) S.c->rejected += 1;
    if (h <= P.min_step) {
      S.status = conv_fail_here ? ST_CONV_FAIL : ST_STEP_LIMIT;
      S.active = false;
      S.h = h_next;
      return false;
    }
  }
  S.h = h_next;
  // dense output decision (stepper.py:634-645, stored slot never overwritten)
  return P.dense_mode == 0 ? (S.o->idx < P.ndo) && (S.o->dnext <= S.t) : ok && landing;
}

// Counts an attempt with its six coupling solves.
__device__ __forceinline__ void count_attempt(const ScalarState& S, int sweeps, int conv_fail_here) {
  S.o->steps += 1;
  if (S.lead) {
    S.c->lin_iters += sweeps;
    S.c->conv_ok += 6 - conv_fail_here;
    S.c->conv_fail += conv_fail_here;
  }
}

// After a dense store (if any): advance the schedule and test termination
// (stepper.py:651-662).
__device__ __forceinline__ void after_store(ScalarState& S, const Params& P, bool stored) {
  if (!S.active) return;
  if (stored) {
    S.o->idx += 1;
    if (P.dense_mode == 0) {
      const double nx = S.t + S.c->ddt;
      S.o->dnext = nx < S.c->t_end ? nx : S.c->t_end;
    }
  }
  if (S.t >= S.c->t_end) {
    S.status = ST_SUCCESS;
    S.active = false;
  } else if (fabs(S.g_old) < P.etol) {
    S.status = ST_EVENT;
    S.active = false;
  }
}

}  // namespace cbc
