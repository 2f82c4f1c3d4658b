// solo_core.cuh -- CKM1D step for systems of a single bubble with the Richardson
// solve: one lane per system, 32 systems per warp.
//
// Without partners there is nothing to exchange: no shuffle, no shared record, no
// reduction.  (The one-lane-per-bubble form spent them all the same: 9.7 us an
// attempt alone, now 5.3; 300,000 systems 0.194 ns an attempt, now 0.162.  For two
// bubbles per lane the sweep itself gets faster, 51 cycles against 75, but the tests'
// selects double per lane and the whole attempt does not: 15.0 us with 32 systems a
// warp against 12.5 with 16.)  The
// iteration's solution is its right-hand side; the loop is kept because its
// count and its outcome are results (a residual that is not a number never
// converges).
//
// Same operations in the same order as ckm1d_core.cuh.
#pragma once

#include "cold_core.cuh"

namespace cbc {

constexpr int SOLO_THREADS = 128;  // largest block
// Blocks per SM that the registers are limited for: 128 a thread.  Shared memory
// admits four with one harmonic, three with two (15 KB a warp).
constexpr int SOLO_BLOCKS = 4;

// Shared memory of a warp, in doubles: every lane uses its own columns.
struct SoloSmem {
  double* up;    // [13][32] bubble constants
  double* ks;    // [5][4][32] stage derivatives k1..k5
  LaneCold* own; // [32]
  Cold* cold;    // [32]
  double* hc;    // [7 nk][32] harmonic constants
};

__host__ __device__ inline int solo_smem_doubles(int nk) {
  return (13 + 20 + HC_PER_K * nk) * 32 + 32 * (int)((sizeof(LaneCold) + sizeof(Cold)) / 8);
}

__device__ __forceinline__ SoloSmem solo_smem(double* base, int nk) {
  SoloSmem w;
  w.up = base + (threadIdx.x >> 5) * solo_smem_doubles(nk);
  w.ks = w.up + 13 * 32;
  w.own = reinterpret_cast<LaneCold*>(w.ks + 20 * 32);
  w.cold = reinterpret_cast<Cold*>(w.own + 32);
  w.hc = reinterpret_cast<double*>(w.cold + 32);
  return w;
}

// Constants of this lane's bubble (13 values, `stride` apart).
__device__ __forceinline__ void solo_store_bubble(const SoloSmem& W, int lane, const double* up13, long long stride) {
#pragma unroll
  for (int p = 0; p < 13; ++p) W.up[p * 32 + lane] = up13[p * stride];
}

// Right-hand side for one field form (rhs_form in ckm1d_core.cuh).
template <int NKC, int ACC, bool FAST>
__device__ __forceinline__ void solo_rhs_form(const Params& P, const SoloSmem& W, int lane, const Cold& cold, bool on,
                                              double t, const double y[4], double dy[4], bool& in_range, bool& conv,
                                              int& iters) {
  const auto hc = [&](int k, int c) { return W.hc[(HC_PER_K * k + c) * 32 + lane]; };
  const auto up = [&](int p) { return W.up[p * 32 + lane]; };
  const double u7 = up(7);
  const double D = fma(-(u7 * y[0]), y[2], y[0]) + up(4) * u7;
  in_range = state_in_range(y[0], y[1], D);
  const OwnTerms o = own_terms<NKC, ACC, FAST, false>(P, hc, cold.sp0, t, y[0], y[1], D, 0, 0);
  double b0, b1;
  implicit_rhs(o, PairSums{0.0, 0.0, 0.0, 0.0, 0.0}, up, cold.sp3, y[0], y[2], y[3], b0, b1);
  // relaxed Richardson from v = b without partners: r = b - v
  const double rt = P.lin_rtol2 * fma(b0, b0, b1 * b1);
  const double tol2 = rt > P.lin_atol2 ? rt : P.lin_atol2;
  double vr = b0, vt = b1;
  bool found = !on;
  iters = 0;
  for (int it = 0; it < P.lin_max_iter; ++it) {
    if (__all_sync(FULL, found)) break;
    const double r0 = b0 - fma(0.0, o.rD, vr), r1 = b1 - (0.0 + vt);
    iters = found ? iters : it + 1;
    found = found | (fma(r0, r0, r1 * r1) < tol2);
    vr = found ? vr : fma(P.omega, r0, vr);
    vt = found ? vt : fma(P.omega, r1, vt);
  }
  conv = found;
  dy[0] = y[2];
  dy[1] = y[3];
  dy[2] = vr;
  dy[3] = vt;
}

// One adaptive Cash-Karp step of every active lane's system (step in
// ckm1d_core.cuh).  Returns true if a dense sample must be stored after it.
__device__ __forceinline__ bool solo_step(const Params& P, const SoloSmem& W, int lane, BubbleState& S) {
  const bool on = S.active;
  bool landing;
  double t_land;
  const double h = attempt_step(S, P, landing, t_land);
  double* ks = W.ks + lane;     // ks[(st * 4 + c) * 32]
  int conv_fail_here, sweeps;
  double kk[4];
  // the general functions where some lane's system is outside the range of the
  // interleaved ones; made again with them when some lane's state left it
  const bool outside = __any_sync(FULL, on & !(S.t + h <= S.c->fast_until));
  for (bool general = outside;; general = true) {
    bool in_range = true;
    conv_fail_here = sweeps = 0;
#pragma unroll 1
    for (int st = 0; st < 6; ++st) {
      double ys[4];
      stage_state(st, ks, 32, h, S.y, ys);
      const double ts = (st == 0) ? S.t : fma(kStageA[st], h, S.t);
      bool cv, ok;
      int it;
      if (general)
        solo_rhs_form<0, -1, false>(P, W, lane, *S.c, on, ts, ys, kk, ok, cv, it);
      else if (P.nk == 2 && P.ac == 2)
        solo_rhs_form<2, 2, true>(P, W, lane, *S.c, on, ts, ys, kk, ok, cv, it);
      else if (P.nk == 2 && P.ac == 1)
        solo_rhs_form<2, 1, true>(P, W, lane, *S.c, on, ts, ys, kk, ok, cv, it);
      else
        solo_rhs_form<0, -1, true>(P, W, lane, *S.c, on, ts, ys, kk, ok, cv, it);
      if (st < 5) {
#pragma unroll
        for (int c = 0; c < 4; ++c) ks[(st * 4 + c) * 32] = kk[c];
      }
      in_range = in_range & ok;
      sweeps += it;
      conv_fail_here += cv ? 0 : 1;
    }
    if (general) break;
    if (__all_sync(FULL, !on | in_range)) break;
  }
  double yn[4], ratio;
  bool fin, okerr;
  candidate<true>(P, on, h, S.y, ks, 32, kk, yn, fin, okerr, ratio);
  if (!on) return false;
  count_attempt(S, sweeps, conv_fail_here);
  bool accepted;
  // no neighbour: the event value is 1e30
  const bool store = finish_step(S, P, h, landing, t_land, fin, okerr, ratio, 1e30, conv_fail_here, accepted);
  if (accepted) {
#pragma unroll
    for (int c = 0; c < 4; ++c) S.y[c] = yn[c];
  }
  return store;
}

}  // namespace cbc
