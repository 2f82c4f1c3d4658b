// wide_core.cuh -- CKM1D step for systems of 9 to 16 bubbles with the Richardson
// coupling solve: one lane per bubble, two or three systems per warp.
//
// The 4 (K - 1) partner coefficients of a lane stay in registers (120 of them at
// K = 16).  Read from shared memory at every sweep, 32 bytes a partner beside the
// 16 of the partner's iterate, they bounded the solve: 4,736 x K = 16 filling the
// GPU took 50.8 ns an attempt, now 25.2; a single system alone 48 us, now 38.7.  To make
// room the scalars of a system, which an attempt touches once, live in shared
// memory (cold_core.cuh).  K = 16 has a kernel of its own; any other K runs one
// padded to 16 with zero coefficients and zero partners, without a branch per
// partner (K = 11 alone: 99 us with the branches, now 56 to 58).  Registers and
// shared memory (24 KB a warp) admit two blocks of four warps per SM: two warps a
// scheduler.
#pragma once

#include "cold_core.cuh"

namespace cbc {

constexpr int WIDE = 16;           // partners are padded to this many bubbles
constexpr int WIDE_THREADS = 128;  // largest block
constexpr int WIDE_VALUES = 66;    // one exchange buffer: 2 K values per system, the last ones zero

// Per-warp shared memory, in doubles.
struct WideSmem {
  double* up;      // [13][32]  bubble constants, lane-private columns
  double* ks;      // [5][4][32] stage derivatives k1..k5, lane-private columns
  double* xv;      // [2][33] double2 partner-state exchange records; record 32 is zero
  double* xr;      // [2][2][WIDE_VALUES] exchange buffers of the Richardson iterates
  double* cm;      // [3][15][32] coupling coefficients of each lane's partners (zero past K - 1)
  LaneCold* own;   // [32]
  Cold* cold;      // [G] scalars of each group's system
  double* hc;      // [7 nk][G] harmonic constants of each group
};

constexpr int WIDE_FIXED = 13 * 32 + 20 * 32 + 2 * 2 * 33 + 4 * WIDE_VALUES + 3 * (WIDE - 1) * 32 +
                           32 * (int)(sizeof(LaneCold) / 8);

__host__ __device__ inline int wide_smem_doubles(int K, int nk) {
  const int n = WIDE_FIXED + (int)(sizeof(Cold) / 8) * (32 / K) + HC_PER_K * nk * (32 / K);
  return (n + 1) & ~1;
}

// The regions of this warp, all constant offsets from one base but the last one.
__device__ __forceinline__ WideSmem wide_smem(double* base, int K, int nk) {
  WideSmem w;
  w.up = base + (threadIdx.x >> 5) * wide_smem_doubles(K, nk);
  w.ks = w.up + 13 * 32;
  w.xv = w.ks + 20 * 32;
  w.xr = w.xv + 2 * 2 * 33;
  w.cm = w.xr + 4 * WIDE_VALUES;
  w.own = reinterpret_cast<LaneCold*>(w.cm + 3 * (WIDE - 1) * 32);
  w.cold = reinterpret_cast<Cold*>(w.own + 32);
  w.hc = reinterpret_cast<double*>(w.cold + 32 / K);
  const int lane = threadIdx.x & 31;
  if (lane < 2) reinterpret_cast<double2*>(w.xv)[33 * lane + 32] = make_double2(0.0, 0.0);
  if (lane < 4) w.xr[WIDE_VALUES * lane + 64] = 0.0;
  __syncwarp();
  return w;
}

__device__ __forceinline__ double upv(const WideSmem& w, const Geo& g, int p) { return w.up[p * 32 + g.lane]; }

// This lane's bubble constants (13, `stride` apart) and coupling coefficients.
__device__ __forceinline__ void wide_store_bubble(const WideSmem& w, const Geo& g, const double* up13,
                                                  long long stride, const MView& M) {
#pragma unroll
  for (int p = 0; p < 13; ++p) w.up[p * 32 + g.lane] = up13[p * stride];
  for (int d = 1; d < WIDE; ++d) {
    const int j = partner_lane(g, d) - g.base;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      w.cm[(c * (WIDE - 1) + d - 1) * 32 + g.lane] = d < g.K ? M.m[c * M.sc + j * M.sj] : 0.0;
  }
}

// Record of partner d: lanes outside every group read their own, past the last
// partner it is the zero record.
__device__ __forceinline__ int wide_rec(const Geo& g, int d) {
  return d >= g.K ? 32 : (g.valid ? partner_lane(g, d) : g.lane);
}

// Terms of the right-hand side up to the coupling solve, the partners four at a
// time so that their reciprocals interleave.
template <int NKC, int ACC, bool FAST>
__device__ __forceinline__ void wide_rhs_terms(const Geo& g, const Params& P, const WideSmem& W, const Cold& cold,
                                               double t, const double y[4], double D, double& b0, double& b1,
                                               double& cpf0, double (&Am)[WIDE], double (&Bm)[WIDE],
                                               double (&Cm)[WIDE], double (&Dm)[WIDE]) {
  const auto hc = [&](int k, int c) { return W.hc[(HC_PER_K * k + c) * g.G + g.grp]; };
  const OwnTerms o = own_terms<NKC, ACC, FAST, true>(P, hc, cold.sp0, t, y[0], y[1], D, g.base, g.li);
  PairSums ps{0.0, 0.0, 0.0, 0.0, 0.0};
  const double2* xv2 = reinterpret_cast<const double2*>(W.xv);
#pragma unroll
  for (int d0 = 1; d0 < WIDE; d0 += 4) {
    // each batch after the one before it: all interleaved need more registers
    // than there are
    __syncwarp();
    PartnerTerms q[4];
    double ad[4], rd[4], sg[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      ad[i] = 1.0;
      if (d0 + i < WIDE) {
        const int src = wide_rec(g, d0 + i);
        q[i] = partner_terms(xv2[src], xv2[33 + src]);
        pair_distance(y[1], q[i].x1, ad[i], sg[i]);
      }
    }
    f_rcp<FAST>(ad, rd);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int d = d0 + i;
      if (d < WIDE) {
        const double* m = W.cm + (d - 1) * 32 + g.lane;
        const double m0 = m[0], m1 = m[(WIDE - 1) * 32], m2 = m[2 * (WIDE - 1) * 32];
        const PairTerms pt = pair_terms(q[i], rd[i], sg[i], m0, m1);
        ps.g0 = fma(-m0, pt.t0, ps.g0);
        ps.g1 = fma(-0.5 * m0, pt.t1, ps.g1);
        ps.tn = fma(m1, pt.t2, ps.tn);
        ps.tg2 = fma(m1, pt.t1, ps.tg2);
        ps.tg3 = fma(m2, pt.t1, ps.tg3);
        Am[d] = pt.a;
        Bm[d] = pt.b;
        Cm[d] = pt.c;
        Dm[d] = pt.d;
      }
    }
  }
  implicit_rhs(o, ps, [&](int p) { return upv(W, g, p); }, cold.sp3, y[0], y[2], y[3], b0, b1);
  cpf0 = o.rD;
}

// Puts this lane's iterate into exchange buffer `buf` before a sweep, at li and
// li + K of its group's values, so that partner d is the value d further (282
// cycles a sweep at K = 16 in isolation; by shuffle 378; stored once 269, but the
// partners' indices take registers that the coefficients leave no room for).
// Two buffers used in turn need one __syncwarp a sweep.
__device__ __forceinline__ void wide_exchange(const Geo& g, const WideSmem& W, int buf, double vr, double vt) {
  if (g.valid) {
    double* xr = W.xr + 2 * WIDE_VALUES * buf + g.grp * 2 * g.K + g.li;
    xr[0] = xr[g.K] = vr;
    xr[WIDE_VALUES] = xr[WIDE_VALUES + g.K] = vt;
  }
  __syncwarp();
}

// Residual of the iterate in buffer `buf` (residual in ckm1d_core.cuh); partners
// past K read zeros and have zero coefficients.
template <int KC>
__device__ __forceinline__ void wide_residual(const Geo& g, const WideSmem& W, int buf, const double (&Am)[WIDE],
                                              const double (&Bm)[WIDE], const double (&Cm)[WIDE],
                                              const double (&Dm)[WIDE], double cpf0, double b0, double b1, double vr,
                                              double vt, double& r0, double& r1) {
  double ar[4] = {0.0, 0.0, 0.0, 0.0}, at[4] = {0.0, 0.0, 0.0, 0.0};
  const double* xr = W.xr + 2 * WIDE_VALUES * buf;
  const double* own = xr + (g.valid ? g.grp * 2 * g.K + g.li : 0);
#pragma unroll
  for (int d = 1; d < WIDE; ++d) {
    const double* q = KC > 0 || d < g.K ? own + d : xr + 64;
    const double x = q[0], z = q[WIDE_VALUES];
    const int c = (d - 1) & 3;
    ar[c] = fma(Bm[d], z, ar[c]);
    at[c] = fma(Dm[d], z, at[c]);
    ar[c] = fma(Am[d], x, ar[c]);
    at[c] = fma(Cm[d], x, at[c]);
  }
  const double sr = tree_open(ar, 4);
  const double st = tree_open(at, 4);
  r0 = b0 - fma(sr, cpf0, vr);
  r1 = b1 - (st + vt);
}

// Right-hand side (rhs in ckm1d_core.cuh).
template <int KC>
__device__ __forceinline__ void wide_rhs(const Geo& g, const Params& P, const WideSmem& W, const Cold& cold, bool on,
                                         double t, const double y[4], double dy[4], bool& conv, int& iters) {
  double2* xv2 = reinterpret_cast<double2*>(W.xv);
  __syncwarp();
  xv2[g.lane] = make_double2(y[0], y[1]);
  xv2[33 + g.lane] = make_double2(y[2], y[3]);
  __syncwarp();
  const double u7 = upv(W, g, 7);
  const double D = fma(-(u7 * y[0]), y[2], y[0]) + upv(W, g, 4) * u7;
  const bool general = on & !(state_in_range(y[0], y[1], D) & (fabs(t) <= cold.fast_until));
  double b0, b1, cpf0, Am[WIDE], Bm[WIDE], Cm[WIDE], Dm[WIDE];
  // some lane's arguments are outside the range of the interleaved functions
  if (__any_sync(FULL, general))
    wide_rhs_terms<0, -1, false>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else if (P.nk == 2 && P.ac == 2)
    wide_rhs_terms<2, 2, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else if (P.nk == 2 && P.ac == 1)
    wide_rhs_terms<2, 1, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else
    wide_rhs_terms<0, -1, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);

  // relaxed Richardson from v = b, two sweeps per vote (see rhs_form in
  // ckm1d_core.cuh)
  const double rt = P.lin_rtol2 * group_sum<WIDE>(fma(b0, b0, b1 * b1), g);
  const double tol2 = rt > P.lin_atol2 ? rt : P.lin_atol2;
  double vr = b0, vt = b1, ans_r = b0, ans_t = b1, r0, r1;
  bool found = !on;
  iters = 0;
  const int maxit = P.lin_max_iter;
  wide_exchange(g, W, 1, vr, vt);
  wide_residual<KC>(g, W, 1, Am, Bm, Cm, Dm, cpf0, b0, b1, vr, vt, r0, r1);
  for (int it = 0; it < maxit; it += 2) {
    if (__all_sync(FULL, found)) break;
    const double br = fma(P.omega, r0, vr), bt = fma(P.omega, r1, vt);
    double q0, q1, s0, s1;
    wide_exchange(g, W, 0, br, bt);
    wide_residual<KC>(g, W, 0, Am, Bm, Cm, Dm, cpf0, b0, b1, br, bt, q0, q1);
    const bool two = it + 1 < maxit;
    const double wr = fma(P.omega, q0, br), wt = fma(P.omega, q1, bt);
    wide_exchange(g, W, 1, wr, wt);
    wide_residual<KC>(g, W, 1, Am, Bm, Cm, Dm, cpf0, b0, b1, wr, wt, s0, s1);
    double rna = fma(r0, r0, r1 * r1), rnb = fma(q0, q0, q1 * q1);
    if (KC == WIDE) {     // full power-of-two groups: butterfly, the same sums
#pragma unroll
      for (int w = 1; w < WIDE; w <<= 1) {
        rna = rna + __shfl_xor_sync(FULL, rna, w);
        rnb = rnb + __shfl_xor_sync(FULL, rnb, w);
      }
    } else {
      rna = group_sum<WIDE>(rna, g);
      rnb = group_sum<WIDE>(rnb, g);
    }
    const bool hita = !found & (rna < tol2);
    iters = found ? iters : it + 1;
    ans_r = hita ? vr : ans_r;
    ans_t = hita ? vt : ans_t;
    found = found | hita;
    const bool hitb = two & !found & (rnb < tol2);
    iters = (found | !two) ? iters : it + 2;
    ans_r = hitb ? br : ans_r;
    ans_t = hitb ? bt : ans_t;
    found = found | hitb;
    vr = two ? wr : br;
    vt = two ? wt : bt;
    r0 = s0;
    r1 = s1;
  }
  conv = found;
  dy[0] = y[2];
  dy[1] = y[3];
  dy[2] = found ? ans_r : vr;
  dy[3] = found ? ans_t : vt;
}

// One adaptive Cash-Karp step for every active group of the warp (step in
// ckm1d_core.cuh).
template <int KC>
__device__ __forceinline__ bool wide_step(const Geo& g, const Params& P, const WideSmem& W, BubbleState& S) {
  const bool on = S.active;
  bool landing;
  double t_land;
  const double h = attempt_step(S, P, landing, t_land);
  double* ks = W.ks + g.lane;   // ks[(st * 4 + c) * 32]
  int conv_fail_here = 0, sweeps = 0;
  double kk[4];
#pragma unroll 1
  for (int st = 0; st < 6; ++st) {
    double ys[4];
    stage_state(st, ks, 32, h, S.y, ys);
    const double ts = (st == 0) ? S.t : fma(kStageA[st], h, S.t);
    bool cv;
    int it;
    wide_rhs<KC>(g, P, W, *S.c, on, ts, ys, kk, cv, it);
    if (st < 5) {
#pragma unroll
      for (int c = 0; c < 4; ++c) ks[(st * 4 + c) * 32] = kk[c];
    }
    sweeps += it;
    conv_fail_here += cv ? 0 : 1;
  }
  double yn[4], ratio_l;
  bool fin, ok_l;
  candidate<true>(P, on, h, S.y, ks, 32, kk, yn, fin, ok_l, ratio_l);
  const bool finite = group_all(fin, g);
  const double g_new = group_event<WIDE>(yn, upv(W, g, 12), g, P.col);
  const double ratio = group_min<WIDE>(ratio_l, g);
  const bool okerr = group_all(ok_l, g);
  if (!on) return false;
  count_attempt(S, sweeps, conv_fail_here);
  bool accepted;
  const bool store = finish_step(S, P, h, landing, t_land, finite, okerr, ratio, g_new, conv_fail_here, accepted);
  if (accepted) {
#pragma unroll
    for (int c = 0; c < 4; ++c) S.y[c] = yn[c];
  }
  return store;
}

}  // namespace cbc
