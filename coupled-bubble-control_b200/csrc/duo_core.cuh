// duo_core.cuh -- CKM1D step for systems of 17 to 32 bubbles with the Richardson
// coupling solve: two lanes per bubble, one block of two warps per system.
//
// With one lane per bubble the 4 (K - 1) partner coefficients of a lane do not
// fit the registers beyond K = 16; read from shared memory at every sweep
// (48 bytes a partner with the partner's iterate, two of them multiply-adds) they
// bound the solve: at K = 32 a sweep moves 46 KB through the 128 bytes a cycle
// of an SM, 372 cycles, which is what three systems per SM measured (1,116 a
// sweep).  Here each lane of the pair holds the coefficients of two of the four
// accumulation chains in registers (lane 0: partners d = 1, 2 mod 4, lane 1:
// d = 3, 0 mod 4), so only the iterates move: 16 bytes a partner, and the two
// half sums meet in one shuffle.  An attempt before and after: K = 32 alone 80 us, now
// 47, GPU full 230 ns, now 118; K = 20 164 us and 396 ns, now 57 and 123.
//
// Same operations in the same order as the one-lane form (ckm1d_core.cuh): the
// chains and their tree, the ordered sums over the partners (lane 0 sums the two
// radial ones, lane 1 the three translational ones, each over all partners,
// with the terms of the other lane's partners shuffled over), the pairwise tree of
// the norms.  Every value that decides control flow is the same in all 64
// threads, so the team needs no votes, only barriers around its exchanges.
#pragma once

#include "cold_core.cuh"

namespace cbc {

constexpr int DUO_THREADS = 64;   // of a team: one system
constexpr int DUO_BLOCKS = 4;     // teams per SM the registers are limited for

// TEAMS: systems of a block.  One, or as many as an SM has registers for where
// the block has to hold its SM alone (latency lanes: blocks of one team each are
// spread over as many SMs, beside other buckets' work).  One lane SM with 6,000
// systems of 8 bubbles on the others: an attempt of four systems of K = 32 66 us
// each, of one 42; K = 20 72 and 56.
template <int TEAMS>
struct DuoGeo {
  int K;
  int tid;     // thread of the team
  int team;
  int i;       // bubble of this thread
  int c;       // lane of the pair
  bool valid;  // i < K
};

template <int TEAMS>
__device__ __forceinline__ DuoGeo<TEAMS> make_duo_geo(int K) {
  DuoGeo<TEAMS> g;
  g.K = K;
  g.tid = TEAMS > 1 ? threadIdx.x % DUO_THREADS : threadIdx.x;
  g.team = TEAMS > 1 ? threadIdx.x / DUO_THREADS : 0;
  g.i = g.tid >> 1;
  g.c = g.tid & 1;
  g.valid = g.i < K;
  return g;
}

// Barrier of the team's two warps, and the same with an OR over their threads.
template <int TEAMS>
__device__ __forceinline__ void duo_sync(const DuoGeo<TEAMS>& g) {
  if constexpr (TEAMS == 1) __syncthreads();
  else asm volatile("barrier.sync %0, %1;" ::"r"(1 + g.team), "n"(DUO_THREADS) : "memory");
}
template <int TEAMS>
__device__ __forceinline__ bool duo_sync_or(const DuoGeo<TEAMS>& g, bool v) {
  if constexpr (TEAMS == 1) {
    return __syncthreads_or(v) != 0;
  } else {
    int r;
    asm volatile(
        "{\n"
        "  .reg .pred p, q;\n"
        "  setp.ne.s32 p, %1, 0;\n"
        "  barrier.red.or.pred q, %2, %3, p;\n"
        "  selp.s32 %0, 1, 0, q;\n"
        "}"
        : "=r"(r)
        : "r"((int)v), "r"(1 + g.team), "n"(DUO_THREADS)
        : "memory");
    return r != 0;
  }
}

// Shared memory of a team, in doubles.
struct DuoSmem {
  double* hc;    // [7 nk]    harmonic constants
  double* up;    // [13][32]  bubble constants
  double* ks;    // [5][4][32] stage derivatives k1..k5
  double* xv;    // [2][33] double2 partner states; record 32 is zero
  double* xr;    // [2][66] double2 iterates, bubble i at i and i + K; record 65 is zero
  double* rr;    // [2][32]   squared residuals
  double* cm;    // [3][32][32] coupling coefficients of partner d = 1..32 (zero past K - 1)
  double* red;   // [2][4]    per-warp results of the step's reductions
  int* claim;    // [2]       for the batched worker
  LaneCold* own; // [64]
  Cold* cold;    // scalars of the system
};

__host__ __device__ inline int duo_smem_doubles(int nk) {
  return ((HC_PER_K * nk + 1) & ~1) + 13 * 32 + 20 * 32 + 2 * 2 * 33 + 2 * 2 * 66 + 64 + 3 * 32 * 32 + 8 + 1 +
         DUO_THREADS * (int)(sizeof(LaneCold) / 8) + (int)(sizeof(Cold) / 8);
}
static_assert((1 + DUO_THREADS * sizeof(LaneCold) / 8 + sizeof(Cold) / 8) % 2 == 0, "teams start 16-byte aligned");

template <int TEAMS>
__device__ __forceinline__ DuoSmem duo_smem(const DuoGeo<TEAMS>& g, double* p, int nk) {
  DuoSmem w;
  w.up = p + g.team * duo_smem_doubles(nk);
  w.ks = w.up + 13 * 32;
  w.xv = w.ks + 20 * 32;
  w.xr = w.xv + 2 * 2 * 33;
  w.rr = w.xr + 2 * 2 * 66;
  w.cm = w.rr + 64;
  w.red = w.cm + 3 * 32 * 32;
  w.claim = reinterpret_cast<int*>(w.red + 8);
  w.own = reinterpret_cast<LaneCold*>(w.red + 9);
  w.cold = reinterpret_cast<Cold*>(w.own + DUO_THREADS);
  w.hc = reinterpret_cast<double*>(w.cold + 1);
  if (g.tid < 2) {
    reinterpret_cast<double2*>(w.xv)[33 * g.tid + 32] = make_double2(0.0, 0.0);
    reinterpret_cast<double2*>(w.xr)[66 * g.tid + 65] = make_double2(0.0, 0.0);
  }
  w.rr[g.tid] = 0.0;
  duo_sync(g);
  return w;
}

// Constants of this thread's bubble (from its column of the caller's 13 rows)
// and its coupling coefficients M(c, j, i) for the partners j = (i + d) mod K;
// each lane of the pair writes half of them.  m points at M(0, 0, i).
template <int TEAMS>
__device__ __forceinline__ void duo_store_bubble(const DuoSmem& W, const DuoGeo<TEAMS>& g, const double* up13,
                                                  long long up_stride, const MView& M) {
  if (g.valid)
    for (int p = g.c; p < 13; p += 2) W.up[p * 32 + g.i] = up13[p * up_stride];
  for (int d = 1 + g.c; d <= 32; d += 2) {
    const int j = g.i + d < g.K ? g.i + d : g.i + d - g.K;
    for (int c = 0; c < 3; ++c)
      W.cm[(c * 32 + d - 1) * 32 + g.i] = g.valid && d < g.K ? M.m[c * M.sc + j * M.sj] : 0.0;
  }
}

// Terms of the right-hand side (rhs_terms of the one-lane form).  Coefficient
// s = 2 m + e of a lane (m = 0..7, e = 0, 1) belongs to partner
// d = 4 m + 2 c + e + 1; partners past K - 1 are the zero record with zero
// coefficients, which adds nothing (straight-line code for 32 bubbles takes 46 us
// an attempt, with a branch per four partners for K = 20 it took 75).
template <int NKC, int ACC, bool FAST, int TEAMS>
__device__ __forceinline__ void duo_rhs_terms(const DuoGeo<TEAMS>& g, const Params& P, const DuoSmem& W, const Cold& cold,
                                               double t, const double y[4], double D, double& b0, double& b1,
                                               double& cpf0, double (&Am)[16], double (&Bm)[16], double (&Cm)[16],
                                               double (&Dm)[16]) {
  const auto hc = [&](int k, int c) { return W.hc[HC_PER_K * k + c]; };
  const OwnTerms o = own_terms<NKC, ACC, FAST, true>(P, hc, cold.sp0, t, y[0], y[1], D, g.tid & 30, g.c);
  const double2* xv2 = reinterpret_cast<const double2*>(W.xv);
  // lane 0 sums g0 and g1, lane 1 sums tn, tg2 and tg3
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  const double kf = g.c ? 1.0 : -0.5;
#pragma unroll
  for (int m = 0; m < 8; ++m) {
    __syncwarp();    // each batch after the one before it: all interleaved need too many registers
    {
      PartnerTerms q[2];
      double ad[2], rd[2], sg[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int d = 4 * m + 2 * g.c + e + 1;
        const int j = g.i + d < g.K ? g.i + d : g.i + d - g.K;
        const int src = g.valid && d < g.K ? j : 32;
        q[e] = partner_terms(xv2[src], xv2[33 + src]);
        pair_distance(y[1], q[e].x1, ad[e], sg[e]);
      }
      f_rcp<FAST>(ad, rd);
      double T1[4], TB[4];     // t1 and (lane 0: t0, lane 1: t2) of partners 4 m + 1 .. 4 m + 4
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = 4 * m + 2 * g.c + e;
        const PairTerms pt = pair_terms(q[e], rd[e], sg[e], W.cm[row * 32 + g.i], W.cm[(32 + row) * 32 + g.i]);
        Am[2 * m + e] = pt.a;
        Bm[2 * m + e] = pt.b;
        Cm[2 * m + e] = pt.c;
        Dm[2 * m + e] = pt.d;
        const double o1 = __shfl_xor_sync(FULL, pt.t1, 1), ob = __shfl_xor_sync(FULL, g.c ? pt.t0 : pt.t2, 1);
        const double mine = g.c ? pt.t2 : pt.t0;
        T1[e] = g.c ? o1 : pt.t1;
        TB[e] = g.c ? ob : mine;
        T1[2 + e] = g.c ? pt.t1 : o1;
        TB[2 + e] = g.c ? mine : ob;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int row = 4 * m + u;
        const double mc = W.cm[(32 * g.c + row) * 32 + g.i], m2 = W.cm[(64 + row) * 32 + g.i];
        s0 = fma(g.c ? mc : -mc, TB[u], s0);
        s1 = fma(kf * mc, T1[u], s1);
        s2 = fma(m2, T1[u], s2);
      }
    }
  }
  const double o0 = __shfl_xor_sync(FULL, s0, 1), o1 = __shfl_xor_sync(FULL, s1, 1), o2 = __shfl_xor_sync(FULL, s2, 1);
  PairSums ps;
  ps.g0 = g.c ? o0 : s0;
  ps.g1 = g.c ? o1 : s1;
  ps.tn = g.c ? s0 : o0;
  ps.tg2 = g.c ? s1 : o1;
  ps.tg3 = g.c ? s2 : o2;
  implicit_rhs(o, ps, [&](int p) { return W.up[p * 32 + g.i]; }, cold.sp3, y[0], y[2], y[3], b0, b1);
  cpf0 = o.rD;
}

// Writes this thread's iterate and its bubble's squared residual to buffer
// `buf` and waits for the team.  Two buffers used in turn need one barrier a
// sweep.
template <int TEAMS>
__device__ __forceinline__ void duo_exchange(const DuoGeo<TEAMS>& g, const DuoSmem& W, int buf, double vr, double vt,
                                              double rr) {
  if (g.valid) {
    reinterpret_cast<double2*>(W.xr)[66 * buf + g.i + (g.c ? g.K : 0)] = make_double2(vr, vt);
    if (g.c == 0) W.rr[32 * buf + g.i] = rr;
  }
  duo_sync(g);
}

// Pairwise tree over the 32 (zero padded) squared residuals of buffer `buf`,
// the same value in every thread.
template <int TEAMS>
__device__ __forceinline__ double duo_norm(const DuoGeo<TEAMS>& g, const DuoSmem& W, int buf) {
  double v = W.rr[32 * buf + (g.tid & 31)];
#pragma unroll
  for (int w = 1; w < 32; w <<= 1) v = v + __shfl_xor_sync(FULL, v, w);
  return v;
}

// Residual of the iterate in buffer `buf` (residual of the one-lane form): the
// lane's two chains, joined with the other lane's.
template <int TEAMS>
__device__ __forceinline__ void duo_residual(const DuoGeo<TEAMS>& g, const DuoSmem& W, int buf, const double (&Am)[16],
                                              const double (&Bm)[16], const double (&Cm)[16], const double (&Dm)[16],
                                              double cpf0, double b0, double b1, double vr, double vt, double& r0,
                                              double& r1) {
  const double2* xr = reinterpret_cast<const double2*>(W.xr) + 66 * buf;
  double ar[2] = {0.0, 0.0}, at[2] = {0.0, 0.0};
#pragma unroll
  for (int m = 0; m < 8; ++m) {
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int d = 4 * m + 2 * g.c + e + 1, s = 2 * m + e;
      const double2 v = xr[g.valid && d < g.K ? g.i + d : 65];
      ar[e] = fma(Bm[s], v.y, ar[e]);
      at[e] = fma(Dm[s], v.y, at[e]);
      ar[e] = fma(Am[s], v.x, ar[e]);
      at[e] = fma(Cm[s], v.x, at[e]);
    }
  }
  double sr = ar[0] + ar[1], st = at[0] + at[1];
  sr = sr + __shfl_xor_sync(FULL, sr, 1);
  st = st + __shfl_xor_sync(FULL, st, 1);
  r0 = b0 - fma(sr, cpf0, vr);
  r1 = b1 - (st + vt);
}

template <int TEAMS>
__device__ __forceinline__ void duo_rhs(const DuoGeo<TEAMS>& g, const Params& P, const DuoSmem& W, const Cold& cold,
                                         double t, const double y[4], double dy[4], bool& conv, int& iters) {
  double2* xv2 = reinterpret_cast<double2*>(W.xv);
  if (g.valid) {
    if (g.c == 0) xv2[g.i] = make_double2(y[0], y[1]);
    else xv2[33 + g.i] = make_double2(y[2], y[3]);
  }
  const double u7 = W.up[7 * 32 + g.i];
  const double D = fma(-(u7 * y[0]), y[2], y[0]) + W.up[4 * 32 + g.i] * u7;
  const bool general = g.valid & !(state_in_range(y[0], y[1], D) & (fabs(t) <= cold.fast_until));
  double b0, b1, cpf0, Am[16], Bm[16], Cm[16], Dm[16];
  if (duo_sync_or(g, general))
    duo_rhs_terms<0, -1, false>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else if (P.nk == 2 && P.ac == 2)
    duo_rhs_terms<2, 2, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else if (P.nk == 2 && P.ac == 1)
    duo_rhs_terms<2, 1, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  else
    duo_rhs_terms<0, -1, true>(g, P, W, cold, t, y, D, b0, b1, cpf0, Am, Bm, Cm, Dm);
  dy[0] = y[2];
  dy[1] = y[3];

  // relaxed Richardson from v = b: iterate it is tested while it + 1 is swept
  const int maxit = P.lin_max_iter;
  double vr = b0, vt = b1, r0, r1;
  duo_exchange(g, W, 1, vr, vt, fma(b0, b0, b1 * b1));
  const double rt = P.lin_rtol2 * duo_norm(g, W, 1);
  const double tol2 = rt > P.lin_atol2 ? rt : P.lin_atol2;
  duo_residual(g, W, 1, Am, Bm, Cm, Dm, cpf0, b0, b1, vr, vt, r0, r1);
  conv = false;
  iters = maxit;
  for (int it = 0;; ++it) {
    const double ur = fma(P.omega, r0, vr), ut = fma(P.omega, r1, vt);
    duo_exchange(g, W, it & 1, ur, ut, fma(r0, r0, r1 * r1));
    double q0, q1;
    const double nb = duo_norm(g, W, it & 1);
    duo_residual(g, W, it & 1, Am, Bm, Cm, Dm, cpf0, b0, b1, ur, ut, q0, q1);
    if (it < maxit && nb < tol2) {
      conv = true;
      iters = it + 1;
    }
    if (conv || it >= maxit) break;
    vr = ur;
    vt = ut;
    r0 = q0;
    r1 = q1;
  }
  dy[2] = vr;
  dy[3] = vt;
}

// event_fun over the team (group_event of the one-lane form) and the step's
// reductions: finiteness, acceptance, smallest ratio, event value.
template <int TEAMS>
__device__ __forceinline__ double duo_event(const DuoGeo<TEAMS>& g, const DuoSmem& W, const double y[4], double col,
                                             bool& fin, bool& ok, double& ratio) {
  double2* xv2 = reinterpret_cast<double2*>(W.xv);
  const double ri = y[0] * W.up[12 * 32 + g.i];
  if (g.valid && g.c == 0) xv2[g.i] = make_double2(ri, y[1]);
  duo_sync(g);
  double gap = 1e30;
  if (g.i + 1 < g.K) {
    const double2 n = xv2[g.i + 1];
    gap = fabs(y[1] - n.y) - (ri + n.x) * col;
  }
  if (!(gap < 1e30)) gap = 1e30;
  if (!g.valid) ratio = 1.0e30;
#pragma unroll
  for (int w = 2; w < 32; w <<= 1) {
    const double a = __shfl_xor_sync(FULL, gap, w), b = __shfl_xor_sync(FULL, ratio, w);
    if (a < gap) gap = a;
    if (b < ratio) ratio = b;
  }
  const unsigned bad_fin = __ballot_sync(FULL, g.valid && !fin), bad_ok = __ballot_sync(FULL, g.valid && !ok);
  double* red = W.red + 4 * (g.tid >> 5);
  if ((g.tid & 31) == 0) {
    red[0] = gap;
    red[1] = ratio;
    red[2] = bad_fin ? 1.0 : 0.0;
    red[3] = bad_ok ? 1.0 : 0.0;
  }
  duo_sync(g);
  const double* a = W.red;
  gap = a[4] < a[0] ? a[4] : a[0];
  ratio = a[5] < a[1] ? a[5] : a[1];
  fin = a[2] + a[6] == 0.0;
  ok = a[3] + a[7] == 0.0;
  return gap;
}

// One adaptive Cash-Karp step of the team's system.  Returns true if a dense
// sample must be stored after it.
template <int TEAMS>
__device__ __forceinline__ bool duo_step(const DuoGeo<TEAMS>& g, const Params& P, const DuoSmem& W, BubbleState& S) {
  bool landing;
  double t_land;
  const double h = attempt_step(S, P, landing, t_land);
  double* ks = W.ks + g.i;
  int conv_fail_here = 0, sweeps = 0;
  double kk[4];
#pragma unroll 1
  for (int st = 0; st < 6; ++st) {
    double ys[4];
    stage_state(st, ks, 32, h, S.y, ys);
    const double ts = (st == 0) ? S.t : fma(kStageA[st], h, S.t);
    bool cv;
    int it;
    duo_rhs(g, P, W, *S.c, ts, ys, kk, cv, it);
    __syncwarp();
    if (st < 5 && g.c == 0) {
#pragma unroll
      for (int c = 0; c < 4; ++c) ks[(st * 4 + c) * 32] = kk[c];
    }
    __syncwarp();
    sweeps += it;
    conv_fail_here += cv ? 0 : 1;
  }
  double yn[4], ratio;
  bool fin, ok;
  candidate<true>(P, g.valid, h, S.y, ks, 32, kk, yn, fin, ok, ratio);
  const double g_new = duo_event(g, W, yn, P.col, fin, ok, ratio);
  count_attempt(S, sweeps, conv_fail_here);
  bool accepted;
  const bool store = finish_step(S, P, h, landing, t_land, fin, ok, ratio, g_new, conv_fail_here, accepted);
  if (accepted) {
#pragma unroll
    for (int c = 0; c < 4; ++c) S.y[c] = yn[c];
  }
  return store;
}

}  // namespace cbc
