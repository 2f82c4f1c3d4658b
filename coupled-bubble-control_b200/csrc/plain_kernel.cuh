// plain_kernel.cuh -- reference-layout CKM1D integrator (the drop-in solver).
//
// plain_kernel<KB, KC> is the one-launch-per-K form: a static mapping of
// systems to warps over the caller's reference-layout buffers, advancing each
// system by at most `budget` steps.  It replaces the fused kernel of the
// reference (backends/numba/rkck45_coupled_numba_stepper.py:116-706).
#pragma once

#include "cbc_internal.h"
#include "duo_core.cuh"
#include "plain.h"
#include "solo_core.cuh"
#include "wide_core.cuh"

namespace cbc {

// Dense sample `slot` of bubble i (state y) of system s at time t.
__device__ __forceinline__ void ref_store_dense(const RefLayout& L, double t, const double y[4], int i, long long s,
                                                int slot) {
  const long long NST = (long long)L.ns * L.tile;
  if (i == 0) L.dense_time[(long long)slot * L.ns + s] = t;
#pragma unroll
  for (int c = 0; c < 4; ++c) L.dense_state[((long long)slot * 4 + c) * NST + s * L.tile + i] = y[c];
}

// State of the bubble at `off`, from and to the buffers.
__device__ __forceinline__ void ref_load_state(const RefLayout& L, long long off, double y[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) y[c] = L.actual_state[c * (long long)L.ns * L.tile + off];
}
__device__ __forceinline__ void ref_write_state(const RefLayout& L, const double y[4], long long off) {
#pragma unroll
  for (int c = 0; c < 4; ++c) L.actual_state[c * (long long)L.ns * L.tile + off] = y[c];
}

__device__ __forceinline__ double ref_prev_time(const RefLayout& L, const Params& P, long long s, int idx) {
  return (P.ndo > 0 && idx > 0) ? L.dense_time[(long long)(idx - 1) * L.ns + s] : 0.0;
}

__device__ __forceinline__ double ref_fast_until(const RefLayout& L, const Params& P, long long s, double t) {
  return fast_until(L.system_params[0 * (long long)L.ns + s], L.system_params[1 * (long long)L.ns + s],
                    L.system_params[2 * (long long)L.ns + s], L.control_params + s, P.nk, L.ns, t);
}

// Scalars of system s into a lane's state, and the prologue: scalars in
// registers, or in shared memory.
__device__ __forceinline__ void ref_load(const RefLayout& L, const Params& P, long long s, LaneState& S) {
  S.sp0 = L.system_params[0 * (long long)L.ns + s];
  S.sp3 = L.system_params[3 * (long long)L.ns + s];
  S.t = L.actual_time[s];
  S.t_end = L.time_end[s];
  S.t_begin = L.time_begin[s];
  S.h = L.time_step[s];
  S.idx = (P.ndo > 0) ? L.dense_index[s] : 0;
  prologue(S, P, L.actual_event[s], ref_prev_time(L, P, s, S.idx), L.status[s]);
}
__device__ __forceinline__ void ref_load(const RefLayout& L, const Params& P, long long s, ScalarState& S) {
  const double t_end = L.time_end[s];
  S.t = L.actual_time[s];
  S.h = L.time_step[s];
  S.o->idx = (P.ndo > 0) ? L.dense_index[s] : 0;
  if (S.lead) {
    S.c->sp0 = L.system_params[0 * (long long)L.ns + s];
    S.c->sp3 = L.system_params[3 * (long long)L.ns + s];
    S.c->fast_until = ref_fast_until(L, P, s, S.t);
  }
  prologue(S, P, t_end, L.time_begin[s], L.actual_event[s], ref_prev_time(L, P, s, S.o->idx), L.status[s]);
}

__device__ __forceinline__ void ref_store_harmonics(const RefLayout& L, const Params& P, long long s, double* hc,
                                                    int stride) {
  store_harmonics(hc, stride, L.system_params[1 * (long long)L.ns + s], L.system_params[2 * (long long)L.ns + s],
                  L.system_params[4 * (long long)L.ns + s], L.control_params + s, P.nk, L.ns);
}

// Scalars and counters of system s (one lane of the system).
__device__ __forceinline__ void ref_write_scalars(const RefLayout& L, const Params& P, long long s, double t, double h,
                                                  double event, int status, int idx, int steps, int rejected,
                                                  int conv_ok, int conv_fail, long long lin_iters,
                                                  int* active_counter) {
  L.actual_time[s] = t;
  L.time_step[s] = h;
  L.actual_event[s] = event;
  L.status[s] = status;
  if (P.ndo > 0) L.dense_index[s] = idx;
  if (L.total_steps) L.total_steps[s] += steps;
  if (L.rejected_steps) L.rejected_steps[s] += rejected;
  if (L.conv_success) L.conv_success[s] += conv_ok;
  if (L.conv_failures) L.conv_failures[s] += conv_fail;
  if (L.lin_iters) L.lin_iters[s] += lin_iters;
  if (status == ST_ACTIVE && active_counter) atomicAdd(active_counter, 1);
}
__device__ __forceinline__ void ref_write_scalars(const RefLayout& L, const Params& P, long long s, const LaneState& S,
                                                  int* active_counter) {
  ref_write_scalars(L, P, s, S.t, S.h, S.g_old, S.status, S.idx, S.steps, S.rejected, S.conv_ok, S.conv_fail,
                    S.lin_iters, active_counter);
}
__device__ __forceinline__ void ref_write_scalars(const RefLayout& L, const Params& P, long long s,
                                                  const ScalarState& S, int* active_counter) {
  ref_write_scalars(L, P, s, S.t, S.h, S.g_old, S.status, S.o->idx, S.o->steps, S.c->rejected, S.c->conv_ok,
                    S.c->conv_fail, S.c->lin_iters, active_counter);
}

// One lane per bubble: 2 to 8 bubbles, and the direct solve (ckm1d_core.cuh).
template <int KB, int KC, int LIN>
__global__ void __launch_bounds__(128, min_blocks_for(KB))
    plain_kernel(RefLayout L, Params P, long long budget, int final_launch, int* active_counter) {
  extern __shared__ __align__(16) double smem[];
  const Geo g = make_geo(KC > 0 ? KC : L.ups);
  const WarpSmem W = warp_smem(smem, g.K, P.nk, LIN);
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long s = warp * g.G + g.grp;
  const bool have = g.valid && s < L.ns;
  const long long NST = (long long)L.ns * L.tile;
  const long long lane_off = s * L.tile + g.li;

  LaneState S;
  S.active = false;
  S.status = ST_ACTIVE;
  if (have) {
    ref_load_state(L, lane_off, S.y);
    store_bubble_consts(W, g, L.unit_params + lane_off, NST);
    store_coupling(W, g, MView{L.coupling + lane_off, (long long)L.ups * NST, NST});
    ref_load(L, P, s, S);
    if (g.li == 0) {
      ref_store_harmonics(L, P, s, W.hc + g.grp, g.G);
      if constexpr (LIN == LIN_RICHARDSON) fast_until_of(W, g, P.nk) = ref_fast_until(L, P, s, S.t);
    }
  }
  __syncwarp();
  if (have && first_sample(S, P)) {
    ref_store_dense(L, S.t, S.y, g.li, s, S.idx);
    first_stored(S, P);
  }
  {
    const double g0 = group_event<KB>(S.y, upv(W, g, 12), g, P.col);
    if (S.active) S.g_old = g0;
  }

  for (long long it = 0; it < budget; ++it) {
    if (!__any_sync(FULL, S.active)) break;
    const bool st = step<KB, KC, LIN, KB == 2 && LIN == LIN_RICHARDSON>(g, P, W, S);
    if (st) ref_store_dense(L, S.t, S.y, g.li, s, S.idx);
    after_store(S, P, st);
  }

  if (have) {
    if (S.status == ST_ACTIVE && final_launch) S.status = ST_MAX_STEPS;
    ref_write_state(L, S.y, lane_off);
    if (g.li == 0) ref_write_scalars(L, P, s, S, active_counter);
  }
}

// The same for 9 to 16 bubbles with the Richardson solve (wide_core.cuh).
template <int KC>
__global__ void __launch_bounds__(WIDE_THREADS, 1)
    plain_wide_kernel(RefLayout L, Params P, long long budget, int final_launch, int* active_counter) {
  extern __shared__ __align__(16) double smem[];
  const Geo g = make_geo(KC > 0 ? KC : L.ups);
  const WideSmem W = wide_smem(smem, g.K, P.nk);
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long s = warp * g.G + g.grp;
  const bool have = g.valid && s < L.ns;
  const long long NST = (long long)L.ns * L.tile;
  const long long lane_off = s * L.tile + g.li;

  BubbleState S;
  S.c = W.cold + g.grp;
  S.o = W.own + g.lane;
  S.lead = have && g.li == 0;
  S.active = false;
  S.status = ST_ACTIVE;
  if (have) {
    ref_load_state(L, lane_off, S.y);
    ref_load(L, P, s, S);
    wide_store_bubble(W, g, L.unit_params + lane_off, NST,
                      MView{L.coupling + lane_off, (long long)L.ups * NST, NST});
    if (g.li == 0) ref_store_harmonics(L, P, s, W.hc + g.grp, g.G);
  }
  __syncwarp();
  if (have && first_sample(S, P)) {
    ref_store_dense(L, S.t, S.y, g.li, s, S.o->idx);
    first_stored(S, P);
  }
  {
    const double g0 = group_event<WIDE>(S.y, upv(W, g, 12), g, P.col);
    if (S.active) S.g_old = g0;
  }
  for (long long it = 0; it < budget; ++it) {
    if (!__any_sync(FULL, S.active)) break;
    const bool st = wide_step<KC>(g, P, W, S);
    if (st) ref_store_dense(L, S.t, S.y, g.li, s, S.o->idx);
    after_store(S, P, st);
  }
  if (have) {
    if (S.status == ST_ACTIVE && final_launch) S.status = ST_MAX_STEPS;
    ref_write_state(L, S.y, lane_off);
    if (g.li == 0) ref_write_scalars(L, P, s, S, active_counter);
  }
}

// The same for a single bubble per system with the Richardson solve: one system
// per lane (solo_core.cuh).
template <int KC>
__global__ void __launch_bounds__(SOLO_THREADS, SOLO_BLOCKS)
    plain_solo_kernel(RefLayout L, Params P, long long budget, int final_launch, int* active_counter) {
  extern __shared__ __align__(16) double smem[];
  const SoloSmem W = solo_smem(smem, P.nk);
  const int lane = threadIdx.x & 31;
  const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long NST = (long long)L.ns * L.tile;
  const bool have = s < L.ns;
  BubbleState S;
  S.c = W.cold + lane;
  S.o = W.own + lane;
  S.lead = true;
  S.active = false;
  S.status = ST_ACTIVE;
  if (have) {
    ref_load(L, P, s, S);
    ref_load_state(L, s * L.tile, S.y);
    solo_store_bubble(W, lane, L.unit_params + s * L.tile, NST);
    ref_store_harmonics(L, P, s, W.hc + lane, 32);
    if (first_sample(S, P)) {
      ref_store_dense(L, S.t, S.y, 0, s, S.o->idx);
      first_stored(S, P);
    }
    if (S.active) S.g_old = 1e30;
  }
  for (long long it = 0; it < budget; ++it) {
    if (!__any_sync(FULL, S.active)) break;
    const bool st = solo_step(P, W, lane, S);
    if (st) ref_store_dense(L, S.t, S.y, 0, s, S.o->idx);
    after_store(S, P, st);
  }
  if (have) {
    if (S.status == ST_ACTIVE && final_launch) S.status = ST_MAX_STEPS;
    ref_write_state(L, S.y, s * L.tile);
    ref_write_scalars(L, P, s, S, active_counter);
  }
}

// The same for 17 to 32 bubbles per system with the Richardson solve: one system
// per block of two warps (duo_core.cuh).
template <int KC>
__global__ void __launch_bounds__(DUO_THREADS, DUO_BLOCKS)
    plain_duo_kernel(RefLayout L, Params P, long long budget, int final_launch, int* active_counter) {
  extern __shared__ __align__(16) double smem[];
  const DuoGeo<1> g = make_duo_geo<1>(KC > 0 ? KC : L.ups);
  const DuoSmem W = duo_smem(g, smem, P.nk);
  const long long s = blockIdx.x;
  const long long NST = (long long)L.ns * L.tile;
  const long long lane_off = s * L.tile + (g.valid ? g.i : 0);
  const bool mine = g.valid && g.c == 0;

  BubbleState S;
  S.c = W.cold;
  S.o = W.own + g.tid;
  S.lead = g.tid == 0;
  ref_load_state(L, lane_off, S.y);
  ref_load(L, P, s, S);
  duo_store_bubble(W, g, L.unit_params + lane_off, NST, MView{L.coupling + lane_off, (long long)L.ups * NST, NST});
  if (g.tid == 0) ref_store_harmonics(L, P, s, W.hc, 1);
  __syncthreads();
  if (first_sample(S, P)) {
    if (mine) ref_store_dense(L, S.t, S.y, g.i, s, S.o->idx);
    first_stored(S, P);
  }
  {
    bool f = true, k = true;
    double r = 1.0;
    const double g0 = duo_event(g, W, S.y, P.col, f, k, r);
    if (S.active) S.g_old = g0;
  }
  for (long long it = 0; it < budget && S.active; ++it) {
    const bool st = duo_step(g, P, W, S);
    if (st && mine) ref_store_dense(L, S.t, S.y, g.i, s, S.o->idx);
    after_store(S, P, st);
  }
  if (S.status == ST_ACTIVE && final_launch) S.status = ST_MAX_STEPS;
  if (mine) ref_write_state(L, S.y, lane_off);
  if (g.tid == 0) ref_write_scalars(L, P, s, S, active_counter);
}

template <int KB, int KC>
cudaError_t launch_plain_k(const RefLayout& L, const Params& P, long long budget, int final_launch, int* counter,
                           cudaStream_t stream) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  int cap = 0;
  e = cudaDeviceGetAttribute(&cap, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) return e;
  return dispatch_lin(P.lin, [&](auto lin) {
    constexpr int LIN = decltype(lin)::value;
    const int threads = block_threads_for(L.ups, P.nk, LIN, (size_t)cap, 128);
    const int per_block = systems_per_block(L.ups, LIN, threads, 32);
    const long long blocks = ((long long)L.ns + per_block - 1) / per_block;
    const size_t shmem = kernel_smem(L.ups, P.nk, LIN, threads);
    const auto launch = [&](auto kernel) {
      if (shmem > 48 * 1024) {
        const cudaError_t ce = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shmem);
        if (ce != cudaSuccess) return ce;
      }
      kernel<<<(unsigned)blocks, threads, shmem, stream>>>(L, P, budget, final_launch, counter);
      return cudaGetLastError();
    };
    if constexpr (KC == 1 && LIN == LIN_RICHARDSON) return launch(plain_solo_kernel<KC>);
    else if constexpr (KB == 16 && LIN == LIN_RICHARDSON) return launch(plain_wide_kernel<KC>);
    else if constexpr (KB == 32 && LIN == LIN_RICHARDSON) return launch(plain_duo_kernel<KC>);
    else return launch(plain_kernel<KB, KC, LIN>);
  });
}

}  // namespace cbc
