// ensemble_kernel.cuh -- batched mixed-K integrator: persistent, work-stealing kernels
// over a ragged ensemble, launched together (optionally as one CUDA graph).
//
// The reference can only integrate one (NS, K) ensemble per kernel build
// (all shapes are compile-time macros, backends/cupy_cuda/kernel_loader.py:35-63;
// one thread per bubble padded to TILE = next_pow2(K), specs.py:40-52) and
// relaunches every kernel_steps steps with a host synchronisation.  Here:
//   * systems of any K <= 32 live in one ragged ensemble (CSR offsets);
//   * a work list orders the systems by K bucket, longest expected work first;
//   * each warp holds floor(32/K) system slots; whenever a system finishes,
//     its slot writes the result back and claims the next system of its bucket
//     with one atomicAdd per warp, so lanes never idle while work remains (above
//     16 bubbles with the Richardson solve a team of two warps holds one system);
//   * one persistent kernel per K bucket, of the form for its bubble count,
//     launched on forked streams so the buckets overlap and a bucket's tail is
//     filled by the next bucket's warps.
// Integration arithmetic is the same device code as the reference-layout
// kernels, so results are bit-identical to the CPU oracle.
#pragma once

#include "cbc_internal.h"
#include "ensemble.h"
#include "duo_core.cuh"
#include "solo_core.cuh"
#include "warp_turn.h"
#include "wide_core.cuh"

namespace cbc {

// Dense sample `slot` of bubble i (row boff + i, state y) of system s at time t.
__device__ __forceinline__ void ens_store_dense(const EnsLayout& E, double t, const double y[4], long long boff, int i,
                                                int s, int slot) {
  if (i == 0) E.dense_time[(long long)slot * E.ns + s] = t;
  double2* d = reinterpret_cast<double2*>(E.dense_state + ((long long)slot * E.nb + boff + i) * 4);
  d[0] = make_double2(y[0], y[1]);
  d[1] = make_double2(y[2], y[3]);
}

// State of the bubble in row `row`, from and to memory.
__device__ __forceinline__ void ens_load_state(const EnsLayout& E, long long row, double y[4]) {
  const double2* st = reinterpret_cast<const double2*>(E.state + row * 4);
  const double2 s01 = st[0], s23 = st[1];
  y[0] = s01.x;
  y[1] = s01.y;
  y[2] = s23.x;
  y[3] = s23.y;
}
__device__ __forceinline__ void ens_write_state(const EnsLayout& E, long long row, const double y[4]) {
  double2* st = reinterpret_cast<double2*>(E.state + row * 4);
  st[0] = make_double2(y[0], y[1]);
  st[1] = make_double2(y[2], y[3]);
}

// Time of the last stored dense sample (0 if none).
__device__ __forceinline__ double ens_prev_time(const EnsLayout& E, const Params& P, int s, int idx) {
  return (P.ndo > 0 && idx > 0) ? E.dense_time[(long long)(idx - 1) * E.ns + s] : 0.0;
}

// Scalars of system s into a lane's state, and the prologue: scalars in
// registers, or in shared memory.
__device__ __forceinline__ void ens_load_scalars(const EnsLayout& E, const Params& P, int s, ScalarState& S) {
  const double* sp = E.system_params + (long long)s * E.sp_stride;
  const double t_end = E.t_end[s];
  S.t = E.t[s];
  S.h = E.h[s];
  S.o->idx = (P.ndo > 0) ? E.dense_index[s] : 0;
  if (S.lead) {
    S.c->sp0 = sp[0];
    S.c->sp3 = sp[3];
    S.c->boff = E.bubble_offset[s];
    S.c->fast_until = fast_until(sp[0], sp[1], sp[2], E.control_params + (long long)s * E.cp_stride, P.nk, 1, S.t);
  }
  prologue(S, P, t_end, E.t_begin[s], E.event[s], ens_prev_time(E, P, s, S.o->idx), E.status[s]);
}

// Steps that count against max_steps from before this call (steps_total).
__device__ __forceinline__ long long ens_base(const EnsLayout& E, int s, int steps_total) {
  return (steps_total && E.steps) ? (long long)E.steps[s] : 0;
}
__device__ __forceinline__ void ens_step_base(const EnsLayout& E, int s, int steps_total, long long max_steps,
                                              ScalarState& S) {
  const long long base = ens_base(E, s, steps_total);
  if (S.lead) S.c->step_base = base;
  if (S.active && base >= max_steps) {
    S.status = ST_MAX_STEPS;
    S.active = false;
  }
}

// Scalars and counters of system s (one lane of the system).
__device__ __forceinline__ void ens_write_scalars(const EnsLayout& E, const Params& P, int s, double t, double h,
                                                  double event, int status, int idx, int steps, int rejected,
                                                  int conv_ok, int conv_fail, long long lin_iters) {
  if (E.trace_done_ns) E.trace_done_ns[s] = global_ns();
  E.t[s] = t;
  E.h[s] = h;
  E.event[s] = event;
  E.status[s] = status;
  if (P.ndo > 0) E.dense_index[s] = idx;
  if (E.steps) E.steps[s] += steps;
  if (E.rejected) E.rejected[s] += rejected;
  if (E.conv_ok) E.conv_ok[s] += conv_ok;
  if (E.conv_fail) E.conv_fail[s] += conv_fail;
  if (E.lin_iters) E.lin_iters[s] += lin_iters;
}
__device__ __forceinline__ void ens_write_scalars(const EnsLayout& E, const Params& P, int s, const ScalarState& S) {
  ens_write_scalars(E, P, s, S.t, S.h, S.g_old, S.status, S.o->idx, S.o->steps, S.c->rejected, S.c->conv_ok,
                    S.c->conv_fail, S.c->lin_iters);
}

// ---- 2 to 8 bubbles, and the direct solve for any number (ckm1d_core.cuh) ----

// Loads system s into this lane's slot (lane li of the group) and runs the
// prologue.  Called only by lanes whose group claimed s.
template <int LIN>
__device__ __forceinline__ void lane_load(const EnsLayout& E, const Params& P, const Geo& g, int s, LaneState& S,
                                         const WarpSmem& W, long long& boff) {
  boff = E.bubble_offset[s];
  if (g.li == 0 && E.trace_load_ns) E.trace_load_ns[s] = global_ns();
  const long long b = boff + g.li;
  ens_load_state(E, b, S.y);
  store_bubble_consts(W, g, E.unit_params + b * E.up_stride, 1);
  const double* sp = E.system_params + (long long)s * E.sp_stride;
  S.sp0 = sp[0];
  S.sp3 = sp[3];
  S.t = E.t[s];
  S.t_end = E.t_end[s];
  S.t_begin = E.t_begin[s];
  S.h = E.h[s];
  S.idx = (P.ndo > 0) ? E.dense_index[s] : 0;
  prologue(S, P, E.event[s], ens_prev_time(E, P, s, S.idx), E.status[s]);
  store_coupling(W, g, MView{E.coupling + E.coupling_offset[s] + g.li, (long long)g.K * g.K, g.K});
  if (g.li == 0) {
    const double* cp = E.control_params + (long long)s * E.cp_stride;
    store_harmonics(W.hc + g.grp, g.G, sp[1], sp[2], sp[4], cp, P.nk, 1);
    if constexpr (LIN == LIN_RICHARDSON)
      fast_until_of(W, g, P.nk) = fast_until(sp[0], sp[1], sp[2], cp, P.nk, 1, S.t);
  }
}

__device__ __forceinline__ void lane_writeback(const EnsLayout& E, const Params& P, const Geo& g, int s,
                                              long long boff, LaneState& S) {
  ens_write_state(E, boff + g.li, S.y);
  if (g.li == 0)
    ens_write_scalars(E, P, s, S.t, S.h, S.g_old, S.status, S.idx, S.steps, S.rejected, S.conv_ok, S.conv_fail,
                      S.lin_iters);
}

// Persistent worker: warps claim systems of bucket [begin, end) of the work
// list until it is empty.  All systems of a bucket have the same K (<= KB).
template <int KB, int KC, int LIN, int MB>
__global__ void __launch_bounds__(128, min_blocks_variant(KB, MB))
    ensemble_kernel(EnsLayout E, Params P, const int* __restrict__ order, int begin, int end, int K, int* head,
                    long long max_steps, int steps_total, const long long* epoch, long long budget_ns,
                    int slots) {
  extern __shared__ __align__(16) double smem[];
  const Geo g = make_geo(KC > 0 ? KC : K, slots);
  const WarpSmem W = warp_smem(smem, g.K, P.nk, LIN);
  const int lane = threadIdx.x & 31;
  const bool leader = g.valid && g.li == 0;

  LaneState S;
  S.active = false;
  S.status = ST_ACTIVE;
  S.steps = 0;
  int sys = -1;           // system in this lane's slot (-1: none)
  long long boff = 0;
  long long step_base = 0;  // steps the system had accumulated before it was loaded (steps_total)
  bool drained = false;   // work list exhausted for this warp (warp-uniform)
  const long long deadline = budget_ns > 0 ? epoch[0] + budget_ns : 0;
  bool sliced_out = false;  // time slice over (warp-uniform); independent of drained

  while (true) {
    // ---- time slice over: stop every slot after its current step ----
    if (deadline != 0 && !sliced_out) {
      long long now = 0;
      if (lane == 0) now = global_ns();
      now = __shfl_sync(FULL, now, 0);
      if (now >= deadline) {
        sliced_out = true;
        drained = true;
      }
    }
    if (sliced_out && S.active) {
      S.status = ST_MAX_STEPS;
      S.active = false;
    }
    // ---- retire finished systems and refill empty slots (warp-uniform) ----
    const bool retire = g.valid && sys >= 0 && !S.active;
    if (__any_sync(FULL, retire)) {
      if (retire) lane_writeback(E, P, g, sys, boff, S);
      if (retire) sys = -1;
    }
    const bool want = leader && sys < 0 && !drained;
    const unsigned wmask = __ballot_sync(FULL, want);
    if (wmask) {
      int base_idx = 0;
      if (lane == 0) base_idx = atomicAdd(head, __popc(wmask));
      base_idx = __shfl_sync(FULL, base_idx, 0);
      int claim = -1;
      if (want) {
        const int idx = begin + base_idx + __popc(wmask & ((1u << lane) - 1u));
        claim = (idx < end) ? order[idx] : -1;
      }
      if (__any_sync(FULL, want && claim < 0)) drained = true;
      // hand the claimed system id to every lane of the group
      // (both shuffles are executed by every lane: never inside a
      // short-circuit or a divergent branch)
      const int got = __shfl_sync(FULL, claim, g.base);
      const int leader_wanted = __shfl_sync(FULL, (int)want, g.base);
      const bool fresh = g.valid && sys < 0 && got >= 0 && leader_wanted != 0;
      if (fresh) {
        sys = got;
        lane_load<LIN>(E, P, g, sys, S, W, boff);
        step_base = (steps_total && E.steps) ? (long long)E.steps[sys] : 0;
        if (S.active && step_base >= max_steps) {
          S.status = ST_MAX_STEPS;
          S.active = false;
        }
      }
      __syncwarp();
      // first dense sample and initial event value for the fresh systems
      if (fresh && S.active && P.ndo > 0) {
        bool stq;
        if (P.dense_mode == 0) stq = (S.idx < P.ndo) && (S.dnext <= S.t);
        else stq = (S.idx < P.ndo) && (S.t >= grid_time(S, S.idx, P.ndo));
        if (stq) {
          ens_store_dense(E, S.t, S.y, boff, g.li, sys, S.idx);
          S.idx += 1;
          if (P.dense_mode == 0) {
            const double nx = S.t + S.ddt;
            S.dnext = nx < S.t_end ? nx : S.t_end;
          }
        }
      }
      const double g0 = group_event<KB>(S.y, upv(W, g, 12), g, P.col);
      if (fresh && S.active) S.g_old = g0;
      // systems that arrive already finished go straight back out
      continue;
    }
    if (!__any_sync(FULL, S.active)) {
      if (!__any_sync(FULL, sys >= 0)) break;  // nothing left in any slot
      continue;
    }
    // ---- one Cash-Karp step for every active slot ----
    const bool stq = step<KB, KC, LIN>(g, P, W, S);
    if (stq) ens_store_dense(E, S.t, S.y, boff, g.li, sys, S.idx);
    after_store(S, P, stq);
    if (S.active && S.steps + step_base >= max_steps) {
      S.status = ST_MAX_STEPS;
      S.active = false;
    }
  }
}

// 9 to 16 bubbles with the Richardson solve (wide_core.cuh):
template <int KC>
struct WideForm {
  Geo g;
  WideSmem W;
  BubbleState S;

  __device__ __forceinline__ WideForm(double* smem, int K, int nk, int slots)
      : g(make_geo(KC > 0 ? KC : K, slots)), W(wide_smem(smem, g.K, nk)) {
    S.c = W.cold + g.grp;
    S.o = W.own + g.lane;
    S.lead = g.valid && g.li == 0;
    S.active = false;
    S.status = ST_ACTIVE;
  }
  __device__ __forceinline__ void load(const EnsLayout& E, const Params& P, int s, int steps_total,
                                       long long max_steps) {
    const long long row = E.bubble_offset[s] + g.li;
    ens_load_state(E, row, S.y);
    ens_load_scalars(E, P, s, S);
    wide_store_bubble(W, g, E.unit_params + row * E.up_stride, 1,
                      MView{E.coupling + E.coupling_offset[s] + g.li, (long long)g.K * g.K, g.K});
    const double* sp = E.system_params + (long long)s * E.sp_stride;
    if (S.lead)
      store_harmonics(W.hc + g.grp, g.G, sp[1], sp[2], sp[4], E.control_params + (long long)s * E.cp_stride, P.nk, 1);
    ens_step_base(E, s, steps_total, max_steps, S);
  }
  __device__ __forceinline__ void begin(const EnsLayout& E, const Params& P, bool fresh, int s) {
    if (fresh && first_sample(S, P)) {
      ens_store_dense(E, S.t, S.y, S.c->boff, g.li, s, S.o->idx);
      first_stored(S, P);
    }
    const double g0 = group_event<WIDE>(S.y, upv(W, g, 12), g, P.col);
    if (fresh && S.active) S.g_old = g0;
  }
  __device__ __forceinline__ void write(const EnsLayout& E, const Params& P, int s) {
    ens_write_state(E, S.c->boff + g.li, S.y);
    if (S.lead) ens_write_scalars(E, P, s, S);
  }
  __device__ __forceinline__ void stop() {
    S.status = ST_MAX_STEPS;
    S.active = false;
  }
  __device__ __forceinline__ void advance(const EnsLayout& E, const Params& P, int s, long long max_steps) {
    const bool stq = wide_step<KC>(g, P, W, S);
    if (stq) ens_store_dense(E, S.t, S.y, S.c->boff, g.li, s, S.o->idx);
    after_store(S, P, stq);
    if (S.active && S.o->steps + S.c->step_base >= max_steps) stop();
  }
};

// Persistent worker: warps claim systems of bucket [begin, end) of the work
// list until it is empty.  All systems of a bucket have the same K.
template <class Form>
__device__ __forceinline__ void ensemble_worker(Form& f, const EnsLayout& E, const Params& P,
                                                const int* __restrict__ order, int begin, int end, int* head,
                                                long long max_steps, int steps_total, const long long* epoch,
                                                long long budget_ns) {
  const Geo& g = f.g;
  const int lane = threadIdx.x & 31;
  const bool leader = g.valid && g.li == 0;
  int sys = -1;           // system in this lane's slot (-1: none)
  bool drained = false;   // work list exhausted for this warp (warp-uniform)
  const long long deadline = budget_ns > 0 ? epoch[0] + budget_ns : 0;
  bool sliced_out = false;  // time slice over (warp-uniform); independent of drained

  while (true) {
    // ---- time slice over: stop every slot after its current step ----
    if (deadline != 0 && !sliced_out) {
      long long now = 0;
      if (lane == 0) now = global_ns();
      now = __shfl_sync(FULL, now, 0);
      if (now >= deadline) {
        sliced_out = true;
        drained = true;
      }
    }
    if (sliced_out && f.S.active) f.stop();
    // ---- retire finished systems and refill empty slots (warp-uniform) ----
    const bool retire = g.valid && sys >= 0 && !f.S.active;
    if (__any_sync(FULL, retire)) {
      if (retire) {
        f.write(E, P, sys);
        sys = -1;
      }
      __syncwarp();
    }
    const bool want = leader && sys < 0 && !drained;
    const unsigned wmask = __ballot_sync(FULL, want);
    if (wmask) {
      int base_idx = 0;
      if (lane == 0) base_idx = atomicAdd(head, __popc(wmask));
      base_idx = __shfl_sync(FULL, base_idx, 0);
      int claim = -1;
      if (want) {
        const int idx = begin + base_idx + __popc(wmask & ((1u << lane) - 1u));
        claim = (idx < end) ? order[idx] : -1;
      }
      if (__any_sync(FULL, want && claim < 0)) drained = true;
      // hand the claimed system id to every lane of the group
      // (both shuffles are executed by every lane: never inside a
      // short-circuit or a divergent branch)
      const int got = __shfl_sync(FULL, claim, g.base);
      const int leader_wanted = __shfl_sync(FULL, (int)want, g.base);
      const bool fresh = g.valid && sys < 0 && got >= 0 && leader_wanted != 0;
      if (fresh) {
        sys = got;
        if (leader && E.trace_load_ns) E.trace_load_ns[sys] = global_ns();
        f.load(E, P, sys, steps_total, max_steps);
      }
      __syncwarp();
      f.begin(E, P, fresh, sys);
      // systems that arrive already finished go straight back out
      continue;
    }
    if (!__any_sync(FULL, f.S.active)) {
      if (!__any_sync(FULL, sys >= 0)) break;  // nothing left in any slot
      continue;
    }
    // ---- one Cash-Karp step for every active slot ----
    f.advance(E, P, sys, max_steps);
  }
}

template <int KC>
__global__ void __launch_bounds__(WIDE_THREADS, 1)
    ensemble_wide_kernel(EnsLayout E, Params P, const int* __restrict__ order, int begin, int end, int K, int* head,
                         long long max_steps, int steps_total, const long long* epoch, long long budget_ns,
                         int slots) {
  extern __shared__ __align__(16) double smem[];
  WideForm<KC> f(smem, K, P.nk, slots);
  ensemble_worker(f, E, P, order, begin, end, head, max_steps, steps_total, epoch, budget_ns);
}

// The same for a single bubble per system with the Richardson solve: one system
// per lane (solo_core.cuh).  slots: lanes of a warp that take systems.
template <int KC>
__global__ void __launch_bounds__(SOLO_THREADS, SOLO_BLOCKS)
    ensemble_solo_kernel(EnsLayout E, Params P, const int* __restrict__ order, int begin, int end, int* head,
                         long long max_steps, int steps_total, const long long* epoch, long long budget_ns,
                         int slots) {
  extern __shared__ __align__(16) double smem[];
  const SoloSmem W = solo_smem(smem, P.nk);
  const int lane = threadIdx.x & 31;
  BubbleState S;
  S.c = W.cold + lane;
  S.o = W.own + lane;
  S.lead = true;
  S.active = false;
  S.status = ST_ACTIVE;
  int sys = -1;           // system of this lane (-1: none)
  bool drained = lane >= slots;
  const long long deadline = budget_ns > 0 ? epoch[0] + budget_ns : 0;

  while (true) {
    // time slice over: stop every system after its current step, claim no more
    if (deadline != 0) {
      long long now = 0;
      if (lane == 0) now = global_ns();
      now = __shfl_sync(FULL, now, 0);
      if (now >= deadline) {
        drained = true;
        if (S.active) {
          S.status = ST_MAX_STEPS;
          S.active = false;
        }
      }
    }
    const unsigned active = __ballot_sync(FULL, S.active), held = __ballot_sync(FULL, sys >= 0),
                   done = __ballot_sync(FULL, drained);
    const Turn turn = next_turn(active, held, done);
    if (turn == Turn::exit) break;
    // retire finished systems and refill empty lanes
    if (turn == Turn::refill) {
      if (sys >= 0 && !S.active) {
        ens_write_state(E, S.c->boff, S.y);
        ens_write_scalars(E, P, sys, S);
        sys = -1;
      }
      const bool want = sys < 0 && !drained;
      const unsigned wmask = __ballot_sync(FULL, want);
      if (wmask) {
        int base_idx = 0;
        if (lane == 0) base_idx = atomicAdd(head, __popc(wmask));
        base_idx = __shfl_sync(FULL, base_idx, 0);
        if (want) {
          const int idx = begin + base_idx + __popc(wmask & ((1u << lane) - 1u));
          if (idx < end) {
            sys = order[idx];
            const long long row = E.bubble_offset[sys];
            if (E.trace_load_ns) E.trace_load_ns[sys] = global_ns();
            ens_load_scalars(E, P, sys, S);
            ens_load_state(E, row, S.y);
            solo_store_bubble(W, lane, E.unit_params + row * E.up_stride, 1);
            const double* sp = E.system_params + (long long)sys * E.sp_stride;
            store_harmonics(W.hc + lane, 32, sp[1], sp[2], sp[4], E.control_params + (long long)sys * E.cp_stride,
                            P.nk, 1);
            ens_step_base(E, sys, steps_total, max_steps, S);
            // first dense sample and initial event value
            if (first_sample(S, P)) {
              ens_store_dense(E, S.t, S.y, S.c->boff, 0, sys, S.o->idx);
              first_stored(S, P);
            }
            if (S.active) S.g_old = 1e30;
          } else {
            drained = true;
          }
        }
      }
      __syncwarp();
      continue;    // systems that arrived already finished go straight back out
    }
    // one Cash-Karp step for every active lane
    const bool stq = solo_step(P, W, lane, S);
    if (stq) ens_store_dense(E, S.t, S.y, S.c->boff, 0, sys, S.o->idx);
    after_store(S, P, stq);
    if (S.active && S.o->steps + S.c->step_base >= max_steps) {
      S.status = ST_MAX_STEPS;
      S.active = false;
    }
  }
}

// The same for 17 to 32 bubbles per system with the Richardson solve: one system
// per team of two warps (duo_core.cuh), TEAMS of them to a block, each claiming
// for itself.  KC: exact K, or 0 (read at run time).
template <int KC, int TEAMS>
__global__ void __launch_bounds__(DUO_THREADS * TEAMS, DUO_BLOCKS / TEAMS)
    ensemble_duo_kernel(EnsLayout E, Params P, const int* __restrict__ order, int begin, int end, int K, int* head,
                         long long max_steps, int steps_total, const long long* epoch, long long budget_ns) {
  extern __shared__ __align__(16) double smem[];
  const DuoGeo<TEAMS> g = make_duo_geo<TEAMS>(KC > 0 ? KC : K);
  const DuoSmem W = duo_smem(g, smem, P.nk);
  // [0] claimed system, [1] whether the time slice is over.  A block of one team keeps
  // them in static shared memory (run-time K spills 50 bytes then, 130 in dynamic
  // memory: GPU full 122.2 ns an attempt against 123.5 for K = 20); a lane's block
  // requests all that its SM has and may have none.
  int* claim = W.claim;
  if constexpr (TEAMS == 1) {
    __shared__ int words[2];
    claim = words;
  }
  const long long deadline = budget_ns > 0 ? epoch[0] + budget_ns : 0;
  BubbleState S;
  S.c = W.cold;
  S.o = W.own + g.tid;
  S.lead = g.tid == 0;
  while (true) {
    // claim the next system; none once the slice is over
    if (g.tid == 0) {
      int idx = -1;
      if (deadline == 0 || global_ns() < deadline) {
        const int n = begin + atomicAdd(head, 1);
        if (n < end) idx = order[n];
      }
      claim[0] = idx;
    }
    duo_sync(g);
    const int sys = claim[0];
    if (sys < 0) break;
    const long long row = E.bubble_offset[sys] + (g.valid ? g.i : 0);
    if (g.tid == 0 && E.trace_load_ns) E.trace_load_ns[sys] = global_ns();
    ens_load_state(E, row, S.y);
    ens_load_scalars(E, P, sys, S);
    duo_store_bubble(W, g, E.unit_params + row * E.up_stride, 1,
                      MView{E.coupling + E.coupling_offset[sys] + (g.valid ? g.i : 0), (long long)g.K * g.K, g.K});
    const double* sp = E.system_params + (long long)sys * E.sp_stride;
    if (g.tid == 0)
      store_harmonics(W.hc, 1, sp[1], sp[2], sp[4], E.control_params + (long long)sys * E.cp_stride, P.nk, 1);
    ens_step_base(E, sys, steps_total, max_steps, S);
    duo_sync(g);
    if (first_sample(S, P)) {
      if (g.valid && g.c == 0) ens_store_dense(E, S.t, S.y, S.c->boff, g.i, sys, S.o->idx);
      first_stored(S, P);
    }
    {
      bool f = true, k = true;
      double r = 1.0;
      const double g0 = duo_event(g, W, S.y, P.col, f, k, r);
      if (S.active) S.g_old = g0;
    }
    while (S.active) {
      if (deadline != 0) {     // time slice over: stop after the current step
        if (g.tid == 0) claim[1] = global_ns() >= deadline;
        duo_sync(g);
        if (claim[1]) {
          S.status = ST_MAX_STEPS;
          S.active = false;
          break;
        }
      }
      const bool stq = duo_step(g, P, W, S);
      if (stq && g.valid && g.c == 0) ens_store_dense(E, S.t, S.y, S.c->boff, g.i, sys, S.o->idx);
      after_store(S, P, stq);
      if (S.active && S.o->steps + S.c->step_base >= max_steps) {
        S.status = ST_MAX_STEPS;
        S.active = false;
      }
    }
    if (g.valid && g.c == 0) ens_write_state(E, S.c->boff + g.i, S.y);
    if (g.tid == 0) ens_write_scalars(E, P, sys, S);
  }
}

// Every batched kernel asks for the same (maximum) shared-memory carveout, so
// that blocks of different bucket kernels can share an SM: with per-kernel
// carveouts an SM configured for one kernel takes no block of another until it
// drains, which serialises the buckets.
template <class Kernel>
cudaError_t configure_kernel(Kernel kernel, size_t shmem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       (int)cudaSharedmemCarveoutMaxShared);
  // the opt-in limit is raised to the device maximum (never lowered again), so
  // a launch captured earlier with a larger request stays valid
  if (e == cudaSuccess && shmem > 48 * 1024) {
    int dev = 0;
    e = cudaGetDevice(&dev);
    const size_t cap = max_block_smem(dev);
    if (e == cudaSuccess) {
      if (shmem > cap) return cudaErrorInvalidValue;
      e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cap);
    }
  }
  return e;
}

template <int KB, int KC>
cudaError_t launch_ensemble_k(const EnsLayout& E, const Params& P, const int* order, int begin, int end, int K,
                              int* head, long long max_steps, int steps_total, const long long* epoch,
                              long long budget_ns, int blocks, int threads, cudaStream_t stream, size_t smem_bytes,
                              int slots, int mb) {
  return dispatch_lin(P.lin, [&](auto lin) {
    return dispatch_mb(KB <= 8 ? mb : 0, [&](auto mbv) {
      constexpr int LIN = decltype(lin)::value, MB = KB <= 8 ? decltype(mbv)::value : 0;
      size_t shmem = kernel_smem(K, P.nk, LIN, threads);
      if (smem_bytes > shmem) shmem = smem_bytes;
      if constexpr (KC == 1 && LIN == LIN_RICHARDSON) {
        const auto kernel = ensemble_solo_kernel<KC>;
        const cudaError_t e = configure_kernel(kernel, shmem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, shmem, stream>>>(E, P, order, begin, end, head, max_steps, steps_total, epoch,
                                                   budget_ns, slots);
      } else if constexpr (KB == 32 && LIN == LIN_RICHARDSON) {
        const auto kernel = threads == DUO_THREADS ? ensemble_duo_kernel<KC, 1> : ensemble_duo_kernel<KC, DUO_BLOCKS>;
        const cudaError_t e = configure_kernel(kernel, shmem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, shmem, stream>>>(E, P, order, begin, end, K, head, max_steps, steps_total, epoch,
                                                   budget_ns);
      } else if constexpr (KB == 16 && LIN == LIN_RICHARDSON) {
        const auto kernel = ensemble_wide_kernel<KC>;
        const cudaError_t e = configure_kernel(kernel, shmem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, shmem, stream>>>(E, P, order, begin, end, K, head, max_steps, steps_total, epoch,
                                                   budget_ns, slots);
      } else {
        const auto kernel = ensemble_kernel<KB, KC, LIN, MB>;
        const cudaError_t e = configure_kernel(kernel, shmem);
        if (e != cudaSuccess) return e;
        kernel<<<blocks, threads, shmem, stream>>>(E, P, order, begin, end, K, head, max_steps, steps_total, epoch,
                                                   budget_ns, slots);
      }
      return cudaGetLastError();
    });
  });
}

template <int KB, int KC>
cudaError_t occupancy_k(int K, int nk, int threads, int lin, int mb, int* n) {
  const size_t shmem = kernel_smem(K, nk, lin, threads);
  return dispatch_lin(lin, [&](auto li) {
    return dispatch_mb(KB <= 8 ? mb : 0, [&](auto mbv) {
      constexpr int LIN = decltype(li)::value, MB = KB <= 8 ? decltype(mbv)::value : 0;
      if constexpr (KC == 1 && LIN == LIN_RICHARDSON) {
        const auto kernel = ensemble_solo_kernel<KC>;
        configure_kernel(kernel, shmem);
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kernel, threads, shmem);
      } else if constexpr (KB == 32 && LIN == LIN_RICHARDSON) {
        const auto kernel = ensemble_duo_kernel<KC, 1>;
        configure_kernel(kernel, shmem);
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kernel, threads, shmem);
      } else if constexpr (KB == 16 && LIN == LIN_RICHARDSON) {
        const auto kernel = ensemble_wide_kernel<KC>;
        configure_kernel(kernel, shmem);
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kernel, threads, shmem);
      } else {
        const auto kernel = ensemble_kernel<KB, KC, LIN, MB>;
        configure_kernel(kernel, shmem);
        return cudaOccupancyMaxActiveBlocksPerMultiprocessor(n, kernel, threads, shmem);
      }
    });
  });
}

}  // namespace cbc
