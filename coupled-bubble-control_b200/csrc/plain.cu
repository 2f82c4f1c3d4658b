// plain.cu -- the reference-layout solve and the context entry points of
// libcbc_b200.so.  cbc_solve replaces the host launch loop of the reference
// (backends/numba/rkck45_coupled_numba_solver.py:29-91); its kernels are in
// plain_kernel.cuh.
#include <new>

#include "cbc_internal.h"
#include "plain.h"

namespace cbc {

cudaError_t launch_plain_any(const RefLayout& L, const Params& P, long long budget, int final_launch,
                             int* counter, cudaStream_t stream) {
  return dispatch_k(L.ups, [&](auto kb, auto kc) {
    return launch_plain_k<decltype(kb)::value, decltype(kc)::value>(L, P, budget, final_launch, counter, stream);
  });
}

}  // namespace cbc

using namespace cbc;

extern "C" {

// Raised with every change of the kernels: launch shapes tuned on one version are
// not used by another (the tuner's table has it in its keys).
int32_t cbc_version(void) { return 101; }

int32_t cbc_create(cbc_context** out, int32_t device) {
  if (!out) return fail(nullptr, CBC_E_INVALID, "out is NULL");
  *out = nullptr;
  int ndev = 0;
  cudaError_t e = cudaGetDeviceCount(&ndev);
  if (e != cudaSuccess) return fail(nullptr, CBC_E_CUDA, "cudaGetDeviceCount: %s", cudaGetErrorString(e));
  if (device < 0 || device >= ndev) return fail(nullptr, CBC_E_INVALID, "device %d out of range (%d devices)", device, ndev);
  cbc_context* ctx = new (std::nothrow) cbc_context();
  if (!ctx) return fail(nullptr, CBC_E_NOMEM, "context allocation failed");
  ctx->device = device;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(device);
  cudaDeviceGetAttribute(&ctx->sm_count, cudaDevAttrMultiProcessorCount, device);
  e = cudaMalloc(&ctx->d_counter, sizeof(int));
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_head, kScheduleBytes);
  if (e == cudaSuccess) e = cudaMallocHost(&ctx->h_counter, sizeof(int));
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev0);
  if (e == cudaSuccess) e = cudaEventCreate(&ctx->ev1);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&ctx->fork, cudaEventDisableTiming);
  int prio_low = 0, prio_high = 0;
  if (e == cudaSuccess) e = cudaDeviceGetStreamPriorityRange(&prio_low, &prio_high);
  for (int i = 0; i < CBC_SIDE_STREAMS && e == cudaSuccess; ++i) {
    e = cudaEventCreateWithFlags(&ctx->join[i], cudaEventDisableTiming);
    // first half: higher priority (bucket start grids); second half: lowest
    // priority (backfill grids only take SMs no start grid is waiting for)
    const int prio = i < CBC_SIDE_STREAMS / 2 ? prio_high : prio_low;
    if (e == cudaSuccess) e = cudaStreamCreateWithPriority(&ctx->side[i], cudaStreamNonBlocking, prio);
  }
  if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&ctx->capture, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = noalloc_scratch_address(device, &ctx->noalloc_scratch);
  cudaSetDevice(prev);
  if (e != cudaSuccess) {
    cbc_destroy(ctx);
    return fail(nullptr, CBC_E_CUDA, "context set-up failed: %s", cudaGetErrorString(e));
  }
  *out = ctx;
  return CBC_OK;
}

int32_t cbc_destroy(cbc_context* ctx) {
  if (!ctx) return CBC_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(ctx->device);
  if (ctx->d_counter) cudaFree(ctx->d_counter);
  if (ctx->d_head) cudaFree(ctx->d_head);
  if (ctx->h_counter) cudaFreeHost(ctx->h_counter);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->fork) cudaEventDestroy(ctx->fork);
  for (int i = 0; i < CBC_SIDE_STREAMS; ++i) {
    if (ctx->join[i]) cudaEventDestroy(ctx->join[i]);
    if (ctx->side[i]) cudaStreamDestroy(ctx->side[i]);
  }
  if (ctx->capture) cudaStreamDestroy(ctx->capture);
  cudaSetDevice(prev);
  delete ctx;
  return CBC_OK;
}

const char* cbc_last_error(const cbc_context* ctx) {
  if (ctx) return ctx->err.c_str();
  return global_error().c_str();
}

int32_t cbc_solve(cbc_context* ctx, const cbc_spec* spec, const cbc_buffers* b, int64_t max_steps,
                  int32_t kernel_steps, int32_t launch_mode, void* stream_, cbc_solve_stats* stats) {
  if (!ctx) return fail(nullptr, CBC_E_INVALID, "context is NULL");
  ctx->err.clear();
  int32_t rc = check_spec(ctx, spec);
  if (rc) return rc;
  if (!b) return fail(ctx, CBC_E_INVALID, "buffers is NULL");
  if (max_steps < 1 || kernel_steps < 1) return fail(ctx, CBC_E_INVALID, "max_steps and kernel_steps must be >= 1");
  if (launch_mode != CBC_LAUNCH_RELAUNCH && launch_mode != CBC_LAUNCH_SINGLE)
    return fail(ctx, CBC_E_INVALID, "unknown launch mode %d", launch_mode);
  if (!b->actual_time || !b->time_end || !b->time_begin || !b->time_step || !b->actual_state || !b->unit_params ||
      !b->system_params || !b->control_params || !b->coupling_matrices || !b->actual_event || !b->status_flags)
    return fail(ctx, CBC_E_INVALID, "a required buffer pointer is NULL");
  if (spec->ndo > 0 && (!b->dense_index || !b->dense_time || !b->dense_state))
    return fail(ctx, CBC_E_INVALID, "ndo > 0 needs dense_index, dense_time and dense_state");

  RefLayout L;
  L.ns = spec->ns;
  L.ups = spec->ups;
  L.tile = spec->tile;
  L.actual_time = b->actual_time;
  L.time_end = b->time_end;
  L.time_begin = b->time_begin;
  L.time_step = b->time_step;
  L.actual_state = b->actual_state;
  L.unit_params = b->unit_params;
  L.system_params = b->system_params;
  L.control_params = b->control_params;
  L.coupling = b->coupling_matrices;
  L.dense_index = b->dense_index;
  L.dense_time = b->dense_time;
  L.dense_state = b->dense_state;
  L.actual_event = b->actual_event;
  L.status = b->status_flags;
  L.total_steps = b->total_steps;
  L.rejected_steps = b->rejected_steps;
  L.conv_success = b->convergence_success;
  L.conv_failures = b->convergence_failures;
  L.lin_iters = (long long*)b->lin_iters;
  const Params P = make_params(*spec);
  cudaStream_t stream = (cudaStream_t)stream_;

  int prev = 0;
  cudaGetDevice(&prev);
  if (prev != ctx->device) CBC_CUDA_TRY(ctx, cudaSetDevice(ctx->device));
  struct Restore {
    int d;
    ~Restore() { cudaSetDevice(d); }
  } restore{prev};

  const long long launches = (max_steps + kernel_steps - 1) / kernel_steps;
  int32_t n = 0;
  double dev_ms = 0.0;
  int32_t left = -1;
  if (launch_mode == CBC_LAUNCH_SINGLE) {
    CBC_CUDA_TRY(ctx, cudaEventRecord(ctx->ev0, stream));
    CBC_CUDA_TRY(ctx, launch_plain_any(L, P, launches * (long long)kernel_steps, 1, nullptr, stream));
    ++ctx->launches;
    CBC_CUDA_TRY(ctx, cudaEventRecord(ctx->ev1, stream));
    n = 1;
    if (stats) {
      CBC_CUDA_TRY(ctx, cudaEventSynchronize(ctx->ev1));
      float ms = 0.f;
      cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
      dev_ms = ms;
    }
  } else {
    // the reference host loop: launch, synchronise, stop when every system is done
    for (long long l = 0; l < launches; ++l) {
      const int final_launch = (l + 1 == launches);
      CBC_CUDA_TRY(ctx, cudaMemsetAsync(ctx->d_counter, 0, sizeof(int), stream));
      CBC_CUDA_TRY(ctx, cudaEventRecord(ctx->ev0, stream));
      CBC_CUDA_TRY(ctx, launch_plain_any(L, P, kernel_steps, final_launch, ctx->d_counter, stream));
      ++ctx->launches;
      CBC_CUDA_TRY(ctx, cudaEventRecord(ctx->ev1, stream));
      CBC_CUDA_TRY(ctx, cudaMemcpyAsync(ctx->h_counter, ctx->d_counter, sizeof(int), cudaMemcpyDeviceToHost, stream));
      CBC_CUDA_TRY(ctx, cudaStreamSynchronize(stream));
      float ms = 0.f;
      cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1);
      dev_ms += ms;
      ++n;
      left = *ctx->h_counter;
      if (left == 0) break;
    }
  }
  if (stats) {
    stats->launches = n;
    stats->active_left = left;
    stats->device_ms = dev_ms;
  }
  return CBC_OK;
}

}  // extern "C"
