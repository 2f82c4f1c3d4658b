// plain.h -- device view of the reference-layout buffers and the launcher of
// the reference-layout kernels.
#pragma once

namespace cbc {

struct RefLayout {
  int ns, ups, tile;
  double* actual_time;
  const double* time_end;
  const double* time_begin;
  double* time_step;
  double* actual_state;
  const double* unit_params;
  const double* system_params;
  const double* control_params;
  const double* coupling;
  int* dense_index;
  double* dense_time;
  double* dense_state;
  double* actual_event;
  int* status;
  int* total_steps;
  int* rejected_steps;
  int* conv_success;
  int* conv_failures;
  long long* lin_iters;
};

// Launches the kernel of one instantiation (KB, KC; see dispatch_k): defined in
// plain_kernel.cuh, instantiated by kernels_k.cu.
template <int KB, int KC>
cudaError_t launch_plain_k(const RefLayout& L, const Params& P, long long budget, int final_launch, int* counter,
                           cudaStream_t stream);

}  // namespace cbc
