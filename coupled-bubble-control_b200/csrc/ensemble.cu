// ensemble.cu -- host side of the batched kernels: dispatch over the bubble
// count of a bucket, occupancy, the device clock stamp.  The kernels are in
// ensemble_kernel.cuh, compiled once per bubble count by kernels_k.cu.
#include "cbc_internal.h"
#include "ensemble.h"

namespace cbc {

size_t max_block_smem(int device) {
  int v = 0;
  cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  return (size_t)v;
}

__global__ void stamp_kernel(long long* epoch) { *epoch = global_ns(); }

cudaError_t launch_stamp(long long* epoch, cudaStream_t stream) {
  stamp_kernel<<<1, 1, 0, stream>>>(epoch);
  return cudaGetLastError();
}

cudaError_t launch_ensemble_bucket(const EnsLayout& E, const Params& P, const int* order, int begin, int end,
                                   int K, int* head, long long max_steps, int steps_total,
                                   const long long* epoch, long long budget_ns, int blocks, int threads,
                                   cudaStream_t stream, size_t smem_bytes, int slots, int mb) {
  return dispatch_k(K, [&](auto kb, auto kc) {
    return launch_ensemble_k<decltype(kb)::value, decltype(kc)::value>(E, P, order, begin, end, K, head, max_steps,
                                                                      steps_total, epoch, budget_ns, blocks, threads,
                                                                      stream, smem_bytes, slots, mb);
  });
}

int resident_blocks(int K, int nk, int threads, int lin, int mb) {
  int n = 0;
  const cudaError_t e = dispatch_k(K, [&](auto kb, auto kc) {
    return occupancy_k<decltype(kb)::value, decltype(kc)::value>(K, nk, threads, lin, mb, &n);
  });
  return (e == cudaSuccess && n > 0) ? n : 1;
}

}  // namespace cbc
