// kernels_k.cu -- the batched and reference-layout kernels of one
// instantiation: compiled once per (CBC_KB, CBC_KC) pair of dispatch_k, so that
// the instantiations build in parallel.
// Above 8 bubbles the matrix rows of a lane fill its registers, and tables that
// the compiler may fold cost more of them (9 to 15 bubbles: 88 bytes spilled, 64
// without; 17 to 31: 54, 50; direct solve: 254 registers, 194).  Up to 8 bubbles it is
// the other way round (2 bubbles: 0 bytes folded, 20 without; direct solve 0, 218).
#if CBC_KB >= 16
#define CBCM_TABLE_CONST
#endif
#include "ensemble_kernel.cuh"
#include "plain_kernel.cuh"

namespace cbc {

template cudaError_t launch_ensemble_k<CBC_KB, CBC_KC>(const EnsLayout&, const Params&, const int*, int, int, int,
                                                       int*, long long, int, const long long*, long long, int, int,
                                                       cudaStream_t, size_t, int, int);
template cudaError_t occupancy_k<CBC_KB, CBC_KC>(int, int, int, int, int, int*);
template cudaError_t launch_plain_k<CBC_KB, CBC_KC>(const RefLayout&, const Params&, long long, int, int*,
                                                    cudaStream_t);

}  // namespace cbc
