// Fixed-point complex128 row passes, kernel shape 0: explicit instantiation.
#define SGPE_FX_KERNELS
#include "sgpe_launch.cuh"

namespace sgpe {
template cudaError_t launch_row_fx_s<0>(const RowArgs<double>*, int, int, int, cudaStream_t);
}  // namespace sgpe
