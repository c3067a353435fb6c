// Fixed-point complex128 column passes, kernel shape 0: explicit instantiation.
#define SGPE_FX_KERNELS
#include "sgpe_launch.cuh"

namespace sgpe {
template cudaError_t launch_col_fx_s<0>(const ColArgs<double>*, int, int, int, cudaStream_t);
}  // namespace sgpe
