// Fixed-point complex128 passes, kernel shapes 1 and 2: explicit instantiation.
#define SGPE_FX_KERNELS
#include "sgpe_launch.cuh"

namespace sgpe {
template cudaError_t launch_row_fx_s<1>(const RowArgs<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_row_fx_s<2>(const RowArgs<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_col_fx_s<1>(const ColArgs<double>*, int, int, int, cudaStream_t);
template cudaError_t launch_col_fx_s<2>(const ColArgs<double>*, int, int, int, cudaStream_t);
}  // namespace sgpe
