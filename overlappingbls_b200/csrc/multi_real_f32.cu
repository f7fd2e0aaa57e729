// Multi-field derivatives, pads and unpads for float.
#include "multi.cuh"
namespace obl {
template cudaError_t launch_rows_multi_real<float>(int, int, const RowArgs<float> &, const MultiPtr<float> &, int, cudaStream_t);
template cudaError_t launch_cols_multi_real<float>(int, int, const ColArgs<float> &, const MultiPtr<float> &, int, cudaStream_t);
}
