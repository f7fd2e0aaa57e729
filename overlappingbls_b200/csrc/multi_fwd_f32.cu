// Multi-field forward transforms for float.
#include "multi.cuh"
namespace obl {
template cudaError_t launch_rows_multi_fwd<float>(int, const RowArgs<float> &, const MultiPtr<float> &, int, cudaStream_t);
template cudaError_t launch_cols_multi_fwd<float>(int, const ColArgs<float> &, const MultiPtr<float> &, int, cudaStream_t);
}
