// Multi-field forward transforms for double.
#include "multi.cuh"
namespace obl {
template cudaError_t launch_rows_multi_fwd<double>(int, const RowArgs<double> &, const MultiPtr<double> &, int, cudaStream_t);
template cudaError_t launch_cols_multi_fwd<double>(int, const ColArgs<double> &, const MultiPtr<double> &, int, cudaStream_t);
}
