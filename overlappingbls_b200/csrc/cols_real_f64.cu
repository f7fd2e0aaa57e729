// Real column (y-direction) kernel instantiations for double.
#include "lines_dispatch.cuh"
namespace obl {
template cudaError_t launch_cols_real<double>(int, int, const ColArgs<double> &, cudaStream_t);
}
