// Multi-output row and column kernels of the step for float.
#include "fused_launch.cuh"
namespace obl {
template struct RowsFwd3Launch<float>;
template struct ColsFwdLaunch<float>;
}
