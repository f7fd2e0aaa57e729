// Multi-output row and column kernels of the step for double.
#include "fused_launch.cuh"
namespace obl {
template struct RowsFwd3Launch<double>;
template struct ColsFwdLaunch<double>;
}
