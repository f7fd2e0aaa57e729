// Multi-output row, column and inverse kernels of the step for float.
#include "fused_launch.cuh"
namespace obl {
template struct RowsFwd3Launch<float>;
template struct ColsFwdLaunch<float>;
template struct PinvLaunch<float>;
}
