// Inverse passes of the pressure for float.
#include "fused_launch.cuh"
namespace obl {
template struct PinvLaunch<float>;
}
