// Inverse passes of the pressure for double.
#include "fused_launch.cuh"
namespace obl {
template struct PinvLaunch<double>;
}
