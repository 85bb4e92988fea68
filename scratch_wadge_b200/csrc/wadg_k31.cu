// the 3D kernels of degree 1
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 3, 1)
}  // namespace wadg
