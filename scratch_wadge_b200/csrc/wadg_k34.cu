// the 3D kernels of degree 4
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 3, 4)
}  // namespace wadg
