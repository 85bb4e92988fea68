// the 3D kernels of degree 2
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 3, 2)
}  // namespace wadg
