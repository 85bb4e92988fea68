// the 2D kernels of degree 4
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 2, 4)
}  // namespace wadg
