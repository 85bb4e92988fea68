// the 2D kernels of degree 3
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 2, 3)
}  // namespace wadg
