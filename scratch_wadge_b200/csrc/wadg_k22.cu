// the 2D kernels of degree 2
#include "wadg_launch.cuh"

namespace wadg {
WADG_LAUNCHES_DEGREE(, 2, 2)
}  // namespace wadg
