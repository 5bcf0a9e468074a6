// The fused hexahedron kernels of mixed-precision plans.
#include "hex_launch.cuh"

namespace dgb {
DGB_HEX_LAUNCHES_F32()
}
