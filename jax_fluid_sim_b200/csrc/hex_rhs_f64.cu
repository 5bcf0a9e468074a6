// The fused hexahedron kernels in float64.
#include "hex_launch.cuh"

namespace dgb {
DGB_HEX_LAUNCHES(, double)
}
