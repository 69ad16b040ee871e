// generic_r13.cu -- the generic passes with compile-time butterflies up to
// radix 13 (generic_launch.cuh).
#include "generic_launch.cuh"

namespace m3d {
M3D_GEN_ALL(, 13)
}  // namespace m3d
