// generic_r31.cu -- the generic passes with compile-time butterflies up to
// radix 31 (generic_launch.cuh, zmid_launch.cuh).
#include "zmid_launch.cuh"

namespace m3d {
M3D_GEN_ALL(, 31)
M3D_GEN_ZMID_ALL(, 31)
}  // namespace m3d
