// ryser_cube_int_n32.cu -- column-cube walks (int32 x) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_int_n32(int i) { return cube_pick<3, 32>(i); }
}  // namespace perm
