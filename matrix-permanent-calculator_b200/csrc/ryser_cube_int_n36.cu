// ryser_cube_int_n36.cu -- column-cube walks (int32 x) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_int_n36(int i) { return cube_pick<3, 36>(i); }
}  // namespace perm
