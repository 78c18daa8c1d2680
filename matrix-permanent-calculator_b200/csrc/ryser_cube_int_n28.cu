// ryser_cube_int_n28.cu -- column-cube walks (int32 x) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_int_n28(int i) { return cube_pick<3, 28>(i); }
}  // namespace perm
