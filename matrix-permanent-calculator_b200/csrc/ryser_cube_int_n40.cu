// ryser_cube_int_n40.cu -- column-cube walks (int32 x) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_int_n40(int i) { return cube_pick<3, 40>(i); }
}  // namespace perm
