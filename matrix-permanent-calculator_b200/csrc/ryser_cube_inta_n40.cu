// ryser_cube_inta_n40.cu -- column-cube walks (int32 x with sum |term|) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_inta_n40(int i) { return cube_pick<4, 40>(i); }
}  // namespace perm
