// ryser_cube_inta_n32.cu -- column-cube walks (int32 x with sum |term|) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_inta_n32(int i) { return cube_pick<4, 32>(i); }
}  // namespace perm
