// ryser_cube_inta_n28.cu -- column-cube walks (int32 x with sum |term|) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_inta_n28(int i) { return cube_pick<4, 28>(i); }
}  // namespace perm
