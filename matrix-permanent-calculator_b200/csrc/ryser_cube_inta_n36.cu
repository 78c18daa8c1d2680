// ryser_cube_inta_n36.cu -- column-cube walks (int32 x with sum |term|) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_inta_n36(int i) { return cube_pick<4, 36>(i); }
}  // namespace perm
