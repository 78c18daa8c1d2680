// ryser_cube_sdd_n32.cu -- column-cube walks (split-dd) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n32(int i) { return cube_pick<2, 32>(i); }
}  // namespace perm
