// ryser_cube_sdd_n36.cu -- column-cube walks (split-dd) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n36(int i) { return cube_pick<2, 36>(i); }
}  // namespace perm
