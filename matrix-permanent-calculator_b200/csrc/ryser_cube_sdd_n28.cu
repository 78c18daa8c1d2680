// ryser_cube_sdd_n28.cu -- column-cube walks (split-dd) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n28(int i) { return cube_pick<2, 28>(i); }
}  // namespace perm
