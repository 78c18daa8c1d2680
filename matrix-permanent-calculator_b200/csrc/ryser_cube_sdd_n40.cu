// ryser_cube_sdd_n40.cu -- column-cube walks (split-dd) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n40(int i) { return cube_pick<2, 40>(i); }
}  // namespace perm
