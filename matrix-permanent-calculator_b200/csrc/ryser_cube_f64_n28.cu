// ryser_cube_f64_n28.cu -- column-cube walks (FP64 x) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n28(int i) { return cube_pick<0, 28>(i); }
}  // namespace perm
