// ryser_cube_f64_n36.cu -- column-cube walks (FP64 x) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n36(int i) { return cube_pick<0, 36>(i); }
}  // namespace perm
