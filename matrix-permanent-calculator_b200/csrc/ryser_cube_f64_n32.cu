// ryser_cube_f64_n32.cu -- column-cube walks (FP64 x) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n32(int i) { return cube_pick<0, 32>(i); }
}  // namespace perm
