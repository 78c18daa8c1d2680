// ryser_cube_f64a_n36.cu -- column-cube walks (FP64 x with sum |term|) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64a_n36(int i) { return cube_pick<1, 36>(i); }
}  // namespace perm
