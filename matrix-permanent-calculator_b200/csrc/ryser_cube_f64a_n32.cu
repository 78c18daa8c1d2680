// ryser_cube_f64a_n32.cu -- column-cube walks (FP64 x with sum |term|) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64a_n32(int i) { return cube_pick<1, 32>(i); }
}  // namespace perm
