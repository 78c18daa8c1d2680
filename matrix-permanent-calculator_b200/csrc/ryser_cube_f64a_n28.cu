// ryser_cube_f64a_n28.cu -- column-cube walks (FP64 x with sum |term|) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64a_n28(int i) { return cube_pick<1, 28>(i); }
}  // namespace perm
