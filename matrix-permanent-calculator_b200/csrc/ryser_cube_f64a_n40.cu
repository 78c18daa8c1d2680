// ryser_cube_f64a_n40.cu -- column-cube walks (FP64 x with sum |term|) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64a_n40(int i) { return cube_pick<1, 40>(i); }
}  // namespace perm
