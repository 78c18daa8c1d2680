// ryser_cube_f64_n40.cu -- column-cube walks (FP64 x) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n40(int i) { return cube_pick<0, 40>(i); }
}  // namespace perm
