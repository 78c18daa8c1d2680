// ryser_cube_intc_n40.cu -- column-cube walks (certified int32 x) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_intc_n40(int i) { return cube_pick<5, 40>(i); }
}  // namespace perm
