// ryser_cube_intc_n36.cu -- column-cube walks (certified int32 x) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_intc_n36(int i) { return cube_pick<5, 36>(i); }
}  // namespace perm
