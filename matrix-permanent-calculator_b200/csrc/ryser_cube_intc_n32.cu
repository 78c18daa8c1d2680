// ryser_cube_intc_n32.cu -- column-cube walks (certified int32 x) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_intc_n32(int i) { return cube_pick<5, 32>(i); }
}  // namespace perm
