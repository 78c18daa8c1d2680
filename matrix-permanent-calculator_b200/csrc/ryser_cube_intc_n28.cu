// ryser_cube_intc_n28.cu -- column-cube walks (certified int32 x) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_intc_n28(int i) { return cube_pick<5, 28>(i); }
}  // namespace perm
