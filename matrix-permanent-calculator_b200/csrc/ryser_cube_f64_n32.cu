// ryser_cube_f64_n32.cu -- column-cube walks (FP64 x) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n32(int i) {
  return cube_f64_pick<cube_first<32>()>(i, std::make_index_sequence<cube_count<32>()>());
}
}  // namespace perm
