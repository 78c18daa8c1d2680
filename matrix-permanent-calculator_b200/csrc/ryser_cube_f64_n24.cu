// ryser_cube_f64_n24.cu -- column-cube walks (FP64 x) of the shapes of 24 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n24(int i) {
  return cube_f64_pick<cube_first<24>()>(i, std::make_index_sequence<cube_count<24>()>());
}
}  // namespace perm
