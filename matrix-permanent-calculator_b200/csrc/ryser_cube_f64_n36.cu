// ryser_cube_f64_n36.cu -- column-cube walks (FP64 x) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n36(int i) {
  return cube_f64_pick<cube_first<36>()>(i, std::make_index_sequence<cube_count<36>()>());
}
}  // namespace perm
