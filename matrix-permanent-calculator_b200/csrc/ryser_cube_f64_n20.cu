// ryser_cube_f64_n20.cu -- column-cube walks (FP64 x) of the shapes of 20 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_f64_n20(int i) {
  return cube_f64_pick<cube_first<20>()>(i, std::make_index_sequence<cube_count<20>()>());
}
}  // namespace perm
