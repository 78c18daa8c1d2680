// ryser_cube_sdd_n36.cu -- column-cube walks (split-dd) of the shapes of 36 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n36(int i) {
  return cube_sdd_pick<cube_first<36>()>(i, std::make_index_sequence<cube_count<36>()>());
}
}  // namespace perm
