// ryser_cube_sdd_n24.cu -- column-cube walks (split-dd) of the shapes of 24 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n24(int i) {
  return cube_sdd_pick<cube_first<24>()>(i, std::make_index_sequence<cube_count<24>()>());
}
}  // namespace perm
