// ryser_cube_sdd_n28.cu -- column-cube walks (split-dd) of the shapes of 28 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n28(int i) {
  return cube_sdd_pick<cube_first<28>()>(i, std::make_index_sequence<cube_count<28>()>());
}
}  // namespace perm
