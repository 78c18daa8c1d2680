// ryser_cube_sdd_n20.cu -- column-cube walks (split-dd) of the shapes of 20 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n20(int i) {
  return cube_sdd_pick<cube_first<20>()>(i, std::make_index_sequence<cube_count<20>()>());
}
}  // namespace perm
