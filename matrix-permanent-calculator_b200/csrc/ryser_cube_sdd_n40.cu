// ryser_cube_sdd_n40.cu -- column-cube walks (split-dd) of the shapes of 40 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n40(int i) {
  return cube_sdd_pick<cube_first<40>()>(i, std::make_index_sequence<cube_count<40>()>());
}
}  // namespace perm
