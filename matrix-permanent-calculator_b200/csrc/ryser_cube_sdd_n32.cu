// ryser_cube_sdd_n32.cu -- column-cube walks (split-dd) of the shapes of 32 rows.
#include "cube_inst.cuh"

namespace perm {
const void* cube_sdd_n32(int i) {
  return cube_sdd_pick<cube_first<32>()>(i, std::make_index_sequence<cube_count<32>()>());
}
}  // namespace perm
