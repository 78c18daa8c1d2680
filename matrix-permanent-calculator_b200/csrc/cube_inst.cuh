// cube_inst.cuh -- instances of the column-cube walks (ryser_cube.cuh) for
// the shapes of one size; each ryser_cube_*_n<size>.cu compiles one table.
#pragma once
#include <utility>

#include "ryser_cube.cuh"

namespace perm {

template <int kSize>
constexpr int cube_first() {
  for (int i = 0; i < kCubeSizeCount; i++)
    if (kCubeSizes[i] == kSize) return kCubeFirst[i];
  return -1;
}
template <int kSize>
constexpr int cube_count() {
  for (int i = 0; i < kCubeSizeCount; i++)
    if (kCubeSizes[i] == kSize) return kCubeFirst[i + 1] - kCubeFirst[i];
  return 0;
}
// table of one kind: 0 FP64, 1 FP64 with sum |term|, 2 split-dd, 3 int32, 4
// int32 with sum |term|, 5 certified int32
template <int kKind, int kShape>
const void* cube_instance() {
  if constexpr (kKind == 0) return reinterpret_cast<const void*>(&ryser_cube_kernel<kShape, false>);
  if constexpr (kKind == 1) return reinterpret_cast<const void*>(&ryser_cube_kernel<kShape, true>);
  if constexpr (kKind == 2) return reinterpret_cast<const void*>(&ryser_cube_sdd_kernel<kShape>);
  if constexpr (kKind == 3) return reinterpret_cast<const void*>(&ryser_cube_int_kernel<kShape, false, false>);
  if constexpr (kKind == 4) return reinterpret_cast<const void*>(&ryser_cube_int_kernel<kShape, false, true>);
  if constexpr (kKind == 5) return reinterpret_cast<const void*>(&ryser_cube_int_kernel<kShape, true, false>);
}
template <int kKind, int kFirst, size_t... kI>
const void* cube_table(int i, std::index_sequence<kI...>) {
  static const void* const table[] = {cube_instance<kKind, kFirst + (int)kI>()...};
  return table[i];
}
template <int kKind, int kSize>
const void* cube_pick(int i) {
  return cube_table<kKind, cube_first<kSize>()>(i, std::make_index_sequence<cube_count<kSize>()>());
}

}  // namespace perm
