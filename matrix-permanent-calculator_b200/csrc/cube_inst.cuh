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
template <int kFirst, size_t... kI>
const void* cube_f64_pick(int i, std::index_sequence<kI...>) {
  static const void* const table[] = {reinterpret_cast<const void*>(&ryser_cube_kernel<kFirst + (int)kI>)...};
  return table[i];
}
template <int kFirst, size_t... kI>
const void* cube_sdd_pick(int i, std::index_sequence<kI...>) {
  static const void* const table[] = {reinterpret_cast<const void*>(&ryser_cube_sdd_kernel<kFirst + (int)kI>)...};
  return table[i];
}

}  // namespace perm
