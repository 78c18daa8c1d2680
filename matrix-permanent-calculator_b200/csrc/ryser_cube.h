// ryser_cube.h -- launch arguments of the column-cube walks (ryser_cube.cuh).
#pragma once
#include <cstddef>
#include <cstdint>

#include "cube_shapes.h"

namespace perm {

struct dd;

// Threads per CTA, one CTA per SM (ryser_cube.cuh).
constexpr int kCubeThreads = 256;
constexpr int kCubeWarps = kCubeThreads / 32;
// Words a block leaves in `partials`: its total, and its warps' sums of |term|.
constexpr int kCubeWords = 2 + kCubeWarps;
// Rows whose product the certified integer walk keeps in FP64 exactly.
constexpr int kCubeExactRows = 8;

struct CubeWalk {
  const void* img;  // columns 4..n-1 in slot order: FP64, split-dd coarse parts then remainders, or int32
  int n;
  int m;                     // log2 of the range alignment, in outer Gray indices
  uint64_t block0, nblocks;  // aligned blocks of 2^m outer indices of this launch
  uint64_t seg;              // cubes between two recomputations of b
  dd* partials;  // the blocks' totals, then kCubeWarps doubles a block: sum |term| (walks that sum it)
  unsigned* ticket;
  double* out;
  int* err;
  uint32_t inject;  // failure injection (tests): staging expects this many extra bytes
};

// The sums of the fast columns over their signs, with the last column of a
// row's set plus (2^|T| / 2 per row), in kernel order: of x, of split x, of
// y = 2x.
struct CubeArgs : CubeWalk {
  double c[kCubeMaxSums];  // halved
};
struct CubeSddArgs : CubeWalk {
  double c[kCubeMaxSums], cl[kCubeMaxSums];  // halved: of the coarse parts, of the remainders
};
struct CubeIntArgs : CubeWalk {
  int ci[kCubeMaxSums];
  double cd[kCubeMaxWide];  // of the rows left over from the int32 products
};

inline size_t cube_smem_bytes(int rows, size_t column_bytes, int n, bool remainders) {
  return (size_t)rows * (column_bytes * (size_t)(n - 4) + (remainders ? sizeof(double) * kCubeThreads : 0)) + 32 * 16 + 16;
}

}  // namespace perm
