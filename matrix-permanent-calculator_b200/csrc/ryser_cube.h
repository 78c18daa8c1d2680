// ryser_cube.h -- launch arguments of the column-cube walks (ryser_cube.cuh).
#pragma once
#include <cstddef>
#include <cstdint>

#include "cube_shapes.h"

namespace perm {

struct dd;

constexpr int kCubeThreads = 256;  // per CTA, one CTA per SM (ryser_cube.cuh)

struct CubeArgs {
  const double* img;  // columns 4..n-1 in slot order (split-dd: coarse parts, then remainders)
  int n;
  int m;                     // log2 of the range alignment, in outer Gray indices
  uint64_t block0, nblocks;  // aligned blocks of 2^m outer indices of this launch
  uint64_t seg;              // cubes between two recomputations of b
  dd* partials;
  unsigned* ticket;
  double* out;
  double* sums;  // certified walks: sums[0] += sum |term| (zeroed by the host)
  int* err;
  uint32_t inject;  // failure injection (tests): staging expects this many extra bytes
  double c[kCubeMaxSums];   // sums of the fast columns over their signs, halved (plus last
                            // column: row of class T has 2^|T| / 2), kernel order
  double cl[kCubeMaxSums];  // split-dd: of their remainders
};

inline size_t cube_smem_bytes(bool pair, int n, int rows) {
  return sizeof(double) * (size_t)rows * ((pair ? 2 : 1) * (size_t)(n - 4) + (pair ? kCubeThreads : 0)) + 32 * 16 + 16;
}

}  // namespace perm
