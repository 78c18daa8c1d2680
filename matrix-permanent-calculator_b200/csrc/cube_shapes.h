// cube_shapes.h -- row shapes of the column-cube walk (ryser_cube.cuh): how
// many rows each class of rows has, as compile-time constants, so that a
// kernel keeps its rows in registers and its loops unroll.
//
// A row's class is the set of fast columns (of four, bits 0..3) where it is
// nonzero.  A row may also sit in the slot of any larger set (its extra
// entries there are zeros), and unused slots hold rows of the constant 1, so
// a few shapes per size serve every matrix whose four chosen columns fit.
// The shapes were picked greedily from the class counts of random matrices of
// density 0.15..0.95 (a third at 0.5): with 12 to 14 shapes per size the
// cheapest that fits needs 1.07 to 1.11 times the operations of a
// shape made for the matrix (one shape: 1.7 times, 6 shapes: 1.15).
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define PERM_HD __host__ __device__
#else
#define PERM_HD
#endif

namespace perm {

struct CubeShape {
  uint8_t rows[16];  // by class
};

// Shapes of kCubeSizes[i] rows are kCubeShapes[kCubeFirst[i] .. kCubeFirst[i + 1]),
// cheapest first; comments: row values and FP64 operations per 16 terms.
constexpr int kCubeSizeCount = 6;
constexpr int kCubeSizes[kCubeSizeCount] = {20, 24, 28, 32, 36, 40};
constexpr int kCubeFirst[kCubeSizeCount + 1] = {0, 12, 24, 38, 52, 66, 80};
constexpr int kCubeShapeCount = 80;
constexpr CubeShape kCubeShapes[kCubeShapeCount] = {
    // up to 20 rows
    {{13, 3, 0, 1, 0, 0, 0, 0, 2, 1, 0, 0, 0, 0, 0, 0}},  // 31 values, 90 operations
    {{13, 2, 0, 1, 2, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 29 values, 100 operations
    {{11, 2, 0, 1, 2, 0, 0, 0, 1, 1, 0, 0, 2, 0, 0, 0}},  // 37 values, 118 operations
    {{9, 2, 2, 0, 0, 2, 2, 0, 1, 2, 0, 0, 0, 0, 0, 0}},  // 43 values, 136 operations
    {{4, 3, 1, 1, 0, 2, 3, 0, 4, 1, 0, 1, 0, 0, 0, 0}},  // 56 values, 167 operations
    {{3, 1, 3, 1, 0, 3, 2, 0, 2, 2, 1, 1, 0, 0, 1, 0}},  // 67 values, 194 operations
    {{4, 1, 1, 1, 0, 3, 1, 2, 2, 2, 2, 0, 0, 0, 1, 0}},  // 72 values, 203 operations
    {{2, 1, 0, 2, 1, 3, 2, 1, 0, 2, 3, 1, 1, 0, 1, 0}},  // 82 values, 235 operations
    {{0, 2, 1, 2, 0, 3, 2, 1, 1, 3, 0, 2, 0, 1, 2, 0}},  // 96 values, 258 operations
    {{3, 1, 0, 2, 0, 0, 0, 3, 0, 1, 0, 1, 2, 2, 3, 2}},  // 129 values, 314 operations
    {{0, 1, 0, 1, 0, 0, 1, 4, 0, 0, 1, 2, 0, 5, 2, 3}},  // 166 values, 390 operations
    {{0, 0, 0, 0, 0, 0, 2, 2, 0, 1, 0, 2, 0, 3, 1, 9}},  // 220 values, 492 operations
    // up to 24 rows
    {{18, 1, 0, 1, 2, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 32 values, 105 operations
    {{12, 2, 4, 0, 0, 1, 1, 0, 3, 1, 0, 0, 0, 0, 0, 0}},  // 42 values, 135 operations
    {{6, 5, 4, 1, 0, 1, 3, 0, 3, 1, 0, 0, 0, 0, 0, 0}},  // 54 values, 165 operations
    {{5, 3, 1, 1, 0, 2, 3, 0, 3, 3, 1, 0, 0, 0, 2, 0}},  // 75 values, 212 operations
    {{3, 3, 3, 1, 0, 3, 2, 0, 4, 1, 1, 1, 0, 0, 2, 0}},  // 79 values, 222 operations
    {{3, 0, 2, 2, 0, 3, 1, 1, 3, 4, 4, 0, 0, 0, 1, 0}},  // 85 values, 234 operations
    {{2, 4, 2, 3, 0, 2, 3, 1, 2, 2, 0, 0, 2, 0, 1, 0}},  // 82 values, 237 operations
    {{2, 2, 2, 2, 1, 3, 3, 1, 2, 2, 0, 1, 1, 0, 2, 0}},  // 92 values, 259 operations
    {{1, 2, 0, 2, 2, 0, 0, 2, 0, 3, 1, 4, 2, 2, 3, 0}},  // 129 values, 326 operations
    {{0, 0, 0, 3, 1, 3, 0, 3, 0, 3, 1, 3, 1, 1, 3, 2}},  // 158 values, 386 operations
    {{0, 0, 0, 1, 0, 2, 0, 5, 0, 0, 1, 4, 0, 4, 3, 4}},  // 208 values, 476 operations
    {{1, 0, 0, 1, 0, 0, 0, 4, 0, 0, 0, 3, 0, 4, 2, 9}},  // 253 values, 560 operations
    // up to 28 rows
    {{18, 3, 3, 0, 2, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 38 values, 135 operations
    {{15, 3, 3, 1, 3, 0, 0, 0, 3, 0, 0, 0, 0, 0, 0, 0}},  // 43 values, 148 operations
    {{8, 4, 4, 2, 5, 0, 0, 0, 3, 1, 0, 0, 1, 0, 0, 0}},  // 56 values, 181 operations
    {{6, 4, 2, 4, 4, 0, 1, 0, 4, 1, 1, 0, 1, 0, 0, 0}},  // 66 values, 207 operations
    {{4, 4, 1, 1, 0, 4, 3, 1, 6, 2, 1, 0, 0, 0, 1, 0}},  // 86 values, 239 operations
    {{6, 4, 1, 3, 2, 0, 3, 1, 1, 2, 1, 0, 2, 1, 1, 0}},  // 90 values, 255 operations
    {{5, 2, 4, 3, 0, 3, 1, 1, 2, 1, 1, 0, 2, 2, 1, 0}},  // 97 values, 272 operations
    {{2, 5, 1, 2, 2, 0, 4, 1, 2, 3, 2, 1, 1, 1, 1, 0}},  // 102 values, 283 operations
    {{2, 3, 1, 1, 0, 3, 4, 3, 1, 4, 3, 0, 2, 0, 1, 0}},  // 112 values, 305 operations
    {{3, 2, 0, 2, 0, 2, 4, 2, 2, 1, 2, 3, 1, 2, 2, 0}},  // 131 values, 340 operations
    {{0, 0, 3, 3, 0, 4, 2, 1, 0, 3, 3, 1, 2, 3, 2, 1}},  // 146 values, 370 operations
    {{0, 1, 1, 2, 0, 1, 4, 3, 1, 4, 0, 3, 2, 2, 1, 3}},  // 178 values, 434 operations
    {{0, 0, 0, 1, 0, 2, 1, 4, 0, 1, 2, 4, 0, 5, 4, 4}},  // 228 values, 528 operations
    {{0, 0, 0, 0, 0, 0, 0, 5, 0, 0, 0, 4, 1, 3, 3, 12}},  // 316 values, 688 operations
    // up to 32 rows
    {{18, 5, 4, 0, 0, 0, 1, 0, 4, 0, 0, 0, 0, 0, 0, 0}},  // 48 values, 145 operations
    {{22, 2, 2, 0, 0, 2, 1, 0, 2, 1, 0, 0, 0, 0, 0, 0}},  // 50 values, 149 operations
    {{17, 4, 3, 1, 3, 0, 0, 0, 3, 0, 0, 0, 1, 0, 0, 0}},  // 51 values, 166 operations
    {{15, 2, 3, 2, 3, 1, 1, 0, 3, 1, 0, 0, 1, 0, 0, 0}},  // 61 values, 192 operations
    {{7, 6, 4, 2, 4, 0, 2, 0, 3, 2, 1, 0, 1, 0, 0, 0}},  // 73 values, 224 operations
    {{7, 3, 2, 1, 0, 4, 3, 2, 2, 3, 4, 0, 0, 0, 1, 0}},  // 105 values, 278 operations
    {{3, 2, 3, 3, 4, 4, 2, 1, 3, 3, 0, 1, 2, 0, 1, 0}},  // 107 values, 296 operations
    {{4, 3, 3, 4, 2, 2, 3, 0, 0, 3, 2, 0, 3, 2, 1, 0}},  // 112 values, 307 operations
    {{4, 1, 3, 5, 1, 2, 3, 1, 2, 2, 1, 1, 2, 3, 1, 0}},  // 126 values, 337 operations
    {{3, 1, 1, 4, 1, 1, 2, 2, 0, 2, 3, 1, 4, 3, 1, 3}},  // 177 values, 438 operations
    {{2, 1, 0, 4, 1, 1, 3, 4, 0, 1, 1, 3, 2, 4, 3, 2}},  // 198 values, 479 operations
    {{1, 1, 1, 3, 0, 2, 1, 2, 0, 1, 0, 5, 2, 2, 4, 7}},  // 257 values, 594 operations
    {{0, 1, 1, 2, 0, 3, 2, 3, 0, 1, 0, 4, 1, 3, 4, 7}},  // 264 values, 608 operations
    {{0, 0, 0, 1, 0, 0, 0, 5, 0, 0, 0, 5, 0, 4, 3, 14}},  // 364 values, 788 operations
    // up to 36 rows
    {{24, 3, 3, 1, 0, 0, 2, 0, 3, 0, 0, 0, 0, 0, 0, 0}},  // 54 values, 155 operations
    {{22, 3, 3, 1, 4, 0, 0, 0, 2, 1, 0, 0, 0, 0, 0, 0}},  // 54 values, 171 operations
    {{20, 3, 3, 1, 4, 0, 1, 0, 2, 2, 0, 0, 0, 0, 0, 0}},  // 60 values, 185 operations
    {{12, 6, 5, 1, 5, 0, 1, 0, 3, 1, 1, 0, 1, 0, 0, 0}},  // 70 values, 217 operations
    {{10, 4, 1, 3, 4, 2, 2, 0, 2, 1, 3, 1, 2, 0, 1, 0}},  // 100 values, 283 operations
    {{6, 3, 3, 5, 2, 3, 2, 1, 3, 1, 2, 0, 2, 2, 1, 0}},  // 120 values, 327 operations
    {{4, 2, 3, 3, 2, 3, 4, 2, 4, 4, 0, 1, 2, 1, 1, 0}},  // 130 values, 345 operations
    {{4, 2, 3, 5, 3, 2, 2, 2, 2, 4, 0, 2, 2, 1, 2, 0}},  // 140 values, 365 operations
    {{3, 3, 2, 5, 3, 2, 1, 2, 0, 2, 4, 1, 2, 3, 2, 1}},  // 163 values, 414 operations
    {{2, 2, 2, 3, 2, 3, 2, 3, 1, 1, 3, 3, 3, 3, 2, 1}},  // 180 values, 451 operations
    {{0, 1, 1, 2, 1, 4, 1, 5, 0, 3, 4, 3, 1, 4, 4, 2}},  // 226 values, 542 operations
    {{1, 1, 0, 1, 0, 0, 2, 6, 1, 3, 0, 5, 0, 5, 6, 5}},  // 285 values, 646 operations
    {{0, 0, 0, 1, 0, 1, 1, 6, 0, 1, 0, 6, 0, 4, 4, 12}},  // 368 values, 812 operations
    {{0, 0, 0, 0, 0, 1, 1, 4, 0, 0, 0, 5, 0, 3, 3, 19}},  // 432 values, 932 operations
    // up to 40 rows
    {{25, 4, 4, 0, 3, 0, 0, 0, 3, 1, 0, 0, 0, 0, 0, 0}},  // 57 values, 178 operations
    {{21, 5, 5, 0, 4, 0, 0, 0, 4, 1, 0, 0, 0, 0, 0, 0}},  // 61 values, 190 operations
    {{18, 5, 4, 1, 5, 0, 1, 0, 3, 2, 0, 0, 1, 0, 0, 0}},  // 72 values, 215 operations
    {{11, 6, 5, 2, 5, 2, 1, 0, 5, 1, 1, 0, 1, 0, 0, 0}},  // 85 values, 256 operations
    {{6, 6, 4, 2, 2, 5, 2, 1, 4, 1, 4, 0, 3, 0, 0, 0}},  // 114 values, 319 operations
    {{4, 4, 4, 3, 2, 5, 4, 1, 2, 4, 4, 0, 2, 0, 1, 0}},  // 132 values, 357 operations
    {{4, 2, 4, 5, 3, 3, 4, 1, 3, 3, 2, 1, 3, 2, 0, 0}},  // 140 values, 373 operations
    {{6, 4, 3, 3, 1, 3, 4, 1, 2, 3, 1, 2, 3, 1, 3, 0}},  // 150 values, 391 operations
    {{3, 4, 1, 2, 3, 4, 5, 1, 2, 2, 4, 4, 2, 2, 1, 0}},  // 163 values, 420 operations
    {{2, 1, 1, 3, 1, 4, 5, 4, 1, 5, 2, 3, 1, 3, 4, 0}},  // 202 values, 499 operations
    {{4, 1, 2, 3, 1, 4, 3, 3, 1, 3, 2, 3, 2, 3, 3, 2}},  // 210 values, 513 operations
    {{0, 2, 0, 3, 0, 4, 3, 3, 0, 1, 3, 6, 3, 3, 3, 6}},  // 288 values, 666 operations
    {{0, 2, 0, 1, 0, 1, 0, 8, 0, 1, 1, 5, 0, 5, 7, 9}},  // 364 values, 810 operations
    {{0, 0, 0, 1, 0, 0, 0, 6, 0, 0, 1, 4, 0, 5, 4, 19}},  // 464 values, 1000 operations
};

// Classes in the order the kernel multiplies them (ryser_cube.cuh).
PERM_HD constexpr int cube_class(int i) { return (int)((0xB98DC4EA62F75310ull >> (4 * i)) & 15); }
PERM_HD constexpr int cube_bits(int cls) { return (cls & 1) + ((cls >> 1) & 1) + ((cls >> 2) & 1) + ((cls >> 3) & 1); }
PERM_HD constexpr int cube_rows(const CubeShape& s) {
  int n = 0;
  for (int t = 0; t < 16; t++) n += s.rows[t];
  return n;
}
// first slot of the i-th class in kernel order
PERM_HD constexpr int cube_slot(const CubeShape& s, int i) {
  int n = 0;
  for (int t = 0; t < i; t++) n += s.rows[cube_class(t)];
  return n;
}
// first fast-column sum of that class: a row of class T has 2^|T| / 2
PERM_HD constexpr int cube_sum(const CubeShape& s, int i) {
  int n = 0;
  for (int t = 0; t < i; t++) n += s.rows[cube_class(t)] * ((1 << cube_bits(cube_class(t))) / 2);
  return n;
}
// row values per 16 terms
PERM_HD constexpr int cube_values(const CubeShape& s) {
  int n = 0;
  for (int t = 0; t < 16; t++) n += s.rows[t] << cube_bits(t);
  return n;
}
constexpr int kCubeMaxSums = 256;  // largest number of fast-column sums of a shape

}  // namespace perm
