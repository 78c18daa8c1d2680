// cube_shapes.h -- row shapes of the column-cube walk (ryser_cube.cuh): how
// many rows each class of rows has, as compile-time constants, so that a
// kernel keeps its rows in registers and its loops unroll.
//
// A row's class is the set of fast columns (of four, bits 0..3) where it is
// nonzero.  A row may also sit in the slot of any larger set (its extra
// entries there are zeros), and unused slots hold rows of the constant 1, so
// a few shapes per size serve every matrix whose four chosen columns fit.
// The shapes were picked greedily, then improved by moving single slots, over
// the class counts of random matrices of density 0.15..0.95 (half of them near
// 0.5): with 22 shapes per size the cheapest that fits needs 1.07 to 1.09 times
// the operations of a shape made for the matrix (one shape: 1.7 times).
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
constexpr int kCubeSizeCount = 4;
constexpr int kCubeSizes[kCubeSizeCount] = {28, 32, 36, 40};
constexpr int kCubeFirst[kCubeSizeCount + 1] = {0, 22, 44, 66, 88};
constexpr int kCubeShapeCount = 88;
constexpr CubeShape kCubeShapes[kCubeShapeCount] = {
    // up to 28 rows
    {{19, 2, 0, 2, 3, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 41 values, 113 operations
    {{16, 2, 0, 3, 3, 0, 0, 0, 4, 0, 0, 0, 0, 0, 0, 0}},  // 46 values, 126 operations
    {{12, 2, 0, 3, 5, 0, 0, 0, 5, 1, 0, 0, 0, 0, 0, 0}},  // 52 values, 142 operations
    {{11, 4, 4, 1, 3, 0, 1, 0, 2, 1, 0, 0, 1, 0, 0, 0}},  // 53 values, 159 operations
    {{9, 6, 3, 1, 2, 0, 2, 0, 3, 1, 1, 0, 0, 0, 0, 0}},  // 57 values, 173 operations
    {{6, 0, 5, 3, 4, 2, 1, 0, 3, 3, 0, 0, 1, 0, 0, 0}},  // 70 values, 200 operations
    {{5, 4, 2, 2, 2, 2, 3, 0, 2, 3, 0, 0, 2, 0, 1, 0}},  // 81 values, 225 operations
    {{6, 3, 3, 2, 0, 2, 3, 1, 1, 2, 2, 0, 3, 0, 0, 0}},  // 84 values, 232 operations
    {{5, 5, 1, 2, 3, 0, 3, 2, 2, 1, 0, 1, 2, 0, 1, 0}},  // 91 values, 241 operations
    {{4, 3, 2, 2, 3, 4, 1, 0, 1, 1, 3, 1, 2, 1, 0, 0}},  // 90 values, 248 operations
    {{4, 4, 2, 3, 3, 0, 2, 0, 1, 2, 1, 1, 3, 1, 1, 0}},  // 92 values, 248 operations
    {{2, 3, 2, 4, 0, 2, 2, 1, 2, 3, 2, 0, 4, 0, 1, 0}},  // 100 values, 268 operations
    {{3, 2, 2, 3, 2, 3, 1, 1, 2, 1, 2, 2, 2, 1, 1, 0}},  // 107 values, 283 operations
    {{0, 5, 1, 2, 2, 2, 4, 1, 0, 2, 4, 1, 2, 2, 0, 0}},  // 112 values, 293 operations
    {{2, 2, 4, 3, 0, 2, 2, 1, 2, 3, 1, 1, 1, 2, 2, 0}},  // 114 values, 296 operations
    {{2, 1, 0, 4, 0, 4, 2, 2, 1, 3, 3, 1, 2, 0, 3, 0}},  // 126 values, 318 operations
    {{2, 1, 2, 3, 1, 0, 3, 2, 1, 3, 0, 2, 2, 3, 3, 0}},  // 136 values, 334 operations
    {{1, 0, 0, 3, 0, 1, 2, 3, 1, 2, 3, 2, 2, 5, 3, 0}},  // 159 values, 383 operations
    {{1, 0, 0, 2, 0, 0, 3, 3, 1, 1, 1, 4, 2, 5, 2, 3}},  // 199 values, 459 operations
    {{0, 1, 0, 1, 0, 1, 0, 5, 1, 1, 0, 4, 0, 4, 5, 5}},  // 240 values, 535 operations
    {{1, 0, 0, 0, 0, 0, 2, 3, 1, 1, 0, 5, 0, 3, 3, 9}},  // 271 values, 591 operations
    {{0, 0, 0, 0, 0, 0, 1, 3, 0, 0, 0, 3, 0, 5, 2, 14}},  // 332 values, 707 operations
    // up to 32 rows
    {{23, 2, 0, 2, 3, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 45 values, 121 operations
    {{19, 3, 0, 2, 5, 0, 0, 0, 3, 0, 0, 0, 0, 0, 0, 0}},  // 49 values, 133 operations
    {{19, 3, 4, 0, 3, 0, 0, 0, 2, 1, 0, 0, 0, 0, 0, 0}},  // 47 values, 143 operations
    {{16, 3, 5, 1, 2, 0, 0, 0, 3, 1, 0, 0, 1, 0, 0, 0}},  // 54 values, 160 operations
    {{11, 5, 6, 1, 5, 0, 0, 0, 2, 1, 0, 0, 1, 0, 0, 0}},  // 59 values, 175 operations
    {{13, 4, 3, 1, 2, 0, 2, 0, 2, 2, 1, 0, 1, 1, 0, 0}},  // 71 values, 201 operations
    {{6, 4, 6, 3, 2, 2, 2, 0, 2, 1, 1, 0, 2, 1, 0, 0}},  // 86 values, 242 operations
    {{5, 3, 5, 3, 4, 1, 2, 0, 2, 3, 0, 0, 2, 1, 1, 0}},  // 93 values, 253 operations
    {{5, 4, 2, 3, 2, 2, 3, 0, 3, 2, 2, 1, 2, 1, 0, 0}},  // 99 values, 269 operations
    {{5, 3, 3, 3, 2, 2, 3, 1, 3, 1, 0, 2, 3, 0, 1, 0}},  // 107 values, 281 operations
    {{4, 4, 3, 2, 0, 3, 4, 1, 2, 3, 0, 1, 3, 1, 1, 0}},  // 114 values, 294 operations
    {{5, 2, 2, 3, 3, 2, 3, 0, 1, 3, 2, 1, 2, 1, 2, 0}},  // 113 values, 297 operations
    {{2, 3, 2, 3, 3, 3, 1, 2, 3, 2, 2, 1, 3, 1, 1, 0}},  // 120 values, 314 operations
    {{2, 3, 3, 3, 0, 3, 2, 2, 3, 3, 0, 1, 3, 1, 3, 0}},  // 132 values, 332 operations
    {{2, 3, 1, 2, 2, 2, 2, 2, 1, 4, 3, 3, 3, 0, 2, 0}},  // 136 values, 346 operations
    {{0, 2, 3, 3, 0, 3, 3, 2, 3, 2, 1, 3, 2, 3, 2, 0}},  // 152 values, 377 operations
    {{3, 0, 0, 3, 0, 3, 1, 4, 1, 2, 4, 2, 3, 3, 2, 1}},  // 173 values, 413 operations
    {{0, 0, 1, 4, 0, 2, 2, 6, 1, 4, 1, 2, 2, 2, 4, 1}},  // 192 values, 455 operations
    {{0, 1, 1, 2, 1, 4, 1, 4, 1, 2, 2, 4, 2, 1, 3, 3}},  // 204 values, 483 operations
    {{0, 0, 0, 0, 1, 1, 1, 5, 0, 2, 0, 5, 1, 4, 7, 5}},  // 270 values, 601 operations
    {{0, 0, 0, 3, 0, 1, 1, 3, 0, 0, 0, 4, 0, 6, 5, 9}},  // 308 values, 671 operations
    {{0, 0, 0, 0, 0, 0, 1, 5, 0, 0, 0, 4, 0, 4, 3, 15}},  // 372 values, 791 operations
    // up to 36 rows
    {{25, 2, 0, 2, 4, 0, 0, 0, 3, 0, 0, 0, 0, 0, 0, 0}},  // 51 values, 135 operations
    {{21, 5, 3, 0, 2, 0, 1, 0, 4, 0, 0, 0, 0, 0, 0, 0}},  // 53 values, 157 operations
    {{19, 4, 3, 1, 3, 0, 1, 0, 5, 0, 0, 0, 0, 0, 0, 0}},  // 57 values, 167 operations
    {{17, 4, 5, 1, 4, 0, 0, 0, 2, 2, 0, 0, 1, 0, 0, 0}},  // 63 values, 181 operations
    {{7, 7, 5, 1, 5, 0, 1, 0, 5, 2, 0, 0, 3, 0, 0, 0}},  // 79 values, 223 operations
    {{11, 4, 3, 3, 2, 0, 2, 1, 3, 2, 0, 0, 3, 1, 1, 0}},  // 99 values, 259 operations
    {{7, 5, 4, 2, 4, 0, 3, 1, 2, 3, 1, 0, 2, 1, 1, 0}},  // 105 values, 279 operations
    {{5, 2, 4, 4, 4, 3, 3, 0, 4, 2, 2, 0, 2, 1, 0, 0}},  // 105 values, 285 operations
    {{5, 4, 6, 2, 2, 2, 3, 1, 2, 3, 0, 1, 3, 1, 1, 0}},  // 117 values, 305 operations
    {{5, 3, 3, 4, 1, 4, 3, 0, 0, 3, 4, 1, 4, 1, 0, 0}},  // 123 values, 321 operations
    {{3, 2, 4, 4, 2, 2, 3, 2, 3, 3, 2, 0, 4, 1, 1, 0}},  // 129 values, 335 operations
    {{2, 0, 2, 6, 0, 4, 4, 1, 4, 4, 2, 1, 4, 1, 1, 0}},  // 142 values, 358 operations
    {{3, 3, 3, 3, 1, 4, 3, 2, 1, 3, 4, 0, 2, 2, 2, 0}},  // 143 values, 363 operations
    {{2, 2, 3, 6, 3, 2, 2, 2, 1, 3, 2, 1, 3, 3, 1, 0}},  // 148 values, 374 operations
    {{3, 2, 1, 4, 3, 4, 2, 2, 2, 3, 4, 0, 1, 1, 3, 1}},  // 155 values, 387 operations
    {{0, 1, 2, 2, 0, 1, 3, 7, 1, 5, 3, 2, 2, 4, 2, 1}},  // 208 values, 493 operations
    {{0, 0, 2, 2, 0, 4, 2, 5, 0, 5, 3, 3, 1, 3, 4, 2}},  // 224 values, 521 operations
    {{2, 1, 0, 3, 0, 2, 1, 5, 1, 3, 1, 4, 0, 5, 4, 4}},  // 254 values, 578 operations
    {{0, 0, 0, 1, 1, 0, 5, 5, 0, 1, 2, 4, 2, 6, 3, 6}},  // 286 values, 641 operations
    {{0, 0, 0, 2, 0, 2, 1, 5, 0, 2, 0, 5, 0, 3, 5, 11}},  // 348 values, 759 operations
    {{0, 0, 0, 2, 0, 0, 0, 5, 0, 1, 0, 3, 0, 4, 5, 16}},  // 404 values, 863 operations
    {{0, 0, 0, 0, 0, 1, 0, 4, 0, 0, 0, 5, 0, 3, 4, 19}},  // 436 values, 923 operations
    // up to 40 rows
    {{28, 4, 3, 0, 3, 0, 0, 0, 2, 0, 0, 0, 0, 0, 0, 0}},  // 52 values, 152 operations
    {{23, 4, 4, 1, 4, 0, 0, 0, 4, 0, 0, 0, 0, 0, 0, 0}},  // 59 values, 171 operations
    {{19, 6, 5, 0, 5, 0, 0, 0, 2, 1, 0, 0, 2, 0, 0, 0}},  // 67 values, 191 operations
    {{17, 7, 4, 1, 4, 0, 2, 0, 3, 0, 0, 0, 2, 0, 0, 0}},  // 73 values, 205 operations
    {{13, 6, 5, 3, 4, 0, 1, 0, 4, 1, 0, 0, 2, 1, 0, 0}},  // 87 values, 237 operations
    {{10, 6, 4, 3, 4, 1, 2, 1, 4, 1, 2, 0, 1, 1, 0, 0}},  // 102 values, 278 operations
    {{7, 5, 5, 3, 4, 2, 2, 0, 3, 2, 3, 1, 2, 1, 0, 0}},  // 113 values, 303 operations
    {{6, 4, 3, 2, 3, 4, 4, 1, 3, 4, 3, 0, 2, 0, 1, 0}},  // 124 values, 326 operations
    {{4, 4, 3, 2, 5, 4, 2, 1, 3, 3, 4, 1, 3, 0, 1, 0}},  // 130 values, 340 operations
    {{4, 2, 6, 3, 3, 4, 3, 2, 3, 3, 3, 1, 2, 1, 0, 0}},  // 136 values, 352 operations
    {{4, 3, 5, 3, 2, 3, 5, 1, 1, 5, 0, 2, 4, 1, 1, 0}},  // 146 values, 368 operations
    {{4, 3, 2, 3, 3, 2, 3, 2, 4, 4, 2, 3, 3, 1, 1, 0}},  // 152 values, 384 operations
    {{3, 4, 2, 3, 3, 2, 4, 2, 2, 1, 2, 4, 5, 1, 2, 0}},  // 165 values, 411 operations
    {{0, 5, 4, 4, 2, 3, 3, 2, 1, 2, 3, 3, 3, 3, 2, 0}},  // 176 values, 435 operations
    {{0, 2, 2, 3, 0, 5, 2, 4, 3, 3, 4, 3, 5, 1, 2, 1}},  // 198 values, 477 operations
    {{2, 2, 1, 4, 2, 4, 3, 3, 1, 2, 3, 4, 3, 2, 2, 2}},  // 210 values, 502 operations
    {{0, 1, 1, 3, 0, 3, 4, 4, 0, 3, 2, 6, 2, 5, 4, 2}},  // 256 values, 591 operations
    {{3, 0, 0, 2, 0, 2, 2, 5, 1, 2, 2, 5, 0, 5, 5, 6}},  // 301 values, 673 operations
    {{0, 0, 0, 1, 0, 0, 2, 9, 0, 0, 2, 6, 2, 6, 4, 8}},  // 356 values, 779 operations
    {{1, 0, 0, 0, 0, 0, 0, 5, 1, 4, 2, 5, 0, 5, 5, 12}},  // 379 values, 819 operations
    {{0, 0, 0, 3, 0, 1, 0, 5, 0, 0, 0, 4, 0, 4, 4, 19}},  // 456 values, 971 operations
    {{1, 0, 0, 0, 0, 0, 1, 3, 0, 1, 0, 5, 0, 4, 4, 21}},  // 473 values, 1007 operations
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
constexpr int kCubeMaxSums = 256;  // at least the fast-column sums of any shape
// Integer walks: rows of a class outside its int32 runs of 4 and 3 rows,
// their first FP64 sum (2^|T| / 2 per row), and the factors of a term (runs
// and left-over rows).
PERM_HD constexpr int cube_left(int rows) { return rows % 4 == 3 ? 0 : rows % 4; }
PERM_HD constexpr int cube_left_sum(const CubeShape& s, int i) {
  int n = 0;
  for (int t = 0; t < i; t++) n += cube_left(s.rows[cube_class(t)]) * ((1 << cube_bits(cube_class(t))) / 2);
  return n;
}
PERM_HD constexpr int cube_factors(const CubeShape& s) {
  int n = 0;
  for (int t = 0; t < 16; t++) n += (s.rows[t] + 1) / 4 + cube_left(s.rows[t]);
  return n;
}
constexpr int kCubeMaxWide = 84;  // 2 rows in each of the 16 classes: 2 x 80 / 2

}  // namespace perm
