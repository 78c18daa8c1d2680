// cube_plan.h -- host-side layout of the column-cube walks (ryser_cube.cuh):
// which four columns are summed at once, which compiled shape holds the row
// classes they make, and which row sits in which slot.  Host only.
#pragma once
#include <vector>

#include "cube_shapes.h"

namespace perm {

struct CubeLayout {
  int shape = -1;             // index into kCubeShapes, -1: none fits or none is cheap enough
  double cost = 0;            // cube_shape_cost of the shape
  std::vector<double> mat;    // row-major n x n: the fast columns first, rows in slot order
                              // (the matrix or its transpose; same permanent)
  int exp2 = 0;               // the permanent is mat's times 2^exp2 (rows of extreme sizes are scaled)
  std::vector<int> slot_row;  // row of `mat` in each slot, -1: a row of the constant 1
};

// Which of a matrix and its transpose (same permanent, other terms) a walk may
// take.  Every error is a fraction of the terms' absolute sum.  The size of a
// row is a factor of every term and costs nothing, but columns of different
// sizes make that sum larger without limit, so the transpose of a matrix whose
// rows differ in size must not be walked, and that of a matrix whose columns do
// (by 8 bits in all, in sums and in norms) is the one to walk.
enum class WalkSide { kMatrix, kEither, kTranspose };
WalkSide walk_side(const std::vector<double>& a, int n);

// The cheapest compiled shape, of at most max_cost, that holds the rows of some
// four columns of the n x n row-major matrix or, with `transpose`, of its
// transpose; false when there is none (orders outside 9..40 and matrices with
// infinities or NaNs among them).  The transpose saves another 3..6% of the
// operations; even where walk_side allows either, its terms' absolute sum may be
// a few times larger, so it is only for double-double walks.
bool cube_layout(const std::vector<double>& a, int n, double max_cost, bool transpose, CubeLayout* layout);

// FP64 operations per 16 terms of a shape's FP64 walk, and the same weighted
// by the rate its size reaches, as operations at a rate of 0.82: fitted to
// 0.80..0.85 up to 130 row values, 0.73 at 198, 0.65 at 257, 0.62 at 364, all of
// the FP64 peak that dependent chains of FMAs measure (0.92 of the pipe's).
double cube_shape_ops(int shape);
double cube_shape_cost(int shape);

}  // namespace perm
