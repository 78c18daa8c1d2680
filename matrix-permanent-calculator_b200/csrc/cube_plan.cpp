// cube_plan.cpp -- host-side layout of the column-cube walks (cube_plan.h).
#include "cube_plan.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <initializer_list>

namespace perm {

namespace {

struct Quad {
  int values = 0;  // sum over rows of 2^|T|
  bool transpose = false;
  uint8_t c[4];
};

// Up-sets of the 16 classes (every family that holds with a set all its
// supersets): rows fit a shape exactly when no up-set has more rows than
// slots (Hall's condition, since a row of class T may use any superset).
struct UpSets {
  static constexpr int kPad = 176;  // 167 non-empty ones, padded for whole-vector compares
  int count = 0;
  uint64_t lo[kPad], hi[kPad];                 // byte masks over classes 0..7 and 8..15
  uint8_t caps[kCubeShapeCount][kPad];
  uint8_t perm[24][16];   // class under each order of the columns
  uint8_t column[24][4];  // new place of each column
  UpSets() {
    memset(lo, 0, sizeof lo);
    memset(hi, 0, sizeof hi);
    memset(caps, 0, sizeof caps);
    for (int f = 1; f < (1 << 16); f++) {
      bool up = true;
      for (int t = 0; t < 16 && up; t++)
        if ((f >> t) & 1)
          for (int k = 0; k < 4; k++) up = up && ((f >> (t | (1 << k))) & 1);
      if (!up) continue;
      for (int t = 0; t < 8; t++) {
        if ((f >> t) & 1) lo[count] |= 0xffull << (8 * t);
        if ((f >> (t + 8)) & 1) hi[count] |= 0xffull << (8 * t);
      }
      count++;
    }
    for (int s = 0; s < kCubeShapeCount; s++) sums(kCubeShapes[s].rows, caps[s]);
    int p[4] = {0, 1, 2, 3}, i = 0;
    do {
      for (int t = 0; t < 16; t++) {
        int r = 0;
        for (int k = 0; k < 4; k++)
          if ((t >> k) & 1) r |= 1 << p[k];
        perm[i][t] = (uint8_t)r;
      }
      for (int k = 0; k < 4; k++) column[i][k] = (uint8_t)p[k];
      i++;
    } while (std::next_permutation(p, p + 4));
  }
  // rows in each up-set (at most 64: byte sums do not overflow)
  void sums(const uint8_t* rows, uint8_t* out) const {
    uint64_t a, b;
    memcpy(&a, rows, 8);
    memcpy(&b, rows + 8, 8);
    for (int u = 0; u < count; u++)
      out[u] = (uint8_t)((((a & lo[u]) + (b & hi[u])) * 0x0101010101010101ull) >> 56);
  }
};
const UpSets& up_sets() {
  static const UpSets u;
  return u;
}

// Every four of the `candidates` sparsest columns with their row values:
// sum_j 2^|T_j| = sum over subsets U of the four of the rows nonzero in all
// of U.  Keeps the `keep` cheapest.
void collect_quads(const std::vector<uint64_t>& sup, int n, int candidates, bool transpose, size_t keep, int max_values,
                   std::vector<Quad>* out) {
  std::vector<int> ord(n);
  for (int k = 0; k < n; k++) ord[k] = k;
  std::stable_sort(ord.begin(), ord.end(),
                   [&](int x, int y) { return __builtin_popcountll(sup[x]) < __builtin_popcountll(sup[y]); });
  const int K = std::min(n, candidates);
  int one[64], two[64][64];
  uint64_t s[64];
  for (int i = 0; i < K; i++) {
    s[i] = sup[ord[i]];
    one[i] = __builtin_popcountll(s[i]);
    for (int j = 0; j < i; j++) two[i][j] = __builtin_popcountll(s[i] & s[j]);
  }
  auto cheaper = [](const Quad& x, const Quad& y) { return x.values < y.values; };
  int limit = max_values;
  for (int i = 3; i < K; i++)
    for (int j = 2; j < i; j++) {
      const uint64_t ij = s[i] & s[j];
      const int vij = n + one[i] + one[j] + two[i][j];
      if (vij > limit) continue;
      for (int k = 1; k < j; k++) {
        const uint64_t ijk = ij & s[k], ik = s[i] & s[k], jk = s[j] & s[k];
        const int vijk = vij + one[k] + two[i][k] + two[j][k] + __builtin_popcountll(ijk);
        if (vijk > limit) continue;
        for (int l = 0; l < k; l++) {
          const int v = vijk + one[l] + two[i][l] + two[j][l] + two[k][l] + __builtin_popcountll(ij & s[l]) +
                        __builtin_popcountll(ik & s[l]) + __builtin_popcountll(jk & s[l]) +
                        __builtin_popcountll(ijk & s[l]);
          if (v > limit) continue;
          out->push_back({v, transpose, {(uint8_t)ord[i], (uint8_t)ord[j], (uint8_t)ord[k], (uint8_t)ord[l]}});
          if (out->size() >= 4 * keep) {
            std::nth_element(out->begin(), out->begin() + keep, out->end(), cheaper);
            out->resize(keep);
            limit = std::min(limit, std::max_element(out->begin(), out->end(), cheaper)->values);
          }
        }
      }
    }
}

// Scale of the terms of a walk of the matrix, or of its transpose: log2 of the
// products over its rows of their absolute sums and of their Euclidean norms.
struct TermScale {
  double sum = 0.0, norm = 0.0;
};
TermScale term_scale(const std::vector<double>& a, int n, bool transpose) {
  TermScale t;
  for (int i = 0; i < n; i++) {
    const double* row = a.data() + (transpose ? i : (size_t)i * n);
    const size_t step = transpose ? n : 1;
    double sum = 0.0, squares = 0.0;
    for (int k = 0; k < n; k++) sum += std::fabs(row[k * step]);
    for (int k = 0; k < n; k++) {
      const double v = row[k * step] / sum;
      squares += v * v;
    }
    const double l = std::log2(sum);
    t.sum += l;
    t.norm += l + 0.5 * std::log2(squares);
  }
  return t;
}

// Rows of very different sizes: sorted into the classes of a cube their products
// could leave the range of FP64, which in the caller's order they may not.  So
// where the absolute sums above 1 multiply to more than 2^900 or those below 1
// to less than 2^-700 (low parts of double-double products are 2^-106 of the
// high ones, and cancelling rows smaller than their sums), every row is divided
// by the power of two of its sum; *exp2 is the exponent the permanent lost.
// False for rows this cannot be done to exactly (not finite, or with entries
// that would become subnormal).
bool bring_into_range(std::vector<double>* mat, int n, int* exp2) {
  *exp2 = 0;
  int up = 0, down = 0;
  std::vector<int> e(n, 0);
  for (int i = 0; i < n; i++) {
    double sum = 0.0;
    for (int k = 0; k < n; k++) sum += std::fabs((*mat)[(size_t)i * n + k]);
    if (!std::isfinite(sum)) return false;
    if (sum == 0.0) continue;
    e[i] = std::ilogb(sum);
    up += std::max(e[i] + 1, 0);
    down += std::min(e[i], 0);
  }
  if (up <= 900 && down >= -700) return true;
  for (int i = 0; i < n; i++) {
    for (int k = 0; k < n; k++) {
      double& v = (*mat)[(size_t)i * n + k];
      if (v != 0.0 && std::ilogb(v) - e[i] < -1000) return false;
      v = std::ldexp(v, -e[i]);
    }
    *exp2 += e[i];
  }
  return true;
}

}  // namespace

// Three bits are allowed, in which 98% (order 36, density 0.2, values (0,1]) to
// 100% (order 30, 0/1) of matrices whose rows and columns have no sizes of their
// own pass (one bit: 75%, and the others' walks took up to 1.2 times as long).
// Of 30000 matrices of order 13 with rows, columns or blocks scaled by up to
// 10^4, the transposes that passed had sums of |term| at most 46 times the
// matrix's, 8 times in 98 of 100, which double-double sums have to spare.
WalkSide walk_side(const std::vector<double>& a, int n) {
  const TermScale own = term_scale(a, n, false), other = term_scale(a, n, true);
  if (!(other.sum <= own.sum + 3.0 && other.norm <= own.norm + 3.0)) return WalkSide::kMatrix;
  return other.sum < own.sum - 8.0 && other.norm < own.norm - 8.0 ? WalkSide::kTranspose : WalkSide::kEither;
}

double cube_shape_ops(int shape) {
  const CubeShape& s = kCubeShapes[shape];
  auto w = [&](int i) { return 1 << cube_bits(cube_class(i)); };
  auto k = [&](int i) { return (int)s.rows[cube_class(i)]; };
  double ops = cube_rows(s);  // updates of b
  for (int i = 0; i < 16; i++) ops += k(i) * (i ? 2 * w(i) : 1);
  // class arrays: the first row of a chain only sets it; {02} and {13} are
  // merged into 8 values, the second chain into 16
  auto chain = [&](std::initializer_list<int> order, int extra) {
    bool unset = true;
    for (int i : order) {
      if (!k(i)) continue;
      if (i == extra)
        ops += unset ? -w(i) : 8 - w(i);
      else if (unset)
        ops -= w(i);
      unset = false;
    }
    return !unset;
  };
  chain({1, 2, 3, 4, 5}, 3);
  if (chain({6, 7, 8, 9}, 8)) ops += 16;
  if (chain({10, 11, 12}, -1)) ops += 8;  // fused with the differences
  chain({0, 13, 14, 15}, -1);
  return ops + 8 + 8 + 3;  // differences over column 2, products with the last chain, sum
}

double cube_shape_cost(int shape) {
  return cube_shape_ops(shape) * (1.0 + std::max(0, cube_values(kCubeShapes[shape]) - 130) / 600.0);
}

bool cube_layout(const std::vector<double>& a, int n, double max_cost, bool transpose, CubeLayout* layout) {
  layout->shape = -1;
  if (n < 9 || n > kCubeSizes[kCubeSizeCount - 1]) return false;
  int size = 0;
  while (kCubeSizes[size] < n) size++;
  // Where at most one slot would stay unused, shapes of the next size are
  // cheaper for some matrices (by 10% on average at order 32, density 0.7);
  // below order 31 the 20 us of trying them cost more.
  const bool next = n >= 31 && kCubeSizes[size] - n <= 1;
  const int first = kCubeFirst[size], last = kCubeFirst[std::min(size + 1 + next, kCubeSizeCount)];
  static const struct Costs {
    double v[kCubeShapeCount];
    int values[kCubeShapeCount], at_least[kCubeShapeCount][5] = {};
    uint8_t both[kCubeShapeCount][16] = {};    // slots of the classes with columns k and l
    uint8_t fullest[kCubeShapeCount][4] = {};  // of those with column k, ascending
    Costs() {
      for (int s = 0; s < kCubeShapeCount; s++) {
        v[s] = cube_shape_cost(s);
        values[s] = cube_values(kCubeShapes[s]);
        for (int t = 0; t < 16; t++)
          for (int b = cube_bits(t); b >= 0; b--) at_least[s][b] += kCubeShapes[s].rows[t];
        for (int kl = 0; kl < 16; kl++)
          for (int t = 0; t < 16; t++)
            if (((t >> (kl / 4)) & 1) && ((t >> (kl % 4)) & 1)) both[s][kl] += kCubeShapes[s].rows[t];
        for (int k = 0; k < 4; k++) fullest[s][k] = both[s][5 * k];
        std::sort(fullest[s], fullest[s] + 4);
      }
    }
  } costs;
  int max_values = 0;
  for (int s = first; s < last; s++)
    if (costs.v[s] <= max_cost) max_values = std::max(max_values, cube_values(kCubeShapes[s]));
  if (!max_values) return false;

  std::vector<uint64_t> cols(n, 0), rows(n, 0);
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++)
      if (a[(size_t)j * n + k] != 0.0) {
        cols[k] |= 1ull << j;
        rows[j] |= 1ull << k;
      }
  // a wider search pays for longer walks: 70 sets of columns (some 20 us; the
  // transpose's as many again) come within 4% of the operations of 4845 (130 us)
  const int candidates = n < 28 ? 8 : n < 32 ? 10 : n < 34 ? 14 : 20;
  const size_t keep = n < 28 ? 6 : n < 32 ? 8 : n < 34 ? 16 : 32;
  std::vector<Quad> quads;
  quads.reserve(4 * keep);
  collect_quads(cols, n, candidates, false, keep, max_values, &quads);
  if (transpose) collect_quads(rows, n, candidates, true, keep, max_values, &quads);
  std::sort(quads.begin(), quads.end(), [](const Quad& x, const Quad& y) { return x.values < y.values; });
  if (quads.size() > keep) quads.resize(keep);

  const UpSets& U = up_sets();
  Quad best_quad;
  int best_perm = 0;
  double best = max_cost;
  for (const Quad& q : quads) {
    const std::vector<uint64_t>& sup = q.transpose ? rows : cols;
    uint8_t count[16] = {};
    int at_least[5] = {};  // rows nonzero in at least t of the four
    for (int j = 0; j < n; j++) {
      int t = 0;
      for (int k = 0; k < 4; k++) t |= (int)((sup[q.c[k]] >> j) & 1) << k;
      count[t]++;
      for (int b = cube_bits(t); b >= 0; b--) at_least[b]++;
    }
    // rows nonzero in column k, and in columns k and l
    uint8_t need[16], fullest[4];
    for (int k = 0; k < 4; k++)
      for (int l = 0; l < 4; l++) need[4 * k + l] = (uint8_t)__builtin_popcountll(sup[q.c[k]] & sup[q.c[l]]);
    for (int k = 0; k < 4; k++) fullest[k] = need[5 * k];
    std::sort(fullest, fullest + 4);
    // shapes that could beat the best and have room in every layer of the
    // lattice and for every column; only those are tried under the 24 orders
    int tryable[kCubeShapeCount], tries = 0;
    for (int s = first; s < last; s++) {
      if (costs.v[s] > best || (layout->shape >= 0 && costs.v[s] >= best) || costs.values[s] < q.values) continue;
      bool room = true;
      for (int t = 1; t <= 4; t++) room = room && at_least[t] <= costs.at_least[s][t];
      for (int k = 0; k < 4; k++) room = room && fullest[k] <= costs.fullest[s][k];
      if (room) tryable[tries++] = s;
    }
    for (int p = 0; p < 24 && tries; p++) {
      uint8_t have[16], sum[UpSets::kPad];
      bool summed = false;
      for (int i = 0; i < tries; i++) {
        const int s = tryable[i];
        // the columns' and pairs' own counts first: most orders fail here
        bool fits = true;
        for (int k = 0; k < 4 && fits; k++)
          for (int l = 0; l <= k; l++)
            if (need[4 * k + l] > costs.both[s][4 * U.column[p][k] + U.column[p][l]]) {
              fits = false;
              break;
            }
        if (!fits) continue;
        if (!summed) {
          for (int t = 0; t < 16; t++) have[U.perm[p][t]] = count[t];
          memset(sum, 0, sizeof sum);
          U.sums(have, sum);
          summed = true;
        }
        uint8_t over = 0;
        for (int u = 0; u < UpSets::kPad; u++) over |= (uint8_t)(sum[u] > U.caps[s][u]);
        if (over) continue;
        best = costs.v[s];
        layout->shape = s;
        best_quad = q;
        best_perm = p;
        tries = 0;
        for (int x = 0; x < i; x++)
          if (costs.v[tryable[x]] < best) tryable[tries++] = tryable[x];
        break;
      }
    }
  }
  if (layout->shape < 0) return false;
  layout->cost = best;

  // Rows to slots: a row of class T into any class containing T (augmenting
  // paths; the shape fits, so every row finds a place).
  const std::vector<uint64_t>& sup = best_quad.transpose ? rows : cols;
  const CubeShape& shape = kCubeShapes[layout->shape];
  uint8_t fast[4];  // column of `a` (or row, transposed) behind each fast column
  for (int k = 0; k < 4; k++) {
    int to = 0;
    while (U.perm[best_perm][1 << k] != (1 << to)) to++;
    fast[to] = best_quad.c[k];
  }
  std::vector<int> cls(n), place(n, -1);
  for (int j = 0; j < n; j++) {
    cls[j] = 0;
    for (int k = 0; k < 4; k++) cls[j] |= (int)((sup[fast[k]] >> j) & 1) << k;
  }
  std::vector<std::vector<int>> in(16);
  for (int j = 0; j < n; j++) {
    bool seen[16] = {};
    struct Augment {
      std::vector<std::vector<int>>& in;
      std::vector<int>&cls, &place;
      const CubeShape& shape;
      bool* seen;
      bool go(int row) {
        for (int bits = 0; bits <= 4; bits++)
          for (int t = 0; t < 16; t++) {
            if (cube_bits(t) != bits || (t & cls[row]) != cls[row] || seen[t] || !shape.rows[t]) continue;
            seen[t] = true;
            if ((int)in[t].size() < shape.rows[t]) {
              in[t].push_back(row);
              place[row] = t;
              return true;
            }
            for (size_t i = 0; i < in[t].size(); i++) {
              const int other = in[t][i];
              if (go(other)) {
                in[t][i] = row;
                place[row] = t;
                return true;
              }
            }
          }
        return false;
      }
    } augment{in, cls, place, shape, seen};
    if (!augment.go(j)) {
      layout->shape = -1;
      return false;
    }
  }
  auto at = [&](int j, int k) { return best_quad.transpose ? a[(size_t)k * n + j] : a[(size_t)j * n + k]; };
  std::vector<int> col_order(fast, fast + 4), row_order;
  for (int k = 0; k < n; k++)
    if (std::find(fast, fast + 4, (uint8_t)k) == fast + 4) col_order.push_back(k);
  layout->slot_row.assign(cube_rows(shape), -1);
  for (int i = 0; i < 16; i++) {
    const int t = cube_class(i), slot = cube_slot(shape, i);
    for (size_t r = 0; r < in[t].size(); r++) {
      layout->slot_row[slot + r] = (int)row_order.size();
      row_order.push_back(in[t][r]);
    }
  }
  layout->mat.resize((size_t)n * n);
  for (int i = 0; i < n; i++)
    for (int k = 0; k < n; k++) layout->mat[(size_t)i * n + k] = at(row_order[i], col_order[k]);
  if (bring_into_range(&layout->mat, n, &layout->exp2)) return true;
  layout->shape = -1;
  return false;
}

}  // namespace perm
