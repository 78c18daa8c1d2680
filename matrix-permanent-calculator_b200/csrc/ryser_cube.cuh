// ryser_cube.cuh -- dense exact permanents with four columns summed at once:
// the "column cube" walk.
//
// Ryser's sum over the signs s of columns 0..n-2, x_j = (a_j,n-1 + sum_k s_k
// a_jk) / 2 (the reference walks them one sign at a time in Gray order,
// kernel_xshared_coalescing_mshared, gpu_exact_dense.cu:330-399).  Here all
// 16 sign choices of four "fast" columns are evaluated together, and only the
// other n - 5 columns are walked in Gray order: b_j = (a_j,n-1 + sum over the
// walked columns) / 2 is updated once per 16 terms.
//
// What makes it cheap is that zeros in the fast columns split the rows into
// 16 classes: a row whose nonzeros among them are the set T takes only
// 2^|T| values b + c over the 16 sign choices (c: the fast columns' sums, the
// same for every thread), so it costs 2^|T| additions and multiplies instead
// of 16.  The products of a class are an array over the signs of T, which is
// copied (widened) into the array of a larger class or multiplied into it:
//
//   {} > {0} > {01} (x {02}) > {012} > {0123} = top
//   {1} > {12} (x {13}) > {123}, {2} > {23} > {023}      multiplied into top
//   {3} > {03} > {013}: top is summed over s_2 first, then multiplied
//
// The host picks the four columns, of the matrix or of its transpose, whose
// rows fit the cheapest of the compiled shapes (cube_shapes.h).  At density
// 1/2 that leaves about 0.2 x 16 n row values per 16 terms: for an order-32
// matrix 284 FP64 operations instead of 1024 for the plain walk, and 640 for
// the three-level row layout this replaced (n = 32, density 1/2: 6.38 ms
// then, 2.3..2.7 ms by shape now).
//
// Bound: the FP64 pipe, 80..85% of it on order-32 shapes up to 130 row values
// (the rest are fixed latencies between dependent products: 2.4 warps' worth
// of independent work per scheduler), falling to 62% at 360 values.  The sums
// c are kernel parameters, read as constant operands of the additions: from
// shared memory they would take more cycles than the arithmetic (a 64-bit
// broadcast load takes two, an addition and a multiply one; 3.5..3.9 ms at
// n = 32).  One CTA of 256 threads per SM (up to 255 registers) hides more
// latency by independent products than more threads do with fewer registers
// (n = 30, 105 row values: 0.59 ms; 2 CTAs of 128: 0.64; 12 warps of 168
// registers: 0.70).
#pragma once
#include <type_traits>

#include "cube_shapes.h"
#include "ryser_cube.h"
#include "ryser_dense_sdd.cuh"

namespace perm {

// Index of entry s of an array over the signs of a set within an array over
// a smaller set (all sets list their columns in ascending order).
__device__ constexpr int cube_drop(int s, int set, int sub) {
  int r = 0, o = 0;
  for (int k = 0, b = 0; k < 4; k++) {
    if (!((set >> k) & 1)) continue;
    if ((sub >> k) & 1) r |= ((s >> b) & 1) << o++;
    b++;
  }
  return r;
}

// Product arrays and row values of a walk: FP64, or split x with
// double-double products (pair).
template <bool kPair>
struct CubeNum;
template <>
struct CubeNum<false> {
  double hi;
  __device__ __forceinline__ void mul(const CubeNum& x) { hi = hi * x.hi; }
};
template <>
struct CubeNum<true> {
  double hi, lo;
  __device__ __forceinline__ void mul(const CubeNum& x) {
    dd t = {hi, lo};
    pair_mul(t, x.hi, x.lo);
    hi = t.hi;
    lo = t.lo;
  }
};

template <int kSet, bool kPair>
struct CubeArray {
  static constexpr int kW = 1 << cube_bits(kSet);
  CubeNum<kPair> v[kW];
};

// to = from widened to a larger set, or multiplied into it
template <int kTo, int kFrom, bool kPair>
__device__ __forceinline__ void cube_widen(CubeArray<kTo, kPair>& to, const CubeArray<kFrom, kPair>& from) {
#pragma unroll
  for (int s = 0; s < CubeArray<kTo, kPair>::kW; s++) to.v[s] = from.v[cube_drop(s, kTo, kFrom)];
}
template <int kTo, int kFrom, bool kPair>
__device__ __forceinline__ void cube_merge(CubeArray<kTo, kPair>& to, const CubeArray<kFrom, kPair>& from) {
#pragma unroll
  for (int s = 0; s < CubeArray<kTo, kPair>::kW; s++) to.v[s].mul(from.v[cube_drop(s, kTo, kFrom)]);
}

// The products of one cube, and their signed sum.  `row(slot)` returns a
// row's b; `kShape` gives the class sizes.
template <int kShape, bool kPair, class Row>
struct Cube {
  using Num = CubeNum<kPair>;
  const CubeArgs& a;
  Row row;

  template <int kI>
  static constexpr int count() {
    return kCubeShapes[kShape].rows[cube_class(kI)];
  }

  // multiplies the rows of class kI into p (which is unset when kFirst)
  template <int kI, bool kFirst>
  __device__ __forceinline__ void rows(CubeArray<cube_class(kI), kPair>& p) const {
    constexpr int W = CubeArray<cube_class(kI), kPair>::kW, H = W / 2;
    constexpr int kSlot = cube_slot(kCubeShapes[kShape], kI), kSum = cube_sum(kCubeShapes[kShape], kI);
#pragma unroll
    for (int r = 0; r < count<kI>(); r++) {
      const Num b = row(kSlot + r);
#pragma unroll
      for (int s = 0; s < W; s++) {
        Num x = b;
        if constexpr (W > 1) {
          // the sums with the last column's sign plus; minus is their mirror image
          const int q = kSum + r * H + (s >= H ? s - H : H - 1 - s);
          x.hi = s >= H ? __dadd_rn(b.hi, a.c[q]) : __dsub_rn(b.hi, a.c[q]);
          if constexpr (kPair) x.lo = s >= H ? __dadd_rn(b.lo, a.cl[q]) : __dsub_rn(b.lo, a.cl[q]);
        }
        if (kFirst && r == 0)
          p.v[s] = x;
        else
          p.v[s].mul(x);
      }
    }
  }

  // {k} > {kl} (x extra) > {klm}: classes kI, kI + 1, (kX), kL of the kernel
  // order; true when it has any rows
  template <int kI0, int kI1, int kX, int kI2>
  static constexpr bool any() {
    return count<kI0>() + count<kI1>() + (kX >= 0 ? count<(kX >= 0 ? kX : 0)>() : 0) + count<kI2>() > 0;
  }
  template <int kI0, int kI1, int kX, int kI2, int kFrom, bool kUnset>
  __device__ __forceinline__ void chain(CubeArray<cube_class(kI2), kPair>& p3,
                                        const CubeArray<kFrom, kPair>& from) const {
    constexpr int A = cube_class(kI0), B = cube_class(kI1), C = cube_class(kI2);
    constexpr bool f1 = kUnset && count<kI0>() == 0, f2 = f1 && count<kI1>() == 0;
    CubeArray<A, kPair> p1;
    if constexpr (!kUnset) cube_widen(p1, from);
    rows<kI0, kUnset>(p1);
    CubeArray<B, kPair> p2;
    if constexpr (!f1) cube_widen(p2, p1);
    rows<kI1, f1>(p2);
    if constexpr (!f2) cube_widen(p3, p2);
    if constexpr (kX >= 0) {
      constexpr int kXi = kX >= 0 ? kX : 0;
      if constexpr (count<kXi>() > 0) {
        CubeArray<cube_class(kXi), kPair> x;
        rows<kXi, true>(x);
        if constexpr (f2)
          cube_widen(p3, x);
        else
          cube_merge(p3, x);
        rows<kI2, false>(p3);
        return;
      }
    }
    rows<kI2, f2>(p3);
  }

  // top[16] and the last chain's array over {0, 1, 3}
  __device__ __forceinline__ void products(CubeArray<15, kPair>& top, CubeArray<11, kPair>& last) const {
    static_assert(count<13>() + count<14>() + count<15>() > 0 && count<0>() + count<1>() + count<2>() + count<4>() > 0,
                  "shapes have rows in the first and the last chain");
    {
      CubeArray<0, kPair> p0;
      rows<0, true>(p0);
      CubeArray<7, kPair> p3;
      chain<1, 2, 3, 4, 0, count<0>() == 0>(p3, p0);
      cube_widen(top, p3);
      rows<5, false>(top);
    }
    const CubeArray<0, kPair> none = {};
    if constexpr (any<6, 7, 8, 9>()) {
      CubeArray<14, kPair> p3;
      chain<6, 7, 8, 9, 0, true>(p3, none);
      cube_merge(top, p3);
    }
    if constexpr (any<10, 11, -1, 12>()) {
      CubeArray<13, kPair> p3;
      chain<10, 11, -1, 12, 0, true>(p3, none);
      cube_merge(top, p3);
    }
    chain<13, 14, -1, 15, 0, true>(last, none);
  }
};

// Adds the 16 signed terms last x top to (H, L) (Sum2, over column 2's sign
// first) and their absolute values to m1.
__device__ __forceinline__ void cube_sum_dd(const CubeArray<15, true>& top, const CubeArray<11, true>& last, bool odd,
                                            double& H, double& L, double& m1) {
  double gs = 0.0, gc = 0.0;
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const int lo = (s & 3) | ((s & 4) << 1);  // sign of column 2 minus
    const CubeNum<true>&t0 = top.v[lo], &t1 = top.v[lo | 4];
    dd d = two_sum(t0.hi, -t1.hi);
    d.lo = __dadd_rn(d.lo, __dsub_rn(t0.lo, t1.lo));
    m1 = __fma_rn(fabs(last.v[s].hi), __dadd_rn(fabs(t0.hi), fabs(t1.hi)), m1);
    pair_mul(d, last.v[s].hi, last.v[s].lo);
    if (__popc(s) & 1) d = {-d.hi, -d.lo};
    if (s == 0)
      gs = d.hi, gc = d.lo;
    else
      sum2_add(gs, gc, d.hi, d.lo);
  }
  sum2_add(H, L, odd ? -gs : gs, odd ? -gc : gc);
}

// Range of outer Gray indices of this thread, and the loop over it:
// start(h) sets b for outer index h, flip(h) moves it from h - 1 to h,
// cube(h) adds the 16 terms of h.
template <class Start, class Flip, class Eval>
__device__ __forceinline__ void cube_walk(const CubeArgs& a, Start start, Flip flip, Eval cube) {
  const uint64_t TT = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t q = a.nblocks / TT, r = a.nblocks % TT;
  const uint64_t b0 = q * tid + (r * tid) / TT, b1 = q * (tid + 1) + (r * (tid + 1)) / TT;
  const uint64_t e = (a.block0 + b1) << a.m;
  // b is recomputed from the matrix every `seg` cubes, so that the roundings
  // of its updates do not add up over the whole range
  for (uint64_t h = (a.block0 + b0) << a.m; h < e;) {
    const uint64_t stop = e - h > a.seg ? h + a.seg : e;
    start(h);
#pragma unroll 1
    for (;;) {
      cube(h);
      if (++h == stop) break;
      flip(h);
    }
  }
}

// FP64 walk.
template <int kShape>
__global__ void __launch_bounds__(kCubeThreads, 1) ryser_cube_kernel(const __grid_constant__ CubeArgs a) {
  constexpr int N = cube_rows(kCubeShapes[kShape]);
  static_assert(N % 2 == 0, "columns are read two rows at a time");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nc = a.n - 4;  // columns 4..n-1, the last one never flips
  double* sC = reinterpret_cast<double*>(smem_raw);
  dd* red = reinterpret_cast<dd*>(sC + (size_t)nc * N);
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 32);
  const bool staged = stage_to_smem(sC, a.img, (uint32_t)(sizeof(double) * nc * N), bar, a.err, a.inject);
  Acc acc;
  if (staged) {
    double b[N];
    auto add = [&](const double* c, double s) {
#pragma unroll
      for (int j = 0; j < N; j += 2) {
        const double2 v = lds2(c + j);
        b[j] = __fma_rn(s, v.x, b[j]);
        b[j + 1] = __fma_rn(s, v.y, b[j + 1]);
      }
    };
    auto row = [&](int j) { return CubeNum<false>{b[j]}; };
    const Cube<kShape, false, decltype(row)> cube{a, row};
    cube_walk(
        a,
        [&](uint64_t h) {
          const uint64_t g = h ^ (h >> 1);
#pragma unroll
          for (int j = 0; j < N; j++) b[j] = 0.0;
          add(sC + (size_t)(nc - 1) * N, 0.5);
#pragma unroll 1
          for (int k = 0; k < nc - 1; k++) add(sC + (size_t)k * N, ((g >> k) & 1) ? 0.5 : -0.5);
        },
        [&](uint64_t h) {
          const int k = __ffsll((long long)h) - 1;
          add(sC + (size_t)k * N, ((h >> (k + 1)) & 1) ? -1.0 : 1.0);
        },
        [&](uint64_t h) {
          CubeArray<15, false> top;
          CubeArray<11, false> last;
          cube.products(top, last);
          double even = 0.0, odd = 0.0;
#pragma unroll
          for (int s = 0; s < 8; s++) {
            const int lo = (s & 3) | ((s & 4) << 1);  // sign of column 2 minus
            const double d = top.v[lo].hi - top.v[lo | 4].hi;
            double& t = (__popc(s) & 1) ? odd : even;
            t = s < 2 ? last.v[s].hi * d : __fma_rn(last.v[s].hi, d, t);
          }
          const double t = even - odd;
          acc.add((h & 1) ? -t : t);
        });
  }
  const dd bt = block_reduce_dd(acc.value(), red);
  grid_finish_dd(bt, a.partials, a.ticket, a.out, (a.n & 1) ? 2.0 : -2.0, red);
}

// Split-dd walk (ryser_dense_sdd.cuh): b's exact coarse parts in registers,
// its remainders in shared memory ([slot][thread], conflict-free), which
// leaves room for the double-double arrays without spills.  6 FP64 operations
// per row value; 61..84% of the FP64 pipe (n = 34, density 1/2: 49 ms, in the
// three-level row layout before 102 ms).  With all of b in shared memory, read
// and updated in one pass, it was 9% slower (more wavefronts), with 12 warps
// of 168 registers 9% (spills).
template <int kShape>
__global__ void __launch_bounds__(kCubeThreads, 1) ryser_cube_sdd_kernel(const __grid_constant__ CubeArgs a) {
  constexpr int N = cube_rows(kCubeShapes[kShape]);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nc = a.n - 4;
  double* sC = reinterpret_cast<double*>(smem_raw);  // coarse columns, then their remainders
  const double* sD = sC + (size_t)nc * N;
  double* sL = sC + 2 * (size_t)nc * N;
  dd* red = reinterpret_cast<dd*>(sL + (size_t)N * kCubeThreads);
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 32);
  const bool staged = stage_to_smem(sC, a.img, (uint32_t)(sizeof(double) * 2 * nc * N), bar, a.err, a.inject);
  double H = 0.0, L = 0.0, m1 = 0.0;
  if (staged) {
    double b[N];
    double* bl = sL + threadIdx.x;
    auto add = [&](int k, double s) {
#pragma unroll
      for (int j = 0; j < N; j += 2) {
        const double2 v = lds2(sC + (size_t)k * N + j), w = lds2(sD + (size_t)k * N + j);
        b[j] = __fma_rn(s, v.x, b[j]);
        b[j + 1] = __fma_rn(s, v.y, b[j + 1]);
        bl[j * kCubeThreads] = __fma_rn(s, w.x, bl[j * kCubeThreads]);
        bl[(j + 1) * kCubeThreads] = __fma_rn(s, w.y, bl[(j + 1) * kCubeThreads]);
      }
    };
    auto row = [&](int j) { return CubeNum<true>{b[j], bl[j * kCubeThreads]}; };
    const Cube<kShape, true, decltype(row)> cube{a, row};
    cube_walk(
        a,
        [&](uint64_t h) {
          const uint64_t g = h ^ (h >> 1);
#pragma unroll
          for (int j = 0; j < N; j++) b[j] = bl[j * kCubeThreads] = 0.0;
          add(nc - 1, 0.5);
#pragma unroll 1
          for (int k = 0; k < nc - 1; k++) add(k, ((g >> k) & 1) ? 0.5 : -0.5);
        },
        [&](uint64_t h) {
          const int k = __ffsll((long long)h) - 1;
          add(k, ((h >> (k + 1)) & 1) ? -1.0 : 1.0);
        },
        [&](uint64_t h) {
          CubeArray<15, true> top;
          CubeArray<11, true> last;
          cube.products(top, last);
          cube_sum_dd(top, last, (h & 1) != 0, H, L, m1);
        });
  }
  DenseSddArgs f = {};  // the shared tail's destinations
  f.partials = a.partials;
  f.ticket = a.ticket;
  f.out = a.out;
  f.sums = a.sums;
  sdd_finish(H, L, m1, f, red, (a.n & 1) ? 2.0 : -2.0);
}

}  // namespace perm
