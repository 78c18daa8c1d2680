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
//   {0} > {01} (x {02}) > {012} > {0123} = top, {1} > {12} (x {13}) > {123}
//   {2} > {23} > {023}, {} > {3} > {03} > {013}
//
// The first two are multiplied into top, the third with the difference over
// the sign of column 2, the last with the sum of the rest.
//
// The host picks the four columns (for the certified walks, of the matrix or of
// its transpose) whose rows fit the cheapest of the compiled shapes
// (cube_shapes.h).  At density
// 1/2 that leaves about 0.2 x 16 n row values per 16 terms: for an order-32
// matrix some 300 FP64 operations instead of 1024 for the plain walk, and 640
// for the three-level row layout this replaced (n = 32, density 1/2: 5.8..6.4 ms
// then, 2.3..3.6 ms by shape now).
//
// Bound: the FP64 pipe, 74..83% of it at orders 32..34 up to 130 row values,
// 72% at 142, 60..65% at 200..290 (the rest are fixed latencies between dependent
// products: 2.4 warps' worth of independent work per scheduler).  The sums
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
#include "ryser_dense_int.cuh"
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

// A product: FP64, or a double-double pair.  kRows template arguments count
// the rows multiplied so far: 0 means unset, and products of up to kExact rows
// are exact in FP64 (lo is 0 and not kept).
struct CubeF64 {
  double hi;
  template <int kRows>
  __device__ __forceinline__ void mul(double x) {
    hi = hi * x;
  }
  template <int kRows, int kOther>
  __device__ __forceinline__ void mul(const CubeF64& x) {
    hi = hi * x.hi;
  }
};

template <int kExact>
struct CubeDd {
  double hi, lo;
  // by an exact value x of one or more rows, kRows in all afterwards
  template <int kRows, int kBefore>
  __device__ __forceinline__ void mul_exact(double x) {
    const double h = __dmul_rn(hi, x);
    if constexpr (kRows > kExact) {
      const double e = __fma_rn(hi, x, -h);
      lo = kBefore <= kExact ? e : __fma_rn(lo, x, e);
    }
    hi = h;
  }
  // by another product of kOther rows
  template <int kRows, int kOther>
  __device__ __forceinline__ void mul(const CubeDd& x) {
    if constexpr (kOther <= kExact) {
      mul_exact<kRows + kOther, kRows>(x.hi);
    } else {
      const double h = __dmul_rn(hi, x.hi);
      double l = __fma_rn(hi, x.hi, -h);
      l = __fma_rn(hi, x.lo, l);
      if constexpr (kRows > kExact) l = __fma_rn(lo, x.hi, l);
      hi = h;
      lo = l;
    }
  }
};

template <int kSet, class Num>
struct CubeArray {
  static constexpr int kW = 1 << cube_bits(kSet);
  Num v[kW];
};

// to = from widened to a larger set, or multiplied into it
template <int kTo, int kFrom, class Num>
__device__ __forceinline__ void cube_widen(CubeArray<kTo, Num>& to, const CubeArray<kFrom, Num>& from) {
#pragma unroll
  for (int s = 0; s < CubeArray<kTo, Num>::kW; s++) to.v[s] = from.v[cube_drop(s, kTo, kFrom)];
}
template <int kRows, int kOther, int kTo, int kFrom, class Num>
__device__ __forceinline__ void cube_merge(CubeArray<kTo, Num>& to, const CubeArray<kFrom, Num>& from) {
#pragma unroll
  for (int s = 0; s < CubeArray<kTo, Num>::kW; s++)
    to.v[s].template mul<kRows, kOther>(from.v[cube_drop(s, kTo, kFrom)]);
}

// The products of one cube.  `src` multiplies the rows of a class into an
// array: src.rows<kI, kDone>(p), kDone rows being in p already.
template <int kShape, class Num, class Source>
struct Cube {
  const Source& src;

  template <int kI>
  static constexpr int count() {
    return kI < 0 ? 0 : kCubeShapes[kShape].rows[cube_class(kI < 0 ? 0 : kI)];
  }

  // {k} > {kl} (x another pair) > {klm}: classes kI0, kI1, kX (-1: none) and
  // kI2 of the kernel order, starting from an array of kDone rows
  template <int kI0, int kI1, int kX, int kI2>
  static constexpr int total() {
    return count<kI0>() + count<kI1>() + count<kX>() + count<kI2>();
  }
  template <int kI0, int kI1, int kX, int kI2, int kFrom, int kDone>
  __device__ __forceinline__ void chain(CubeArray<cube_class(kI2), Num>& p3, const CubeArray<kFrom, Num>& from) const {
    constexpr int n1 = kDone + count<kI0>(), n2 = n1 + count<kI1>(), n3 = n2 + count<kX>();
    CubeArray<cube_class(kI0), Num> p1;
    if constexpr (kDone > 0) cube_widen(p1, from);
    src.template rows<kI0, kDone>(p1);
    CubeArray<cube_class(kI1), Num> p2;
    if constexpr (n1 > 0) cube_widen(p2, p1);
    src.template rows<kI1, n1>(p2);
    if constexpr (n2 > 0) cube_widen(p3, p2);
    if constexpr (n3 > n2) {
      CubeArray<cube_class(kX < 0 ? 0 : kX), Num> x;
      src.template rows<(kX < 0 ? 0 : kX), 0>(x);
      if constexpr (n2 == 0)
        cube_widen(p3, x);
      else
        cube_merge<n2, n3 - n2>(p3, x);
    }
    src.template rows<kI2, n3>(p3);
  }

  static constexpr int kFirst = total<1, 2, 3, 4>() + count<5>();  // rows of top
  static constexpr int kSecond = total<6, 7, 8, 9>();
  static constexpr int kThird = total<10, 11, -1, 12>();
  static constexpr int kLast = count<0>() + total<13, 14, -1, 15>();
  static_assert(total<1, 2, 3, 4>() > 0 && kLast > 0, "shapes have rows in the first and the last chain");

  // top[16]: the first and second chain and the rows of {0123}; the arrays of
  // the third ({0, 2, 3}; unset without rows) and the last chain ({0, 1, 3}),
  // which also takes the rows of {}: the chains are about as long then, and
  // more of their products stay below 2^53 for integers
  __device__ __forceinline__ void products(CubeArray<15, Num>& top, CubeArray<13, Num>& third,
                                           CubeArray<11, Num>& last) const {
    const CubeArray<0, Num> none = {};
    {
      CubeArray<7, Num> p3;
      chain<1, 2, 3, 4, 0, 0>(p3, none);
      cube_widen(top, p3);
      src.template rows<5, total<1, 2, 3, 4>()>(top);
    }
    if constexpr (kSecond > 0) {
      CubeArray<14, Num> p3;
      chain<6, 7, 8, 9, 0, 0>(p3, none);
      cube_merge<kFirst, kSecond>(top, p3);
    }
    if constexpr (kThird > 0) chain<10, 11, -1, 12, 0, 0>(third, none);
    CubeArray<0, Num> p0;
    src.template rows<0, 0>(p0);
    chain<13, 14, -1, 15, 0, count<0>()>(last, p0);
  }
};

// Rows of FP64 x: b + c with c a constant operand.  `row(slot)` returns b.
template <int kShape, class Row>
struct CubeRowsF64 {
  const CubeArgs& a;
  Row row;
  template <int kI, int kDone>
  __device__ __forceinline__ void rows(CubeArray<cube_class(kI), CubeF64>& p) const {
    constexpr int W = CubeArray<cube_class(kI), CubeF64>::kW, H = W / 2;
    constexpr int kSlot = cube_slot(kCubeShapes[kShape], kI), kSum = cube_sum(kCubeShapes[kShape], kI);
    constexpr int K = kCubeShapes[kShape].rows[cube_class(kI)];
#pragma unroll
    for (int r = 0; r < K; r++) {
      const double b = row(kSlot + r);
#pragma unroll
      for (int s = 0; s < W; s++) {
        double x = b;
        // the sums with the last column's sign plus; minus is their mirror image
        if constexpr (W > 1)
          x = s >= H ? __dadd_rn(b, a.c[kSum + r * H + s - H]) : __dsub_rn(b, a.c[kSum + r * H + H - 1 - s]);
        if (kDone == 0 && r == 0)
          p.v[s].hi = x;
        else
          p.v[s].hi = p.v[s].hi * x;
      }
    }
  }
};

// Rows of split x: pairs with exact coarse parts.  `row(slot)` returns (b, its remainder).
template <int kShape, class Row>
struct CubeRowsSdd {
  const CubeSddArgs& a;
  Row row;
  template <int kI, int kDone>
  __device__ __forceinline__ void rows(CubeArray<cube_class(kI), CubeDd<0>>& p) const {
    constexpr int W = CubeArray<cube_class(kI), CubeDd<0>>::kW, H = W / 2;
    constexpr int kSlot = cube_slot(kCubeShapes[kShape], kI), kSum = cube_sum(kCubeShapes[kShape], kI);
    constexpr int K = kCubeShapes[kShape].rows[cube_class(kI)];
#pragma unroll
    for (int r = 0; r < K; r++) {
      const CubeDd<0> b = row(kSlot + r);
#pragma unroll
      for (int s = 0; s < W; s++) {
        CubeDd<0> x = b;
        if constexpr (W > 1) {
          const int q = kSum + r * H + (s >= H ? s - H : H - 1 - s);
          x.hi = s >= H ? __dadd_rn(b.hi, a.c[q]) : __dsub_rn(b.hi, a.c[q]);
          x.lo = s >= H ? __dadd_rn(b.lo, a.cl[q]) : __dsub_rn(b.lo, a.cl[q]);
        }
        if (kDone == 0 && r == 0)
          p.v[s] = x;
        else
          p.v[s].template mul<1, 1>(x);
      }
    }
  }
};

// Rows of an integer matrix, y = 2x in int32 (registers).  Runs of 4 rows of
// a class (and a last run of 3) are multiplied in int32 and converted once per
// value: the host checks |product| < 2^31.  The one or two rows left over are
// converted once and added and multiplied in FP64: a run that short costs
// more in conversions (two cycles each per warp and SM) than it saves.  Both
// are exact.
template <int kShape, class Num, class Row>
struct CubeRowsInt {
  const CubeIntArgs& a;
  Row row;

  template <int kRows, int kBefore>
  __device__ __forceinline__ static void put(Num& p, double x) {
    if constexpr (kBefore == 0)
      p.hi = x;
    else if constexpr (std::is_same_v<Num, CubeF64>)
      p.hi = p.hi * x;
    else
      p.template mul_exact<kRows, kBefore>(x);
  }
  template <int kI, int kR, int kDone>
  __device__ __forceinline__ void from(CubeArray<cube_class(kI), Num>& p) const {
    constexpr int W = CubeArray<cube_class(kI), Num>::kW, H = W / 2;
    constexpr int K = kCubeShapes[kShape].rows[cube_class(kI)], kLeft = K - kR;
    constexpr int kSlot = cube_slot(kCubeShapes[kShape], kI), kSum = cube_sum(kCubeShapes[kShape], kI);
    if constexpr (kLeft >= 3) {
      constexpr int G = kLeft >= 4 ? 4 : 3;
#pragma unroll
      for (int s = 0; s < W; s++) {
        uint32_t y[4];
#pragma unroll
        for (int t = 0; t < G; t++) {
          const int b = row(kSlot + kR + t), q = kSum + (kR + t) * H;
          if constexpr (W > 1)
            y[t] = (uint32_t)(s >= H ? b + a.ci[q + s - H] : b - a.ci[q + H - 1 - s]);
          else
            y[t] = (uint32_t)b;
        }
        const uint32_t v = G == 4 ? (y[0] * y[1]) * (y[2] * y[3]) : (y[0] * y[1]) * y[2];
        put<kDone + G, kDone>(p.v[s], __int2double_rn((int)v));
      }
      from<kI, kR + G, kDone + G>(p);
    } else if constexpr (kLeft > 0) {
      constexpr int kLeftSum = cube_left_sum(kCubeShapes[kShape], kI) + (kR - (K - cube_left(K))) * H;
      const double b = __int2double_rn(row(kSlot + kR));
#pragma unroll
      for (int s = 0; s < W; s++) {
        double x = b;
        if constexpr (W > 1) x = s >= H ? __dadd_rn(b, a.cd[kLeftSum + s - H]) : __dsub_rn(b, a.cd[kLeftSum + H - 1 - s]);
        put<kDone + 1, kDone>(p.v[s], x);
      }
      from<kI, kR + 1, kDone + 1>(p);
    }
  }
  template <int kI, int kDone>
  __device__ __forceinline__ void rows(CubeArray<cube_class(kI), Num>& p) const {
    from<kI, 0, kDone>(p);
  }
};

// Adds the 16 signed terms last x top to (H, L) (Sum2, over column 2's sign
// first) and their absolute values to m1.  Exact products keep no low part.
template <bool kTopExact, bool kLastExact, class Num>
__device__ __forceinline__ void cube_sum_dd(const CubeArray<15, Num>& top, const CubeArray<11, Num>& last, bool odd,
                                            double& H, double& L, double& m1) {
  dd t[8];
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const int lo = (s & 3) | ((s & 4) << 1);  // sign of column 2 minus
    const Num &t0 = top.v[lo], &t1 = top.v[lo | 4];
    dd d = two_sum(t0.hi, -t1.hi);
    if constexpr (!kTopExact) d.lo = __dadd_rn(d.lo, __dsub_rn(t0.lo, t1.lo));
    m1 = __fma_rn(fabs(last.v[s].hi), __dadd_rn(fabs(t0.hi), fabs(t1.hi)), m1);
    if constexpr (kLastExact) {
      const double h = __dmul_rn(d.hi, last.v[s].hi);
      d.lo = __fma_rn(d.lo, last.v[s].hi, __fma_rn(d.hi, last.v[s].hi, -h));
      d.hi = h;
    } else {
      pair_mul(d, last.v[s].hi, last.v[s].lo);
    }
    if (__popc(s) & 1) d = {-d.hi, -d.lo};
    t[s] = d;
  }
  // pairwise: every rounding error of the high parts goes to the low part
#pragma unroll
  for (int w = 4; w >= 1; w >>= 1) {
#pragma unroll
    for (int s = 0; s < w; s++) {
      dd r = two_sum(t[s].hi, t[s + w].hi);
      r.lo = __dadd_rn(r.lo, __dadd_rn(t[s].lo, t[s + w].lo));
      t[s] = r;
    }
  }
  sum2_add(H, L, odd ? -t[0].hi : t[0].hi, odd ? -t[0].lo : t[0].lo);
}

// Adds the 16 signed terms top x third x last to acc: over column 2's sign
// first, then column 0's, then the other two, as one sum or (kTwo) as two.
//
// What the error comes from are the roundings of the largest terms, which for
// matrices without negative entries are those of plus signs alone.  So every
// difference of products is fused on the side of the plus sign, and only the
// minus side's product is rounded by itself; integer walks, whose row layouts
// round less than those of FP64 x, add two sums.  Errors then are no larger than
// the row layouts' (rms in units of 2^-53 sum |term|, orders 25..28: values
// 1..4, 600 matrices each, 0.074/0.064/0.061/0.058 against
// 0.082/0.076/0.068/0.070; FP32 values, 360 matrices each,
// 0.154/0.124/0.125/0.120 against 0.177/0.162/0.144/0.125).  With the minus sides
// fused and one sum the integers' were above them (0.088/0.084/0.076/0.069), and
// with one sum now they are 4% larger than with two, in 1% less time; four sums
// are 5% below two, in 3% more time.  The sign as a factor of fused additions
// pays for the second sum: selected, one sum takes as long (n = 30..37).
// kAbs: the terms' absolute values are added to m1.
template <bool kThird, bool kAbs, bool kTwo>
__device__ __forceinline__ void cube_add_f64(const CubeArray<15, CubeF64>& top, const CubeArray<13, CubeF64>& third,
                                             const CubeArray<11, CubeF64>& last, bool odd, Acc& acc, double& m1) {
  double d[8];
#pragma unroll
  for (int s = 0; s < 8; s++) {
    const int t0 = (s & 3) | ((s & 4) << 1), t1 = t0 | 4;  // column 2 minus, plus
    if constexpr (kThird) {
      const int a0 = (s & 1) | (s & 4), a1 = a0 | 2;
      const double p = __dmul_rn(top.v[t0].hi, third.v[a0].hi);
      d[s] = __fma_rn(top.v[t1].hi, third.v[a1].hi, -p);
      if constexpr (kAbs)
        m1 = __fma_rn(fabs(last.v[s].hi), __fma_rn(fabs(top.v[t1].hi), fabs(third.v[a1].hi), fabs(p)), m1);
    } else {
      d[s] = __dsub_rn(top.v[t1].hi, top.v[t0].hi);
      if constexpr (kAbs)
        m1 = __fma_rn(fabs(last.v[s].hi), __dadd_rn(fabs(top.v[t0].hi), fabs(top.v[t1].hi)), m1);
    }
  }
  double t[4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int s = 2 * q;
    t[q] = __fma_rn(last.v[s + 1].hi, d[s + 1], -__dmul_rn(last.v[s].hi, d[s]));
  }
  // terms with an even number of minus signs among the four columns count plus
  const double sign = odd ? -1.0 : 1.0, large = __dsub_rn(t[3], t[2]), small = __dsub_rn(t[0], t[1]);
  if constexpr (kTwo) {
    acc.add(large, sign);
    acc.add(small, sign);
  } else {
    acc.add(__dadd_rn(large, small), sign);
  }
}

// Range of outer Gray indices of this thread, and the loop over it:
// start(h) sets b for outer index h, flip(h) moves it from h - 1 to h,
// cube(h) adds the 16 terms of h.
template <class Start, class Flip, class Eval>
__device__ __forceinline__ void cube_walk(const CubeWalk& a, Start start, Flip flip, Eval cube) {
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

// The thread totals' sum to *out and, with abs_sum, every warp's sum of m1 to
// the words behind the blocks' totals, which are added in their order afterwards
// (by the host, or by cube_sums_kernel in a batch), so that a walk's error estimate
// is the same every time.  The form matters to the register allocation of the
// certified walks: added here by the block that finishes last, or stored without
// the fence (the kernel's end makes the stores visible too), they were up to 4 or 5%
// slower by shape; so they are within 0.7% of atomic additions in any order.
__device__ __forceinline__ void cube_finish(const CubeWalk& a, dd total, bool abs_sum, double m1, double factor, dd* red) {
  double* sums = reinterpret_cast<double*>(a.partials + gridDim.x);
  if (abs_sum) {
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) m1 += __shfl_down_sync(0xffffffffu, m1, d);
    if ((threadIdx.x & 31) == 0) {
      sums[blockIdx.x * kCubeWarps + (threadIdx.x >> 5)] = m1;
      __threadfence();
    }
  }
  const dd bt = block_reduce_dd(total, red);
  grid_finish_dd(bt, a.partials, a.ticket, a.out, factor, red);
}

// FP64 walk; kAbs: its sum |term| as well (16 of some 250 operations).
template <int kShape, bool kAbs>
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
  double m1 = 0.0;
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
    auto row = [&](int j) { return b[j]; };
    const CubeRowsF64<kShape, decltype(row)> src{a, row};
    const Cube<kShape, CubeF64, decltype(src)> cube{src};
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
          CubeArray<15, CubeF64> top;
          CubeArray<13, CubeF64> third;
          CubeArray<11, CubeF64> last;
          cube.products(top, third, last);
          cube_add_f64<(decltype(cube)::kThird > 0), kAbs, false>(top, third, last, (h & 1) != 0, acc, m1);
        });
  }
  cube_finish(a, acc.value(), kAbs, m1, (a.n & 1) ? 2.0 : -2.0, red);
}

// Split-dd walk (ryser_dense_sdd.cuh): b's exact coarse parts in registers,
// its remainders in shared memory ([slot][thread], conflict-free), which
// leaves room for the double-double arrays without spills.  6 FP64 operations
// per row value; 61..84% of the FP64 pipe (n = 34, density 1/2: 49 ms, in the
// three-level row layout before 102 ms).  With all of b in shared memory, read
// and updated in one pass, it was 9% slower (more wavefronts), with 12 warps
// of 168 registers 9% (spills).
template <int kShape>
__global__ void __launch_bounds__(kCubeThreads, 1) ryser_cube_sdd_kernel(const __grid_constant__ CubeSddArgs a) {
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
    auto row = [&](int j) { return CubeDd<0>{b[j], bl[j * kCubeThreads]}; };
    const CubeRowsSdd<kShape, decltype(row)> src{a, row};
    const Cube<kShape, CubeDd<0>, decltype(src)> cube{src};
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
          using C = decltype(cube);
          CubeArray<15, CubeDd<0>> top;
          CubeArray<13, CubeDd<0>> third;
          CubeArray<11, CubeDd<0>> last;
          cube.products(top, third, last);
          if constexpr (C::kThird > 0) cube_merge<C::kFirst + C::kSecond, C::kThird>(top, third);
          cube_sum_dd<false, false>(top, last, (h & 1) != 0, H, L, m1);
        });
  }
  cube_finish(a, two_sum(H, L), true, m1, (a.n & 1) ? 2.0 : -2.0, red);
}

// Integer walks: y in int32 registers, columns as int32 in shared memory.
// FP64 products (kDd false), or double-double products and sum with a
// certified error (ryser_dense_intc.cuh), where products of up to
// kCubeExactRows rows are kept in FP64 exactly (checked by the host).
// FP64 products, order-40 shape of 140 values: 186 cycles per warp and cube,
// 0.64 instructions issued per cycle and scheduler, FP64 pipe 46%, conversions
// 30% (n = 40, density 1/2: 375 in the three-level row layout before).  In a
// program of this walk alone, one sum a cube, 182:
// constants of both signs instead of mirrored ones 200 (the compiler loads
// them to registers early); left-over rows added to the bit pattern of 2^52 + b
// instead of converted: 187; 12 warps of 168 registers: 185 and spills in the
// larger shapes.  Certified: 364 cycles, of which the double-double arrays and
// sum are two thirds of the FP64 operations (12 warps: 381).
template <int kShape, bool kDd, bool kAbs>
__global__ void __launch_bounds__(kCubeThreads, 1) ryser_cube_int_kernel(const __grid_constant__ CubeIntArgs a) {
  using Num = std::conditional_t<kDd, CubeDd<kCubeExactRows>, CubeF64>;
  constexpr int N = cube_rows(kCubeShapes[kShape]);
  static_assert(N % 4 == 0, "columns are read four rows at a time");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nc = a.n - 4;
  int* sC = reinterpret_cast<int*>(smem_raw);
  dd* red = reinterpret_cast<dd*>(sC + (size_t)nc * N);
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 32);
  const bool staged = stage_to_smem(sC, a.img, (uint32_t)(sizeof(int) * nc * N), bar, a.err, a.inject);
  Acc acc;
  double H = 0.0, L = 0.0, m1 = 0.0;
  if (staged) {
    int b[N];
    auto add = [&](int k, int s) {
#pragma unroll
      for (int j = 0; j < N; j += 4) {
        const int4 v = lds4i(sC + (size_t)k * N + j);
        b[j] += s * v.x;
        b[j + 1] += s * v.y;
        b[j + 2] += s * v.z;
        b[j + 3] += s * v.w;
      }
    };
    auto row = [&](int j) { return b[j]; };
    const CubeRowsInt<kShape, Num, decltype(row)> src{a, row};
    const Cube<kShape, Num, decltype(src)> cube{src};
    cube_walk(
        a,
        [&](uint64_t h) {
          const uint64_t g = h ^ (h >> 1);
#pragma unroll
          for (int j = 0; j < N; j++) b[j] = 0;
          add(nc - 1, 1);
#pragma unroll 1
          for (int k = 0; k < nc - 1; k++) add(k, ((g >> k) & 1) ? 1 : -1);
        },
        [&](uint64_t h) {
          const int k = __ffsll((long long)h) - 1;
          add(k, ((h >> (k + 1)) & 1) ? -2 : 2);
        },
        [&](uint64_t h) {
          using C = decltype(cube);
          CubeArray<15, Num> top;
          CubeArray<13, Num> third;
          CubeArray<11, Num> last;
          cube.products(top, third, last);
          if constexpr (kDd) {
            if constexpr (C::kThird > 0) cube_merge<C::kFirst + C::kSecond, C::kThird>(top, third);
            cube_sum_dd<C::kFirst + C::kSecond + C::kThird <= kCubeExactRows, C::kLast <= kCubeExactRows>(
                top, last, (h & 1) != 0, H, L, m1);
          } else {
            cube_add_f64<(C::kThird > 0), kAbs, true>(top, third, last, (h & 1) != 0, acc, m1);
          }
        });
  }
  // prod y = 2^n prod x
  const double factor = ((a.n & 1) ? 2.0 : -2.0) * ldexp(1.0, -a.n);
  cube_finish(a, kDd ? two_sum(H, L) : acc.value(), kDd || kAbs, m1, factor, red);
}

}  // namespace perm
