// engine.cu -- host side of the permanent engine: device contexts, launch
// planning, the C ABI declared in include/perman_b200.h.
//
// Replaces the reference's host wrappers (gpu_exact_dense.cu:641-699,
// gpu_exact_sparse.cu:1124-1190, gpu_approximation_dense.cu:374-409, 528-571,
// gpu_approximation_sparse.cu:455-495, 608-661).  Differences by design:
//  * a context owns the stream and all scratch, allocated once, so a call does
//    no cudaMalloc/cudaFree (the reference allocates and frees per call and
//    hard-codes cudaSetDevice(1));
//  * every CUDA call is checked and reported through a status code and a
//    per-context message (the reference checks none);
//  * results come back as one double-double (16 bytes) reduced on the device
//    instead of 524,288 partials summed on the host;
//  * launch shapes are chosen from the device's SM count and the kernel's
//    occupancy instead of a fixed <<<2048, 256>>>.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include "../../include/perman_b200.h"
#include "batch.h"
#include "cube_plan.h"
#include "host_pool.h"
#include "matrix_io.h"
#include "mc.h"
#include "mc_sparse.h"
#include "perman_common.cuh"
#include "ryser_cube.h"
#include "ryser_dense.cuh"
#include "ryser_dense_dd.cuh"
#include "ryser_dense_split.cuh"
#include "ryser_dense_tc.cuh"
#include "ryser_dense_int.cuh"
#include "ryser_dense_intc.cuh"
#include "ryser_dense_int_sparse.cuh"
#include "ryser_dense_intc_sparse.cuh"
#include "ryser_dense_2l.cuh"
#include "ryser_dense_sdd.cuh"
#include "skipper.h"

namespace perm {
const void* dense_kernel_0(int n);
const void* dense_kernel_1(int n);
const void* dense_kernel_2(int n);
const void* dense_kernel_3(int n);
const void* dense_kernel_4(int n);

const void* dense_int_kernel_g3(int n);
const void* dense_int_kernel_g4(int n);
const void* dense_int_kernel_g5(int n);
const void* dense_int_kernel_g6(int n);

const void* dense_dd_kernel(int n);
const void* dense_2l_kernel_r16(int n);
const void* dense_2l_kernel_r20(int n);
const void* dense_2l_kernel_r24(int n);
const void* dense_2l_kernel_r28(int n);
const void* dense_3l_kernel_r20(int n, int r1);
const void* dense_3l_kernel_r24(int n, int r1);
const void* dense_3l_kernel_r28(int n, int r1);
const void* dense_3l_kernel_r32(int n, int r1);
const void* dense_3l_kernel_r36(int n, int r1);

// FP64-X walk in the two-level row layout (ryser_dense_2l.cuh): orders
// 20..48, 16..28 inner rows
constexpr int k2lInner[4] = {16, 20, 24, 28};
// FP64-X three-level layout (ryser_dense_3l_kernel<N, R1, R2>): second
// levels ending at R2, first levels R1 in 8..20
constexpr int kFp3lR2[5] = {20, 24, 28, 32, 36};
static const void* dense_3l_kernel(int n, int r1, int r2) {
  switch (r2) {
    case 20: return dense_3l_kernel_r20(n, r1);
    case 24: return dense_3l_kernel_r24(n, r1);
    case 28: return dense_3l_kernel_r28(n, r1);
    case 32: return dense_3l_kernel_r32(n, r1);
    case 36: return dense_3l_kernel_r36(n, r1);
    default: return nullptr;
  }
}
static const void* dense_2l_kernel(int n, int inner) {
  switch (inner) {
    case 16: return dense_2l_kernel_r16(n);
    case 20: return dense_2l_kernel_r20(n);
    case 24: return dense_2l_kernel_r24(n);
    case 28: return dense_2l_kernel_r28(n);
    default: return nullptr;
  }
}
const void* dense_split_kernel(int n);

const void* dense_intc_kernel_g3(int n);
const void* dense_intc_kernel_g4(int n);
const void* dense_intc_kernel_g5(int n);
const void* dense_intc_kernel_g6(int n);
const void* dense_int_3l_kernel_g4(int n, int ng1, int ng2);
const void* dense_int_3l_kernel_g5(int n, int ng1, int ng2);
const void* dense_int_3l_kernel_g6(int n, int ng1, int ng2);
const void* dense_int_sparse_kernel_g4(int n, int ngo);
const void* dense_int_sparse_kernel_g5(int n, int ngo);
const void* dense_int_sparse_kernel_g6(int n, int ngo);
const void* dense_intc_3l_kernel_g4p(int n, int ng1, int ng2);
const void* dense_intc_3l_kernel_g5(int n, int ng1, int ng2);
const void* dense_intc_3l_kernel_g6p(int n, int ng1, int ng2);
const void* dense_intc_sparse_kernel_g4p(int n, int ngo);
const void* dense_intc_sparse_kernel_g5(int n, int ngo);
const void* dense_intc_sparse_kernel_g6p(int n, int ngo);
const void* dense_intc_pair_kernel_g4(int n);
const void* dense_intc_pair_kernel_g5(int n);
const void* dense_intc_pair_kernel_g6(int n);

const void* dense_sdd_kernel(int n);
const void* sparse_sdd_kernel_r6(int n);
const void* sparse_sdd_kernel_r8(int n);
const void* sparse_sdd_kernel_r12(int n);
const void* sparse_sdd_kernel_r16(int n);
const void* sparse_sdd_kernel_r20(int n);
const void* sparse_sdd_kernel_r24(int n);
const void* sparse_sdd_kernel_r28(int n);
const void* sdd_3l_kernel_r16(int n, int r1);
const void* sdd_3l_kernel_r20(int n, int r1);
const void* sdd_3l_kernel_r24(int n, int r1);
const void* sdd_3l_kernel_r28(int n, int r1);

// ryser_cube_<kind>_n<size>.cu
#define PERM_CUBE_KIND(kind)            \
  const void* cube_##kind##_n28(int i); \
  const void* cube_##kind##_n32(int i); \
  const void* cube_##kind##_n36(int i); \
  const void* cube_##kind##_n40(int i);
PERM_CUBE_KIND(f64)
PERM_CUBE_KIND(f64a)
PERM_CUBE_KIND(sdd)
PERM_CUBE_KIND(int)
PERM_CUBE_KIND(inta)
PERM_CUBE_KIND(intc)
#undef PERM_CUBE_KIND
const void* dense_tc_kernel_g3(int n);
const void* dense_tc_kernel_g4(int n);
const void* dense_tc_kernel_g5(int n);
const void* dense_tc_kernel_g6(int n);

static int cube_size(int shape) {
  int i = 0;
  while (shape >= kCubeFirst[i + 1]) i++;
  return i;
}
// kinds of column-cube walks, in the order of their occupancy tables
enum CubeKind { kCubeF64, kCubeF64Abs, kCubeSdd, kCubeInt, kCubeIntAbs, kCubeIntc, kCubeKinds };
static const void* cube_kernel(int shape, int kind) {
  using Pick = const void* (*)(int);
#define PERM_CUBE_KIND(kind) \
  {cube_##kind##_n28, cube_##kind##_n32, cube_##kind##_n36, cube_##kind##_n40}
  static const Pick pick[kCubeKinds][kCubeSizeCount] = {PERM_CUBE_KIND(f64), PERM_CUBE_KIND(f64a), PERM_CUBE_KIND(sdd),
                                                        PERM_CUBE_KIND(int), PERM_CUBE_KIND(inta), PERM_CUBE_KIND(intc)};
#undef PERM_CUBE_KIND
  const int i = cube_size(shape);
  return pick[kind][i](shape - kCubeFirst[i]);
}

static const void* dense_tc_kernel(int n, int g) {
  switch (g) {
    case 3: return dense_tc_kernel_g3(n);
    case 4: return dense_tc_kernel_g4(n);
    case 5: return dense_tc_kernel_g5(n);
    case 6: return dense_tc_kernel_g6(n);
    default: return nullptr;
  }
}

static const void* dense_int_kernel(int n, int g) {
  switch (g) {
    case 3: return dense_int_kernel_g3(n);
    case 4: return dense_int_kernel_g4(n);
    case 5: return dense_int_kernel_g5(n);
    case 6: return dense_int_kernel_g6(n);
    default: return nullptr;
  }
}

// int32-X walk in the two-level row layout (ryser_dense_int_sparse.cuh):
// orders 20..48, groups of 4..6 rows, 1..3 outer groups
constexpr int kIntSparseMinN = 20, kIntSparseMaxN = 48, kIntSparseMaxOuter = 3;
static const void* dense_int_sparse_kernel(int n, int g, int ngo) {
  switch (g) {
    case 4: return dense_int_sparse_kernel_g4(n, ngo);
    case 5: return dense_int_sparse_kernel_g5(n, ngo);
    case 6: return dense_int_sparse_kernel_g6(n, ngo);
    default: return nullptr;
  }
}

// certified int32-X walk in the two-level row layout: groups of 4 and 6 in
// int64 pairs, groups of 5 alone (family index 0, 1, 2)
static int intc_sparse_family(int g, int pair) {
  return (g == 4 && pair) ? 0 : (g == 5 && !pair) ? 1 : (g == 6 && pair) ? 2 : -1;
}
static const void* dense_intc_sparse_kernel(int n, int g, int pair, int ngo) {
  switch (intc_sparse_family(g, pair)) {
    case 0: return dense_intc_sparse_kernel_g4p(n, ngo);
    case 1: return dense_intc_sparse_kernel_g5(n, ngo);
    case 2: return dense_intc_sparse_kernel_g6p(n, ngo);
    default: return nullptr;
  }
}

// int32-X walk in the three-level row layout: orders 28..48, groups of 4..6,
// 2..4 groups on the first level (column 0), 1..2 on the second (columns 1, 2)
constexpr int kInt3lMinN = 28;
static const void* dense_int_3l_kernel(int n, int g, int ng1, int ng2) {
  switch (g) {
    case 4: return dense_int_3l_kernel_g4(n, ng1, ng2);
    case 5: return dense_int_3l_kernel_g5(n, ng1, ng2);
    case 6: return dense_int_3l_kernel_g6(n, ng1, ng2);
    default: return nullptr;
  }
}

static const void* dense_intc_3l_kernel(int n, int g, int pair, int ng1, int ng2) {
  switch (intc_sparse_family(g, pair)) {
    case 0: return dense_intc_3l_kernel_g4p(n, ng1, ng2);
    case 1: return dense_intc_3l_kernel_g5(n, ng1, ng2);
    case 2: return dense_intc_3l_kernel_g6p(n, ng1, ng2);
    default: return nullptr;
  }
}

static const void* dense_intc_kernel(int n, int g, int pair) {
  if (pair) {
    switch (g) {
      case 4: return dense_intc_pair_kernel_g4(n);
      case 5: return dense_intc_pair_kernel_g5(n);
      case 6: return dense_intc_pair_kernel_g6(n);
      default: return nullptr;
    }
  }
  switch (g) {
    case 3: return dense_intc_kernel_g3(n);
    case 4: return dense_intc_kernel_g4(n);
    case 5: return dense_intc_kernel_g5(n);
    case 6: return dense_intc_kernel_g6(n);
    default: return nullptr;
  }
}

// Inner-row counts of the sparse split-dd layout (ryser_sparse_sdd_kernel<N, R>).
// 20..28: the rolled step loop (two-level rows of dense matrices)
constexpr int kSparseInner[7] = {6, 8, 12, 16, 20, 24, 28};

// Three-level split-dd layout (ryser_sdd_3l_kernel<N, R1, R2>): second-level
// ends R2 and first-level ends R1 < R2 (multiples of 4).
constexpr int kSdd3lR2[4] = {16, 20, 24, 28};
constexpr int kSdd3lMinN = 24;

static const void* sdd_kernel(int n, int inner, int inner1) {
  if (inner1) {
    switch (inner) {
      case 16: return sdd_3l_kernel_r16(n, inner1);
      case 20: return sdd_3l_kernel_r20(n, inner1);
      case 24: return sdd_3l_kernel_r24(n, inner1);
      case 28: return sdd_3l_kernel_r28(n, inner1);
      default: return nullptr;
    }
  }
  switch (inner) {
    case 0: return dense_sdd_kernel(n);
    case 6: return sparse_sdd_kernel_r6(n);
    case 8: return sparse_sdd_kernel_r8(n);
    case 12: return sparse_sdd_kernel_r12(n);
    case 16: return sparse_sdd_kernel_r16(n);
    case 20: return sparse_sdd_kernel_r20(n);
    case 24: return sparse_sdd_kernel_r24(n);
    case 28: return sparse_sdd_kernel_r28(n);
    default: return nullptr;
  }
}

static const void* dense_kernel(int n) {
  if (n >= 1 && n <= 20) return dense_kernel_0(n);
  if (n <= 32) return dense_kernel_1(n);
  if (n <= 42) return dense_kernel_2(n);
  if (n <= 52) return dense_kernel_3(n);
  if (n <= 64) return dense_kernel_4(n);
  return nullptr;
}

// Estimates of sum_S |term(S)| and sum_S term(S)^2 over the 2^(n-1) column
// subsets S of the walk, stratified by |S|: class k holds C(n-1, k) subsets
// and gets `per_class` threads.  A class no larger than that is enumerated
// exactly (the r-th k-subset in colex order, by unranking); a
// larger one is sampled uniformly (Floyd's k-subset algorithm on a
// splitmix64 stream) and each sample weighted C(n-1, k) / per_class.  Term
// magnitudes depend strongly on |S| (|S| = 0 is the all-minus subset, often
// the largest term), so a plain uniform sample of Gray indices either misses
// the heavy classes or, hitting one, overstates the sums by 2^(n-1)/samples.
// Each thread builds x(S) from scratch in FP64; block b leaves its weighted sums
// of |prod x_j| and of its square in out[2 b] and out[2 b + 1].
__device__ __forceinline__ uint64_t splitmix64(uint64_t& state) {
  uint64_t z = (state += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void __launch_bounds__(256) ryser_abs_sample_kernel(const double* colA, int n, int np, int per_class,
                                                                uint64_t seed, double* out) {
  __shared__ double sA[64 * 64];
  __shared__ double x0[64];
  __shared__ double red[8], red2[8];
  for (int idx = threadIdx.x; idx < n * np; idx += blockDim.x) sA[idx] = colA[idx];
  __syncthreads();
  if (threadIdx.x < n) {
    const int j = threadIdx.x;
    double rs = 0.0;
    for (int k = 0; k < n; k++) rs += sA[k * np + j];
    x0[j] = sA[(n - 1) * np + j] - rs * 0.5;
  }
  __syncthreads();
  const int m = n - 1;
  double local = 0.0, local2 = 0.0;
  const uint64_t s = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = (int)(s / (uint64_t)per_class);
  const uint64_t r = s % (uint64_t)per_class;
  if (k <= m) {
    double c = 1.0;  // C(m, k)
    for (int t = 1; t <= k; t++) c = c * (double)(m - k + t) / (double)t;
    uint64_t g = 0;
    double w = 0.0;
    if (c <= (double)per_class) {
      if ((double)r < c) {
        // colex unranking: the largest element i is the largest with
        // C(i, kk) <= rank; cb tracks C(i, kk) down the loop (small exact integers)
        double cb = (k <= m - 1) ? c * (double)(m - k) / (double)m : 0.0;  // C(m - 1, k)
        uint64_t rank = r;
        int kk = k;
        for (int i = m - 1; i >= 0 && kk > 0; i--) {
          if ((double)rank >= cb) {
            rank -= (uint64_t)cb;
            g |= 1ull << i;
            if (i > 0) cb = cb * (double)kk / (double)i;
            kk--;
          } else if (i > 0) {
            cb = cb * (double)(i - kk) / (double)i;
          }
        }
        w = 1.0;
      }
    } else {
      uint64_t st = seed ^ (s * 0xD1B54A32D192ED03ull);
      for (int j = m - k; j < m; j++) {
        const uint32_t t = (uint32_t)(((splitmix64(st) >> 32) * (uint64_t)(j + 1)) >> 32);
        g |= ((g >> t) & 1) ? (1ull << j) : (1ull << t);
      }
      w = c / (double)per_class;
    }
    if (w > 0.0) {
      double p = 1.0;
      for (int j = 0; j < n; j++) {
        double xj = x0[j];
        for (int kk = 0; kk < m; kk++)
          if ((g >> kk) & 1) xj += sA[kk * np + j];
        p *= xj;
      }
      local = w * fabs(p);
      local2 = w * p * p;
    }
  }
  for (int d = 16; d >= 1; d >>= 1) {
    local += __shfl_down_sync(0xffffffffu, local, d);
    local2 += __shfl_down_sync(0xffffffffu, local2, d);
  }
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5] = local;
    red2[threadIdx.x >> 5] = local2;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0, t2 = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      t += red[w];
      t2 += red2[w];
    }
    out[2 * blockIdx.x] = t;
    out[2 * blockIdx.x + 1] = t2;
  }
}

// Size estimate of perm(A) for a nonnegative matrix, for the accuracy
// policy's choice of its first walk: Rasmussen's estimator with weights.
// Row i picks an unused column c with probability a_ic / R_i (R_i: the row's
// sum over unused columns) and multiplies the trial weight by R_i, so the
// expected weight is perm(A).  One trial per thread on a splitmix64 stream;
// weights are kept as log2 and scaled by 2^-log2_ub (log2_ub: log2 of the
// product of the row sums, an upper bound of every weight), so the scaled
// weights lie in [0, 1] and their block sums are added to *out.  A trial
// whose row sum vanishes has weight 0.
__global__ void __launch_bounds__(256) weighted_rasmussen_kernel(const double* colA, int n, int np, int trials,
                                                                 uint64_t seed, double log2_ub, double* out) {
  __shared__ double sA[64 * 64];
  __shared__ double red[8];
  for (int idx = threadIdx.x; idx < n * np; idx += blockDim.x) sA[idx] = colA[idx];
  __syncthreads();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  double w = 0.0;
  if (t < trials) {
    uint64_t st = seed ^ ((uint64_t)t * 0xD1B54A32D192ED03ull);
    uint64_t used = 0;
    double lw = 0.0;
    bool alive = true;
    for (int i = 0; i < n && alive; i++) {
      double r = 0.0;
      for (int c = 0; c < n; c++)
        if (!((used >> c) & 1)) r += sA[c * np + i];
      if (!(r > 0.0)) {
        alive = false;
        break;
      }
      lw += log2(r);
      const double u = r * ((double)(splitmix64(st) >> 11) * 0x1.0p-53);
      double acc = 0.0;
      int pick = -1;
      for (int c = 0; c < n; c++) {
        if ((used >> c) & 1) continue;
        const double v = sA[c * np + i];
        if (v > 0.0) {
          pick = c;
          acc += v;
          if (acc > u) break;
        }
      }
      used |= 1ull << pick;  // r > 0: some unused column is positive
    }
    if (alive) w = exp2(lw - log2_ub);
  }
  for (int d = 16; d >= 1; d >>= 1) w += __shfl_down_sync(0xffffffffu, w, d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x == 0) {
    double b = 0.0;
    for (int k = 0; k < (int)(blockDim.x >> 5); k++) b += red[k];
    atomicAdd(out, b);
  }
}

__global__ void fp64_peak_kernel(double* out, int iters, double a, double b) {
  double x0 = threadIdx.x * 1e-9, x1 = x0 + 1e-3, x2 = x0 + 2e-3, x3 = x0 + 3e-3;
  double x4 = x0 + 4e-3, x5 = x0 + 5e-3, x6 = x0 + 6e-3, x7 = x0 + 7e-3;
  for (int i = 0; i < iters; i++) {
#pragma unroll
    for (int u = 0; u < 16; u++) {
      x0 = fma(x0, a, b);
      x1 = fma(x1, a, b);
      x2 = fma(x2, a, b);
      x3 = fma(x3, a, b);
      x4 = fma(x4, a, b);
      x5 = fma(x5, a, b);
      x6 = fma(x6, a, b);
      x7 = fma(x7, a, b);
    }
  }
  double s = ((x0 + x1) + (x2 + x3)) + ((x4 + x5) + (x6 + x7));
  if (s == 12345.678) out[0] = s;  // keeps the chains live
}
}  // namespace perm

using namespace perm;

struct DenseOperand;
struct perm_matrix;

// Result words of a call; behind them are the column cubes' partials (kCubeWords a
// block, at most kCubeBlocks blocks an SM), or the moment sample's (2 a block).
constexpr int kOutWords = 16;
constexpr int kCubeBlocks = 2048 / kCubeThreads;
constexpr int kSamplesPerClass = 8192;  // term-moment sample: threads per subset-size class
// Blocks of the sample of an order-n matrix: classes |S| = 0 .. n-1.
constexpr int moment_blocks(int n) { return n * kSamplesPerClass / 256; }

// Smallest order of the column-cube walks: the shards of shard_bounds are
// whole cubes of 16 terms from here on, and below it the search for four
// columns (some 30 us on the host) costs what the walk gains.
constexpr int kCubeMinN = 25;
// ... and of the accuracy policy's whole FP64 walks: the cube sums its own
// |term|, the row layouts pay for a sample (20..60 us; real, density 1/2: n = 20
// 95 against 57 us, n = 23 115 and 60).  Below 20 every FP64 walk is the
// one-level one, as perm_exact_dense_noalloc's is.
constexpr int kCubeSumMinN = 20;
// Shortest lane range, as a power of two, that small batches are cut to.
constexpr int kBatchMinM = 7;
// In a batch's graph the column-cube walks run in kBatchBranches parallel
// branches, largest first, each with a CTA per 64 cubes of its threads, so
// that small ones share the device: smallest order, and at most so many walks
// (the largest orders), since a graph node takes some 10 us to instantiate.
// 1024 matrices of orders 12..28: 24.9 ms from order 25 on, 23.4 from 24, 22.7
// from 23, 22.3 from 22, 21.9 from 21 (and 3 ms more of set-up); 8 branches
// 22.4, 32 branches 22.1.
constexpr int kBatchCubeMinN = 22;
constexpr int kBatchBranches = 16;
constexpr size_t kBatchMaxCubes = 4096;

struct perm_ctx {
  int device = 0;
  int num_sms = 0;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  // scratch, allocated once
  dd* partials = nullptr;  // kMaxBlocks dd
  unsigned* ticket = nullptr;
  // One block, read back by one copy: [0..7] results, [8] d_err, [9..10]
  // d_counters, [12..14] d_est, from kOutWords on the partial sums of column cubes
  // or of the term-moment sample.
  double* d_out = nullptr;
  int* d_err = nullptr;
  unsigned long long* d_counters = nullptr;  // [0] queue head, [1] visited
  double* h_out = nullptr;                   // pinned copy of the block
  // growable staging
  unsigned char* d_stage = nullptr;
  size_t d_stage_cap = 0;
  unsigned char* h_stage = nullptr;
  size_t h_stage_cap = 0;
  double* d_trials = nullptr;
  size_t d_trials_cap = 0;
  // occupancy per kernel family and order: [0] FP64-X, [G] int32-X, [7] dd,
  // [8 + G - 3] tensor core, [12] split X, [13 + G - 3] certified int32-X,
  // [17] split-dd dense, [18 + i] split-dd sparse with kSparseInner[i] inner rows
  // (i < 4; [43 + i - 4] for the others), [46 + i] FP64-X in the two-level
  // layout with k2lInner[i] inner rows, [50 + 6 (G - 4) + 2 (ng1 - 2) + ng2 - 1]
  // int32-X in the three-level layout, [68 + 6 family + 2 (ng1 - 2) + ng2 - 1]
  // certified int32-X in the three-level layout, [86 + 4 (R2 / 4 - 4) +
  // R1 / 4 - 2] split-dd in the three-level layout, [102 + 4 i + R1 / 4 - 2]
  // FP64 X in the three-level layout with kFp3lR2[i],
  // [22 + G - 4] certified int32-X with exact pairs of groups, [25 + 3 (G - 4)
  // + ngo - 1] int32-X in the two-level row layout, [34 + 3 family + ngo - 1]
  // certified int32-X in the two-level layout
  int dense_occ[122][PERM_MAX_EXACT_N + 1] = {};
  int cube_occ[kCubeKinds][kCubeShapeCount] = {};  // column-cube walks
  int batch_m[kBatchMaxOrder + 1] = {};          // autotuned lane-range exponents (0: default)
  int dense_pref[PERM_MAX_EXACT_N + 1] = {};     // autotuned kernel for integer inputs (0: built-in choice)
  double rel_target = 1e-10;                     // rerun in double-double above this estimate (<=0: never)
  double* d_est = nullptr;  // [0..1] sample-kernel / walk moment accumulators, [2] size-estimate sum
  double split_m1 = 0, split_m2 = 0;             // last split-X walk: sum |term|, sum term^2
  double walk_m1 = 0;                            // last certified (int32-X dd or split-dd) walk: sum |term|
  uint64_t walk_terms_per_thread = 0;            // ... and its longest thread range
  int inject_timeouts = 0;                       // failure injection: launches left to inject into
  int batch_occ[kBatchVariantCount] = {};  // CTAs per SM of each batch kernel variant
  int batch_variant = 0;                   // autotuned batch kernel variant (kBatchVariants)
  std::string err;
  std::mutex mu;
};

static const int kMaxBlocks = 8192;
// Column-cube walks recompute b after this many cubes (2^12 terms): its
// updates' roundings add up over 256 steps, in the row layouts over up to 2^12,
// and the n (n - 5) additions are below 2% of the segment.
constexpr uint64_t kCubeSegment = 256;

static int fail(perm_ctx* ctx, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (ctx) ctx->err = buf;
  return code;
}
static int fail_cuda(perm_ctx* ctx, cudaError_t e, const char* what) {
  cudaGetLastError();  // clear sticky-free errors
  return fail(ctx, e == cudaErrorMemoryAllocation ? PERM_ENOMEM : PERM_ECUDA, "%s: %s (%s)", what,
              cudaGetErrorName(e), cudaGetErrorString(e));
}
#define CU(ctx, expr)                                     \
  do {                                                    \
    cudaError_t _e = (expr);                              \
    if (_e != cudaSuccess) return fail_cuda(ctx, _e, #expr); \
  } while (0)

static int ensure_stage(perm_ctx* ctx, size_t bytes) {
  bytes = (bytes + 255) & ~(size_t)255;
  if (bytes > ctx->d_stage_cap) {
    if (ctx->d_stage) cudaFree(ctx->d_stage);
    ctx->d_stage = nullptr;
    ctx->d_stage_cap = 0;
    CU(ctx, cudaMalloc(&ctx->d_stage, bytes));
    ctx->d_stage_cap = bytes;
  }
  if (bytes > ctx->h_stage_cap) {
    if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
    ctx->h_stage = nullptr;
    ctx->h_stage_cap = 0;
    CU(ctx, cudaMallocHost(&ctx->h_stage, bytes));
    ctx->h_stage_cap = bytes;
  }
  return PERM_OK;
}

static double elem(const void* mat, int dtype, size_t idx) {
  switch (dtype) {
    case PERM_F32: return (double)static_cast<const float*>(mat)[idx];
    case PERM_I32: return (double)static_cast<const int*>(mat)[idx];
    default: return static_cast<const double*>(mat)[idx];
  }
}

// Column-major, even-stride copy of a row-major host matrix.
static void pack_columns(const void* mat, int n, int dtype, double* dst) {
  const int np = (n + 1) & ~1;
  for (int k = 0; k < n; k++) {
    for (int j = 0; j < n; j++) dst[(size_t)k * np + j] = elem(mat, dtype, (size_t)j * n + k);
    for (int j = n; j < np; j++) dst[(size_t)k * np + j] = 0.0;
  }
}

// Raise a kernel's dynamic shared-memory limit to the device's opt-in
// maximum, once per (device, kernel).  The limit is a per-function setting
// shared by every thread of the process: setting it to each call's own size
// would let a concurrent call shrink it between another call's set and
// launch, so it is only ever raised, to one fixed value.
static int allow_smem(perm_ctx* ctx, const void* fn, size_t need) {
  static std::mutex mu;
  static std::vector<std::pair<std::pair<int, const void*>, size_t>> done;
  std::lock_guard<std::mutex> lock(mu);
  for (auto& d : done)
    if (d.first.first == ctx->device && d.first.second == fn) {
      if (need > d.second) return fail(ctx, PERM_EUNSUPPORTED, "kernel needs %zu B of shared memory (max %zu)", need, d.second);
      return PERM_OK;
    }
  int optin = 0;
  CU(ctx, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, ctx->device));
  cudaFuncAttributes fa;
  CU(ctx, cudaFuncGetAttributes(&fa, fn));
  const size_t maxdyn = (size_t)optin > fa.sharedSizeBytes ? (size_t)optin - fa.sharedSizeBytes : 0;
  CU(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)maxdyn));
  done.push_back({{ctx->device, fn}, maxdyn});
  if (need > maxdyn) return fail(ctx, PERM_EUNSUPPORTED, "kernel needs %zu B of shared memory (max %zu)", need, maxdyn);
  return PERM_OK;
}

// ---------------------------------------------------------------------------
// context
// ---------------------------------------------------------------------------
extern "C" int perm_version(void) { return 10000; }

extern "C" int perm_device_count(void) {
  int c = 0;
  if (cudaGetDeviceCount(&c) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  return c;
}

extern "C" const char* perm_status_string(int s) {
  switch (s) {
    case PERM_OK: return "ok";
    case PERM_EINVAL: return "invalid argument";
    case PERM_ECUDA: return "CUDA error";
    case PERM_ENOMEM: return "out of memory";
    case PERM_EUNSUPPORTED: return "unsupported";
    case PERM_ETIMEOUT: return "device wait timed out";
    case PERM_EIO: return "matrix input error";
    default: return "unknown status";
  }
}

extern "C" const char* perm_ctx_last_error(const perm_ctx* ctx) { return ctx ? ctx->err.c_str() : ""; }

extern "C" void perm_ctx_destroy(perm_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->device);
  if (ctx->stream) cudaStreamSynchronize(ctx->stream);
  cudaFree(ctx->partials);
  cudaFree(ctx->ticket);
  cudaFree(ctx->d_out);
  cudaFree(ctx->d_stage);
  cudaFree(ctx->d_trials);
  if (ctx->h_out) cudaFreeHost(ctx->h_out);
  if (ctx->h_stage) cudaFreeHost(ctx->h_stage);
  if (ctx->ev0) cudaEventDestroy(ctx->ev0);
  if (ctx->ev1) cudaEventDestroy(ctx->ev1);
  if (ctx->stream) cudaStreamDestroy(ctx->stream);
  delete ctx;
}

static int ctx_init(perm_ctx* ctx, int device) {
  int count = 0;
  CU(ctx, cudaGetDeviceCount(&count));
  if (device < 0 || device >= count)
    return fail(ctx, PERM_EINVAL, "device %d not in [0, %d)", device, count);
  ctx->device = device;
  CU(ctx, cudaSetDevice(device));
  cudaDeviceProp prop;
  CU(ctx, cudaGetDeviceProperties(&prop, device));
  if (prop.major != 10)
    return fail(ctx, PERM_EUNSUPPORTED, "device %d is sm_%d%d; this build targets sm_100a (B200)", device,
                prop.major, prop.minor);
  ctx->num_sms = prop.multiProcessorCount;
  CU(ctx, cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
  CU(ctx, cudaEventCreate(&ctx->ev0));
  CU(ctx, cudaEventCreate(&ctx->ev1));
  CU(ctx, cudaMalloc(&ctx->partials, sizeof(dd) * kMaxBlocks * 2));
  CU(ctx, cudaMalloc(&ctx->ticket, sizeof(unsigned) * 4));
  const size_t out_words = kOutWords + std::max((size_t)ctx->num_sms * kCubeBlocks * kCubeWords,
                                                (size_t)2 * moment_blocks(PERM_MAX_EXACT_N));
  CU(ctx, cudaMalloc(&ctx->d_out, sizeof(double) * out_words));
  ctx->d_err = reinterpret_cast<int*>(ctx->d_out + 8);
  ctx->d_counters = reinterpret_cast<unsigned long long*>(ctx->d_out + 9);
  ctx->d_est = ctx->d_out + 12;
  CU(ctx, cudaMemset(ctx->ticket, 0, sizeof(unsigned) * 4));
  CU(ctx, cudaMemset(ctx->d_out, 0, sizeof(double) * out_words));
  CU(ctx, cudaMallocHost(&ctx->h_out, sizeof(double) * out_words));
  return PERM_OK;
}

extern "C" int perm_ctx_create(int device, perm_ctx** out) {
  if (!out) return PERM_EINVAL;
  *out = nullptr;
  perm_ctx* ctx = new perm_ctx();
  int rc = ctx_init(ctx, device);
  if (rc != PERM_OK) {
    // keep the message for the caller through a static copy
    static thread_local std::string last;
    last = ctx->err;
    fprintf(stderr, "perm_ctx_create: %s\n", last.c_str());
    perm_ctx_destroy(ctx);
    return rc;
  }
  *out = ctx;
  return PERM_OK;
}

// Reads back the result block (results, error flag, counters, moments) after
// the stream drains, with `partials` words of partial sums; `meanwhile` runs on
// the host before the wait.
template <class Meanwhile>
static int finish_and_read(perm_ctx* ctx, int partials, Meanwhile meanwhile) {
  CU(ctx, cudaMemcpyAsync(ctx->h_out, ctx->d_out, sizeof(double) * (kOutWords + partials), cudaMemcpyDeviceToHost,
                          ctx->stream));
  meanwhile();
  CU(ctx, cudaStreamSynchronize(ctx->stream));
  CU(ctx, cudaGetLastError());
  int errflag = 0;
  memcpy(&errflag, ctx->h_out + 8, sizeof(int));
  if (errflag) {
    cudaMemsetAsync(ctx->d_err, 0, sizeof(int), ctx->stream);
    cudaStreamSynchronize(ctx->stream);
    return fail(ctx, PERM_ETIMEOUT, "%s wait timed out on device %d",
                errflag == 3 ? "tensor-core pipeline" : "shared-memory staging", ctx->device);
  }
  return PERM_OK;
}

static int finish_and_read(perm_ctx* ctx) {
  return finish_and_read(ctx, 0, [] {});
}

// ---------------------------------------------------------------------------
// dense exact
// ---------------------------------------------------------------------------
// A dense operand in its device image: FP64 columns (np = n rounded up to
// even) for the FP64-X kernel, or doubled int32 columns plus y0 (np4 = n
// rounded up to a multiple of 4) for the int32-X kernel.
struct DenseOperand {
  int n = 0, variant = PERM_KERNEL_DENSE, group = 0;
  int pair = 0;   // certified int32-X walk: consecutive groups multiplied in exact FP64 pairs
  int ngo = 0;    // int32-X walk: outer product groups of the two-level row layout (0: one level)
  int ng1 = 0, ng2 = 0;  // int32-X walk: groups of the three-level layout's first and second level (0: not)
  int inner = 0;  // split-dd and FP64 X: rows 0..inner-1 hold the support of columns 0..2 (0: one level)
  int inner1 = 0;  // split-dd three-level layout: rows 0..inner1-1 hold column 0's support (0: not)
  int shape = -1;  // column-cube walk (ryser_cube.cuh): its shape, -1: one of the row layouts above
  bool abs_sum = false;  // ... which sums |term| too (FP64 walk; the certified ones always do)
  int exp2 = 0;  // ... whose results are multiplied by 2^exp2
  std::vector<double> sums;  // ... and the fast columns' sums, then (split-dd) those of their remainders
  std::vector<unsigned char> image;
};

// Row absolute sums of an integer-valued matrix with |a| < 2^24 (each bounds
// |y_j| = |2 x_j| along the whole walk); false for other matrices.
static bool int_row_abs(const std::vector<double>& a, int n, std::vector<double>& rowabs) {
  rowabs.assign(n, 0.0);
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++) {
      const double v = a[(size_t)j * n + k];
      if (v != std::floor(v) || std::fabs(v) >= 16777216.0) return false;
      rowabs[j] += std::fabs(v);
    }
  return true;
}

// Whether every run of `span` consecutive rows starting at multiples of
// `span` has prod(max(sum_k |a_jk|, 1)) below `limit`.
static bool runs_fit(const std::vector<double>& rowabs, int n, int span, double limit) {
  for (int j0 = 0; j0 < n; j0 += span) {
    double b = 1.0;
    for (int t = 0; t < span && j0 + t < n; t++) b *= std::max(rowabs[j0 + t], 1.0);
    if (!(b < limit)) return false;
  }
  return true;
}

// Integer-valued with |a| < 2^24 and a product grouping that provably fits in
// int32: returns the largest group size G in {6,5,4,3} such that every run of
// G consecutive rows has prod(sum_k |a_jk|) < 2^31, or 0.
static int int_group_size(const std::vector<double>& a, int n) {
  if (n < 8) return 0;
  std::vector<double> rowabs;
  if (!int_row_abs(a, n, rowabs)) return 0;
  for (int G = 6; G >= 3; G--)
    if (runs_fit(rowabs, n, G, 2147483648.0)) return G;
  return 0;
}

// Layout of the certified int32-X walk (ryser_dense_intc.cuh): product
// groups of G rows (each |product| < 2^31) whose values enter a
// double-double product, optionally (*pair, orders >= 16, G >= 4) first
// multiplied in consecutive pairs in int64, exact when every run of 2G rows
// has prod(sum_k |a_jk|) < 2^53.  Per Gray step a chain of g groups costs
// n - g int32 multiplies, g conversions and 3g - 4 double-double operations;
// pairs cost n - g multiplies, floor(g/2) 64-bit multiplies, f = ceil(g/2)
// conversions and 3f - 4 operations; the layout with the fewest instructions
// is taken.  Returns G, or 0 when int32 X does not apply.
static int intc_layout(const std::vector<double>& a, int n, int* pair, int* cost_out = nullptr) {
  *pair = 0;
  if (n < 8) return 0;
  std::vector<double> rowabs;
  if (!int_row_abs(a, n, rowabs)) return 0;
  int best_g = 0, best_pair = 0, best_cost = 1 << 30;
  for (int G = 6; G >= 3; G--) {
    if (!runs_fit(rowabs, n, G, 2147483648.0)) continue;
    const int ng = (n + G - 1) / G;
    const int chain = n + 3 * ng - 4;
    if (chain < best_cost) best_g = G, best_pair = 0, best_cost = chain;
    if (n >= 16 && G >= 4 && runs_fit(rowabs, n, 2 * G, 9007199254740992.0)) {
      const int nf = (ng + 1) / 2, paired = n - ng + ng / 2 + 4 * nf - 4;
      if (paired < best_cost) best_g = G, best_pair = 1, best_cost = paired;
    }
  }
  *pair = best_pair;
  if (cost_out) *cost_out = best_cost;
  return best_g;
}

// The tensor-core kernel takes int8 operands: |2a| <= 127, which also keeps
// every row-sum value within its three base digits (|y| <= 63 x 64 = 4032).
static bool tc_eligible(const std::vector<double>& a, int n) {
  if (n < 16 || n > 64) return false;
  for (double v : a)
    if (std::fabs(v) > 63.0) return false;
  return true;
}

// Split-X operand (ryser_dense_split.cuh): every entry a = ah + al with ah on
// its row's grid 2^-q_j, q_j chosen so that partial row sums of coarse parts
// are exact in FP64 (rows scale independently: x_j only sums row j); x0
// likewise, from its double-double value.
// Image: [ah column-major, stride np][al][x0h][x0l].
// Rows whose absolute sum reaches 2^1020 are outside the split: their coarse
// grid 2^-q_j would be coarser than 2^971, and a coarse part rounded up to
// the top of that grid can overflow to infinity.
static bool split_rows_ok(const std::vector<double>& a, int n) {
  for (int j = 0; j < n; j++) {
    double r = 0.0;
    for (int k = 0; k < n; k++) r += std::fabs(a[(size_t)j * n + k]);
    if (!std::isfinite(r) || (r > 0.0 && std::ilogb(r) >= 1020)) return false;
  }
  return true;
}

static int build_split_operand(perm_ctx* ctx, const std::vector<double>& a, int n, DenseOperand* op) {
  if (n < 4 || n > 40) return fail(ctx, PERM_EUNSUPPORTED, "split-X kernel covers orders 4..40 (got %d)", n);
  if (!split_rows_ok(a, n))
    return fail(ctx, PERM_EUNSUPPORTED, "split-X kernel needs row absolute sums below 2^1020");
  // per row: grid 2^-q_j with 2^(51 - q_j) > 4 sum_k |a_jk|, so every partial
  // sum of coarse parts (at most 1.5x the row's absolute sum plus n half
  // grid steps) is an integer multiple of 2^-q_j below 2^51 of them
  std::vector<int> q(n, 0);
  for (int j = 0; j < n; j++) {
    double r = 0.0;
    for (int k = 0; k < n; k++) r += std::fabs(a[(size_t)j * n + k]);
    if (r > 0.0) q[j] = std::min(1000, std::max(-1000, 51 - (std::ilogb(r) + 3)));
  }
  auto coarse = [&q](double v, int j) { return std::ldexp(std::nearbyint(std::ldexp(v, q[j])), -q[j]); };
  const int np = (n + 1) & ~1;
  op->n = n;
  op->variant = PERM_KERNEL_DENSE_SPLIT;
  op->group = 0;
  op->image.assign(sizeof(double) * (2 * (size_t)n * np + 2 * (size_t)np), 0);
  double* img = reinterpret_cast<double*>(op->image.data());
  double* H = img;
  double* L = img + (size_t)n * np;
  double* X0h = L + (size_t)n * np;
  double* X0l = X0h + np;
  for (int k = 0; k < n; k++)
    for (int j = 0; j < n; j++) {
      const double v = a[(size_t)j * n + k], h = coarse(v, j);
      H[(size_t)k * np + j] = h;
      L[(size_t)k * np + j] = v - h;  // exact
    }
  for (int j = 0; j < n; j++) {
    // x0 = a[j][n-1] - rowsum_j / 2 in double-double
    double hi = 0.0, lo = 0.0;
    for (int k = 0; k < n; k++) {
      const double v = a[(size_t)j * n + k], sum = hi + v, bb = sum - hi;
      lo += (hi - (sum - bb)) + (v - bb);
      hi = sum;
    }
    hi *= -0.5;
    lo *= -0.5;
    const double v = a[(size_t)j * n + n - 1], sum = hi + v, bb = sum - hi;
    lo += (hi - (sum - bb)) + (v - bb);
    hi = sum;
    const double h = coarse(hi, j);
    X0h[j] = h;
    X0l[j] = (hi - h) + lo;
  }
  return PERM_OK;
}

// The three columns whose nonzeros lie in the fewest rows: returns the size
// of that row set and the columns.  Exact search over column triples in
// order of increasing column count; a triple's row set is at least as large
// as its largest column, so the search stops once that reaches the best set
// found (for the batch's 8192 matrices this visits a few hundred triples each
// instead of C(n, 3)).
static int sparsest_column_triple(const std::vector<double>& a, int n, int* c3) {
  std::vector<uint64_t> sup(n, 0);
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++)
      if (a[(size_t)j * n + k] != 0.0) sup[k] |= 1ull << j;
  std::vector<int> ord(n);
  for (int k = 0; k < n; k++) ord[k] = k;
  std::stable_sort(ord.begin(), ord.end(),
                   [&](int x, int y) { return __builtin_popcountll(sup[x]) < __builtin_popcountll(sup[y]); });
  int best = n + 1;
  c3[0] = 0;
  c3[1] = 1;
  c3[2] = 2;
  for (int z = 2; z < n; z++) {  // z: the triple's column with the most nonzeros
    if (__builtin_popcountll(sup[ord[z]]) >= best) break;
    for (int y = 1; y < z; y++)
      for (int x = 0; x < y; x++) {
        const int pc = __builtin_popcountll(sup[ord[x]] | sup[ord[y]] | sup[ord[z]]);
        if (pc < best) {
          best = pc;
          int t[3] = {ord[x], ord[y], ord[z]};
          std::sort(t, t + 3);
          c3[0] = t[0];
          c3[1] = t[1];
          c3[2] = t[2];
        }
      }
  }
  return best;
}

// Inner-row count of the sparse split-dd layout for this matrix (0: dense
// layout): the smallest kSparseInner entry that holds the rows of the three
// sparsest columns, for orders 12..40.  Inner-row counts of 20 and more
// (the rolled two-level walk of dense matrices) are taken when their
// (7 (6R + 13) + 12n - 6R + 20) / 8 FP64 operations per step are at most
// 0.85 of the dense layout's 6n + 10 (measured: n = 32 with 20 inner rows
// 27.2 against 38.0 ms, n = 34 with 24 inner rows 123 against 156 ms).
static int sdd_inner_rows(const std::vector<double>& a, int n, int* c3) {
  if (n < 12 || n > 40) return 0;
  const int u = sparsest_column_triple(a, n, c3);
  for (int r : kSparseInner)
    if (u <= r && r + 4 <= n) {
      if (r >= 20 && 7 * (6 * r + 13) + 12 * n - 6 * r + 20 > 0.85 * 8 * (6 * n + 10)) return 0;
      return r;
    }
  return 0;
}

// Split-dd operand (ryser_dense_sdd.cuh): the split-X image, of the matrix
// itself (dense layout) or, when three columns have their nonzeros in at
// most 16 rows, of the matrix with those columns moved to positions 0..2
// and their rows to the top (the sparse layout; the permanent is invariant
// under row and column permutations).
// The sparse layout's permutation: columns c3[0..2] move to positions 0..2
// (the others keep their order), the rows where any of them is nonzero to
// the top (in order), the other rows after them.  The permanent is
// invariant under row and column permutations.
static std::vector<double> sparse_permutation(const double* a, int n, const int* c3) {
  std::vector<int> cols = {c3[0], c3[1], c3[2]}, rows;
  for (int k = 0; k < n; k++)
    if (k != c3[0] && k != c3[1] && k != c3[2]) cols.push_back(k);
  std::vector<char> in_union(n, 0);
  for (int j = 0; j < n; j++)
    for (int t = 0; t < 3; t++)
      if (a[(size_t)j * n + c3[t]] != 0.0) in_union[j] = 1;
  for (int j = 0; j < n; j++)
    if (in_union[j]) rows.push_back(j);
  for (int j = 0; j < n; j++)
    if (!in_union[j]) rows.push_back(j);
  std::vector<double> p((size_t)n * n);
  for (int i = 0; i < n; i++)
    for (int k = 0; k < n; k++) p[(size_t)i * n + k] = a[(size_t)rows[i] * n + cols[k]];
  return p;
}

// Two-level row layout of the int32-X walk (ryser_dense_int_sparse.cuh): the
// three columns whose nonzeros lie in the fewest rows move to positions 0..2
// and those rows to the top (sparse_permutation); the remaining rows form
// ngo whole product groups that columns 0..2 never touch.  Per 8 Gray steps
// the one-level walk with groups of G costs about 8 (2n + ceil(n/G)) integer
// and FP64 instructions, the two-level one 7 (2 RI + ceil(RI/G) + 1) +
// 2n + ceil(n/G) + ngo with RI = n - ngo G inner rows.  Takes the cheapest
// (G, ngo), G in 4..6 up to the one-level G, ngo in 1..3, among layouts
// whose every group product provably fits int32 in this grouping (inner
// groups from row 0, outer groups from row RI); *perm receives the permuted
// matrix.  False when the one-level walk is as cheap.
static bool int_two_level_layout(const std::vector<double>& a, int n, int g1, int* g_out, int* ngo_out,
                                 std::vector<double>* perm) {
  if (n < kIntSparseMinN || n > kIntSparseMaxN || g1 < 4) return false;
  int c3[3];
  const int support = sparsest_column_triple(a, n, c3);
  const int outer = n - support;
  if (outer < 4) return false;
  std::vector<double> p = sparse_permutation(a.data(), n, c3);
  std::vector<double> rowabs;
  if (!int_row_abs(p, n, rowabs)) return false;
  auto fits = [&](int g, int ngo) {
    const int ri = n - g * ngo;
    auto run = [&](int j0, int j1) {
      double b = 1.0;
      for (int j = j0; j < j1; j++) b *= std::max(rowabs[j], 1.0);
      return b < 2147483648.0;
    };
    for (int j = 0; j < ri; j += g)
      if (!run(j, std::min(j + g, ri))) return false;
    for (int t = 0; t < ngo; t++)
      if (!run(ri + t * g, ri + t * g + g)) return false;
    return true;
  };
  const long best_one = 8L * (2 * n + (n + g1 - 1) / g1);
  long best = best_one;
  for (int g = std::min(g1, 6); g >= 4; g--)
    for (int ngo = std::min(kIntSparseMaxOuter, outer / g); ngo >= 1; ngo--) {
      const int ri = n - g * ngo;
      if (ri < 3) continue;
      const long cost = 7L * (2 * ri + (ri + g - 1) / g + 1) + 2 * n + (n + g - 1) / g + ngo;
      if (cost < best && fits(g, ngo)) {
        best = cost;
        *g_out = g;
        *ngo_out = ngo;
      }
    }
  if (best == best_one) return false;
  *perm = std::move(p);
  return true;
}

// Three-level row layout (ryser_dense_int_3l_kernel,
// ryser_dense_intc_3l_kernel): column 0 (flipped at every other Gray step)
// touches rows [0, R1) only, columns 1 and 2 (three steps in eight) rows
// [0, R2) only, with R1 = ng1 g and R2 = R1 + ng2 g; rows of a later level
// may fill an earlier one (their zero entries there make the extra updates
// no-ops).  For levels of g rows, searches every column for column 0 and
// every pair for columns 1, 2 (within `lim`; the int32-X walks: orders
// 28..48, ng1 in 2..4, ng2 in 1..2) for the fewest rows updated per 8
// steps, 4 R1 + 3 R2, and returns the permuted matrix; false when no layout
// fits.
struct LevelLimits {
  int n_lo, n_hi;                              // orders
  int ng1_lo, ng1_hi, ng2_hi, tot_lo, tot_hi;  // first-level and second-level groups, their sum
};
constexpr LevelLimits kIntLevels = {kInt3lMinN, kIntSparseMaxN, 2, 4, 2, 0, 1 << 20};

static bool three_level_permutation(const std::vector<double>& a, int n, int g, int* ng1_out, int* ng2_out,
                                    std::vector<double>* perm, const LevelLimits& lim = kIntLevels) {
  if (n < lim.n_lo || n > lim.n_hi) return false;
  std::vector<uint64_t> sup(n, 0);
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++)
      if (a[(size_t)j * n + k] != 0.0) sup[k] |= 1ull << j;
  long best = -1;
  int bc[3] = {0, 0, 0}, b1 = 0, b2 = 0;
  for (int c0 = 0; c0 < n; c0++) {
    const int ng1 = std::max(lim.ng1_lo, (__builtin_popcountll(sup[c0]) + g - 1) / g);
    if (ng1 > lim.ng1_hi) continue;
    for (int c1 = 0; c1 < n; c1++) {
      if (c1 == c0) continue;
      for (int c2 = c1 + 1; c2 < n; c2++) {
        if (c2 == c0) continue;
        const int u = __builtin_popcountll(sup[c0] | sup[c1] | sup[c2]);
        const int ng2 = std::max({1, lim.tot_lo - ng1, (u - ng1 * g + g - 1) / g});
        if (ng2 > lim.ng2_hi || ng1 + ng2 > lim.tot_hi || (ng1 + ng2) * g + 2 > n) continue;
        const long rows = 4L * ng1 * g + 3L * (ng1 + ng2) * g;
        if (best < 0 || rows < best) {
          best = rows;
          bc[0] = c0, bc[1] = c1, bc[2] = c2, b1 = ng1, b2 = ng2;
        }
      }
    }
  }
  if (best < 0) return false;
  const int r1 = b1 * g, r2 = r1 + b2 * g;
  const uint64_t s0 = sup[bc[0]], s12 = sup[bc[1]] | sup[bc[2]];
  if (__builtin_popcountll(s0 | s12) > r2) return false;
  // rows: level 1 = support of column c0, filled up to R1 with rows of the
  // other two columns' support, then of the rest; level 2 likewise to R2
  std::vector<int> rows, pool;
  for (int j = 0; j < n; j++)
    if ((s0 >> j) & 1) rows.push_back(j);
  for (int j = 0; j < n; j++)
    if (!((s0 >> j) & 1) && ((s12 >> j) & 1)) pool.push_back(j);
  for (int j = 0; j < n; j++)
    if (!(((s0 | s12) >> j) & 1)) pool.push_back(j);
  size_t pi = 0;
  while ((int)rows.size() < r2) rows.push_back(pool[pi++]);
  while (pi < pool.size()) rows.push_back(pool[pi++]);
  std::vector<int> cols = {bc[0], bc[1], bc[2]};
  for (int k = 0; k < n; k++)
    if (k != bc[0] && k != bc[1] && k != bc[2]) cols.push_back(k);
  std::vector<double> p((size_t)n * n);
  for (int i = 0; i < n; i++)
    for (int k = 0; k < n; k++) p[(size_t)i * n + k] = a[(size_t)rows[i] * n + cols[k]];
  *ng1_out = b1;
  *ng2_out = b2;
  *perm = std::move(p);
  return true;
}

// FP64 operations per 8 Gray steps of the split-dd layouts: dense, sparse
// (inner rows r; unrolled below 20, rolled from 20) and three-level
// (ryser_sdd_3l_kernel, levels ending at r1 and r2).
static long sdd_cost(int n, int r, int r1 = 0, int r2 = 0) {
  if (r1) return 24L * r1 + 18L * r2 + 6L * n + 116;
  if (!r) return 8L * (6 * n + 10);
  if (r < 20) return 7L * (6 * r + 9) + 6L * n + 5;
  return 7L * (6 * r + 13) + 12L * n - 6L * r + 20;
}

// Three-level layout of the split-dd walk, levels of 4 rows: first level
// 8..20 rows, second level ending at 16..28, orders 24..40.
constexpr LevelLimits kSddLevels = {kSdd3lMinN, 40, 2, 5, 5, 4, 7};

// Layout of the split-dd walk for this matrix: the sparse layout's inner
// rows (sdd_inner_rows), or the three-level layout when its cost per 8
// steps is lower; *inner = rows in registers (0: dense layout), *inner1 =
// the three-level layout's first level (0: not), *perm = the permuted
// matrix for the sparse and three-level layouts.
static void sdd_choose(const std::vector<double>& a, int n, int* inner, int* inner1, std::vector<double>* perm) {
  int c3[3] = {0, 1, 2};
  *inner = sdd_inner_rows(a, n, c3);
  *inner1 = 0;
  int ng1 = 0, ng2 = 0;
  std::vector<double> three;
  if (three_level_permutation(a, n, 4, &ng1, &ng2, &three, kSddLevels) &&
      sdd_cost(n, 0, 4 * ng1, 4 * (ng1 + ng2)) < sdd_cost(n, *inner)) {
    *inner = 4 * (ng1 + ng2);
    *inner1 = 4 * ng1;
    *perm = std::move(three);
    return;
  }
  if (*inner) *perm = sparse_permutation(a.data(), n, c3);
}

// Three-level layout of the int32-X walk: per 8 steps about
// 4 (2 R1 + 2 ng1) + 3 (2 R2 + 2 (ng1 + ng2) + 1) + 2n + 2 ceil(n/G)
// instructions; G in 4..6 up to the one-level G; the cheapest layout below
// `best_cost` whose groups provably fit int32.
static bool int_three_level_layout(const std::vector<double>& a, int n, int g1, long best_cost, int* g_out,
                                   int* ng1_out, int* ng2_out, std::vector<double>* perm, long* cost_out) {
  if (g1 < 4) return false;
  long best = best_cost;
  for (int g = std::min(g1, 6); g >= 4; g--) {
    int ng1 = 0, ng2 = 0;
    std::vector<double> p;
    if (!three_level_permutation(a, n, g, &ng1, &ng2, &p)) continue;
    const int r1 = ng1 * g, r2 = r1 + ng2 * g;
    const long cost = 4L * (2 * r1 + 2 * ng1) + 3L * (2 * r2 + 2 * (ng1 + ng2) + 1) + 2 * n + 2 * ((n + g - 1) / g);
    if (cost >= best) continue;
    std::vector<double> rowabs;
    if (!int_row_abs(p, n, rowabs) || !runs_fit(rowabs, n, g, 2147483648.0)) continue;
    best = cost;
    *g_out = g;
    *ng1_out = ng1;
    *ng2_out = ng2;
    *perm = std::move(p);
  }
  *cost_out = best;
  return best != best_cost;
}

// Layout of the int32-X walk with product groups of G (int_group_size): one
// level, two levels (int_two_level_layout) or three (int_three_level_layout),
// whichever costs least; *perm receives the permuted matrix of the two- and
// three-level layouts.
struct IntLayout {
  int g, ngo, ng1, ng2;
};
static IntLayout choose_int_layout(const std::vector<double>& a, int n, int G, std::vector<double>* perm,
                                   long* cost_out = nullptr) {
  IntLayout l = {G, 0, 0, 0};
  long cost = 8L * (2 * n + (n + G - 1) / G);
  int g2 = G, ngo2 = 0, g3 = G, a1 = 0, a2 = 0;
  std::vector<double> two, three;
  if (int_two_level_layout(a, n, G, &g2, &ngo2, &two)) {
    const int ri = n - g2 * ngo2;
    cost = 7L * (2 * ri + (ri + g2 - 1) / g2 + 1) + 2 * n + (n + g2 - 1) / g2 + ngo2;
  }
  if (int_three_level_layout(a, n, G, cost, &g3, &a1, &a2, &three, &cost)) {
    l = {g3, 0, a1, a2};
    *perm = std::move(three);
  } else if (ngo2) {
    l = {g2, ngo2, 0, 0};
    *perm = std::move(two);
  }
  if (cost_out) *cost_out = cost;
  return l;
}

// Inner-row count of the FP64-X walk's two-level layout (ryser_dense_2l.cuh;
// 0: one level): the smallest of 16, 20, 24, 28 that holds the rows of the
// three sparsest columns, orders 20..48, when the seven inner steps' 2R + 1
// operations keep the 8-step cost 7 (2R + 1) + 2n within 0.85 of the
// one-level walk's 16n (measured: n = 34 with 24 inner rows 29.6 against
// 37.6 ms, n = 40 with 28, 2120 against 2773 ms).
static int fp64_two_level_rows(const std::vector<double>& a, int n, int* c3) {
  if (n < 20 || n > 48) return 0;
  const int u = sparsest_column_triple(a, n, c3);
  for (int r : k2lInner)
    if (u <= r && r + 4 <= n) return 7 * (2 * r + 1) + 2 * n <= 0.85 * 16 * n ? r : 0;
  return 0;
}

// Three-level layout of the FP64-X walk (ryser_dense_3l_kernel), levels of 4
// rows: first level 8..20 rows, second ending at 20..36, orders 28..48.
constexpr LevelLimits kFp64Levels = {28, 48, 2, 5, 7, 5, 9};

// Layout of the FP64-X walk for this matrix: *inner = the two-level
// layout's inner rows (fp64_two_level_rows) or the three-level layout's
// second level R2, 0 for one level; *inner1 = the three-level layout's
// first level R1 (0: not); *perm = the permuted matrix.  Per 8 steps the
// one-level walk costs 16n operations, the two-level 7 (2R + 1) + 2n, the
// three-level 8 R1 + 6 R2 + 2n + 13; the three-level layout is taken when
// cheapest.
static void fp64_choose(const std::vector<double>& a, int n, int* inner, int* inner1, std::vector<double>* perm,
                        long* cost8 = nullptr) {
  int c3[3] = {0, 1, 2};
  *inner = fp64_two_level_rows(a, n, c3);
  *inner1 = 0;
  const long cost = *inner ? 7L * (2 * *inner + 1) + 2L * n : 16L * n;
  if (cost8) *cost8 = cost;
  int ng1 = 0, ng2 = 0;
  std::vector<double> three;
  if (three_level_permutation(a, n, 4, &ng1, &ng2, &three, kFp64Levels) &&
      32L * ng1 + 24L * (ng1 + ng2) + 2L * n + 13 < cost) {
    *inner = 4 * (ng1 + ng2);
    *inner1 = 4 * ng1;
    *perm = std::move(three);
    if (cost8) *cost8 = 32L * ng1 + 24L * (ng1 + ng2) + 2L * n + 13;
    return;
  }
  if (*inner) *perm = sparse_permutation(a.data(), n, c3);
}

// Two-level row layout of the certified int32-X walk
// (ryser_dense_intc_sparse.cuh): the permutation of int_two_level_layout,
// with groups of 4 or 6 rows in int64 pairs or groups of 5 alone.  Per Gray
// step a level of r rows in g groups with f factors costs r - g int32
// multiplies, its 64-bit pair multiplies, f conversions and 3 double-double
// operations per factor; the inner level runs at every step, the outer one
// and the updates of all n rows at one step in eight.  Takes the cheapest
// layout among those whose group (< 2^31) and pair (< 2^53) products
// provably fit, and only when it beats the one-level layout `one_cost`
// (instructions per 8 steps).  *perm receives the permuted matrix.
static bool intc_two_level_layout(const std::vector<double>& a, int n, long one_cost, int* g_out, int* pair_out,
                                  int* ngo_out, std::vector<double>* perm, long* cost_out = nullptr) {
  if (n < kIntSparseMinN || n > kIntSparseMaxN) return false;
  int c3[3];
  const int support = sparsest_column_triple(a, n, c3);
  const int outer = n - support;
  if (outer < 4) return false;
  std::vector<double> p = sparse_permutation(a.data(), n, c3);
  std::vector<double> rowabs;
  if (!int_row_abs(p, n, rowabs)) return false;
  auto prod = [&](int j0, int j1) {
    double b = 1.0;
    for (int j = j0; j < j1; j++) b *= std::max(rowabs[j], 1.0);
    return b;
  };
  // groups of one level, rows [j0, j1) in runs of g
  auto level_fits = [&](int j0, int j1, int g, bool pair) {
    std::vector<std::pair<int, int>> grp;
    for (int j = j0; j < j1; j += g) grp.push_back({j, std::min(j + g, j1)});
    for (auto& r : grp)
      if (!(prod(r.first, r.second) < 2147483648.0)) return false;
    if (pair)
      for (size_t i = 0; i + 1 < grp.size(); i += 2)
        if (!(prod(grp[i].first, grp[i + 1].second) < 9007199254740992.0)) return false;
    return true;
  };
  auto level_cost = [&](int rows, int g, bool pair) {
    const int ng = (rows + g - 1) / g, f = pair ? (ng + 1) / 2 : ng;
    return (long)(rows - ng) + (pair ? ng / 2 : 0) + f + 3L * f;
  };
  long best = one_cost;
  const int fam_g[3] = {4, 5, 6};
  const bool fam_pair[3] = {true, false, true};
  for (int fam = 0; fam < 3; fam++) {
    const int g = fam_g[fam];
    const bool pair = fam_pair[fam];
    for (int ngo = std::min(kIntSparseMaxOuter, outer / g); ngo >= 1; ngo--) {
      const int ri = n - g * ngo;
      if (ri < 3) continue;
      const long inner = ri + level_cost(ri, g, pair);
      const long cost = 7 * inner + n + level_cost(ri, g, pair) + level_cost(n - ri, g, pair);
      if (cost < best && level_fits(0, ri, g, pair) && level_fits(ri, n, g, pair)) {
        best = cost;
        *g_out = g;
        *pair_out = pair ? 1 : 0;
        *ngo_out = ngo;
      }
    }
  }
  if (best == one_cost) return false;
  *perm = std::move(p);
  if (cost_out) *cost_out = best;
  return true;
}

// Three-level layout of the certified int32-X walk
// (ryser_dense_intc_3l_kernel): the rows of three_level_permutation, with
// the families of the two-level kernel (groups of 4 or 6 in int64 pairs, 5
// alone); per 8 steps 4 (R1 + c1) + 3 (R2 + c1 + c2) + n + c1 + c2 + c3,
// c the level costs of intc_two_level_layout; the cheapest below
// `best_cost` whose groups (< 2^31) and pairs (< 2^53) provably fit.
static bool intc_three_level_layout(const std::vector<double>& a, int n, long best_cost, int* g_out, int* pair_out,
                                    int* ng1_out, int* ng2_out, std::vector<double>* perm, long* cost_out = nullptr) {
  long best = best_cost;
  const int fam_g[3] = {4, 5, 6};
  const bool fam_pair[3] = {true, false, true};
  for (int fam = 0; fam < 3; fam++) {
    const int g = fam_g[fam];
    const bool pair = fam_pair[fam];
    int ng1 = 0, ng2 = 0;
    std::vector<double> p;
    if (!three_level_permutation(a, n, g, &ng1, &ng2, &p)) continue;
    std::vector<double> rowabs;
    if (!int_row_abs(p, n, rowabs)) continue;
    auto prod = [&](int j0, int j1) {
      double b = 1.0;
      for (int j = j0; j < j1; j++) b *= std::max(rowabs[j], 1.0);
      return b;
    };
    auto level_fits = [&](int j0, int j1) {
      std::vector<std::pair<int, int>> grp;
      for (int j = j0; j < j1; j += g) grp.push_back({j, std::min(j + g, j1)});
      for (auto& r : grp)
        if (!(prod(r.first, r.second) < 2147483648.0)) return false;
      if (pair)
        for (size_t i = 0; i + 1 < grp.size(); i += 2)
          if (!(prod(grp[i].first, grp[i + 1].second) < 9007199254740992.0)) return false;
      return true;
    };
    auto lc = [&](int rows) {
      const int ng = (rows + g - 1) / g, f = pair ? (ng + 1) / 2 : ng;
      return (long)(rows - ng) + (pair ? ng / 2 : 0) + f + 3L * f;
    };
    const int r1 = ng1 * g, r2 = r1 + ng2 * g;
    const long c1 = lc(r1), c2 = lc(r2 - r1), c3 = lc(n - r2);
    const long cost = 4 * (r1 + c1) + 3 * (r2 + c1 + c2) + n + c1 + c2 + c3;
    if (cost >= best || !level_fits(0, r1) || !level_fits(r1, r2) || !level_fits(r2, n)) continue;
    best = cost;
    *g_out = g;
    *pair_out = pair ? 1 : 0;
    *ng1_out = ng1;
    *ng2_out = ng2;
    *perm = std::move(p);
  }
  if (cost_out) *cost_out = best;
  return best != best_cost;
}

// Column-major FP64 image, even column stride.
static void build_fp64_image(const std::vector<double>& a, int n, DenseOperand* op) {
  const int np = (n + 1) & ~1;
  op->image.assign(sizeof(double) * (size_t)n * np, 0);
  double* img = reinterpret_cast<double*>(op->image.data());
  for (int k = 0; k < n; k++)
    for (int j = 0; j < n; j++) img[(size_t)k * np + j] = a[(size_t)j * n + k];
}

// Sum of a row's entries in the fast columns of set `cls`; bit b of `signs` is
// the sign of the set's b-th column (1: plus).
template <class Entry>
static double fast_sum(int cls, int signs, Entry entry) {
  double t = 0.0;
  for (int k = 0, b = 0; k < 4; k++)
    if ((cls >> k) & 1) t += ((signs >> b++) & 1) ? entry(k) : -entry(k);
  return t;
}

// Turns the column-major image of a cube layout's matrix (`parts` column sets
// of stride np) into the column-cube walk's operand: columns 4..n-1 in slot
// order, and the sums of columns 0..3 for each row value.  Slots without a
// row hold the constant 1 (2 in the last column, which is halved).
static void build_cube_operand(const CubeLayout& l, int parts, DenseOperand* op) {
  const int n = op->n, np = (n + 1) & ~1;
  const CubeShape& shape = kCubeShapes[l.shape];
  const int N = cube_rows(shape), nc = n - 4;
  const std::vector<unsigned char> columns = std::move(op->image);
  const double* col = reinterpret_cast<const double*>(columns.data());
  op->shape = l.shape;
  op->exp2 = l.exp2;
  op->image.assign(sizeof(double) * parts * nc * N, 0);
  op->sums.assign((size_t)parts * kCubeMaxSums, 0.0);
  double* img = reinterpret_cast<double*>(op->image.data());
  for (int part = 0; part < parts; part++) {
    const double* from = col + (size_t)part * n * np;
    double* to = img + (size_t)part * nc * N;
    for (int slot = 0; slot < N; slot++) {
      const int j = l.slot_row[slot];
      if (j < 0) {
        if (part == 0) to[(size_t)(nc - 1) * N + slot] = 2.0;
        continue;
      }
      for (int k = 0; k < nc; k++) to[(size_t)k * N + slot] = from[(size_t)(k + 4) * np + j];
    }
    for (int i = 1; i < 16; i++) {
      const int cls = cube_class(i), half = (1 << cube_bits(cls)) / 2;
      for (int r = 0; r < shape.rows[cls]; r++) {
        const int j = l.slot_row[cube_slot(shape, i) + r];
        if (j < 0) continue;
        for (int s = 0; s < half; s++) {
          op->sums[(size_t)part * kCubeMaxSums + cube_sum(shape, i) + r * half + s] =
              fast_sum(cls, s + half, [&](int k) { return 0.5 * from[(size_t)k * np + j]; });
        }
      }
    }
  }
}

// The integer walks' operand (int32 columns; slots without a row hold y = 1),
// when the products that the kernel forms in int32 (runs of 4 and 3 rows,
// below 2^31) and, for the certified walk, keeps in FP64 as exact (any
// kCubeExactRows rows, below 2^53) provably fit.
static bool build_cube_int_operand(const CubeLayout& l, DenseOperand* op) {
  const int n = op->n, nc = n - 4;
  const CubeShape& shape = kCubeShapes[l.shape];
  const int N = cube_rows(shape);
  std::vector<double> rowabs;
  if (l.exp2 || !int_row_abs(l.mat, n, rowabs)) return false;
  for (int i = 0; i < 16; i++) {
    const int rows = shape.rows[cube_class(i)], runs = rows - cube_left(rows);
    for (int r = 0; r < runs; r += 4) {
      double b = 1.0;
      for (int t = r; t < std::min(r + 4, runs); t++) {
        const int j = l.slot_row[cube_slot(shape, i) + t];
        if (j >= 0) b *= std::max(rowabs[j], 1.0);
      }
      if (!(b < 2147483648.0)) return false;
    }
  }
  if (op->variant == PERM_KERNEL_DENSE_INT_DD) {
    std::vector<double> large = rowabs;
    std::sort(large.begin(), large.end(), std::greater<double>());
    double b = 1.0;
    for (int t = 0; t < kCubeExactRows; t++) b *= std::max(large[t], 1.0);
    if (!(b < 9007199254740992.0)) return false;
  }
  op->shape = l.shape;
  op->image.assign(sizeof(int) * (size_t)nc * N, 0);
  int* img = reinterpret_cast<int*>(op->image.data());
  for (int slot = 0; slot < N; slot++) {
    const int j = l.slot_row[slot];
    for (int k = 0; k < nc; k++)
      img[(size_t)k * N + slot] = j >= 0 ? (int)l.mat[(size_t)j * n + k + 4] : k == nc - 1 ? 1 : 0;
  }
  // every row's sums, then those of the rows left over from the runs
  op->sums.assign(kCubeMaxSums + kCubeMaxWide, 0.0);
  for (int i = 1; i < 16; i++) {
    const int cls = cube_class(i), half = (1 << cube_bits(cls)) / 2, runs = shape.rows[cls] - cube_left(shape.rows[cls]);
    for (int r = 0; r < shape.rows[cls]; r++) {
      const int j = l.slot_row[cube_slot(shape, i) + r];
      if (j < 0) continue;
      for (int s = 0; s < half; s++) {
        const double t = fast_sum(cls, s + half, [&](int k) { return l.mat[(size_t)j * n + k]; });
        op->sums[cube_sum(shape, i) + r * half + s] = t;
        if (r >= runs) op->sums[kCubeMaxSums + cube_left_sum(shape, i) + (r - runs) * half + s] = t;
      }
    }
  }
  return true;
}

// The FP64 walk's row layout, searched for at most once (the search takes 65 us
// at n = 25, 0.2 ms at n = 33).
struct Fp64Rows {
  int inner = 0, inner1 = 0;
  long cost8 = 0;  // operations per 8 terms; 0: not searched yet
  std::vector<double> perm;
  void choose(const std::vector<double>& a, int n) {
    if (!cost8) fp64_choose(a, n, &inner, &inner1, &perm, &cost8);
  }
};

// The FP64 walk's operand in column cubes; false where a row layout needs
// fewer operations: their walks reach 0.93 (one level) and 0.87 of the FP64
// pipe against 0.82.  One level is 32 n operations per 16 terms.  The smallest
// row layout (levels of 8 and 20 rows) needs 394 + 4n, so cheaper cubes skip
// the search for one; below order 30 the search costs more than it could find
// where the cube needs less than 0.6 of the one-level operations (n = 28,
// density 0.6, 0.25 ms: 0.29 ms with the host's part, 0.34 with the search).
static bool cube_operand_f64(const std::vector<double>& a, int n, Fp64Rows* rows, DenseOperand* op) {
  CubeLayout l;
  if (!cube_layout(a, n, 32.0 * n * 0.82 / 0.93, false, &l)) return false;
  if (l.cost > (n < 30 ? 0.6 * 32.0 * n : (394.0 + 4.0 * n) * 0.82 / 0.87)) {
    rows->choose(a, n);
    if (l.cost / 0.82 > 2.0 * (double)rows->cost8 / (rows->inner ? 0.87 : 0.93)) return false;
  }
  op->n = n;
  op->variant = PERM_KERNEL_DENSE;
  op->group = 0;
  op->inner = op->inner1 = 0;
  build_fp64_image(l.mat, n, op);
  build_cube_operand(l, 1, op);
  return true;
}

// The int32 walks' row layout, searched for at most once (0.25 ms at n = 30).
struct IntRows {
  int group = 0, pair = 0, ngo = 0, ng1 = 0, ng2 = 0;
  long cost = 0;  // instructions per 8 terms; 0: not searched yet
  std::vector<double> mat;  // the permuted matrix; empty: the matrix as it is
  void choose(const std::vector<double>& a, int n, int G, bool certified) {
    if (cost) return;
    if (!certified) {
      const IntLayout l = choose_int_layout(a, n, G, &mat, &cost);
      group = l.g;
      ngo = l.ngo;
      ng1 = l.ng1;
      ng2 = l.ng2;
      if (!ngo && !ng1) mat.clear();
      return;
    }
    int cost1 = 0;
    group = intc_layout(a, n, &pair, &cost1);
    cost = 8L * (n + cost1);
    int g2 = group, p2 = pair, ngo2 = 0;
    std::vector<double> two, three;
    if (intc_two_level_layout(a, n, cost, &g2, &p2, &ngo2, &two, &cost)) {
      group = g2;
      pair = p2;
      ngo = ngo2;
      mat.swap(two);
    }
    int g3 = 0, p3 = 0, a1 = 0, a2 = 0;
    if (intc_three_level_layout(a, n, cost, &g3, &p3, &a1, &a2, &three, &cost)) {
      group = g3;
      pair = p3;
      ngo = 0;
      ng1 = a1;
      ng2 = a2;
      mat.swap(three);
    }
  }
};

// The int32 walks' operand (op->variant: plain or certified) in column cubes,
// where that is the cheaper walk.  Cycles per SM, warp and 16 terms, fitted to
// both walks at orders 30..34 and densities 0.35..0.9 (the fits are good to
// 5%): 40 + 0.39 of the cube's cost against 0.77 of the row layout's
// instructions per 8 terms; certified, 90 + 0.65 against 105 + 0.74.  The
// several-level row layouts need no less than about 0.55 (certified) and 0.6
// of the one-level instructions; only above that are they searched for.
// `transpose`: the transpose may be walked instead (certified walk).
static bool cube_operand_int(const std::vector<double>& a, int n, int G, bool transpose, IntRows* rows,
                             DenseOperand* op) {
  const bool certified = op->variant == PERM_KERNEL_DENSE_INT_DD;
  const double base = certified ? 90.0 : 40.0, per = certified ? 0.65 : 0.39;
  const double row_base = certified ? 105.0 : 0.0, row_per = certified ? 0.74 : 0.77;
  int pair = 0, cost1 = 0;
  if (certified) intc_layout(a, n, &pair, &cost1);
  const double one_level = certified ? 8.0 * (n + cost1) : 8.0 * (2 * n + (n + G - 1) / G);
  CubeLayout cube;
  if (!cube_layout(a, n, (row_base + row_per * one_level - base) / per, transpose, &cube)) return false;
  const double mine = base + per * cube.cost;
  if (mine > row_base + row_per * (certified ? 0.55 : 0.6) * one_level) {
    rows->choose(a, n, G, certified);
    if (mine >= row_base + row_per * (double)rows->cost) return false;
  }
  op->n = n;
  return build_cube_int_operand(cube, op);
}

static std::vector<double> transposed(const std::vector<double>& a, int n) {
  std::vector<double> t(a.size());
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++) t[(size_t)k * n + j] = a[(size_t)j * n + k];
  return t;
}

static int build_sdd_operand(perm_ctx* ctx, std::vector<double> a, int n, bool rows_only, DenseOperand* op) {
  if (n < 4 || n > 40) return fail(ctx, PERM_EUNSUPPORTED, "split-dd kernel covers orders 4..40 (got %d)", n);
  const bool cubes = n >= kCubeMinN && !rows_only;
  WalkSide side = cubes ? walk_side(a, n) : WalkSide::kMatrix;
  if (side != WalkSide::kMatrix) {
    // the callers checked the matrix's rows, not the transpose's
    std::vector<double> t = transposed(a, n);
    if (!split_rows_ok(t, n))
      side = WalkSide::kMatrix;
    else if (side == WalkSide::kTranspose)
      a.swap(t);
  }
  // The column-cube walk (6 operations per row value, 2 per row and about 280
  // for the class arrays and the sum, per 16 terms; 0.63 of the FP64 pipe)
  // unless a row layout is cheaper (per 8 terms, 0.69 dense, 0.56..0.62 the
  // others).  n = 30: 364 values 7.3 ms, dense layout 8.9 ms.  The smallest
  // row layout (sparse, 6 rows) needs 320 + 6n operations per 8 terms; below
  // order 30 it is searched for (50 us) only where the cube needs more than 0.7
  // of the dense layout's time.
  CubeLayout l;
  int inner = 0, inner1 = 0;
  std::vector<double> perm;
  bool cube = cubes && cube_layout(a, n, 1e9, side == WalkSide::kEither, &l);
  bool searched = false;
  if (cube) {
    const double mine = (6.0 * cube_values(kCubeShapes[l.shape]) + 2.0 * n + 280.0) / 0.63;
    if (mine > (n < 30 ? 0.7 * 2.0 * (double)sdd_cost(n, 0) / 0.69 : 2.0 * (320.0 + 6.0 * n) / 0.62)) {
      sdd_choose(a, n, &inner, &inner1, &perm);
      searched = true;
      cube = mine < 2.0 * (double)sdd_cost(n, inner, inner1, inner) / (inner ? 0.62 : 0.69);
    }
  }
  if (cube) {
    const int rc = build_split_operand(ctx, l.mat, n, op);
    if (rc) return rc;
    op->variant = PERM_KERNEL_DENSE_SDD;
    build_cube_operand(l, 2, op);
    return PERM_OK;
  }
  if (!searched) sdd_choose(a, n, &inner, &inner1, &perm);
  const int rc = build_split_operand(ctx, inner ? perm : a, n, op);
  if (rc) return rc;
  op->variant = PERM_KERNEL_DENSE_SDD;
  op->inner = inner;
  op->inner1 = inner1;
  return PERM_OK;
}

// No cube beats the row layouts above density 0.8 or so at orders 20..24.
static bool sparse_enough(const std::vector<double>& a) {
  size_t nonzeros = 0;
  for (double v : a) nonzeros += v != 0.0;
  return nonzeros <= a.size() * 8 / 10;
}

// `own_sum`: the operand is walked in one piece under the accuracy policy;
// `rows_only`: a row layout of the matrix itself, no cubes and no transpose.
static int build_operand(perm_ctx* ctx, const void* mat, int n, int dtype, int variant, DenseOperand* op,
                         bool own_sum = false, bool rows_only = false) {
  std::vector<double> a((size_t)n * n);
  for (size_t i = 0; i < a.size(); i++) a[i] = elem(mat, dtype, i);
  op->n = n;
  const int pref = variant == 0 && n <= PERM_MAX_EXACT_N ? ctx->dense_pref[n] : 0;
  const bool prefer_fp64 = pref == PERM_KERNEL_DENSE;
  if (variant == PERM_KERNEL_DENSE_SPLIT) return build_split_operand(ctx, a, n, op);
  if (variant == PERM_KERNEL_DENSE_SDD) return build_sdd_operand(ctx, a, n, rows_only, op);
  int G = (variant == PERM_KERNEL_DENSE || variant == PERM_KERNEL_DENSE_DD || prefer_fp64) ? 0 : int_group_size(a, n);
  if ((variant == PERM_KERNEL_DENSE_INT || variant == PERM_KERNEL_DENSE_INT_DD) && G == 0)
    return fail(ctx, PERM_EUNSUPPORTED,
                "int32-X kernels need an integer matrix of order >= 8 whose row products fit in int32");
  const bool tc_ok = G && tc_eligible(a, n);
  if (variant == PERM_KERNEL_DENSE_TC && !tc_ok)
    return fail(ctx, PERM_EUNSUPPORTED,
                "tensor-core kernel needs an integer matrix of order 16..64 with |a| <= 63 whose row products "
                "fit in int32");
  if (G) {
    const int np4 = (n + 3) & ~3;
    op->variant = (variant == PERM_KERNEL_DENSE_TC || (variant == 0 && pref == PERM_KERNEL_DENSE_TC && tc_ok))
                      ? PERM_KERNEL_DENSE_TC
                  : variant == PERM_KERNEL_DENSE_INT_DD ? PERM_KERNEL_DENSE_INT_DD
                                                        : PERM_KERNEL_DENSE_INT;
    op->group = G;
    op->pair = 0;
    op->ngo = 0;
    op->ng1 = op->ng2 = 0;
    if (op->variant != PERM_KERNEL_DENSE_TC) {
      IntRows rows;
      // the transpose's search costs more than it saves below order 28
      const bool turn = op->variant == PERM_KERNEL_DENSE_INT_DD && n >= 28 && !rows_only;
      const WalkSide side = turn ? walk_side(a, n) : WalkSide::kMatrix;
      if (side == WalkSide::kTranspose) {
        std::vector<double> t = transposed(a, n);
        if (const int g = int_group_size(t, n)) {
          G = g;
          a.swap(t);
        }
      }
      if (n >= kCubeMinN && !rows_only && cube_operand_int(a, n, G, side == WalkSide::kEither, &rows, op))
        return PERM_OK;
      rows.choose(a, n, G, op->variant == PERM_KERNEL_DENSE_INT_DD);
      op->group = rows.group;
      op->pair = rows.pair;
      op->ngo = rows.ngo;
      op->ng1 = rows.ng1;
      op->ng2 = rows.ng2;
      if (!rows.mat.empty()) a.swap(rows.mat);  // walk the permuted matrix (same permanent)
    }
    op->image.assign(sizeof(int) * (size_t)(n + 1) * np4, 0);
    int* img = reinterpret_cast<int*>(op->image.data());
    for (int k = 0; k < n; k++)
      for (int j = 0; j < n; j++) img[(size_t)k * np4 + j] = 2 * (int)a[(size_t)j * n + k];
    int* y0 = img + (size_t)n * np4;
    for (int j = 0; j < n; j++) {
      long long rs = 0;
      for (int k = 0; k < n; k++) rs += (long long)a[(size_t)j * n + k];
      y0[j] = (int)(2 * (long long)a[(size_t)j * n + n - 1] - rs);
    }
  } else {
    op->variant = variant == PERM_KERNEL_DENSE_DD ? PERM_KERNEL_DENSE_DD : PERM_KERNEL_DENSE;
    op->group = 0;
    op->inner = 0;
    op->inner1 = 0;
    if (op->variant == PERM_KERNEL_DENSE) {
      Fp64Rows rows;
      if (!rows_only && n >= (own_sum && sparse_enough(a) ? kCubeSumMinN : kCubeMinN) &&
          cube_operand_f64(a, n, &rows, op))
        return PERM_OK;
      rows.choose(a, n);
      op->inner = rows.inner;
      op->inner1 = rows.inner1;
      if (op->inner) a.swap(rows.perm);  // walk the permuted matrix (same permanent)
    }
    build_fp64_image(a, n, op);
  }
  return PERM_OK;
}

struct perm_matrix {
  DenseOperand op;
  void* d_image = nullptr;
};

static int cube_kind(const DenseOperand& op) {
  return op.variant == PERM_KERNEL_DENSE_SDD      ? kCubeSdd
         : op.variant == PERM_KERNEL_DENSE_INT    ? kCubeInt
         : op.variant == PERM_KERNEL_DENSE_INT_DD ? kCubeIntc
         : op.abs_sum                             ? kCubeF64Abs
                                                  : kCubeF64;
}
static const void* operand_kernel(const DenseOperand& op) {
  if (op.shape >= 0) return cube_kernel(op.shape, cube_kind(op));
  if (op.variant == PERM_KERNEL_DENSE_INT)
    return op.ng1 ? dense_int_3l_kernel(op.n, op.group, op.ng1, op.ng2)
           : op.ngo ? dense_int_sparse_kernel(op.n, op.group, op.ngo)
                    : dense_int_kernel(op.n, op.group);
  if (op.variant == PERM_KERNEL_DENSE_INT_DD)
    return op.ng1   ? dense_intc_3l_kernel(op.n, op.group, op.pair, op.ng1, op.ng2)
           : op.ngo ? dense_intc_sparse_kernel(op.n, op.group, op.pair, op.ngo)
                    : dense_intc_kernel(op.n, op.group, op.pair);
  if (op.variant == PERM_KERNEL_DENSE_SDD) return sdd_kernel(op.n, op.inner, op.inner1);
  if (op.variant == PERM_KERNEL_DENSE_TC) return dense_tc_kernel(op.n, op.group);
  if (op.variant == PERM_KERNEL_DENSE_DD) return dense_dd_kernel(op.n);
  if (op.variant == PERM_KERNEL_DENSE_SPLIT) return dense_split_kernel(op.n);
  return op.inner1  ? dense_3l_kernel(op.n, op.inner1, op.inner)
         : op.inner ? dense_2l_kernel(op.n, op.inner)
                    : dense_kernel(op.n);
}
static int operand_threads(const DenseOperand& op) {
  if (op.shape >= 0) return kCubeThreads;
  return op.variant == PERM_KERNEL_DENSE_TC ? kTcThreads : 128;
}
static size_t operand_smem(const DenseOperand& op) {
  if (op.shape >= 0)
    return cube_smem_bytes(cube_rows(kCubeShapes[op.shape]),
                           cube_kind(op) >= kCubeInt ? sizeof(int) : (cube_kind(op) == kCubeSdd ? 2 : 1) * sizeof(double),
                           op.n, cube_kind(op) == kCubeSdd);
  if (op.variant == PERM_KERNEL_DENSE_INT || op.variant == PERM_KERNEL_DENSE_INT_DD) return dense_int_smem_bytes(op.n);
  if (op.variant == PERM_KERNEL_DENSE_SDD)
    return op.inner ? sparse_sdd_smem_bytes(op.n, op.inner, 128) : dense_sdd_smem_bytes(op.n);
  if (op.variant == PERM_KERNEL_DENSE_TC) return dense_tc_smem_bytes(op.n);
  if (op.variant == PERM_KERNEL_DENSE_DD) return dense_dd_smem_bytes(op.n);
  if (op.variant == PERM_KERNEL_DENSE_SPLIT) return dense_split_smem_bytes(op.n);
  return dense_smem_bytes(op.n);
}

struct DensePlan {
  int grid = 1, m = 3;
  uint64_t block0 = 0, nblocks = 0;
};

// Shard boundaries depend on (n, shard, nshards) only -- never on the device
// -- so ranks with different grids still partition [0, 2^(n-1)) exactly:
// shards are cut at multiples of 2^ms, ms = max(3, n - 21) (at most 2^20
// shard units), and the kernel's range alignment m never exceeds ms.
static void shard_bounds(int n, int shard, int nshards, uint64_t* first, uint64_t* last, int* ms_out) {
  const uint64_t total = 1ull << (n - 1);
  if (n < 4) {
    *first = shard == 0 ? 0 : total;
    *last = total;
    if (ms_out) *ms_out = 0;
    return;
  }
  const int ms = std::max(3, n - 21);
  const uint64_t units = total >> ms;
  *first = (units * (uint64_t)shard / (uint64_t)nshards) << ms;
  *last = (units * (uint64_t)(shard + 1) / (uint64_t)nshards) << ms;
  if (ms_out) *ms_out = ms;
}

extern "C" int perm_fp64_layout(const double* mat, int n) {
  int levels[2];
  const int rc = perm_fp64_levels(mat, n, levels);
  return rc ? rc : levels[1];
}

extern "C" int perm_fp64_levels(const double* mat, int n, int* levels) {
  if (!mat || !levels || n < 1 || n > PERM_MAX_EXACT_N) return PERM_EINVAL;
  std::vector<double> a(mat, mat + (size_t)n * n);
  std::vector<double> perm;
  fp64_choose(a, n, &levels[1], &levels[0], &perm);
  return PERM_OK;
}

extern "C" int perm_int_layout(const double* mat, int n, int* levels) {
  if (!mat || !levels || n < 1 || n > PERM_MAX_EXACT_N) return PERM_EINVAL;
  std::vector<double> a(mat, mat + (size_t)n * n);
  levels[0] = levels[1] = levels[2] = 0;
  const int g = int_group_size(a, n);
  if (!g) return PERM_EUNSUPPORTED;
  std::vector<double> perm;
  const IntLayout l = choose_int_layout(a, n, g, &perm);
  levels[0] = l.ngo;
  levels[1] = l.ng1;
  levels[2] = l.ng2;
  return l.g;
}

extern "C" int perm_intc_layout(const double* mat, int n, int* pair, int* levels) {
  if (!mat || !pair || !levels || n < 1 || n > PERM_MAX_EXACT_N) return PERM_EINVAL;
  std::vector<double> a(mat, mat + (size_t)n * n);
  levels[0] = levels[1] = levels[2] = 0;
  int cost1 = 0;
  int g = intc_layout(a, n, pair, &cost1);
  if (!g) return PERM_EUNSUPPORTED;
  long cost = 8L * (n + cost1);
  std::vector<double> two, three;
  int g2 = g, p2 = *pair, ngo2 = 0;
  if (intc_two_level_layout(a, n, cost, &g2, &p2, &ngo2, &two, &cost)) {
    g = g2;
    *pair = p2;
    levels[0] = ngo2;
  }
  int g3 = 0, p3 = 0, a1 = 0, a2 = 0;
  if (intc_three_level_layout(a, n, cost, &g3, &p3, &a1, &a2, &three)) {
    g = g3;
    *pair = p3;
    levels[0] = 0;
    levels[1] = a1;
    levels[2] = a2;
  }
  return g;
}

extern "C" int perm_sdd_layout(const double* mat, int n) {
  int levels[2];
  const int rc = perm_sdd_levels(mat, n, levels);
  return rc ? rc : levels[1];
}

extern "C" int perm_sdd_levels(const double* mat, int n, int* levels) {
  if (!mat || !levels || n < 1 || n > PERM_MAX_EXACT_N) return PERM_EINVAL;
  std::vector<double> a(mat, mat + (size_t)n * n);
  if (n < 4 || n > 40 || !split_rows_ok(a, n)) return PERM_EUNSUPPORTED;
  std::vector<double> perm;
  sdd_choose(a, n, &levels[1], &levels[0], &perm);
  return PERM_OK;
}

extern "C" int perm_cube_layout(const double* mat, int n, int variant, double* fp64_ops) {
  if (fp64_ops) *fp64_ops = 0.0;
  if (!mat || n < 1 || n > PERM_MAX_EXACT_N) return -1;
  if (variant != PERM_KERNEL_DENSE && variant != PERM_KERNEL_DENSE_INT && variant != PERM_KERNEL_DENSE_INT_DD &&
      variant != PERM_KERNEL_DENSE_SDD)
    return -1;
  perm_ctx host;  // keeps the message of a refusal
  DenseOperand op;
  if (build_operand(&host, mat, n, PERM_F64, variant, &op) != PERM_OK) return -1;
  if (op.shape >= 0 && fp64_ops) *fp64_ops = cube_shape_ops(op.shape);
  return op.shape;
}

extern "C" int perm_shard_range(int n, int shard, int nshards, uint64_t* first, uint64_t* last) {
  if (n < 1 || n > PERM_MAX_EXACT_N || nshards < 1 || shard < 0 || shard >= nshards || !first || !last)
    return PERM_EINVAL;
  shard_bounds(n, shard, nshards, first, last, nullptr);
  return PERM_OK;
}

// Range alignment (log2, in cubes, at most m_max) of a column-cube walk: a
// thread owns ceil(blocks / threads) blocks of 2^m cubes at most, and leaving a
// block costs about half a cube more, since the lanes then flip different
// columns.
static int cube_align(uint64_t cubes, uint64_t threads, int m_max) {
  double best = -1.0;
  int best_m = 0;
  for (int m = 0; m <= 10 && m <= m_max; m++) {
    const double each = std::ceil((double)(cubes >> m) / (double)threads);
    const double cost = each * (std::ldexp(1.0, m) + 0.5);
    if (best < 0.0 || cost < best) best = cost, best_m = m;
  }
  return best_m;
}

// Launch arguments of a column-cube walk over blocks [block0, block0 +
// nblocks) of 2^m cubes, without its destinations; the walk's own form begins
// with CubeWalk.
union CubeLaunch {
  CubeWalk walk;
  CubeArgs f64;
  CubeSddArgs sdd;
  CubeIntArgs integer;
  CubeLaunch() {}
};
static void cube_args(const DenseOperand& op, const void* d_image, int m, uint64_t block0, uint64_t nblocks,
                      CubeLaunch* u) {
  const int kind = cube_kind(op);
  CubeWalk& w = u->walk;
  w.img = d_image;
  w.n = op.n;
  w.m = m;
  w.block0 = block0;
  w.nblocks = nblocks;
  w.seg = kind >= kCubeInt ? ~0ull : kCubeSegment;
  w.inject = 0;
  if (kind >= kCubeInt) {
    for (int i = 0; i < kCubeMaxSums; i++) u->integer.ci[i] = (int)op.sums[i];
    memcpy(u->integer.cd, op.sums.data() + kCubeMaxSums, sizeof u->integer.cd);
  } else if (kind == kCubeSdd) {
    memcpy(u->sdd.c, op.sums.data(), sizeof u->sdd.c);
    memcpy(u->sdd.cl, op.sums.data() + kCubeMaxSums, sizeof u->sdd.cl);
  } else {
    memcpy(u->f64.c, op.sums.data(), sizeof u->f64.c);
  }
}

static int dense_plan(perm_ctx* ctx, const DenseOperand& op, int shard, int nshards, DensePlan* p) {
  const int n = op.n;
  const void* fn = operand_kernel(op);
  if (!fn) return fail(ctx, PERM_EUNSUPPORTED, "dense exact order %d outside [1, %d]", n, PERM_MAX_EXACT_N);
  int sparse_slot = 0;
  for (int i = 0; i < 7; i++)
    if (op.inner == kSparseInner[i]) sparse_slot = i < 4 ? 18 + i : 43 + i - 4;
  int fp_slot = 0;
  for (int i = 0; i < 4; i++) {
    if (op.inner == k2lInner[i]) fp_slot = 46 + i;
    if (op.inner1 && op.inner == kSdd3lR2[i]) sparse_slot = 86 + 4 * i + op.inner1 / 4 - 2;
  }
  for (int i = 0; i < 5; i++)
    if (op.inner1 && op.inner == kFp3lR2[i]) fp_slot = 102 + 4 * i + op.inner1 / 4 - 2;
  int& occ_slot = op.shape >= 0 ? ctx->cube_occ[cube_kind(op)][op.shape] : ctx->dense_occ[op.variant == PERM_KERNEL_DENSE_INT
                                     ? (op.ng1 ? 50 + 6 * (op.group - 4) + 2 * (op.ng1 - 2) + op.ng2 - 1
                                        : op.ngo ? 25 + 3 * (op.group - 4) + op.ngo - 1
                                                 : op.group)
                                 : op.variant == PERM_KERNEL_DENSE_DD ? 7
                                 : op.variant == PERM_KERNEL_DENSE_TC ? 8 + op.group - 3
                                 : op.variant == PERM_KERNEL_DENSE_SPLIT ? 12
                                 : op.variant == PERM_KERNEL_DENSE_INT_DD
                                     ? (op.ng1 ? 68 + 6 * intc_sparse_family(op.group, op.pair) + 2 * (op.ng1 - 2) +
                                                     op.ng2 - 1
                                        : op.ngo ? 34 + 3 * intc_sparse_family(op.group, op.pair) + op.ngo - 1
                                        : op.pair ? 22 + op.group - 4
                                                  : 13 + op.group - 3)
                                 : op.variant == PERM_KERNEL_DENSE_SDD ? (op.inner ? sparse_slot : 17)
                                 : op.inner ? fp_slot : 0][n];
  if (!occ_slot) {
    int rc = allow_smem(ctx, fn, operand_smem(op));
    if (rc) return rc;
    int occ = 0;
    CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, operand_threads(op), operand_smem(op)));
    occ_slot = std::max(occ, 1);
  }
  if (op.variant == PERM_KERNEL_DENSE_TC) {
    // whole walk only: rounds of 512 subsets, one CTA per SM (it holds all
    // 512 TMEM columns)
    if (shard != 0 || nshards != 1) return fail(ctx, PERM_EINVAL, "tensor-core kernel runs whole walks only");
    const int rb = tc_round_bits(n);
    const uint64_t rounds = 1ull << rb;
    p->grid = (int)std::min<uint64_t>((uint64_t)ctx->num_sms, rounds);
    p->m = n - 1 - rb;
    p->block0 = 0;
    p->nblocks = rounds;
    return PERM_OK;
  }
  uint64_t first = 0, last = 0;
  int ms = 0;
  shard_bounds(n, shard, nshards, &first, &last, &ms);
  if (n < 4) {
    p->grid = 1;
    p->m = 0;
    p->block0 = shard == 0 ? 0 : 1;
    p->nblocks = 0;
    return PERM_OK;
  }
  int grid = std::min(kMaxBlocks, ctx->num_sms * occ_slot);
  if (op.shape >= 0) {
    grid = std::min(grid, ctx->num_sms * kCubeBlocks);
    p->m = 4 + cube_align((last - first) >> 4, (uint64_t)grid * operand_threads(op), nshards == 1 ? n - 5 : ms - 4);
    p->block0 = first >> p->m;
    p->nblocks = (last - first) >> p->m;
    p->grid = (int)std::min<uint64_t>((uint64_t)grid, std::max<uint64_t>(1, (p->nblocks + operand_threads(op) - 1) / operand_threads(op)));
    return PERM_OK;
  }
  // Alignment m <= ms: each thread should own >= 64 aligned blocks when possible.
  const uint64_t len = last - first;
  const uint64_t threads = (uint64_t)grid * 128;
  // FP64 X is recomputed at block boundaries, at most every 2^12 steps (at
  // 2^20 an order-40 walk drifted past its own error bound).
  int m = 3;
  const int m_max = op.variant == PERM_KERNEL_DENSE ? 12 : 20;
  while (m < m_max && m < ms && (len >> (m + 1)) >= threads * 64) m++;
  const uint64_t mine = len >> m;
  if (mine < (uint64_t)grid * 128) grid = (int)std::max<uint64_t>(1, (mine + 127) / 128);
  p->grid = grid;
  p->m = m;
  p->block0 = first >> m;
  p->nblocks = mine;
  return PERM_OK;
}

static int dense_launch(perm_ctx* ctx, const DenseOperand& op, const void* d_image, const DensePlan& p) {
  const int n = op.n;
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  if (op.shape >= 0) {
    const int kind = cube_kind(op);
    CubeLaunch u;
    cube_args(op, d_image, p.m - 4, p.block0, p.nblocks, &u);
    CubeWalk& args = u.walk;
    args.partials = reinterpret_cast<dd*>(ctx->d_out + kOutWords);
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.err = ctx->d_err;
    if (ctx->inject_timeouts > 0 && (kind == kCubeF64 || kind == kCubeF64Abs)) {
      args.inject = 16u;
      ctx->inject_timeouts--;
    }
    void* kargs[] = {&u};
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(operand_threads(op)), kargs, operand_smem(op),
                             ctx->stream));
  } else if (op.variant == PERM_KERNEL_DENSE_TC) {
    DenseTcArgs args;
    args.colI = static_cast<const int*>(d_image);
    args.np4 = (n + 3) & ~3;
    args.round0 = p.block0;
    args.nrounds = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.err = ctx->d_err;
    args.inject = ctx->inject_timeouts > 0 ? 1 : 0;
    if (args.inject) ctx->inject_timeouts--;
    void* kargs[] = {&args};
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(kTcThreads), kargs, operand_smem(op),
                             ctx->stream));
  } else if (op.variant == PERM_KERNEL_DENSE_SPLIT) {
    DenseSplitArgs args;
    args.img = static_cast<const double*>(d_image);
    args.np = (n + 1) & ~1;
    args.m = p.m;
    args.block0 = p.block0;
    args.nblocks = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.sums = ctx->d_est;
    args.err = ctx->d_err;
    void* kargs[] = {&args};
    CU(ctx, cudaMemsetAsync(ctx->d_est, 0, 2 * sizeof(double), ctx->stream));
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(128), kargs, operand_smem(op), ctx->stream));
  } else if (op.variant == PERM_KERNEL_DENSE_INT_DD) {
    DenseIntcArgs args;
    const int np4 = (n + 3) & ~3;
    args.colI = static_cast<const int*>(d_image);
    args.np4 = np4;
    args.m = p.m;
    args.block0 = p.block0;
    args.nblocks = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.sums = ctx->d_est;
    args.err = ctx->d_err;
    void* kargs[] = {&args};
    CU(ctx, cudaMemsetAsync(ctx->d_est, 0, 2 * sizeof(double), ctx->stream));
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(128), kargs, operand_smem(op), ctx->stream));
  } else if (op.variant == PERM_KERNEL_DENSE_SDD) {
    DenseSddArgs args;
    args.img = static_cast<const double*>(d_image);
    args.np = (n + 1) & ~1;
    args.m = p.m;
    args.block0 = p.block0;
    args.nblocks = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.sums = ctx->d_est;
    args.err = ctx->d_err;
    void* kargs[] = {&args};
    CU(ctx, cudaMemsetAsync(ctx->d_est, 0, 2 * sizeof(double), ctx->stream));
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(128), kargs, operand_smem(op), ctx->stream));
  } else if (op.variant == PERM_KERNEL_DENSE_INT) {
    DenseIntArgs args;
    const int np4 = (n + 3) & ~3;
    args.colI = static_cast<const int*>(d_image);
    args.y0 = args.colI + (size_t)n * np4;
    args.np4 = np4;
    args.m = p.m;
    args.block0 = p.block0;
    args.nblocks = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.err = ctx->d_err;
    void* kargs[] = {&args};
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(128), kargs, operand_smem(op), ctx->stream));
  } else {
    DenseArgs args;
    args.colA = static_cast<const double*>(d_image);
    args.np = (n + 1) & ~1;
    args.m = p.m;
    // re-anchor X every >= 2^11 Gray steps (orders <= kAnchorMaxN)
    args.seg_blocks = p.m >= 11 ? 1 : (1ull << (11 - p.m));
    args.block0 = p.block0;
    args.nblocks = p.nblocks;
    args.partials = ctx->partials;
    args.ticket = ctx->ticket;
    args.out = ctx->d_out;
    args.err = ctx->d_err;
    args.inject = ctx->inject_timeouts > 0 && op.variant == PERM_KERNEL_DENSE ? 16u : 0u;
    if (args.inject) ctx->inject_timeouts--;
    void* kargs[] = {&args};
    CU(ctx, cudaLaunchKernel(operand_kernel(op), dim3(p.grid), dim3(128), kargs, operand_smem(op), ctx->stream));
  }
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  return PERM_OK;
}

// The moments from the sample's block sums that were read back, in block order:
// the same every time.
static void add_moments(perm_ctx* ctx, int n) {
  double s1 = 0.0, s2 = 0.0;
  for (int b = 0; b < moment_blocks(n); b++) {
    s1 += ctx->h_out[kOutWords + 2 * b];
    s2 += ctx->h_out[kOutWords + 2 * b + 1];
  }
  ctx->h_out[12] = s1;
  ctx->h_out[13] = s2;
}

// `sampled`: the moment sample was queued behind the walk (row layouts of FP64
// columns).
template <class Meanwhile>
static int dense_collect(perm_ctx* ctx, const DenseOperand& op, const DensePlan& p, perm_result* out,
                         bool sampled, Meanwhile meanwhile) {
  const bool sums = op.variant == PERM_KERNEL_DENSE_SPLIT || op.variant == PERM_KERNEL_DENSE_INT_DD ||
                    op.variant == PERM_KERNEL_DENSE_SDD || op.abs_sum;
  const bool cube_sums = sums && op.shape >= 0;
  int rc = finish_and_read(ctx, cube_sums ? p.grid * kCubeWords : sampled ? 2 * moment_blocks(op.n) : 0, meanwhile);
  if (rc != PERM_OK) return rc;
  if (sampled) add_moments(ctx, op.n);
  if (cube_sums) {
    const double* warps = ctx->h_out + kOutWords + 2 * p.grid;
    double m1 = 0.0;
    for (int w = 0; w < p.grid * kCubeWarps; w++) m1 += warps[w];
    ctx->h_out[12] = m1;
  }
  if (op.variant == PERM_KERNEL_DENSE_SPLIT) {
    ctx->split_m1 = ctx->h_out[12] * 2.0;  // |factor| = 2
    ctx->split_m2 = ctx->h_out[13] * 4.0;
  } else if (sums) {
    // the int32-X walk's terms are prod y = 2^n prod x (|factor| 2^(1-n))
    ctx->walk_m1 = std::ldexp(ctx->h_out[12], op.variant == PERM_KERNEL_DENSE_INT_DD ? 1 - op.n : 1 + op.exp2);
    const uint64_t threads = (uint64_t)p.grid * operand_threads(op);
    ctx->walk_terms_per_thread = ((p.nblocks + threads - 1) / threads) << p.m;
  }
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  const int n = op.n;
  const double hi = std::ldexp(ctx->h_out[0], op.exp2), lo = std::ldexp(ctx->h_out[1], op.exp2);
  out->hi = hi;
  out->lo = lo;
  out->value = hi + lo;
  out->total_steps = std::ldexp(1.0, n - 1);
  out->steps = n < 4 ? (p.block0 == 0 ? out->total_steps : 0.0) : std::ldexp((double)p.nblocks, p.m);
  out->kernel_ms = ms;
  out->kernel = op.variant;
  out->n = n;
  return PERM_OK;
}

static int dense_collect(perm_ctx* ctx, const DenseOperand& op, const DensePlan& p, perm_result* out) {
  return dense_collect(ctx, op, p, out, false, [] {});
}

static int check_dense_args(perm_ctx* ctx, const void* mat, int n, int dtype, const void* out) {
  if (!ctx) return PERM_EINVAL;
  if (!mat || !out) return fail(ctx, PERM_EINVAL, "null matrix or result pointer");
  if (n < 1 || n > PERM_MAX_EXACT_N) return fail(ctx, PERM_EUNSUPPORTED, "order %d outside [1, %d]", n, PERM_MAX_EXACT_N);
  if (dtype != PERM_F64 && dtype != PERM_F32 && dtype != PERM_I32)
    return fail(ctx, PERM_EINVAL, "unknown dtype %d", dtype);
  return PERM_OK;
}

static int check_variant(perm_ctx* ctx, int variant) {
  if (variant != 0 && variant != PERM_KERNEL_DENSE && variant != PERM_KERNEL_DENSE_INT &&
      variant != PERM_KERNEL_DENSE_DD && variant != PERM_KERNEL_DENSE_TC && variant != PERM_KERNEL_DENSE_SPLIT &&
      variant != PERM_KERNEL_DENSE_INT_DD && variant != PERM_KERNEL_DENSE_SDD)
    return fail(ctx, PERM_EINVAL, "unknown dense kernel variant %d", variant);
  return PERM_OK;
}

// Error estimate of a whole-walk result.  The sample kernel estimates
// S1 = sum_i |term(i)| and S2 = sum_i term(i)^2 from terms stratified by
// subset size (the split-X walk sums both exactly); with unit roundoff
// u = 2^-53 and r roundings per term (FP64 X: n x updates and n - 1
// products, r ~ 2n; split X: n combines and n - 1 products, r ~ 2n, each a
// function of the subset alone; int32 X: x and the group products are exact,
// r = ceil(n/G) - 1 FP64 products):
//  * worst: every rounding of every term in the same direction,
//    (r + 16) u S1 / |perm|;
//  * random: four standard deviations of the sum when roundings are
//    independent and uniform (variance u^2 / 3 each), 4 u sqrt(r / 3)
//    sqrt(S2) / |perm|.  Not a bound -- terms with equal values round alike --
//    so it is only used together with an independent second evaluation;
//  * double-double: (4n + 32) u^2 S1 / |perm|;
//  * certified walks (int32 X with double-double products, split-dd), whose
//    S1 is the walk's own exact sum: products of relative error below
//    ~4u^2 per factor (8 ceil(n/G) or 8n in all), Sum2 of the terms (256,
//    plus the low part's own rounding: K^2 for K terms added one by one per
//    thread in the int32-X walk, (K/4)^2 for split-dd's groups of eight),
//    the double-double reductions;
//    for split-dd also the drift of the remainder row sums xl over K updates
//    (64 n^2 K).  Like the double-double bound, of the (hi, lo) pair: value,
//    its sum rounded once, adds at most u.
struct ErrEstimate {
  double s1 = 0, s2 = 0, worst = 0, random = 0;
};

// bounds of `variant`'s rounding error from the sums of |term| and term^2
// (sampled, or the walk's own); k_terms = the longest thread range of a
// certified walk
static void error_bounds(int variant, int group, int n, double value, ErrEstimate* e, uint64_t k_terms = 0,
                         int shape = -1) {
  const double u = std::ldexp(1.0, -53);
  const double av = std::fabs(value), s1 = e->s1, s2 = e->s2;
  if (av == 0.0) {
    e->worst = e->random = s1 > 0 ? INFINITY : 0.0;
    return;
  }
  if (variant == PERM_KERNEL_DENSE_INT_DD || variant == PERM_KERNEL_DENSE_SDD) {
    const double k = (double)k_terms;
    // the column-cube walks take at most n + 5 factors (the rows and the
    // class arrays they are merged through) and sum cubes of 16 terms first
    const bool chain = variant == PERM_KERNEL_DENSE_INT_DD && shape < 0;
    const double prod = chain ? 8.0 * std::ceil((double)n / group) : 8.0 * (shape < 0 ? n : n + 5);
    // low-part rounding: the int32-X walk adds every term to one (hi, lo),
    // split-dd adds groups of eight
    const double lows = chain ? k * k : (k / 4) * (k / 4);
    const double drift = variant == PERM_KERNEL_DENSE_SDD ? 64.0 * n * n * k : 0.0;
    e->worst = e->random = (prod + 256.0 + lows + drift) * u * u * s1 / av;
  } else if (variant == PERM_KERNEL_DENSE_DD) {
    e->worst = e->random = (4.0 * n + 32.0) * u * u * s1 / av;
  } else if (variant == PERM_KERNEL_DENSE_SPLIT) {
    // exact coarse X: one combine per entry and n - 1 product roundings, each
    // a function of the subset alone, so independent from term to term
    e->worst = (2.0 * n + 16.0) * u * s1 / av;
    e->random = 4.0 * u * std::sqrt(2.0 * n / 3.0) * std::sqrt(s2) / av;
  } else if (variant == PERM_KERNEL_DENSE_INT || variant == PERM_KERNEL_DENSE_TC) {
    // (one rounding more in the column-cube walk: the difference over column 2)
    const double groups = shape >= 0 ? cube_factors(kCubeShapes[shape]) + 1.0 : std::ceil((double)n / group);
    e->worst = (groups + 16.0) * u * s1 / av;
    e->random = 4.0 * u * std::sqrt(std::max(1.0, groups - 1.0) / 3.0) * std::sqrt(s2) / av;
  } else {
    e->worst = (2.0 * n + 16.0) * u * s1 / av;
    e->random = 4.0 * u * std::sqrt(2.0 * n / 3.0) * std::sqrt(s2) / av;
  }
}

// Whether the operand's image is the matrix's FP64 columns (what the
// term-moment sample reads).
static bool plain_columns(const DenseOperand& op) {
  return op.shape < 0 && (op.variant == PERM_KERNEL_DENSE || op.variant == PERM_KERNEL_DENSE_DD);
}

// Queues the term-moment sample of the column image d_col_fp64.
static int queue_moments(perm_ctx* ctx, const void* d_col_fp64, int n) {
  const int np = (n + 1) & ~1;
  const int per_class = kSamplesPerClass;
  ryser_abs_sample_kernel<<<moment_blocks(n), 256, 0, ctx->stream>>>(
      static_cast<const double*>(d_col_fp64), n, np, per_class, 0x243F6A8885A308D3ull, ctx->d_out + kOutWords);
  CU(ctx, cudaGetLastError());
  return PERM_OK;
}
// The estimate from the moments in the result block that was read back.
static void estimate_from_moments(perm_ctx* ctx, int n, const DenseOperand& op, double value, ErrEstimate* e) {
  e->s1 = ctx->h_out[12] * 2.0;  // |factor| = 2
  e->s2 = ctx->h_out[13] * 4.0;
  error_bounds(op.variant, op.group, n, value, e, 0, op.shape);
}
static int estimate_error(perm_ctx* ctx, const void* d_col_fp64, int n, const DenseOperand& op, double value,
                          ErrEstimate* e) {
  *e = ErrEstimate();
  if (n < 2) return PERM_OK;
  if (int rc = queue_moments(ctx, d_col_fp64, n)) return rc;
  CU(ctx, cudaMemcpyAsync(ctx->h_out + kOutWords, ctx->d_out + kOutWords, 2 * moment_blocks(n) * sizeof(double),
                          cudaMemcpyDeviceToHost, ctx->stream));
  CU(ctx, cudaStreamSynchronize(ctx->stream));
  add_moments(ctx, n);
  estimate_from_moments(ctx, n, op, value, e);
  return PERM_OK;
}

extern "C" int perm_ctx_inject_wait_timeout(perm_ctx* ctx, int launches) {
  if (!ctx || launches < 0) return PERM_EINVAL;
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->inject_timeouts = launches;
  return PERM_OK;
}

extern "C" int perm_ctx_set_rel_target(perm_ctx* ctx, double rel_target) {
  if (!ctx) return PERM_EINVAL;
  ctx->rel_target = rel_target;
  return PERM_OK;
}

static int stage_operand(perm_ctx* ctx, const DenseOperand& op) {
  int rc = ensure_stage(ctx, op.image.size());
  if (rc) return rc;
  memcpy(ctx->h_stage, op.image.data(), op.image.size());
  CU(ctx, cudaMemcpyAsync(ctx->d_stage, ctx->h_stage, op.image.size(), cudaMemcpyHostToDevice, ctx->stream));
  return PERM_OK;
}

// the whole walk of `op` from the staging buffer (context lock held)
static int run_whole(perm_ctx* ctx, const DenseOperand& op, perm_result* out) {
  int rc = stage_operand(ctx, op);
  if (rc) return rc;
  DensePlan p;
  if ((rc = dense_plan(ctx, op, 0, 1, &p))) return rc;
  if ((rc = dense_launch(ctx, op, ctx->d_stage, p))) return rc;
  return dense_collect(ctx, op, p, out);
}

// Bipartite perfect matching of the nonzero pattern (augmenting paths,
// O(n^3) on the host).  Without one every Gray term sum cancels to exactly 0.
static bool has_perfect_matching(const void* mat, int n, int dtype) {
  std::vector<int> match_col(n, -1);
  std::vector<char> seen(n);
  std::function<bool(int)> augment = [&](int r) -> bool {
    for (int c = 0; c < n; c++) {
      if (elem(mat, dtype, (size_t)r * n + c) == 0.0 || seen[c]) continue;
      seen[c] = 1;
      if (match_col[c] < 0 || augment(match_col[c])) {
        match_col[c] = r;
        return true;
      }
    }
    return false;
  };
  for (int r = 0; r < n; r++) {
    std::fill(seen.begin(), seen.end(), 0);
    if (!augment(r)) return false;
  }
  return true;
}

// Error estimate of the whole-walk result in `out` (computed by `op`'s
// kernel) and, with `policy`, the accuracy policy for the context's target:
//  1. a zero pattern without a perfect matching has permanent exactly 0;
//  2. the worst-case bound meets the target: keep;
//  3. cross-check against B = A^T with its first row times 3
//     (perm(B) = 3 perm(A)): B's x vectors are column sums and the factor 3
//     changes every product's significand, even for symmetric or constant
//     matrices, so B's roundings are independent of A's.  Keep when
//     max(independent-rounding estimate, 16 |perm(A) - perm(B)/3| / |perm(A)|)
//     meets the target;
//  4. otherwise recompute with a certified walk: int32 X with double-double
//     products for integer matrices (orders 8..64), split-dd for the rest
//     (orders 4..40), double-double where neither applies (orders <= 40).
// Step 3 is skipped when its independent-rounding estimate alone misses the
// target, after an int32-X first pass (its certified twin costs about 1.2
// walks, less than a failed cross-check plus the rerun), and when split-dd
// applies and the FP64-X bound is above 4x the target (the cross-check
// rarely passes there).
// A certified walk (int32 X with dd products, split-dd) is its own estimate:
// its bound uses the exact sum |term| the walk accumulated.
// Context lock held.
// `matching`: whether the pattern has a perfect matching (-1: not known yet);
// `sampled`: the term moments of `op`'s matrix are in the result block already;
// `term_sum`: the walk's own sum |term|, where the caller has it (0: not).
static int refine_result(perm_ctx* ctx, const void* mat, int n, int dtype, const DenseOperand& op, bool policy,
                         perm_result* out, int matching = -1, bool sampled = false, double term_sum = 0.0) {
  int rc;
  if (policy && (matching < 0 ? !has_perfect_matching(mat, n, dtype) : !matching)) {
    out->value = out->hi = out->lo = 0.0;
    out->abs_term_sum = out->rel_error_estimate = 0.0;
    return PERM_OK;
  }
  if ((op.variant == PERM_KERNEL_DENSE_INT_DD || op.variant == PERM_KERNEL_DENSE_SDD) &&
      out->steps == out->total_steps) {
    ErrEstimate c;
    c.s1 = ctx->walk_m1;
    error_bounds(op.variant, op.group, n, out->value, &c, ctx->walk_terms_per_thread, op.shape);
    out->abs_term_sum = c.s1;
    out->rel_error_estimate = c.worst;
    return PERM_OK;
  }
  ErrEstimate e;
  if (op.abs_sum && out->steps == out->total_steps) {
    // the walk's own sum |term| decides in most cases; the moments are sampled otherwise
    e.s1 = ctx->walk_m1;
    error_bounds(op.variant, op.group, n, out->value, &e, 0, op.shape);
    out->abs_term_sum = e.s1;
    out->rel_error_estimate = e.worst;
    if (!policy || e.worst <= ctx->rel_target) return PERM_OK;
  }
  const double walked = term_sum > 0.0 ? term_sum : e.s1;
  if (sampled) {
    estimate_from_moments(ctx, n, op, out->value, &e);
  } else {
    // the sample takes an FP64 column image; any other operand is replaced by one
    DenseOperand f;
    const DenseOperand* fp = &op;
    if (!plain_columns(op)) {
      std::vector<double> a((size_t)n * n);
      for (size_t i = 0; i < a.size(); i++) a[i] = elem(mat, dtype, i);
      build_fp64_image(a, n, &f);
      fp = &f;
    }
    if ((rc = stage_operand(ctx, *fp))) return rc;
    if ((rc = estimate_error(ctx, ctx->d_stage, n, op, out->value, &e))) return rc;
  }
  if (walked > 0.0) {
    e.s1 = walked;
    error_bounds(op.variant, op.group, n, out->value, &e, 0, op.shape);
  }
  if (op.variant == PERM_KERNEL_DENSE_SPLIT && out->steps == out->total_steps) {
    // the split walk summed its own |terms| and terms^2: exact moments
    e.s1 = ctx->split_m1;
    e.s2 = ctx->split_m2;
    error_bounds(op.variant, 0, n, out->value, &e);
  }
  out->abs_term_sum = e.s1;
  out->rel_error_estimate = e.worst;
  const double target = ctx->rel_target;
  if (!policy || e.worst <= target || op.variant == PERM_KERNEL_DENSE_DD) return PERM_OK;
  const bool int_first = op.variant == PERM_KERNEL_DENSE_INT || op.variant == PERM_KERNEL_DENSE_TC;
  std::vector<double> av((size_t)n * n);
  for (size_t i = 0; i < av.size(); i++) av[i] = elem(mat, dtype, i);
  // Split-dd (orders 4..40) certifies a real matrix in about 4.2 FP64-X walks.
  // An FP64-X bound well above the target rarely passes an FP64-X
  // cross-check (its correlated X roundings give errors near the bound), so
  // the certified walk then runs at once; closer to the target one FP64-X
  // walk of B is tried first.  Split-X cross-checks of A and B would cost
  // 5.4 walks and can still fail, so the policy does not take them.
  const bool sdd_ok = !int_first && n >= 4 && n <= 40 && split_rows_ok(av, n);
  const bool try_cross = out->value != 0.0 && e.random <= target && !int_first &&
                         !(sdd_ok && e.worst > 4.0 * target);
  if (try_cross) {
    std::vector<double> b((size_t)n * n);
    for (int i2 = 0; i2 < n; i2++)
      for (int j2 = 0; j2 < n; j2++)
        b[(size_t)i2 * n + j2] = elem(mat, dtype, (size_t)j2 * n + i2) * (i2 == 0 ? 3.0 : 1.0);
    DenseOperand t;
    perm_result rt;
    if ((rc = build_operand(ctx, b.data(), n, PERM_F64, 0, &t))) return rc;
    if ((rc = run_whole(ctx, t, &rt))) return rc;
    out->kernel_ms += rt.kernel_ms;
    const double diff = std::fabs(out->value - rt.value / 3.0) / std::fabs(out->value);
    const double est = std::max(e.random, 16.0 * diff);
    if (est <= target) {
      out->rel_error_estimate = est;
      return PERM_OK;
    }
  }
  int cv = 0;
  if (int_group_size(av, n) > 0)
    cv = PERM_KERNEL_DENSE_INT_DD;
  else if (n >= 4 && n <= 40 && split_rows_ok(av, n))
    cv = PERM_KERNEL_DENSE_SDD;
  else if (n <= 40)
    cv = PERM_KERNEL_DENSE_DD;
  else
    return PERM_OK;  // no certified kernel for this matrix: keep the bound
  DenseOperand c_op;
  if ((rc = build_operand(ctx, mat, n, dtype, cv, &c_op))) return rc;
  const double first_ms = out->kernel_ms;
  if ((rc = run_whole(ctx, c_op, out))) return rc;
  out->kernel_ms += first_ms;
  if (cv == PERM_KERNEL_DENSE_DD) {
    if ((rc = estimate_error(ctx, ctx->d_stage, n, c_op, out->value, &e))) return rc;
  } else {
    e.s1 = ctx->walk_m1;
    error_bounds(cv, c_op.group, n, out->value, &e, ctx->walk_terms_per_thread, c_op.shape);
  }
  out->abs_term_sum = e.s1;
  out->rel_error_estimate = e.worst;
  return PERM_OK;
}

// With the accuracy policy on, the kernel a whole-walk call starts with
// when a certified walk is cheap enough to go first: int32 X with
// double-double products for integer matrices (about 1.4 int32-X walks, its
// bound needs no sample), split-dd for real matrices whose three sparsest
// columns touch so few rows R that the (7 (6R + 9) + 6n + 5) / 8 FP64 operations
// per Gray step of its sparse layout are no more than the one-level FP64-X
// walk's 2n (sparse real matrices of order 36: R = 6, 67 against 72).  From
// order 25 both walk column cubes instead; the line between them was drawn for
// the row layouts and not moved.
// 0: the FP64-X / int32-X walk goes first (host checks only;
// policy_predicts_sdd may still choose split-dd for a real matrix).
static int policy_first_kernel(const void* mat, int n, int dtype) {
  std::vector<double> a((size_t)n * n);
  for (size_t i = 0; i < a.size(); i++) a[i] = elem(mat, dtype, i);
  if (int_group_size(a, n) > 0) return PERM_KERNEL_DENSE_INT_DD;
  int c3[3];
  if (!split_rows_ok(a, n)) return 0;
  const int r = sdd_inner_rows(a, n, c3);
  if (r > 0 && 7 * (6 * r + 9) + 6 * n + 5 <= 16 * n) return PERM_KERNEL_DENSE_SDD;
  return 0;
}

constexpr int kPredictMinOrder = 28;      // below, FP64-X walks cost less than the prediction
constexpr int kPredictTrials = 4096;      // size-estimate trials (about +-20% at orders 28..40)
constexpr double kPredictMargin = 1.5;    // predicted FP64-X bound / target that sends a matrix to split-dd

// For a nonnegative real matrix of order kPredictMinOrder..40 whose split
// image exists: predicts the FP64-X walk's worst-case bound before running
// it, (2n + 16) u S1 / |perm|, from the stratified sample of S1 = sum|term|
// and a weighted-Rasmussen estimate of perm(A), and sets *sdd when it is
// above kPredictMargin x the target.  Such a walk would be followed by the
// certified split-dd walk anyway (its bound misses the target and an FP64-X
// cross-check rarely passes there), so split-dd alone costs about 4.2
// FP64-X walks instead of 5.2 to 6.2.  Context lock held.
static int policy_predicts_sdd(perm_ctx* ctx, const void* mat, int n, int dtype, bool* sdd, double* bound) {
  *sdd = false;
  *bound = 0.0;
  if (n < kPredictMinOrder || n > 40 || ctx->rel_target <= 0) return PERM_OK;
  std::vector<double> a((size_t)n * n);
  double log2_ub = 0.0;
  for (int j = 0; j < n; j++) {
    double r = 0.0;
    for (int k = 0; k < n; k++) {
      const double v = elem(mat, dtype, (size_t)j * n + k);
      if (!(v >= 0.0) || !std::isfinite(v)) return PERM_OK;  // nonnegative finite entries only
      a[(size_t)j * n + k] = v;
      r += v;
    }
    if (!(r > 0.0)) return PERM_OK;  // a zero row: the policy returns 0 at once
    log2_ub += std::log2(r);
  }
  if (!split_rows_ok(a, n)) return PERM_OK;
  DenseOperand f;
  build_fp64_image(a, n, &f);
  int rc;
  if ((rc = stage_operand(ctx, f))) return rc;
  const int np = (n + 1) & ~1;
  CU(ctx, cudaMemsetAsync(ctx->d_est + 2, 0, 2 * sizeof(double), ctx->stream));
  if ((rc = queue_moments(ctx, ctx->d_stage, n))) return rc;
  weighted_rasmussen_kernel<<<(kPredictTrials + 255) / 256, 256, 0, ctx->stream>>>(
      reinterpret_cast<const double*>(ctx->d_stage), n, np, kPredictTrials, 0x13198A2E03707344ull, log2_ub,
      ctx->d_est + 2);
  CU(ctx, cudaGetLastError());
  CU(ctx, cudaMemcpyAsync(ctx->h_out, ctx->d_out, sizeof(double) * (kOutWords + 2 * moment_blocks(n)),
                          cudaMemcpyDeviceToHost, ctx->stream));
  CU(ctx, cudaStreamSynchronize(ctx->stream));
  add_moments(ctx, n);
  const double s1 = ctx->h_out[12] * 2.0;  // |factor| = 2
  const double mean_scaled = ctx->h_out[14] / kPredictTrials;
  if (!(mean_scaled > 0.0)) return PERM_OK;  // no trial found a permutation: leave it to the walk
  const double log2_perm = std::log2(mean_scaled) + log2_ub;
  const double log2_bound = std::log2((2.0 * n + 16.0) * std::ldexp(1.0, -53) * s1) - log2_perm;
  *bound = std::exp2(log2_bound);
  *sdd = log2_bound > std::log2(kPredictMargin * ctx->rel_target);
  return PERM_OK;
}

// The policy's first kernel for a whole-walk call (variant 0, target > 0),
// with the device prediction for real matrices.  Context lock NOT held.
static int policy_plan(perm_ctx* ctx, const void* mat, int n, int dtype, int* first, double* bound = nullptr) {
  double b = 0.0;
  if (bound) *bound = 0.0;
  *first = policy_first_kernel(mat, n, dtype);
  if (*first) return PERM_OK;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  bool sdd = false;
  const int rc = policy_predicts_sdd(ctx, mat, n, dtype, &sdd, &b);
  if (bound) *bound = b;
  if (rc) return rc;
  if (sdd) *first = PERM_KERNEL_DENSE_SDD;
  return PERM_OK;
}

extern "C" int perm_exact_dense_plan(perm_ctx* ctx, const void* mat, int n, int dtype, int* kernel,
                                     double* fp64_bound) {
  int rc = check_dense_args(ctx, mat, n, dtype, kernel);
  if (rc) return rc;
  *kernel = 0;
  if (fp64_bound) *fp64_bound = 0.0;
  if (ctx->rel_target <= 0) return PERM_OK;
  return policy_plan(ctx, mat, n, dtype, kernel, fp64_bound);
}

// `rows_only`: walked in a row layout, once (no policy).
static int exact_dense_call(perm_ctx* ctx, const void* mat, int n, int dtype, int variant, int shard, int nshards,
                            bool rows_only, perm_result* out) {
  int rc = check_dense_args(ctx, mat, n, dtype, out);
  if (rc) return rc;
  if ((rc = check_variant(ctx, variant))) return rc;
  if (nshards < 1 || shard < 0 || shard >= nshards)
    return fail(ctx, PERM_EINVAL, "shard %d of %d", shard, nshards);
  DenseOperand op;
  int first = 0;
  const bool policed = variant == 0 && nshards == 1 && ctx->rel_target > 0 && !rows_only;
  if (policed && (rc = policy_plan(ctx, mat, n, dtype, &first))) return rc;
  if ((rc = build_operand(ctx, mat, n, dtype, first ? first : variant, &op, policed, rows_only))) return rc;
  // shards are Gray-index ranges of the walking kernels; the tensor-core
  // kernel's operand image is the int32-X one
  if (nshards > 1 && op.variant == PERM_KERNEL_DENSE_TC) op.variant = PERM_KERNEL_DENSE_INT;
  const bool refine = nshards == 1 && ctx->rel_target >= 0;
  op.abs_sum = refine && op.shape >= 0 && op.variant == PERM_KERNEL_DENSE;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  if ((rc = ensure_stage(ctx, op.image.size()))) return rc;
  memcpy(ctx->h_stage, op.image.data(), op.image.size());
  DensePlan p;
  if ((rc = dense_plan(ctx, op, shard, nshards, &p))) return rc;
  CU(ctx, cudaMemcpyAsync(ctx->d_stage, ctx->h_stage, op.image.size(), cudaMemcpyHostToDevice, ctx->stream));
  if ((rc = dense_launch(ctx, op, ctx->d_stage, p))) return rc;
  // The error estimate's sample follows the walk on the stream where it reads
  // the same image, and the matching check runs while both do: one wait and
  // one copy back for all of it (n = 12, real: 55 us a call, 77 with a copy, a
  // second image and a wait of its own for the sample).
  const bool policy = refine && policed;
  const bool sampled = refine && n >= 2 && plain_columns(op);
  if (sampled && (rc = queue_moments(ctx, ctx->d_stage, n))) return rc;
  int matching = -1;
  if ((rc = dense_collect(ctx, op, p, out, sampled, [&] {
         if (policy) matching = has_perfect_matching(mat, n, dtype);
       })))
    return rc;
  out->abs_term_sum = out->rel_error_estimate = 0;
  if (!refine) return PERM_OK;
  return refine_result(ctx, mat, n, dtype, op, policy, out, matching, sampled);
}

extern "C" int perm_exact_dense_ex(perm_ctx* ctx, const void* mat, int n, int dtype, int variant, int shard,
                                   int nshards, perm_result* out) {
  return exact_dense_call(ctx, mat, n, dtype, variant, shard, nshards, false, out);
}

extern "C" int perm_exact_dense_rows(perm_ctx* ctx, const void* mat, int n, int dtype, int variant, int shard,
                                     int nshards, perm_result* out) {
  return exact_dense_call(ctx, mat, n, dtype, variant, shard, nshards, true, out);
}

extern "C" int perm_exact_dense_refine(perm_ctx* ctx, const void* mat, int n, int dtype, perm_result* io) {
  int rc = check_dense_args(ctx, mat, n, dtype, io);
  if (rc) return rc;
  DenseOperand op;
  if ((rc = build_operand(ctx, mat, n, dtype, 0, &op))) return rc;
  if (op.variant == PERM_KERNEL_DENSE_TC) op.variant = PERM_KERNEL_DENSE_INT;  // what the shards ran
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  io->value = io->hi + io->lo;
  io->n = n;
  io->kernel = op.variant;
  io->steps = io->total_steps = std::ldexp(1.0, n - 1);
  io->abs_term_sum = io->rel_error_estimate = 0;
  if (ctx->rel_target < 0) return PERM_OK;
  return refine_result(ctx, mat, n, dtype, op, ctx->rel_target > 0, io);
}

extern "C" int perm_exact_dense_shard(perm_ctx* ctx, const void* mat, int n, int dtype, int shard,
                                      int nshards, perm_result* out) {
  return perm_exact_dense_ex(ctx, mat, n, dtype, 0, shard, nshards, out);
}

extern "C" int perm_exact_dense(perm_ctx* ctx, const void* mat, int n, int dtype, perm_result* out) {
  return perm_exact_dense_ex(ctx, mat, n, dtype, 0, 0, 1, out);
}

extern "C" int perm_matrix_create_dense_ex(perm_ctx* ctx, const void* mat, int n, int dtype, int variant,
                                           perm_matrix** out) {
  int rc = check_dense_args(ctx, mat, n, dtype, out);
  if (rc) return rc;
  if ((rc = check_variant(ctx, variant))) return rc;
  perm_matrix* m = new perm_matrix();
  if ((rc = build_operand(ctx, mat, n, dtype, variant, &m->op))) {
    delete m;
    return rc;
  }
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  cudaError_t e = cudaMalloc(&m->d_image, m->op.image.size());
  if (e != cudaSuccess) {
    delete m;
    return fail_cuda(ctx, e, "cudaMalloc(resident matrix)");
  }
  e = cudaMemcpy(m->d_image, m->op.image.data(), m->op.image.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    cudaFree(m->d_image);
    delete m;
    return fail_cuda(ctx, e, "cudaMemcpy(resident matrix)");
  }
  *out = m;
  return PERM_OK;
}

extern "C" int perm_matrix_create_dense(perm_ctx* ctx, const void* mat, int n, int dtype, perm_matrix** out) {
  return perm_matrix_create_dense_ex(ctx, mat, n, dtype, 0, out);
}

extern "C" void perm_matrix_destroy(perm_ctx* ctx, perm_matrix* m) {
  if (!m) return;
  if (ctx) cudaSetDevice(ctx->device);
  cudaFree(m->d_image);
  delete m;
}

extern "C" int perm_exact_dense_tc_rounds(perm_ctx* ctx, const void* mat, int n, int dtype, uint64_t round0,
                                          uint64_t nrounds, perm_result* out) {
  int rc = check_dense_args(ctx, mat, n, dtype, out);
  if (rc) return rc;
  DenseOperand op;
  if ((rc = build_operand(ctx, mat, n, dtype, PERM_KERNEL_DENSE_TC, &op))) return rc;
  const uint64_t rounds = 1ull << tc_round_bits(n);
  if (nrounds < 1 || round0 >= rounds || nrounds > rounds - round0)
    return fail(ctx, PERM_EINVAL, "rounds [%llu, +%llu) outside [0, %llu)", (unsigned long long)round0,
                (unsigned long long)nrounds, (unsigned long long)rounds);
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  DensePlan p;
  if ((rc = dense_plan(ctx, op, 0, 1, &p))) return rc;
  p.block0 = round0;
  p.nblocks = nrounds;
  // at least 16 rounds per CTA, so that short ranges run through the
  // in-place round updates and not only the from-scratch first rounds
  p.grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((uint64_t)p.grid, nrounds / 16));
  if ((rc = stage_operand(ctx, op))) return rc;
  if ((rc = dense_launch(ctx, op, ctx->d_stage, p))) return rc;
  rc = dense_collect(ctx, op, p, out);
  out->abs_term_sum = out->rel_error_estimate = 0;
  return rc;
}

extern "C" int perm_exact_dense_resident(perm_ctx* ctx, const perm_matrix* m, perm_result* out) {
  return perm_exact_dense_resident_shard(ctx, m, 0, 1, out);
}

extern "C" int perm_exact_dense_resident_shard(perm_ctx* ctx, const perm_matrix* m, int shard, int nshards,
                                               perm_result* out) {
  if (!ctx || !m || !out) return ctx ? fail(ctx, PERM_EINVAL, "null argument") : PERM_EINVAL;
  if (nshards < 1 || shard < 0 || shard >= nshards) return fail(ctx, PERM_EINVAL, "shard %d of %d", shard, nshards);
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  DensePlan p;
  int rc = dense_plan(ctx, m->op, shard, nshards, &p);
  if (rc) return rc;
  if ((rc = dense_launch(ctx, m->op, m->d_image, p))) return rc;
  rc = dense_collect(ctx, m->op, p, out);
  out->abs_term_sum = out->rel_error_estimate = 0;
  return rc;
}

// Autotuner for the automatic dense-kernel choice on integer inputs: for each
// order in [n_lo, n_hi] (8..40) time the int32-X, FP64-X and (orders >= 16)
// tensor-core kernels on a seeded binary matrix and keep the fastest in the
// context.  choice_out (n_hi - n_lo + 1 ints) receives the kernel ids.
extern "C" int perm_dense_autotune(perm_ctx* ctx, int n_lo, int n_hi, int* choice_out) {
  if (!ctx) return PERM_EINVAL;
  if (n_lo < 8 || n_hi > 40 || n_lo > n_hi) return fail(ctx, PERM_EINVAL, "orders [%d, %d] outside [8, 40]", n_lo, n_hi);
  uint64_t state = 0xD1B54A32D192ED03ull;
  for (int n = n_lo; n <= n_hi; n++) {
    std::vector<double> a((size_t)n * n);
    for (double& v : a) {
      state = state * 6364136223846793005ull + 1442695040888963407ull;
      v = (state >> 63) ? 1.0 : 0.0;
    }
    for (int j = 0; j < n; j++) a[(size_t)j * n + j] = 1.0;  // no empty row or column
    const int variants[3] = {PERM_KERNEL_DENSE_INT, PERM_KERNEL_DENSE, PERM_KERNEL_DENSE_TC};
    const int nv = n >= 16 ? 3 : 2;
    double best_ms[3] = {1e30, 1e30, 1e30};
    for (int v = 0; v < nv; v++) {
      for (int rep = 0; rep < 3; rep++) {
        perm_result r;
        int rc = perm_exact_dense_ex(ctx, a.data(), n, PERM_F64, variants[v], 0, 1, &r);
        if (rc) return rc;
        if (rep) best_ms[v] = std::min(best_ms[v], r.kernel_ms);
      }
    }
    int best = 0;
    for (int v = 1; v < nv; v++)
      if (best_ms[v] < best_ms[best]) best = v;
    ctx->dense_pref[n] = variants[best];
    if (choice_out) choice_out[n - n_lo] = ctx->dense_pref[n];
  }
  return PERM_OK;
}

// ---------------------------------------------------------------------------
// SkipPer
// ---------------------------------------------------------------------------
static inline uint32_t align16(uint32_t v) { return (v + 15u) & ~15u; }

static int run_skipper(perm_ctx* ctx, int n, const int* rptrs, const int* cols, const double* rvals,
                       const int* cptrs, const int* rows, const double* cvals, perm_result* out) {
  const int nnz = rptrs[n];
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  // x0 exactly as the reference SkipPer builds it (algo.h:751-760)
  std::vector<double> x0(n);
  for (int j = 0; j < n; j++) {
    double rs = 0;
    for (int p = rptrs[j]; p < rptrs[j + 1]; p++) rs += rvals[p];
    x0[j] = -rs / 2.0;
  }
  for (int p = cptrs[n - 1]; p < cptrs[n]; p++) x0[rows[p]] += cvals[p];

  SkipArgs a;
  a.wide = 4;
  a.exact = 1;
  double size = 0;
  for (int k = 0; k < n; k++) {
    uint64_t seen = 0;
    for (int p = cptrs[k]; p < cptrs[k + 1]; p++) {
      if ((seen >> rows[p]) & 1) a.wide = 1;
      seen |= 1ull << rows[p];
      if (cvals[p] != std::floor(cvals[p])) a.exact = 0;
      size += std::fabs(cvals[p]);
    }
  }
  for (int p = 0; p < nnz; p++) {
    if (rvals[p] != std::floor(rvals[p])) a.exact = 0;
    size += std::fabs(rvals[p]);
  }
  if (!(size < 0x1p50)) a.exact = 0;
  uint32_t off = align16(sizeof(double) * n);
  a.off_cvals = off;
  off = align16(off + sizeof(double) * nnz);
  a.off_rptrs = off;
  off = align16(off + sizeof(int) * (n + 1));
  a.off_cptrs = off;
  off = align16(off + sizeof(int) * (n + 1));
  a.off_cols = off;
  off = align16(off + sizeof(int) * nnz);
  a.off_rows = off;
  off = align16(off + sizeof(int) * nnz);
  a.pack_bytes = off;
  int rc = ensure_stage(ctx, off);
  if (rc) return rc;
  unsigned char* h = ctx->h_stage;
  memset(h, 0, off);
  memcpy(h, x0.data(), sizeof(double) * n);
  memcpy(h + a.off_cvals, cvals, sizeof(double) * nnz);
  memcpy(h + a.off_rptrs, rptrs, sizeof(int) * (n + 1));
  memcpy(h + a.off_cptrs, cptrs, sizeof(int) * (n + 1));
  memcpy(h + a.off_cols, cols, sizeof(int) * nnz);
  memcpy(h + a.off_rows, rows, sizeof(int) * nnz);

  const int block = 128;
  const size_t smem = skipper_smem_bytes(a.pack_bytes, n, block);
  if (smem > 227 * 1024) return fail(ctx, PERM_EUNSUPPORTED, "SkipPer operand needs %zu B of shared memory", smem);
  if ((rc = allow_smem(ctx, (const void*)skipper_kernel, smem))) return rc;
  int occ = 0;
  CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, skipper_kernel, block, smem));
  occ = std::max(occ, 1);
  const uint64_t total = 1ull << (n - 1);
  int grid = std::min(kMaxBlocks, ctx->num_sms * occ);
  const uint64_t threads = (uint64_t)grid * block;
  // 64 indices or more, 32..64 chunks a thread (n = 36, three nonzeros a row:
  // 8 chunks 2.3..5.1 ms, 32 1.4..2.6, 128 2.3..2.6; n = 27: chunks of 32
  // indices 0.15 ms, 128 0.09; n = 24: 0.06, 0.09)
  uint64_t chunk = 64;
  while (chunk < (1ull << 24) && total / (chunk * 2) >= threads * 32) chunk *= 2;
  a.n = n;
  a.total = total;
  a.chunk = chunk;
  a.nchunks = (total + chunk - 1) / chunk;
  if (a.nchunks < threads) grid = (int)std::max<uint64_t>(1, (a.nchunks + block - 1) / block);
  a.pack = ctx->d_stage;
  a.next_chunk = ctx->d_counters;
  a.visited = ctx->d_counters + 1;
  a.partials = ctx->partials;
  a.ticket = ctx->ticket;
  a.out = ctx->d_out;
  a.err = ctx->d_err;
  CU(ctx, cudaMemcpyAsync(ctx->d_stage, h, off, cudaMemcpyHostToDevice, ctx->stream));
  CU(ctx, cudaMemsetAsync(ctx->d_counters, 0, sizeof(unsigned long long) * 2, ctx->stream));
  void* kargs[] = {&a};
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  CU(ctx, cudaLaunchKernel((const void*)skipper_kernel, dim3(grid), dim3(block), kargs, smem, ctx->stream));
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  rc = finish_and_read(ctx);
  if (rc) return rc;
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  unsigned long long vis = 0;
  memcpy(&vis, ctx->h_out + 10, sizeof vis);
  out->hi = ctx->h_out[0];
  out->lo = ctx->h_out[1];
  out->value = out->hi + out->lo;
  out->steps = (double)vis;
  out->total_steps = std::ldexp(1.0, n - 1);
  out->kernel_ms = ms;
  out->kernel = PERM_KERNEL_SKIPPER;
  out->n = n;
  return PERM_OK;
}

// Whether at least kSkipperZeroFraction of the Gray indices of a fixed
// pseudo-random sample (deterministic) have an x vector with a zero entry.
// SkipPer only pays off when most terms vanish: a visited index costs it
// several times a dense-kernel step, so below kSkipperZeroFraction the register
// kernel runs instead (same matrix, same permanent).  The line was drawn against
// the row layouts; column cubes win somewhat above it too (0/1 matrices, n = 36:
// 1e7..7e7 visited indices 1.5..3.5 ms and 33 in cubes, 1.1e9 of them 43 ms and
// 33; n = 30: 5e6 0.4..0.5 ms, 1.8e7 1.3, cubes 0.51).  Row by row up to the
// first zero, and until the answer is settled (the call beyond the kernel, n =
// 36, three nonzeros a row: 0.55 ms with every x vector built whole, 0.1 so).
static const double kSkipperZeroFraction = 0.75;

static bool mostly_zero_terms(int n, const int* rptrs, const int* cols, const double* rvals, const int* cptrs,
                              const int* rows, const double* cvals, int samples) {
  const int least = (int)std::ceil(kSkipperZeroFraction * samples);
  std::vector<double> x0(n);
  for (int j = 0; j < n; j++) {
    double rs = 0;
    for (int p = rptrs[j]; p < rptrs[j + 1]; p++) rs += rvals[p];
    x0[j] = -rs / 2.0;
  }
  for (int p = cptrs[n - 1]; p < cptrs[n]; p++) x0[rows[p]] += cvals[p];
  const uint64_t total = 1ull << (n - 1);
  uint64_t state = 0x9E3779B97F4A7C15ull;
  int zeros = 0;
  for (int s = 0; s < samples; s++) {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    const uint64_t i = (state >> 1) % total;
    const uint64_t g = i ^ (i >> 1);  // column n-1 is never in it
    for (int j = n - 1; j >= 0; j--) {
      double x = x0[j];
      for (int p = rptrs[j]; p < rptrs[j + 1]; p++)
        if ((g >> cols[p]) & 1) x += rvals[p];
      if (x == 0.0) {
        zeros++;
        break;
      }
    }
    if (zeros >= least || zeros + samples - 1 - s < least) break;
  }
  return zeros >= least;
}

extern "C" int perm_exact_sparse_ex(perm_ctx* ctx, int n, const int* rptrs, const int* cols, const double* rvals,
                                    const int* cptrs, const int* rows, const double* cvals, int variant,
                                    perm_result* out) {
  if (!ctx) return PERM_EINVAL;
  if (!rptrs || !cols || !rvals || !cptrs || !rows || !cvals || !out)
    return fail(ctx, PERM_EINVAL, "null CRS/CCS or result pointer");
  if (n < 1 || n > PERM_MAX_EXACT_N) return fail(ctx, PERM_EUNSUPPORTED, "order %d outside [1, %d]", n, PERM_MAX_EXACT_N);
  const int nnz = rptrs[n];
  if (nnz < 0 || nnz > n * n || cptrs[n] != nnz || rptrs[0] != 0 || cptrs[0] != 0)
    return fail(ctx, PERM_EINVAL, "inconsistent CRS/CCS (rptrs[n]=%d, cptrs[n]=%d)", nnz, cptrs[n]);
  for (int i = 0; i < n; i++)
    if (rptrs[i + 1] < rptrs[i] || cptrs[i + 1] < cptrs[i])
      return fail(ctx, PERM_EINVAL, "pointer arrays must be non-decreasing");
  for (int p = 0; p < nnz; p++)
    if (cols[p] < 0 || cols[p] >= n || rows[p] < 0 || rows[p] >= n)
      return fail(ctx, PERM_EINVAL, "index out of range at entry %d", p);
  if (variant != 0 && variant != PERM_KERNEL_SKIPPER && variant != PERM_KERNEL_DENSE &&
      variant != PERM_KERNEL_DENSE_INT && variant != PERM_KERNEL_DENSE_TC && variant != PERM_KERNEL_DENSE_INT_DD &&
      variant != PERM_KERNEL_DENSE_SDD)
    return fail(ctx, PERM_EINVAL, "unknown sparse kernel variant %d", variant);
  bool skipper = variant == PERM_KERNEL_SKIPPER;
  if (variant == 0) skipper = n < 8 || mostly_zero_terms(n, rptrs, cols, rvals, cptrs, rows, cvals, 2048);
  if (skipper) return run_skipper(ctx, n, rptrs, cols, rvals, cptrs, rows, cvals, out);
  // the matrix the CRS describes, for the register kernels
  std::vector<double> a((size_t)n * n, 0.0);
  for (int i = 0; i < n; i++)
    for (int p = rptrs[i]; p < rptrs[i + 1]; p++) a[(size_t)i * n + cols[p]] = rvals[p];
  return perm_exact_dense_ex(ctx, a.data(), n, PERM_F64, variant == PERM_KERNEL_SKIPPER ? 0 : variant, 0, 1, out);
}

extern "C" int perm_exact_sparse(perm_ctx* ctx, int n, const int* rptrs, const int* cols, const double* rvals,
                                 const int* cptrs, const int* rows, const double* cvals, perm_result* out) {
  return perm_exact_sparse_ex(ctx, n, rptrs, cols, rvals, cptrs, rows, cvals, 0, out);
}

// ---------------------------------------------------------------------------
// Monte Carlo
// ---------------------------------------------------------------------------
static int mc_run(perm_ctx* ctx, const std::vector<uint64_t>& rowmask, const std::vector<double>* dense,
                  int n, bool scaling, int64_t trials, int y, int z, uint64_t seed, double* trial_values,
                  perm_estimate* out, uint64_t trial0 = 0) {
  if (trials < 1) return fail(ctx, PERM_EINVAL, "trials must be >= 1 (got %lld)", (long long)trials);
  if (scaling && (y < 1 || z < 0)) return fail(ctx, PERM_EINVAL, "scale interval must be >= 1 and scale times >= 0");
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  const int np = (n + 1) & ~1;
  McArgs a;
  a.n = n;
  a.np = np;
  a.y = y;
  a.z = z;
  a.mask_bytes = sizeof(uint64_t) * np;
  // 0/1 matrices take the mask-only scaling kernel (same FP64 results)
  bool binary = scaling;
  if (scaling)
    for (double v : *dense)
      if (v != 0.0 && v != 1.0) {
        binary = false;
        break;
      }
  a.pack_bytes = a.mask_bytes + (binary ? a.mask_bytes : scaling ? 2 * sizeof(double) * (size_t)n * np : 0);
  int rc = ensure_stage(ctx, a.pack_bytes);
  if (rc) return rc;
  unsigned char* h = ctx->h_stage;
  memset(h, 0, a.pack_bytes);
  memcpy(h, rowmask.data(), sizeof(uint64_t) * n);
  if (binary) {
    uint64_t* colmask = reinterpret_cast<uint64_t*>(h + a.mask_bytes);
    for (int i = 0; i < n; i++)
      for (int j = 0; j < n; j++)
        if ((*dense)[(size_t)i * n + j] != 0.0) colmask[j] |= 1ull << i;
  } else if (scaling) {
    double* A = reinterpret_cast<double*>(h + a.mask_bytes);
    double* AT = A + (size_t)n * np;
    for (int i = 0; i < n; i++)
      for (int j = 0; j < n; j++) {
        A[(size_t)i * np + j] = (*dense)[(size_t)i * n + j];
        AT[(size_t)j * np + i] = (*dense)[(size_t)i * n + j];
      }
  }
  const size_t smem = mc_smem_bytes(a.pack_bytes, scaling);
  const void* fn = binary ? (const void*)scaling_kernel_binary
                 : scaling ? (const void*)scaling_kernel
                           : (const void*)rasmussen_kernel;
  if ((rc = allow_smem(ctx, fn, smem))) return rc;
  int occ = 0;
  CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kMcBlock, smem));
  occ = std::max(occ, 1);
  const uint64_t warps_needed = (uint64_t)trials;
  int grid = std::min<uint64_t>(std::min(kMaxBlocks, ctx->num_sms * occ), (warps_needed + 7) / 8);
  grid = std::max(grid, 1);
  if (trial_values && (size_t)trials > ctx->d_trials_cap) {
    cudaFree(ctx->d_trials);
    ctx->d_trials = nullptr;
    ctx->d_trials_cap = 0;
    CU(ctx, cudaMalloc(&ctx->d_trials, sizeof(double) * trials));
    ctx->d_trials_cap = trials;
  }
  a.pack = ctx->d_stage;
  a.trials = trials;
  a.trial0 = trial0;
  a.seed = seed;
  a.trial_out = trial_values ? ctx->d_trials : nullptr;
  a.partials = reinterpret_cast<double*>(ctx->partials);
  a.ticket = ctx->ticket;
  a.out = ctx->d_out;
  a.err = ctx->d_err;
  CU(ctx, cudaMemcpyAsync(ctx->d_stage, h, a.pack_bytes, cudaMemcpyHostToDevice, ctx->stream));
  void* kargs[] = {&a};
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  CU(ctx, cudaLaunchKernel(fn, dim3(grid), dim3(kMcBlock), kargs, smem, ctx->stream));
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  if (trial_values)
    CU(ctx, cudaMemcpyAsync(trial_values, ctx->d_trials, sizeof(double) * trials, cudaMemcpyDeviceToHost,
                            ctx->stream));
  rc = finish_and_read(ctx);
  if (rc) return rc;
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  const double T = (double)trials, sum = ctx->h_out[0], sq = ctx->h_out[1];
  out->trials = T;
  out->sum = sum;
  out->sum_sq = sq;
  out->zero_trials = ctx->h_out[2];
  out->mean = sum / T;
  double var = T > 1 ? (sq - sum * out->mean) / (T - 1) : 0.0;
  if (!(var > 0)) var = 0;
  out->std_error = std::sqrt(var / T);
  out->kernel_ms = ms;
  return PERM_OK;
}

static int mc_dense(perm_ctx* ctx, const void* mat, int n, int dtype, bool scaling, int64_t trials, int y,
                    int z, uint64_t seed, double* tv, perm_estimate* out, uint64_t trial0 = 0) {
  if (!ctx) return PERM_EINVAL;
  if (!mat || !out) return fail(ctx, PERM_EINVAL, "null matrix or result pointer");
  if (n < 1 || n > PERM_MAX_MC_N) return fail(ctx, PERM_EUNSUPPORTED, "order %d outside [1, %d]", n, PERM_MAX_MC_N);
  if (dtype != PERM_F64 && dtype != PERM_F32 && dtype != PERM_I32) return fail(ctx, PERM_EINVAL, "unknown dtype %d", dtype);
  std::vector<uint64_t> mask(n, 0);
  std::vector<double> dense((size_t)n * n);
  for (int i = 0; i < n; i++)
    for (int j = 0; j < n; j++) {
      double v = elem(mat, dtype, (size_t)i * n + j);
      dense[(size_t)i * n + j] = v;
      if (v != 0.0) mask[i] |= 1ull << j;
    }
  return mc_run(ctx, mask, &dense, n, scaling, trials, y, z, seed, tv, out, trial0);
}

// Orders above 64: bitset kernel on the packed CRS + CCS of the pattern.
static int mc_sparse_large(perm_ctx* ctx, int n, const int* rptrs, const int* cols, bool scaling, int64_t trials,
                           int y, int z, uint64_t seed, double* tv, perm_estimate* out, uint64_t trial0 = 0) {
  if (trials < 1) return fail(ctx, PERM_EINVAL, "trials must be >= 1 (got %lld)", (long long)trials);
  if (scaling && (y < 1 || z < 0)) return fail(ctx, PERM_EINVAL, "scale interval must be >= 1 and scale times >= 0");
  const int nnz = rptrs[n];
  // CCS rebuilt from the CRS so that both lists are in ascending order
  std::vector<int> cptrs(n + 1, 0), rows(std::max(nnz, 1));
  for (int p = 0; p < nnz; p++) cptrs[cols[p] + 1]++;
  for (int j = 0; j < n; j++) cptrs[j + 1] += cptrs[j];
  std::vector<int> fill(cptrs.begin(), cptrs.end() - 1);
  for (int i = 0; i < n; i++)
    for (int p = rptrs[i]; p < rptrs[i + 1]; p++) rows[fill[cols[p]]++] = i;
  McSparseArgs a;
  a.n = n;
  a.scaling = scaling ? 1 : 0;
  a.y = y;
  a.z = z;
  a.ptr_ints = (n + 1 + 3) & ~3;
  a.idx_ints = (nnz + 3) & ~3;
  a.pack_bytes = (uint32_t)(sizeof(int) * (2 * (size_t)a.ptr_ints + 2 * (size_t)a.idx_ints));
  const size_t smem = mc_sparse_smem_bytes(a.pack_bytes, n, a.scaling);
  if (smem > 227 * 1024)
    return fail(ctx, PERM_EUNSUPPORTED, "order %d with %d nonzeros needs %zu B of shared memory", n, nnz, smem);
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  int rc = ensure_stage(ctx, a.pack_bytes);
  if (rc) return rc;
  int* h = reinterpret_cast<int*>(ctx->h_stage);
  memset(h, 0, a.pack_bytes);
  memcpy(h, rptrs, sizeof(int) * (n + 1));
  memcpy(h + a.ptr_ints, cptrs.data(), sizeof(int) * (n + 1));
  memcpy(h + 2 * a.ptr_ints, cols, sizeof(int) * nnz);
  memcpy(h + 2 * a.ptr_ints + a.idx_ints, rows.data(), sizeof(int) * nnz);
  if ((rc = allow_smem(ctx, (const void*)mc_sparse_kernel, smem))) return rc;
  int occ = 0;
  CU(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, mc_sparse_kernel, kMcSparseBlock, smem));
  occ = std::max(occ, 1);
  const int wpb = kMcSparseBlock / 32;
  int grid = (int)std::min<uint64_t>(std::min(kMaxBlocks, ctx->num_sms * occ), ((uint64_t)trials + wpb - 1) / wpb);
  grid = std::max(grid, 1);
  if (tv && (size_t)trials > ctx->d_trials_cap) {
    cudaFree(ctx->d_trials);
    ctx->d_trials = nullptr;
    ctx->d_trials_cap = 0;
    CU(ctx, cudaMalloc(&ctx->d_trials, sizeof(double) * trials));
    ctx->d_trials_cap = trials;
  }
  a.pack = ctx->d_stage;
  a.trials = trials;
  a.trial0 = trial0;
  a.seed = seed;
  a.trial_out = tv ? ctx->d_trials : nullptr;
  a.partials = reinterpret_cast<double*>(ctx->partials);
  a.ticket = ctx->ticket;
  a.out = ctx->d_out;
  a.err = ctx->d_err;
  CU(ctx, cudaMemcpyAsync(ctx->d_stage, h, a.pack_bytes, cudaMemcpyHostToDevice, ctx->stream));
  void* kargs[] = {&a};
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  CU(ctx, cudaLaunchKernel((const void*)mc_sparse_kernel, dim3(grid), dim3(kMcSparseBlock), kargs, smem, ctx->stream));
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  if (tv) CU(ctx, cudaMemcpyAsync(tv, ctx->d_trials, sizeof(double) * trials, cudaMemcpyDeviceToHost, ctx->stream));
  rc = finish_and_read(ctx);
  if (rc) return rc;
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  const double T = (double)trials, sum = ctx->h_out[0], sq = ctx->h_out[1];
  out->trials = T;
  out->sum = sum;
  out->sum_sq = sq;
  out->zero_trials = ctx->h_out[2];
  out->mean = sum / T;
  double var = T > 1 ? (sq - sum * out->mean) / (T - 1) : 0.0;
  if (!(var > 0)) var = 0;
  out->std_error = std::sqrt(var / T);
  out->kernel_ms = ms;
  return PERM_OK;
}

static int mc_sparse(perm_ctx* ctx, int n, const int* rptrs, const int* cols, bool scaling, int64_t trials,
                     int y, int z, uint64_t seed, double* tv, perm_estimate* out, uint64_t trial0 = 0) {
  if (!ctx) return PERM_EINVAL;
  if (!rptrs || !cols || !out) return fail(ctx, PERM_EINVAL, "null CRS or result pointer");
  if (n < 1 || n > kMcSparseMaxOrder)
    return fail(ctx, PERM_EUNSUPPORTED, "order %d outside [1, %d]", n, kMcSparseMaxOrder);
  if (rptrs[0] != 0) return fail(ctx, PERM_EINVAL, "rptrs[0] must be 0");
  for (int i = 0; i < n; i++) {
    if (rptrs[i + 1] < rptrs[i]) return fail(ctx, PERM_EINVAL, "rptrs must be non-decreasing");
    for (int p = rptrs[i]; p < rptrs[i + 1]; p++) {
      if (cols[p] < 0 || cols[p] >= n) return fail(ctx, PERM_EINVAL, "column index out of range");
      if (p > rptrs[i] && cols[p] <= cols[p - 1]) return fail(ctx, PERM_EINVAL, "CRS columns must ascend within a row");
    }
  }
  if (n > PERM_MAX_MC_N) return mc_sparse_large(ctx, n, rptrs, cols, scaling, trials, y, z, seed, tv, out, trial0);
  std::vector<uint64_t> mask(n, 0);
  std::vector<double> pattern((size_t)n * n, 0.0);
  for (int i = 0; i < n; i++)
    for (int p = rptrs[i]; p < rptrs[i + 1]; p++) {
      mask[i] |= 1ull << cols[p];
      pattern[(size_t)i * n + cols[p]] = 1.0;  // the sparse estimators use the pattern only
    }
  return mc_run(ctx, mask, &pattern, n, scaling, trials, y, z, seed, tv, out, trial0);
}

// Grid-graph input (util.h:403-520): dense 0/1 matrix of an m x n board.
extern "C" int perm_grid_graph(int m, int n, int cap_n, double* out, int* nov_out) {
  if (!out || !nov_out) return PERM_EINVAL;
  HostMatrix g;
  std::string err = grid_graph(m, n, &g);
  if (!err.empty()) {
    fprintf(stderr, "perm_grid_graph: %s\n", err.c_str());
    return PERM_EINVAL;
  }
  if (g.n > cap_n) return PERM_EUNSUPPORTED;
  std::copy(g.a.begin(), g.a.end(), out);
  *nov_out = g.n;
  return PERM_OK;
}

extern "C" int perm_approx_rasmussen(perm_ctx* ctx, const void* mat, int n, int dtype, int64_t trials,
                                     uint64_t seed, double* tv, perm_estimate* out) {
  return mc_dense(ctx, mat, n, dtype, false, trials, 1, 0, seed, tv, out);
}
extern "C" int perm_approx_scaling(perm_ctx* ctx, const void* mat, int n, int dtype, int64_t trials, int y,
                                   int z, uint64_t seed, double* tv, perm_estimate* out) {
  return mc_dense(ctx, mat, n, dtype, true, trials, y, z, seed, tv, out);
}
// Trials [trial0, trial0 + trials) of the same streams: ranges of one
// estimate run on different devices give the per-trial weights of the whole
// run (the estimators' multi-GPU split by trial id).
extern "C" int perm_approx_rasmussen_range(perm_ctx* ctx, const void* mat, int n, int dtype, int64_t trial0,
                                           int64_t trials, uint64_t seed, double* tv, perm_estimate* out) {
  if (!ctx) return PERM_EINVAL;
  if (trial0 < 0) return fail(ctx, PERM_EINVAL, "first trial must be >= 0 (got %lld)", (long long)trial0);
  return mc_dense(ctx, mat, n, dtype, false, trials, 1, 0, seed, tv, out, (uint64_t)trial0);
}
extern "C" int perm_approx_scaling_range(perm_ctx* ctx, const void* mat, int n, int dtype, int64_t trial0,
                                         int64_t trials, int y, int z, uint64_t seed, double* tv,
                                         perm_estimate* out) {
  if (!ctx) return PERM_EINVAL;
  if (trial0 < 0) return fail(ctx, PERM_EINVAL, "first trial must be >= 0 (got %lld)", (long long)trial0);
  return mc_dense(ctx, mat, n, dtype, true, trials, y, z, seed, tv, out, (uint64_t)trial0);
}
extern "C" int perm_approx_rasmussen_sparse(perm_ctx* ctx, int n, const int* rptrs, const int* cols,
                                            int64_t trials, uint64_t seed, double* tv, perm_estimate* out) {
  return mc_sparse(ctx, n, rptrs, cols, false, trials, 1, 0, seed, tv, out);
}
extern "C" int perm_approx_scaling_sparse(perm_ctx* ctx, int n, const int* rptrs, const int* cols,
                                          const int* cptrs, const int* rows, int64_t trials, int y, int z,
                                          uint64_t seed, double* tv, perm_estimate* out) {
  (void)cptrs;
  (void)rows;
  return mc_sparse(ctx, n, rptrs, cols, true, trials, y, z, seed, tv, out);
}
extern "C" int perm_approx_rasmussen_sparse_range(perm_ctx* ctx, int n, const int* rptrs, const int* cols,
                                                  int64_t trial0, int64_t trials, uint64_t seed, double* tv,
                                                  perm_estimate* out) {
  if (!ctx) return PERM_EINVAL;
  if (trial0 < 0) return fail(ctx, PERM_EINVAL, "first trial must be >= 0 (got %lld)", (long long)trial0);
  return mc_sparse(ctx, n, rptrs, cols, false, trials, 1, 0, seed, tv, out, (uint64_t)trial0);
}
extern "C" int perm_approx_scaling_sparse_range(perm_ctx* ctx, int n, const int* rptrs, const int* cols,
                                                int64_t trial0, int64_t trials, int y, int z, uint64_t seed,
                                                double* tv, perm_estimate* out) {
  if (!ctx) return PERM_EINVAL;
  if (trial0 < 0) return fail(ctx, PERM_EINVAL, "first trial must be >= 0 (got %lld)", (long long)trial0);
  return mc_sparse(ctx, n, rptrs, cols, true, trials, y, z, seed, tv, out, (uint64_t)trial0);
}

// ---------------------------------------------------------------------------
// batched exact permanents (one persistent launch, captured in a CUDA graph)
// ---------------------------------------------------------------------------
// One matrix of a batch that walks in column cubes, by a launch of its own in
// the batch's graph.
struct BatchCube {
  DenseOperand op;
  int index = 0;        // position in the caller's batch
  uint64_t offset = 0;  // of its image in d_cubes, bytes
};

// A batch's sums of |term| of its column cubes: one block per cube adds its
// warps' sums in a fixed order.
struct CubeSum {
  uint64_t first;  // of its words in the partials of all cubes
  int count;
  int index;  // of the matrix
};
__global__ void __launch_bounds__(128) cube_sums_kernel(const CubeSum* cubes, const double* partials, double* results) {
  __shared__ double red[4];
  const CubeSum c = cubes[blockIdx.x];
  double s = 0.0;
  const double* warps = partials + c.first + 2 * (c.count / kCubeWarps);
  for (int w = threadIdx.x; w < c.count; w += 128) s += warps[w];
  for (int d = 16; d >= 1; d >>= 1) s += __shfl_down_sync(0xffffffffu, s, d);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) results[3 * (size_t)c.index + 2] = ((red[0] + red[1]) + red[2]) + red[3];
}

struct perm_batch {
  int count = 0;
  uint64_t total_tiles = 0;
  int grid = 1;
  int variant = 0;  // kBatchVariants index
  int sparse = 0;   // matrices walked in the sparse layout
  double* d_operands = nullptr;
  BatchMatrix* d_mats = nullptr;
  dd* d_tile_partials = nullptr;
  double* d_tile_abs = nullptr;
  unsigned* d_mat_done = nullptr;
  unsigned long long* d_next = nullptr;
  double* d_results = nullptr;
  double* h_results = nullptr;  // pinned: (hi, lo, sum |term|) per matrix, then the error flag
  unsigned char* d_cubes = nullptr;  // column images of the column-cube walks
  double* d_cube_partials = nullptr;  // of all cubes
  unsigned* d_cube_tickets = nullptr;  // per branch of the graph
  CubeSum* d_cube_sum = nullptr;      // where each cube's are
  std::vector<double> roundings;  // per matrix: roundings per term
  std::vector<double> abs_scale;  // per matrix: factor of its sum |term|
  std::vector<std::pair<int, int>> exp2;  // matrices whose three results are multiplied by 2^second
  std::vector<int> groups;       // per matrix: 0 = FP64 X, else the int32-X group size
  std::vector<int> shapes;       // per matrix: of its column-cube walk, -1: row layout
  std::vector<int> orders;       // host copies for double-double reruns
  std::vector<uint64_t> offsets;
  std::vector<double> values;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
};

static void batch_free(perm_batch* b) {
  if (!b) return;
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  cudaFree(b->d_operands);
  cudaFree(b->d_mats);
  cudaFree(b->d_tile_partials);
  cudaFree(b->d_tile_abs);
  cudaFree(b->d_mat_done);
  cudaFree(b->d_next);
  cudaFree(b->d_results);
  cudaFree(b->d_cubes);
  cudaFree(b->d_cube_partials);
  cudaFree(b->d_cube_tickets);
  cudaFree(b->d_cube_sum);
  if (b->h_results) cudaFreeHost(b->h_results);
  delete b;
}

// The matrices of a batch that walk in column cubes, with their operands.  The
// searches (some 30 us each) are shared out over up to 8 host threads.
static void batch_cubes(int count, const int* orders, const double* values, std::vector<BatchCube>* out) {
  std::vector<BatchCube> found;
  std::vector<uint64_t> offset;
  uint64_t off = 0;
  for (int i = 0; i < count; i++) {
    if (orders[i] < 1 || orders[i] > kBatchMaxOrder) return;  // refused by the caller
    if (orders[i] >= kBatchCubeMinN) {
      found.emplace_back();
      found.back().index = i;
      offset.push_back(off);
    }
    off += (uint64_t)orders[i] * orders[i];
  }
  if (found.size() > kBatchMaxCubes) {
    std::vector<size_t> by_order(found.size());
    for (size_t k = 0; k < by_order.size(); k++) by_order[k] = k;
    std::stable_sort(by_order.begin(), by_order.end(),
                     [&](size_t x, size_t y) { return orders[found[x].index] > orders[found[y].index]; });
    std::sort(by_order.begin(), by_order.begin() + kBatchMaxCubes);
    size_t kept = 0;
    for (; kept < kBatchMaxCubes; kept++) {
      offset[kept] = offset[by_order[kept]];
      found[kept].index = found[by_order[kept]].index;
    }
    found.resize(kept);
  }
  const size_t threads = std::min<size_t>({found.size() / 8, std::thread::hardware_concurrency(), 8});
  for_each_shared(found.size(), threads ? threads - 1 : 0, [&](size_t k) {
    const int n = orders[found[k].index];
    const std::vector<double> a(values + offset[k], values + offset[k] + (size_t)n * n);
    const int G = int_group_size(a, n);
    DenseOperand& op = found[k].op;
    op.variant = G ? PERM_KERNEL_DENSE_INT : PERM_KERNEL_DENSE;
    IntRows int_rows;
    Fp64Rows rows;
    if (!(G ? cube_operand_int(a, n, G, false, &int_rows, &op) : cube_operand_f64(a, n, &rows, &op))) op.shape = -1;
  });
  for (BatchCube& c : found)
    if (c.op.shape >= 0) out->push_back(std::move(c));
}

static int batch_create_locked(perm_ctx* ctx, int count, const int* orders, const double* values,
                               const int* m_override, perm_batch** out, int variant_override = -1,
                               bool cubes = true) {
  if (count < 1 || !orders || !values || !out) return fail(ctx, PERM_EINVAL, "empty batch or null pointer");
  std::vector<BatchMatrix> mats(count);
  std::vector<uint64_t> src_off(count);
  std::vector<std::vector<double>> sparse_images(count);  // permuted matrices of the sparse layout
  // Larger matrices walk in column cubes where that is cheaper.
  std::vector<BatchCube> cube;
  std::vector<int> cube_of(count, -1);
  try {
    if (cubes) batch_cubes(count, orders, values, &cube);
  } catch (const std::bad_alloc&) {
    return fail(ctx, PERM_ENOMEM, "no host memory for the layouts of %d matrices", count);
  }
  for (size_t k = 0; k < cube.size(); k++) cube_of[cube[k].index] = (int)k;
  uint64_t cube_bytes = 0;
  uint64_t off = 0, img = 0;
  for (int i = 0; i < count; i++) {
    const int n = orders[i];
    if (n < 1 || n > kBatchMaxOrder)
      return fail(ctx, PERM_EUNSUPPORTED, "batch order %d (matrix %d) outside [1, %d]", n, i, kBatchMaxOrder);
    src_off[i] = off;
    off += (uint64_t)n * n;
    BatchMatrix& M = mats[i];
    M.n = n;
    M.index = i;
    M.m = m_override ? m_override[n] : (ctx->batch_m[n] ? ctx->batch_m[n] : batch_default_m(n));
    if (n >= 9 && (M.m < 3 || M.m > n - 6)) M.m = batch_default_m(n);
    M.ntiles = n < 9 ? 1u : (uint32_t)((1ull << (n - 1)) >> (M.m + 5));
    const int np = (n + 1) & ~1;
    M.offset = img;
    img += (uint64_t)n * np;
    // int32 X for integer matrices whose groups of 5 or 6 rows fit in int32
    // (every 0/1 matrix up to order 35); FP64 X otherwise
    M.g = 0;
    M.r = 0;
    if (n >= 9) {
      std::vector<double> a(values + src_off[i], values + src_off[i] + (size_t)n * n);
      const int G = int_group_size(a, n);
      if (G >= 5) M.g = G;
      if (cube_of[i] >= 0) {
        BatchCube& c = cube[cube_of[i]];
        c.offset = cube_bytes;
        cube_bytes += (c.op.image.size() + 255) & ~(uint64_t)255;
        M.g = G;
        img -= (uint64_t)n * np;
        continue;
      }
      // two-level (sparse) layout (orders 12..32) when three columns have
      // their nonzeros in few rows: FP64 X with 8, 16, 20 or 24 inner rows,
      // int32 X (groups of 6) with 6, 12, 18 or 24; taken while the inner
      // steps' 2R + 1 operations keep the 8-step cost 7 (2R + 1) + 2n within
      // 0.85 of the one-level walk's 16n (dense matrices of density up to
      // about 0.55 at these orders)
      if (n >= 12 && n <= 32) {
        int c3[3];
        const int u = sparsest_column_triple(a, n, c3);
        int r = 0;
        if (M.g)
          r = u <= 6 ? 6 : u <= 12 ? 12 : u <= 18 ? 18 : u <= 24 ? 24 : 0;
        else
          r = u <= 8 ? 8 : u <= 16 ? 16 : u <= 20 ? 20 : u <= 24 ? 24 : 0;
        if (r > 16 && 7 * (2 * r + 1) + 2 * n > 0.85 * 16 * n) r = 0;
        if (r && r + 4 <= n) {
          std::vector<double> p = sparse_permutation(a.data(), n, c3);
          if (!M.g || int_group_size(p, n) == 6) {
            M.r = r;
            if (M.g) M.g = 6;
            sparse_images[i] = std::move(p);
          }
        }
      }
    }
  }
  // queue order: most Gray work first (longest-processing-time scheduling)
  std::vector<int> order;
  for (int i = 0; i < count; i++)
    if (cube_of[i] < 0) order.push_back(i);
  // A tile of 2^12 indices per lane takes 0.27 ms whatever else the chip does,
  // so where the batch has few of them the lane ranges are cut, the longest
  // first, until there are 16 tiles an SM (32 and 64 are no better), down to
  // 2^kBatchMinM indices (with 2^6 the columns' staging shows, 2^8 leaves warps
  // idle).  16 matrices of order 18: 285 -> 43 us, 130 of order 18: 286 -> 100,
  // of order 21: 495 -> 422, of orders 15..21: 305 -> 190.
  if (!m_override) {
    int cap = 0;
    for (int i : order) cap = std::max(cap, mats[i].m);
    for (;; cap--) {
      uint64_t have = 0;
      for (int i : order) {
        BatchMatrix& M = mats[i];
        if (M.n >= 9 && M.m > cap) {
          M.m = cap;
          M.ntiles = (uint32_t)((1ull << (M.n - 1)) >> (cap + 5));
        }
        have += M.ntiles;
      }
      if (cap <= kBatchMinM || have >= 16ull * ctx->num_sms) break;
    }
  }
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return mats[x].n > mats[y].n; });
  std::stable_sort(cube.begin(), cube.end(), [](const BatchCube& x, const BatchCube& y) { return x.op.n > y.op.n; });
  const int queued = (int)order.size();
  std::vector<BatchMatrix> q(queued);
  uint64_t tiles = 0;
  for (int r = 0; r < queued; r++) {
    q[r] = mats[order[r]];
    q[r].first_tile = tiles;
    tiles += q[r].ntiles;
  }
  std::vector<double> image(img);
  for (int i = 0; i < count; i++) {
    if (cube_of[i] >= 0) continue;
    const int n = mats[i].n, np = (n + 1) & ~1;
    const double* a = mats[i].r ? sparse_images[i].data() : values + src_off[i];
    double* dst = image.data() + mats[i].offset;
    if (mats[i].g) {
      // doubled int columns (stride np4), then y0 = 2 a[j][n-1] - rowsum_j;
      // (n + 1) np4 words fit in the n np doubles reserved for the matrix
      const int np4 = (n + 3) & ~3;
      int* di = reinterpret_cast<int*>(dst);
      for (int k = 0; k < n; k++)
        for (int j = 0; j < np4; j++) di[(size_t)k * np4 + j] = j < n ? 2 * (int)a[(size_t)j * n + k] : 0;
      for (int j = 0; j < np4; j++) {
        long long rs = 0;
        if (j < n)
          for (int k = 0; k < n; k++) rs += (long long)a[(size_t)j * n + k];
        di[(size_t)n * np4 + j] = j < n ? (int)(2 * (long long)a[(size_t)j * n + n - 1] - rs) : 0;
      }
    } else {
      for (int k = 0; k < n; k++)
        for (int j = 0; j < np; j++) dst[(size_t)k * np + j] = j < n ? a[(size_t)j * n + k] : 0.0;
    }
  }
  perm_batch* b = new perm_batch();
  b->count = count;
  b->total_tiles = tiles;
  int max_n = 0;
  for (int i = 0; i < count; i++) {
    if (cube_of[i] >= 0) continue;
    max_n = std::max(max_n, mats[i].n);
    if (mats[i].r) b->sparse++;
  }
  int vi = variant_override >= 0 ? variant_override : ctx->batch_variant;
  if (vi < 0 || vi >= kBatchVariantCount || kBatchVariants[vi].max_n < max_n) vi = 0;
  b->variant = vi;
  const BatchVariant& V = kBatchVariants[vi];
  b->orders.assign(orders, orders + count);
  b->groups.resize(count);
  b->shapes.assign(count, -1);
  b->roundings.resize(count);
  b->abs_scale.assign(count, 1.0);
  for (int i = 0; i < count; i++) {
    b->groups[i] = mats[i].g;
    b->roundings[i] = mats[i].g ? std::ceil((double)mats[i].n / mats[i].g) : 2.0 * mats[i].n;
  }
  for (const BatchCube& c : cube) {
    // |factor| = 2, of prod y = 2^n prod x in the int32 walk
    b->abs_scale[c.index] = c.op.variant == PERM_KERNEL_DENSE_INT ? std::ldexp(1.0, 1 - c.op.n) : 2.0;
    b->shapes[c.index] = c.op.shape;
    if (c.op.exp2) b->exp2.push_back({c.index, c.op.exp2});
    if (c.op.variant == PERM_KERNEL_DENSE_INT) b->roundings[c.index] = cube_factors(kCubeShapes[c.op.shape]) + 1.0;
  }
  b->offsets = src_off;
  b->values.assign(values, values + off);
  cudaError_t e;
#define BT(expr)                                    \
  do {                                              \
    e = (expr);                                     \
    if (e != cudaSuccess) {                         \
      batch_free(b);                                \
      return fail_cuda(ctx, e, #expr);              \
    }                                               \
  } while (0)
  BT(cudaMalloc(&b->d_operands, sizeof(double) * std::max<uint64_t>(img, 1)));
  BT(cudaMalloc(&b->d_mats, sizeof(BatchMatrix) * std::max(queued, 1)));
  BT(cudaMalloc(&b->d_tile_partials, sizeof(dd) * std::max<uint64_t>(tiles, 1)));
  BT(cudaMalloc(&b->d_tile_abs, sizeof(double) * std::max<uint64_t>(tiles, 1)));
  BT(cudaMalloc(&b->d_mat_done, sizeof(unsigned) * count));
  BT(cudaMalloc(&b->d_next, sizeof(unsigned long long)));
  std::vector<CubeSum> cube_sum;
  auto cube_grid = [&](const BatchCube& c) {
    const uint64_t cubes_n = 1ull << (c.op.n - 5);
    return (int)std::min<uint64_t>((uint64_t)ctx->num_sms, std::max<uint64_t>(1, cubes_n / (64 * kCubeThreads)));
  };
  const size_t result_bytes = sizeof(double) * (3 * (size_t)count + 1);
  BT(cudaMalloc(&b->d_results, result_bytes));
  BT(cudaMemset(b->d_results, 0, result_bytes));
  BT(cudaMallocHost(&b->h_results, result_bytes));
  if (!cube.empty()) {
    std::vector<unsigned char> images(cube_bytes);
    for (const BatchCube& c : cube) memcpy(images.data() + c.offset, c.op.image.data(), c.op.image.size());
    BT(cudaMalloc(&b->d_cubes, cube_bytes));
    BT(cudaMemcpy(b->d_cubes, images.data(), cube_bytes, cudaMemcpyHostToDevice));
    BT(cudaMalloc(&b->d_cube_tickets, sizeof(unsigned) * kBatchBranches));
    BT(cudaMemset(b->d_cube_tickets, 0, sizeof(unsigned) * kBatchBranches));
    cube_sum.reserve(cube.size());
    uint64_t words = 0;
    for (const BatchCube& c : cube) {
      const int grid = cube_grid(c);
      cube_sum.push_back({words, grid * kCubeWarps, c.index});
      words += (uint64_t)grid * kCubeWords;
    }
    BT(cudaMalloc(&b->d_cube_partials, sizeof(double) * words));
    BT(cudaMalloc(&b->d_cube_sum, sizeof(CubeSum) * cube_sum.size()));
    BT(cudaMemcpy(b->d_cube_sum, cube_sum.data(), sizeof(CubeSum) * cube_sum.size(), cudaMemcpyHostToDevice));
    if (int rc2 = allow_smem(ctx, (const void*)cube_sums_kernel, 0)) {  // loads it before the capture
      batch_free(b);
      return rc2;
    }
    for (const BatchCube& c : cube)
      if (int rc2 = allow_smem(ctx, cube_kernel(c.op.shape, cube_kind(c.op) + 1), operand_smem(c.op))) {
        batch_free(b);
        return rc2;
      }
  }
  BT(cudaMemcpy(b->d_operands, image.data(), sizeof(double) * img, cudaMemcpyHostToDevice));
  if (queued) BT(cudaMemcpy(b->d_mats, q.data(), sizeof(BatchMatrix) * queued, cudaMemcpyHostToDevice));
  BT(cudaMemset(b->d_mat_done, 0, sizeof(unsigned) * count));
  if (!ctx->batch_occ[vi]) {
    if (int rc2 = allow_smem(ctx, V.fn, batch_smem_bytes(V))) {
      batch_free(b);
      return rc2;
    }
    int occ = 0;
    BT(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, V.fn, V.block, batch_smem_bytes(V)));
    ctx->batch_occ[vi] = std::max(occ, 1);
  }
  const int wpb = V.block / 32;
  const uint64_t warps = (uint64_t)ctx->num_sms * ctx->batch_occ[vi] * wpb;
  const uint64_t want = std::min<uint64_t>(warps, tiles);
  b->grid = (int)std::max<uint64_t>(1, (want + wpb - 1) / wpb);
  // capture: reset the queue head and the error flag, run, read the results back.
  // The column-cube walks are dealt to parallel branches beside the persistent
  // kernel's: the next walk's CTAs fill the SMs that one leaves.
  BatchArgs args;
  args.operands = b->d_operands;
  args.mats = b->d_mats;
  args.count = queued;
  args.total_tiles = tiles;
  args.next_tile = b->d_next;
  args.tile_partials = b->d_tile_partials;
  args.tile_abs = b->d_tile_abs;
  args.mat_done = b->d_mat_done;
  args.results = b->d_results;
  void* kargs[] = {&args};
  struct Branches {
    cudaStream_t stream[kBatchBranches] = {};
    cudaEvent_t fork = nullptr, join[kBatchBranches] = {};
    ~Branches() {
      for (auto st : stream)
        if (st) cudaStreamDestroy(st);
      for (auto ev : join)
        if (ev) cudaEventDestroy(ev);
      if (fork) cudaEventDestroy(fork);
    }
  } br;
  const int branches = (int)std::min<size_t>(kBatchBranches, cube.size());
  if (branches) BT(cudaEventCreateWithFlags(&br.fork, cudaEventDisableTiming));
  for (int i = 0; i < branches; i++) {
    BT(cudaStreamCreateWithFlags(&br.stream[i], cudaStreamNonBlocking));
    BT(cudaEventCreateWithFlags(&br.join[i], cudaEventDisableTiming));
  }
  BT(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  cudaMemsetAsync(b->d_next, 0, sizeof(unsigned long long), ctx->stream);
  // only the column-cube walks set the error flag (a node of the graph takes 10
  // us: 350 us for 130 matrices of orders 15..21)
  if (branches) {
    cudaMemsetAsync(b->d_results + 3 * (size_t)count, 0, sizeof(double), ctx->stream);
    cudaEventRecord(br.fork, ctx->stream);
  }
  for (int i = 0; i < branches; i++) cudaStreamWaitEvent(br.stream[i], br.fork, 0);
  for (size_t i = 0; i < cube.size(); i++) {
    const BatchCube& c = cube[i];
    const int branch = (int)(i % branches);
    const uint64_t cubes_n = 1ull << (c.op.n - 5);
    const int grid = cube_grid(c);
    const int m = cube_align(cubes_n, (uint64_t)grid * kCubeThreads, c.op.n - 5);
    CubeLaunch u;
    cube_args(c.op, b->d_cubes + c.offset, m, 0, cubes_n >> m, &u);
    u.walk.partials = reinterpret_cast<dd*>(b->d_cube_partials + cube_sum[i].first);
    u.walk.ticket = b->d_cube_tickets + branch;
    u.walk.out = b->d_results + 3 * c.index;
    u.walk.err = reinterpret_cast<int*>(b->d_results + 3 * (size_t)count);
    if (ctx->inject_timeouts > 0 && cube_kind(c.op) == kCubeF64) {
      u.walk.inject = 16u;
      ctx->inject_timeouts--;
    }
    void* cargs[] = {&u};
    cudaLaunchKernel(cube_kernel(c.op.shape, cube_kind(c.op) + 1), dim3(grid), dim3(kCubeThreads), cargs,
                     operand_smem(c.op), br.stream[branch]);
  }
  if (tiles)
    cudaLaunchKernel(V.fn, dim3(b->grid), dim3(V.block), kargs, batch_smem_bytes(V), ctx->stream);
  for (int i = 0; i < branches; i++) {
    cudaEventRecord(br.join[i], br.stream[i]);
    cudaStreamWaitEvent(ctx->stream, br.join[i], 0);
  }
  if (branches)
    cube_sums_kernel<<<(unsigned)cube.size(), 128, 0, ctx->stream>>>(b->d_cube_sum, b->d_cube_partials, b->d_results);
  cudaMemcpyAsync(b->h_results, b->d_results, result_bytes, cudaMemcpyDeviceToHost, ctx->stream);
  BT(cudaStreamEndCapture(ctx->stream, &b->graph));
  BT(cudaGraphInstantiate(&b->exec, b->graph, 0));
#undef BT
  *out = b;
  return PERM_OK;
}

extern "C" int perm_batch_create(perm_ctx* ctx, int count, const int* orders, const double* values,
                                 perm_batch** out) {
  if (!ctx) return PERM_EINVAL;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  return batch_create_locked(ctx, count, orders, values, nullptr, out);
}

static int batch_run_locked(perm_ctx* ctx, perm_batch* b, double* results, double* kernel_ms) {
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  CU(ctx, cudaGraphLaunch(b->exec, ctx->stream));
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  CU(ctx, cudaStreamSynchronize(ctx->stream));
  CU(ctx, cudaGetLastError());
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  int errflag = 0;
  memcpy(&errflag, b->h_results + 3 * (size_t)b->count, sizeof errflag);
  if (errflag) return fail(ctx, PERM_ETIMEOUT, "shared-memory staging wait timed out on device %d", ctx->device);
  if (kernel_ms) *kernel_ms = ms;
  for (const auto& [i, exp2] : b->exp2)
    for (int k = 0; k < 3; k++) b->h_results[3 * i + k] = std::ldexp(b->h_results[3 * i + k], exp2);
  if (results)
    for (int i = 0; i < b->count; i++) {
      results[2 * i] = b->h_results[3 * i];
      results[2 * i + 1] = b->h_results[3 * i + 1];
    }
  return PERM_OK;
}

extern "C" int perm_batch_run_ex(perm_ctx* ctx, perm_batch* b, double* results, double* rel_err, int* reruns,
                                 double* kernel_ms) {
  if (!ctx || !b) return ctx ? fail(ctx, PERM_EINVAL, "null batch") : PERM_EINVAL;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  int rc = batch_run_locked(ctx, b, results, kernel_ms);
  if (rc) return rc;
  // per-matrix worst-case bound from the exact sum of |term| (FP64-X walk);
  // a matrix above the context's target goes through the single-matrix
  // accuracy policy with the batch's value as the first evaluation
  const double u = std::ldexp(1.0, -53);
  int rerun = 0;
  for (int i = 0; i < b->count; i++) {
    const int n = b->orders[i];
    const double v = b->h_results[3 * i] + b->h_results[3 * i + 1];
    const double sa = b->h_results[3 * i + 2] * b->abs_scale[i];
    const int G = b->groups[i];
    const double rounds = b->roundings[i];
    double est = v != 0.0 ? (rounds + 16.0) * u * sa / std::fabs(v) : (sa > 0 ? INFINITY : 0.0);
    if (ctx->rel_target > 0 && est > ctx->rel_target && n >= 2) {
      const double* mat = b->values.data() + b->offsets[i];
      const int kernel = G ? PERM_KERNEL_DENSE_INT : PERM_KERNEL_DENSE;
      // the walk that made the value, whose bound this is; its columns as they
      // are, for the sample of the term moments
      DenseOperand op;
      op.n = n;
      op.variant = kernel;
      op.group = G;
      op.shape = b->shapes[i];
      if (plain_columns(op)) build_fp64_image(std::vector<double>(mat, mat + (size_t)n * n), n, &op);
      perm_result r{};
      r.hi = b->h_results[3 * i];
      r.lo = b->h_results[3 * i + 1];
      r.value = v;
      r.n = n;
      r.kernel = kernel;
      if ((rc = refine_result(ctx, mat, n, PERM_F64, op, true, &r, -1, false, sa))) return rc;
      if (results) {
        results[2 * i] = r.hi;
        results[2 * i + 1] = r.lo;
      }
      est = r.rel_error_estimate;
      if (kernel_ms) *kernel_ms += r.kernel_ms;  // checks and reruns count toward the batch's device time
      rerun++;
    }
    if (rel_err) rel_err[i] = est;
  }
  if (reruns) *reruns = rerun;
  return PERM_OK;
}

extern "C" int perm_batch_run(perm_ctx* ctx, perm_batch* b, double* results, double* kernel_ms) {
  if (!ctx || !b) return ctx ? fail(ctx, PERM_EINVAL, "null batch") : PERM_EINVAL;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  return batch_run_locked(ctx, b, results, kernel_ms);
}

extern "C" void perm_batch_destroy(perm_ctx* ctx, perm_batch* b) {
  if (ctx) cudaSetDevice(ctx->device);
  batch_free(b);
}

extern "C" int perm_batch_exact(perm_ctx* ctx, int count, const int* orders, const double* values, double* results,
                                double* kernel_ms) {
  perm_batch* b = nullptr;
  int rc = perm_batch_create(ctx, count, orders, values, &b);
  if (rc) return rc;
  rc = perm_batch_run(ctx, b, results, kernel_ms);
  perm_batch_destroy(ctx, b);
  return rc;
}

// Autotuner: for each order in [n_lo, n_hi] time a synthetic batch of that
// order (~2^26 Gray steps in total) with each candidate lane-range exponent
// and keep the fastest in the context; m_out (n_hi - n_lo + 1 ints) receives
// the choices.
extern "C" int perm_batch_autotune(perm_ctx* ctx, int n_lo, int n_hi, int* m_out) {
  if (!ctx) return PERM_EINVAL;
  if (n_lo < 1 || n_hi > kBatchMaxOrder || n_lo > n_hi) return fail(ctx, PERM_EINVAL, "orders [%d, %d]", n_lo, n_hi);
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  uint64_t state = 0x243F6A8885A308D3ull;
  for (int n = n_lo; n <= n_hi; n++) {
    if (n < 9) {
      ctx->batch_m[n] = 0;
      if (m_out) m_out[n - n_lo] = 0;
      continue;
    }
    const int count = (int)std::max<uint64_t>(1, (1ull << 26) >> (n - 1));
    std::vector<int> orders(count, n);
    std::vector<double> vals((size_t)count * n * n);
    for (double& v : vals) {
      state = state * 6364136223846793005ull + 1442695040888963407ull;
      v = 1.0 - (double)(state >> 11) * (1.0 / 9007199254740992.0);
    }
    int best_m = batch_default_m(n);
    double best_ms = 1e30;
    for (int m = 3; m <= std::min(16, n - 6); m++) {
      int mo[kBatchMaxOrder + 1] = {};
      mo[n] = m;
      perm_batch* b = nullptr;
      int rc = batch_create_locked(ctx, count, orders.data(), vals.data(), mo, &b, -1, false);
      if (rc) return rc;
      double ms = 1e30, t = 0;
      for (int rep = 0; rep < 3; rep++) {
        rc = batch_run_locked(ctx, b, nullptr, &t);
        if (rc) {
          batch_free(b);
          return rc;
        }
        if (rep) ms = std::min(ms, t);
      }
      batch_free(b);
      if (ms < best_ms * 0.98) {
        best_ms = ms;
        best_m = m;
      }
    }
    ctx->batch_m[n] = best_m;
    if (m_out) m_out[n - n_lo] = best_m;
  }
  // kernel variant (threads per block, register budget, register or
  // shared-memory X) on a mixed batch of these orders, about 2^26 Gray steps
  // per order, half 0/1 and half real matrices at densities 0.3..0.8
  std::vector<int> orders;
  std::vector<double> vals;
  for (int n = std::max(n_lo, 9); n <= n_hi; n++) {
    const int count = (int)std::max<uint64_t>(2, (1ull << 26) >> (n - 1));
    for (int c = 0; c < count; c++) {
      const double d = 0.3 + 0.5 * (c % 6) / 5.0;
      orders.push_back(n);
      for (int e = 0; e < n * n; e++) {
        state = state * 6364136223846793005ull + 1442695040888963407ull;
        const double u1 = (double)(state >> 11) * (1.0 / 9007199254740992.0);
        state = state * 6364136223846793005ull + 1442695040888963407ull;
        const double u2 = 1.0 - (double)(state >> 11) * (1.0 / 9007199254740992.0);
        vals.push_back(u1 < d ? ((c & 1) ? u2 : 1.0) : 0.0);
      }
      for (int j = 0; j < n; j++) vals[vals.size() - (size_t)n * n + (size_t)j * n + j] = 1.0;  // no empty row
    }
  }
  if (!orders.empty()) {
    double best_ms = 1e30;
    int best_v = 0;
    for (int v = 0; v < kBatchVariantCount; v++) {
      if (kBatchVariants[v].max_n < n_hi) continue;
      perm_batch* b = nullptr;
      int rc = batch_create_locked(ctx, (int)orders.size(), orders.data(), vals.data(), nullptr, &b, v, false);
      if (rc) return rc;
      double ms = 1e30, t = 0;
      for (int rep = 0; rep < 3; rep++) {
        rc = batch_run_locked(ctx, b, nullptr, &t);
        if (rc) {
          batch_free(b);
          return rc;
        }
        if (rep) ms = std::min(ms, t);
      }
      batch_free(b);
      if (ms < best_ms * 0.98) {
        best_ms = ms;
        best_v = v;
      }
    }
    ctx->batch_variant = best_v;
  }
  return PERM_OK;
}

extern "C" int perm_batch_use_variant(perm_ctx* ctx, int variant) {
  if (!ctx) return PERM_EINVAL;
  if (variant < 0 || variant >= kBatchVariantCount)
    return fail(ctx, PERM_EINVAL, "batch kernel variant %d outside [0, %d)", variant, kBatchVariantCount);
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->batch_variant = variant;
  return PERM_OK;
}

extern "C" int perm_batch_variant(perm_ctx* ctx, int* variant, int* max_n, int* block, int* min_blocks,
                                  int* shared_x) {
  if (!ctx) return PERM_EINVAL;
  const BatchVariant& V = kBatchVariants[ctx->batch_variant];
  if (variant) *variant = ctx->batch_variant;
  if (max_n) *max_n = V.max_n;
  if (block) *block = V.block;
  if (min_blocks) *min_blocks = V.min_blocks;
  if (shared_x) *shared_x = V.xs;
  return PERM_OK;
}

// ---------------------------------------------------------------------------
// matrix input
// ---------------------------------------------------------------------------
extern "C" int perm_read_matrix(const char* path, int binary, int cap_n, double* out, int* n_out,
                                int* header_nnz, char* type_out) {
  if (!path || !out || !n_out) return PERM_EINVAL;
  HostMatrix m;
  std::string err = read_matrix_file(path, binary != 0, &m);
  if (!err.empty()) {
    fprintf(stderr, "perm_read_matrix: %s\n", err.c_str());
    return PERM_EIO;
  }
  if (m.n > cap_n) return PERM_EUNSUPPORTED;
  std::copy(m.a.begin(), m.a.end(), out);
  *n_out = m.n;
  if (header_nnz) *header_nnz = m.header_nnz;
  if (type_out) snprintf(type_out, 8, "%s", m.type.c_str());
  return PERM_OK;
}

extern "C" int perm_compress(int mode, double* mat, int n, int* cptrs, int* rows, double* cvals, int* rptrs,
                             int* cols, double* rvals) {
  if (!mat || n < 1 || !cptrs || !rows || !cvals || !rptrs || !cols || !rvals) return PERM_EINVAL;
  if (mode < 0 || mode > 2) return PERM_EINVAL;
  Compressed c;
  compress_mode(mode, mat, n, &c);
  std::copy(c.cptrs.begin(), c.cptrs.end(), cptrs);
  std::copy(c.rptrs.begin(), c.rptrs.end(), rptrs);
  std::copy(c.rows.begin(), c.rows.end(), rows);
  std::copy(c.cols.begin(), c.cols.end(), cols);
  std::copy(c.cvals.begin(), c.cvals.end(), cvals);
  std::copy(c.rvals.begin(), c.rvals.end(), rvals);
  return c.nnz();
}

// ---------------------------------------------------------------------------
// measurement
// ---------------------------------------------------------------------------
extern "C" int perm_fp64_peak(perm_ctx* ctx, double* ops, double* kernel_ms) {
  if (!ctx || !ops) return ctx ? fail(ctx, PERM_EINVAL, "null output") : PERM_EINVAL;
  std::lock_guard<std::mutex> lock(ctx->mu);
  CU(ctx, cudaSetDevice(ctx->device));
  const int block = 256, grid = ctx->num_sms * 8, iters = 4096;
  fp64_peak_kernel<<<grid, block, 0, ctx->stream>>>(ctx->d_out, 64, 0.999999999, 1e-9);  // warm-up
  CU(ctx, cudaGetLastError());
  CU(ctx, cudaEventRecord(ctx->ev0, ctx->stream));
  fp64_peak_kernel<<<grid, block, 0, ctx->stream>>>(ctx->d_out, iters, 0.999999999, 1e-9);
  CU(ctx, cudaGetLastError());
  CU(ctx, cudaEventRecord(ctx->ev1, ctx->stream));
  CU(ctx, cudaEventSynchronize(ctx->ev1));
  float ms = 0;
  CU(ctx, cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  const double lane_ops = (double)grid * block * iters * 16.0 * 8.0;
  *ops = lane_ops / (ms * 1e-3);
  if (kernel_ms) *kernel_ms = ms;
  return PERM_OK;
}

// ---------------------------------------------------------------------------
// reference-signature entry points on a process default context
// ---------------------------------------------------------------------------
// Context of the reference-signature entry points.  Like the reference they
// evaluate once and return that value: no error estimate and no accuracy
// policy unless PERM_REL_TARGET sets a target.  PERM_DEVICE picks the device.
static perm_ctx* default_ctx() {
  static std::once_flag once;
  static perm_ctx* ctx = nullptr;
  std::call_once(once, [] {
    const char* d = getenv("PERM_DEVICE");
    int dev = d ? atoi(d) : 0;
    if (perm_ctx_create(dev, &ctx) != PERM_OK) {
      ctx = nullptr;
      return;
    }
    const char* t = getenv("PERM_REL_TARGET");
    perm_ctx_set_rel_target(ctx, t ? atof(t) : -1.0);
  });
  return ctx;
}

static double shim_exact(const void* mat, int nov, int dtype) {
  perm_ctx* ctx = default_ctx();
  if (!ctx) return NAN;
  perm_result r;
  int rc = perm_exact_dense(ctx, mat, nov, dtype, &r);
  if (rc != PERM_OK) {
    fprintf(stderr, "perman_b200: %s\n", perm_ctx_last_error(ctx));
    return NAN;
  }
  return r.value;
}

template <class T>
static double shim_skipper(const T* mat, const int* rptrs, const int* cols, const int* cptrs, const int* rows,
                           const T* cvals, int nov) {
  perm_ctx* ctx = default_ctx();
  if (!ctx) return NAN;
  if (!mat || !rptrs || !cols || !cptrs || !rows || !cvals || nov < 1 || nov > PERM_MAX_EXACT_N) {
    fprintf(stderr, "perman_b200: invalid SkipPer arguments\n");
    return NAN;
  }
  const int nnz = rptrs[nov];
  std::vector<double> rv(std::max(nnz, 1)), cv(std::max(nnz, 1));
  for (int i = 0; i < nov; i++)
    for (int p = rptrs[i]; p < rptrs[i + 1]; p++) rv[p] = (double)mat[(size_t)i * nov + cols[p]];
  for (int p = 0; p < nnz; p++) cv[p] = (double)cvals[p];
  perm_result r;
  int rc = perm_exact_sparse(ctx, nov, rptrs, cols, rv.data(), cptrs, rows, cv.data(), &r);
  if (rc != PERM_OK) {
    fprintf(stderr, "perman_b200: %s\n", perm_ctx_last_error(ctx));
    return NAN;
  }
  return r.value;
}

static uint64_t shim_seed() {
  static std::atomic<uint64_t> calls{0};
  return 0x5EED0000ull + calls.fetch_add(1);
}

static double shim_mc(const void* mat, int nov, int dtype, bool scaling, int times, int y, int z) {
  perm_ctx* ctx = default_ctx();
  if (!ctx) return NAN;
  perm_estimate e;
  int rc = scaling ? perm_approx_scaling(ctx, mat, nov, dtype, times, y, z, shim_seed(), nullptr, &e)
                   : perm_approx_rasmussen(ctx, mat, nov, dtype, times, shim_seed(), nullptr, &e);
  if (rc != PERM_OK) {
    fprintf(stderr, "perman_b200: %s\n", perm_ctx_last_error(ctx));
    return NAN;
  }
  return e.mean;
}

extern "C" {
double gpu_perman64_xshared_coalescing_mshared_int(int* mat, int nov, int, int) { return shim_exact(mat, nov, PERM_I32); }
double gpu_perman64_xshared_coalescing_mshared_float(float* mat, int nov, int, int) { return shim_exact(mat, nov, PERM_F32); }
double gpu_perman64_xshared_coalescing_mshared_double(double* mat, int nov, int, int) { return shim_exact(mat, nov, PERM_F64); }
double gpu_perman64_xshared_coalescing_mshared_skipper_int(int* mat, int* rptrs, int* cols, int* cptrs, int* rows,
                                                           int* cvals, int nov, int, int) {
  return shim_skipper(mat, rptrs, cols, cptrs, rows, cvals, nov);
}
double gpu_perman64_xshared_coalescing_mshared_skipper_float(float* mat, int* rptrs, int* cols, int* cptrs,
                                                             int* rows, float* cvals, int nov, int, int) {
  return shim_skipper(mat, rptrs, cols, cptrs, rows, cvals, nov);
}
double gpu_perman64_xshared_coalescing_mshared_skipper_double(double* mat, int* rptrs, int* cols, int* cptrs,
                                                              int* rows, double* cvals, int nov, int, int) {
  return shim_skipper(mat, rptrs, cols, cptrs, rows, cvals, nov);
}
double gpu_perman64_rasmussen_int(int* mat, int nov, int t) { return shim_mc(mat, nov, PERM_I32, false, t, 1, 0); }
double gpu_perman64_rasmussen_float(float* mat, int nov, int t) { return shim_mc(mat, nov, PERM_F32, false, t, 1, 0); }
double gpu_perman64_rasmussen_double(double* mat, int nov, int t) { return shim_mc(mat, nov, PERM_F64, false, t, 1, 0); }
double gpu_perman64_approximation_int(int* mat, int nov, int t, int y, int z) { return shim_mc(mat, nov, PERM_I32, true, t, y, z); }
double gpu_perman64_approximation_float(float* mat, int nov, int t, int y, int z) { return shim_mc(mat, nov, PERM_F32, true, t, y, z); }
double gpu_perman64_approximation_double(double* mat, int nov, int t, int y, int z) { return shim_mc(mat, nov, PERM_F64, true, t, y, z); }
double gpu_perman64_rasmussen_sparse(int* rptrs, int* cols, int nov, int nnz, int t, int grid_graph) {
  (void)nnz;
  (void)grid_graph;
  perm_ctx* ctx = default_ctx();
  if (!ctx) return NAN;
  perm_estimate e;
  if (perm_approx_rasmussen_sparse(ctx, nov, rptrs, cols, t, shim_seed(), nullptr, &e) != PERM_OK) {
    fprintf(stderr, "perman_b200: %s\n", perm_ctx_last_error(ctx));
    return NAN;
  }
  return e.mean;
}
double gpu_perman64_approximation_sparse(int* cptrs, int* rows, int* rptrs, int* cols, int nov, int nnz, int t,
                                         int y, int z, int grid_graph) {
  (void)nnz;
  (void)grid_graph;
  perm_ctx* ctx = default_ctx();
  if (!ctx) return NAN;
  perm_estimate e;
  if (perm_approx_scaling_sparse(ctx, nov, rptrs, cols, cptrs, rows, t, y, z, shim_seed(), nullptr, &e) != PERM_OK) {
    fprintf(stderr, "perman_b200: %s\n", perm_ctx_last_error(ctx));
    return NAN;
  }
  return e.mean;
}
}  // extern "C"
