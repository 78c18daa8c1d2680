// mc.cu -- Monte-Carlo permanent estimators, one trial per warp.
//
// Rasmussen (replaces kernel_rasmussen, gpu_approximation_dense.cu:156-229, and
// kernel_rasmussen_sparse, gpu_approximation_sparse.cu:198-290): per step take
// the unextracted row with the fewest available nonzeros (lowest index on
// ties), multiply the weight by that count and extract a uniformly chosen
// available column.  An empty row ends the trial with weight 0.
//
// Scaling (replaces kernel_approximation, gpu_approximation_dense.cu:232-369, and
// kernel_approximation_sparse, gpu_approximation_sparse.cu:292-452): same row
// rule; every y steps run z Sinkhorn sweeps (columns then rows) over the
// remaining submatrix in FP64; sample an available column with probability
// proportional to d_r[row] * d_c[col]; weight *= 1 / p.  A zero column or row
// sum ends the trial with weight 0.
//
// Both estimate the permanent of the 0/1 pattern of the matrix (the
// reference's algorithms are documented for binary matrices only).
//
// B200 mapping: a warp runs one trial; lane l owns rows and columns l and
// l + 32, so the minimum-degree row is one popc per lane plus a single
// redux.sync minimum over (count << 8 | row), and each Sinkhorn sweep is a
// column pass (lane = column, walking rows) and a row pass (lane = row, over
// the transposed copy) with no bank conflicts.  Random numbers come from
// Philox4x32-10 keyed by (seed) at counter (trial, step, tag), so trial t is
// reproducible regardless of launch shape.  All FP64 operations use
// explicitly rounded intrinsics in the same order as the CPU restatement, so
// per-trial weights are bit-identical to it.  The trial weight is an FP32
// significand with a separate exponent; trial values are accumulated in FP64.
#include "mc.h"

#include <type_traits>

namespace perm {

namespace {

// idx-th set bit (from 0) of m, the same in every lane: a lane per bit of the
// word that holds it, found by one ballot.
__device__ __forceinline__ int nth_set_bit(uint64_t m, int idx, int lane) {
  const uint32_t lo = (uint32_t)m, hi = (uint32_t)(m >> 32);
  const int in_lo = __popc(lo);
  const bool high = idx >= in_lo;
  const uint32_t w = high ? hi : lo;
  const int k = high ? idx - in_lo : idx;
  const bool hit = ((w >> lane) & 1) && __popc(w & ((1u << lane) - 1)) == k;
  return (high ? 32 : 0) + __ffs(__ballot_sync(0xffffffffu, hit)) - 1;
}

// Row rule of the general scaling estimator: (count << 8 | row) minimum over the
// unextracted rows; returns 0xffffffff if none is left.
__device__ __forceinline__ unsigned min_row_key(const uint64_t* rowmask, int n, uint64_t colext,
                                                uint64_t rowext, int lane) {
  unsigned key = 0xffffffffu;
  int r = lane;
  if (r < n && !((rowext >> r) & 1))
    key = ((unsigned)__popcll(rowmask[r] & ~colext) << 8) | (unsigned)r;
  r = lane + 32;
  if (r < n && !((rowext >> r) & 1)) {
    unsigned k2 = ((unsigned)__popcll(rowmask[r] & ~colext) << 8) | (unsigned)r;
    key = k2 < key ? k2 : key;
  }
  return __reduce_min_sync(0xffffffffu, key);
}

// Block + grid completion of the (sum, sum of squares, zeros) triple.
__device__ __forceinline__ void finish3(double s, double s2, double z, double* slots, const McArgs& a) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    slots[warp * 3 + 0] = s;
    slots[warp * 3 + 1] = s2;
    slots[warp * 3 + 2] = z;
  }
  __syncthreads();
  __shared__ bool is_last;
  if (threadIdx.x == 0) {
    double t0 = 0, t1 = 0, t2 = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
      t0 += slots[w * 3 + 0];
      t1 += slots[w * 3 + 1];
      t2 += slots[w * 3 + 2];
    }
    a.partials[blockIdx.x * 3 + 0] = t0;
    a.partials[blockIdx.x * 3 + 1] = t1;
    a.partials[blockIdx.x * 3 + 2] = t2;
    __threadfence();
    unsigned prev = atomicAdd(a.ticket, 1u);
    is_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last || threadIdx.x != 0) return;
  __threadfence();
  double t0 = 0, t1 = 0, t2 = 0;
  for (unsigned b = 0; b < gridDim.x; b++) {
    t0 += __ldcg(&a.partials[b * 3 + 0]);
    t1 += __ldcg(&a.partials[b * 3 + 1]);
    t2 += __ldcg(&a.partials[b * 3 + 2]);
  }
  a.out[0] = t0;
  a.out[1] = t1;
  a.out[2] = t2;
  *a.ticket = 0u;
  __threadfence();
}

}  // namespace

// Bound: issue slots.  The lanes keep their rows' available columns in
// registers, draw 32 steps' random numbers at once (a lane each) and pick the
// n-th available column by one ballot.  n = 64, density 1/2, 2e5 trials: 3.2 ms
// with one draw and a serial bit search per step, 1.29 ms now.
__global__ void __launch_bounds__(kMcBlock) rasmussen_kernel(McArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const uint64_t* rowmask = reinterpret_cast<const uint64_t*>(smem);
  double* slots = reinterpret_cast<double*>(smem + a.pack_bytes);
  uint64_t* bar = reinterpret_cast<uint64_t*>(slots + (kMcBlock / 32) * 3);
  const bool staged = stage_to_smem(smem, a.pack, a.mask_bytes, bar, a.err);

  const int lane = threadIdx.x & 31;
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  const int n = a.n;
  double s = 0, s2 = 0, zeros = 0;
  if (staged) {
    for (uint64_t q = warp; q < a.trials; q += nwarps) {
      const uint64_t t = a.trial0 + q;
      // this lane's rows, lane and lane + 32: available columns, still there
      uint64_t m0 = lane < n ? rowmask[lane] : 0ull, m1 = lane + 32 < n ? rowmask[lane + 32] : 0ull;
      bool live0 = lane < n, live1 = lane + 32 < n;
      uint64_t colext = 0;
      uint32_t draw = 0;  // this lane's step of the current 32
      WExp w;
      bool ok = true;
      for (int step = 0; step < n; step++) {
        if ((step & 31) == 0) draw = philox_step(a.seed, t, (uint32_t)(step + lane), kTagRasmussen).x;
        // fewest available nonzeros, lowest index on ties
        const unsigned k0 = live0 ? ((unsigned)__popcll(m0) << 8) | (unsigned)lane : 0xffffffffu;
        const unsigned k1 = live1 ? ((unsigned)__popcll(m1) << 8) | (unsigned)(lane + 32) : 0xffffffffu;
        const unsigned key = __reduce_min_sync(0xffffffffu, k0 < k1 ? k0 : k1);
        const int best = (int)(key >> 8), row = (int)(key & 0xffu);
        if (best == 0) {
          ok = false;
          break;
        }
        w.mul((float)best);
        const uint32_t rnd = __shfl_sync(0xffffffffu, draw, step & 31);
        const int idx = (int)(((uint64_t)rnd * (uint64_t)best) >> 32);
        const int col = nth_set_bit(rowmask[row] & ~colext, idx, lane);
        const uint64_t bit = 1ull << col;
        colext |= bit;
        m0 &= ~bit;
        m1 &= ~bit;
        if (row == lane) live0 = false;
        if (row == lane + 32) live1 = false;
      }
      const double v = ok ? w.value() : 0.0;
      if (lane == 0) {
        s += v;
        s2 += v * v;
        zeros += ok ? 0.0 : 1.0;
        if (a.trial_out) a.trial_out[q] = v;
      }
    }
  }
  finish3(s, s2, zeros, slots, a);
}

// The scaling estimator over general matrices.
__device__ __forceinline__ void scaling_trials_general(const McArgs& a, unsigned char* smem) {
  const int n = a.n, np = a.np;
  const uint64_t* rowmask = reinterpret_cast<const uint64_t*>(smem);
  const double* A = reinterpret_cast<const double*>(smem + a.mask_bytes);   // A[i * np + j]
  const double* AT = A + (size_t)n * np;                                       // AT[j * np + i]
  double* dwarp = reinterpret_cast<double*>(smem + a.pack_bytes);
  double* slots = dwarp + (kMcBlock / 32) * kMcWarpDoubles;
  uint64_t* bar = reinterpret_cast<uint64_t*>(slots + (kMcBlock / 32) * 3);
  const bool staged = stage_to_smem(smem, a.pack, a.pack_bytes, bar, a.err);

  const int lane = threadIdx.x & 31;
  double* dr = dwarp + (threadIdx.x >> 5) * kMcWarpDoubles;
  double* dc = dr + 64;
  double* prefix = dc + 64;                               // running sums of the column choice
  int* pcol = reinterpret_cast<int*>(prefix + 64);        // their columns
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  double s = 0, s2 = 0, zeros = 0;
  if (staged) {
    for (uint64_t q = warp; q < a.trials; q += nwarps) {
      const uint64_t t = a.trial0 + q;
      dr[lane] = 1.0;
      dr[lane + 32] = 1.0;
      dc[lane] = 1.0;
      dc[lane + 32] = 1.0;
      __syncwarp();
      uint64_t colext = 0, rowext = 0;
      WExp w;
      bool ok = true;
      for (int it = 0; it < n && ok; it++) {
        const unsigned key = min_row_key(rowmask, n, colext, rowext, lane);
        const int row = (int)(key & 0xffu);
        if (it % a.y == 0) {
          const uint64_t full = n == 64 ? ~0ull : ((1ull << n) - 1);
          const uint64_t rows_left = ~rowext & full, cols_left = ~colext & full;
          const int j0 = lane, j1 = lane + 32;
          const bool c0 = (cols_left >> j0) & 1, c1 = j1 < 64 && ((cols_left >> j1) & 1);
          const bool r0 = (rows_left >> j0) & 1, r1 = j1 < 64 && ((rows_left >> j1) & 1);
          for (int k = 0; k < a.z; k++) {
            // column pass: lane owns columns lane, lane + 32
            double cs0 = 0.0, cs1 = 0.0;
            for (uint64_t m = rows_left; m; m &= m - 1) {
              const int i = __ffsll((long long)m) - 1;
              const double d = dr[i];
              const double* Ai = A + i * np;
              if (c0) cs0 = __dadd_rn(cs0, __dmul_rn(d, Ai[j0]));
              if (c1) cs1 = __dadd_rn(cs1, __dmul_rn(d, Ai[j1]));
            }
            bool fail = (c0 && cs0 == 0.0) || (c1 && cs1 == 0.0);
            if (__any_sync(0xffffffffu, fail)) {
              ok = false;
              break;
            }
            if (c0) dc[j0] = __drcp_rn(cs0);
            if (c1) dc[j1] = __drcp_rn(cs1);
            __syncwarp();
            // row pass: lane owns rows lane, lane + 32
            double rs0 = 0.0, rs1 = 0.0;
            for (uint64_t m = cols_left; m; m &= m - 1) {
              const int j = __ffsll((long long)m) - 1;
              const double d = dc[j];
              const double* ATj = AT + j * np;
              if (r0) rs0 = __dadd_rn(rs0, __dmul_rn(ATj[j0], d));
              if (r1) rs1 = __dadd_rn(rs1, __dmul_rn(ATj[j1], d));
            }
            fail = (r0 && rs0 == 0.0) || (r1 && rs1 == 0.0);
            if (__any_sync(0xffffffffu, fail)) {
              ok = false;
              break;
            }
            if (r0) dr[j0] = __drcp_rn(rs0);
            if (r1) dr[j1] = __drcp_rn(rs1);
            __syncwarp();
          }
          if (!ok) break;
        }
        // column choice: running sums in ascending column order (recorded),
        // the first one above u * sum (one ballot), the last column if none
        const uint64_t avail = rowmask[row] & ~colext;
        const double drow = dr[row];
        double sum = 0.0;
        int cnt = 0;
        for (uint64_t m = avail; m; m &= m - 1, cnt++) {
          const int j = __ffsll((long long)m) - 1;
          sum = __dadd_rn(sum, __dmul_rn(drow, dc[j]));
          if (lane == 0) {
            prefix[cnt] = sum;
            pcol[cnt] = j;
          }
        }
        if (sum == 0.0) {
          ok = false;
          break;
        }
        __syncwarp();
        const u32x4 rnd = philox_step(a.seed, t, (uint32_t)it, kTagScaling);
        const double u = __dmul_rn(__dadd_rn(__dmul_rn((double)(rnd.x >> 5), 67108864.0), (double)(rnd.y >> 6)),
                                   1.0 / 9007199254740992.0);
        const double target = __dmul_rn(u, sum);
        const unsigned lo = __ballot_sync(0xffffffffu, lane < cnt && target < prefix[lane]);
        const unsigned hi = __ballot_sync(0xffffffffu, lane + 32 < cnt && target < prefix[lane + 32]);
        const int pick = lo ? __ffs(lo) - 1 : (hi ? 32 + __ffs(hi) - 1 : cnt - 1);
        const int col = pcol[pick];
        const double sp = __dmul_rn(drow, dc[col]);
        w.mul(__double2float_rn(__ddiv_rn(sum, sp)));
        colext |= 1ull << col;
        rowext |= 1ull << row;
        __syncwarp();
      }
      const double v = ok ? w.value() : 0.0;
      if (lane == 0) {
        s += v;
        s2 += v * v;
        zeros += ok ? 0.0 : 1.0;
        if (a.trial_out) a.trial_out[q] = v;
      }
      __syncwarp();
    }
  }
  finish3(s, s2, zeros, slots, a);
}

// The scaling estimator over 0/1 matrices.  A Sinkhorn sum over a 0/1 matrix
// adds exactly the scaling factors of its 1 entries (a * d = d for a = 1; a
// zero entry adds +0.0 to a non-negative sum), so adding the factors under the
// bits of row and column masks in ascending order gives the general sum's FP64
// value.
//
// The submatrix is kept compact: rows and columns that are left have indices
// 0..k-1 in their old order (so ties and sums keep theirs), lane l owns rows and
// columns l and l + 32, and an extraction deletes a bit from every mask and
// moves the masks and factors above it down by one.  A pass then costs k
// additions a lane and column, and from k = 32 on a lane owns one.
//
// Bound: issue slots (two instructions per entry, a test and a predicated
// addition) and the FP64 chains of the sums.  n = 57, density 1/2, 2e5 trials,
// a sweep of 5 every 4 steps: 37.1 ms over all n entries and two columns a lane
// in every pass, 18.1 ms now (4 CTAs per SM at 64 registers; 3: 18.7, 2: 19.2).
__device__ __forceinline__ uint64_t delete_bit(uint64_t m, int p) {
  const uint64_t low = (1ull << p) - 1;
  return (m & low) | ((m >> 1) & ~low);
}
__device__ __forceinline__ uint32_t delete_bit(uint32_t m, int p) {
  const uint32_t low = (1u << p) - 1;
  return (m & low) | ((m >> 1) & ~low);
}

// Adds d[i] for the set bits i < k of w0 (w1) to s0 (s1), ascending.
template <bool kTwo>
__device__ __forceinline__ void masked_sums(const double* d, uint32_t w0, uint32_t w1, int k, double& s0, double& s1) {
#pragma unroll
  for (int i = 0; i < 32; i += 8) {
    if (i >= k) break;
#pragma unroll
    for (int u = i; u < i + 8; u += 2) {
      const double2 v = *reinterpret_cast<const double2*>(d + u);
      if (w0 & (1u << u)) s0 = __dadd_rn(s0, v.x);
      if (kTwo && (w1 & (1u << u))) s1 = __dadd_rn(s1, v.x);
      if (w0 & (2u << u)) s0 = __dadd_rn(s0, v.y);
      if (kTwo && (w1 & (2u << u))) s1 = __dadd_rn(s1, v.y);
    }
  }
}

// A trial's state; kTwo: more than 32 rows left (64-bit masks, two rows and
// columns a lane).
template <bool kTwo>
struct ScalingState {
  using Mask = std::conditional_t<kTwo, uint64_t, uint32_t>;
  Mask r0, r1, c0, c1;  // masks of this lane's rows (over columns) and columns (over rows)
};

// Sums of the factors `from` under this lane's masks, their reciprocals to
// `to`; false when a sum of the submatrix is zero.
template <bool kTwo, class Mask>
__device__ __forceinline__ bool sinkhorn_pass(const double* from, double* to, Mask m0, Mask m1, int k, int lane) {
  double s0 = 0.0, s1 = 0.0;
  masked_sums<kTwo>(from, (uint32_t)m0, (uint32_t)m1, k, s0, s1);
  if constexpr (kTwo) masked_sums<true>(from + 32, (uint32_t)(m0 >> 32), (uint32_t)(m1 >> 32), k - 32, s0, s1);
  const bool own0 = lane < k, own1 = kTwo && lane + 32 < k;
  if (__any_sync(0xffffffffu, (own0 && s0 == 0.0) || (own1 && s1 == 0.0))) return false;
  if (own0) to[lane] = __drcp_rn(s0);
  if (own1) to[lane + 32] = __drcp_rn(s1);
  __syncwarp();
  return true;
}

// One step with k rows left; false when the trial ends with weight 0.
template <bool kTwo>
__device__ __forceinline__ bool scaling_step(ScalingState<kTwo>& st, double* dr, double* dc, double* prod, int* pcol,
                                             const McArgs& a, int k, bool sweep, uint32_t rx, uint32_t ry, WExp& w,
                                             int lane) {
  using Mask = typename ScalingState<kTwo>::Mask;
  auto bits = [](Mask m) { return kTwo ? __popcll(m) : __popc((uint32_t)m); };
  // fewest available nonzeros, lowest index on ties
  unsigned key = lane < k ? ((unsigned)bits(st.r0) << 8) | (unsigned)lane : 0xffffffffu;
  if (kTwo && lane + 32 < k) {
    const unsigned k1 = ((unsigned)bits(st.r1) << 8) | (unsigned)(lane + 32);
    key = k1 < key ? k1 : key;
  }
  const int row = (int)(__reduce_min_sync(0xffffffffu, key) & 0xffu);
  if (sweep)
    for (int i = 0; i < a.z; i++) {
      if (!sinkhorn_pass<kTwo>(dr, dc, st.c0, st.c1, k, lane)) return false;
      if (!sinkhorn_pass<kTwo>(dc, dr, st.r0, st.r1, k, lane)) return false;
    }
  // column choice: running sums over the row's columns in ascending order
  // (lane t keeps the t-th), the first one above u * sum, the last column if none
  const Mask avail = __shfl_sync(0xffffffffu, kTwo && row >= 32 ? st.r1 : st.r0, row & 31);
  const double drow = dr[row];
  const uint32_t lt = (1u << lane) - 1, lo = (uint32_t)avail, hi = kTwo ? (uint32_t)((uint64_t)avail >> 32) : 0u;
  const int cnt = __popc(lo) + (kTwo ? __popc(hi) : 0);
  if ((lo >> lane) & 1) {
    const int t = __popc(lo & lt);
    prod[t] = __dmul_rn(drow, dc[lane]);
    pcol[t] = lane;
  }
  if (kTwo && ((hi >> lane) & 1)) {
    const int t = __popc(lo) + __popc(hi & lt);
    prod[t] = __dmul_rn(drow, dc[lane + 32]);
    pcol[t] = lane + 32;
  }
  if (lane == 0 && (cnt & 1)) prod[cnt] = 0.0;  // adds nothing
  __syncwarp();
  double sum = 0.0, pre0 = 0.0, pre1 = 0.0;
  for (int t = 0; t < cnt; t += 2) {
    const double2 v = *reinterpret_cast<const double2*>(prod + t);
    const double s = __dadd_rn(sum, v.x);
    sum = __dadd_rn(s, v.y);
    if (!kTwo || t < 32) {
      if (lane == t) pre0 = s;
      if (lane == t + 1) pre0 = sum;
    } else {
      if (lane + 32 == t) pre1 = s;
      if (lane + 32 == t + 1) pre1 = sum;
    }
  }
  if (sum == 0.0) return false;
  const double u = __dmul_rn(__dadd_rn(__dmul_rn((double)(rx >> 5), 67108864.0), (double)(ry >> 6)),
                             1.0 / 9007199254740992.0);
  const double target = __dmul_rn(u, sum);
  const unsigned first = __ballot_sync(0xffffffffu, lane < cnt && target < pre0);
  const unsigned second = kTwo ? __ballot_sync(0xffffffffu, lane + 32 < cnt && target < pre1) : 0u;
  const int pick = first ? __ffs(first) - 1 : (second ? 32 + __ffs(second) - 1 : cnt - 1);
  const int col = pcol[pick];
  w.mul(__double2float_rn(__ddiv_rn(sum, prod[pick])));
  // delete the row and the column
  const double r0 = dr[lane + (lane >= row)], c0 = dc[lane + (lane >= col)];
  double r1 = 0.0, c1 = 0.0;
  if (kTwo) {
    r1 = dr[lane == 31 ? 63 : lane + 32 + (lane + 32 >= row)];
    c1 = dc[lane == 31 ? 63 : lane + 32 + (lane + 32 >= col)];
  }
  __syncwarp();
  dr[lane] = r0;
  dc[lane] = c0;
  if (kTwo) {
    dr[lane + 32] = r1;
    dc[lane + 32] = c1;
  }
  auto drop = [&](Mask& m0, Mask& m1, int bit, int place) {
    m0 = delete_bit(m0, bit);
    if (kTwo) m1 = delete_bit(m1, bit);
    const Mask up0 = __shfl_down_sync(0xffffffffu, m0, 1);
    if (kTwo) {
      const Mask up1 = __shfl_down_sync(0xffffffffu, m1, 1), carry = __shfl_sync(0xffffffffu, m1, 0);
      if (lane >= place) m0 = lane == 31 ? carry : up0;
      if (lane + 32 >= place) m1 = lane == 31 ? (Mask)0 : up1;
    } else {
      if (lane >= place) m0 = lane == 31 ? (Mask)0 : up0;
    }
  };
  drop(st.r0, st.r1, col, row);
  drop(st.c0, st.c1, row, col);
  __syncwarp();
  return true;
}

__device__ __forceinline__ void scaling_trials_binary(const McArgs& a, unsigned char* smem) {
  const int n = a.n, np = a.np;
  const uint64_t* rowmask = reinterpret_cast<const uint64_t*>(smem);
  const uint64_t* colmask = rowmask + np;
  double* dwarp = reinterpret_cast<double*>(smem + a.pack_bytes);
  double* slots = dwarp + (kMcBlock / 32) * kMcWarpDoubles;
  uint64_t* bar = reinterpret_cast<uint64_t*>(slots + (kMcBlock / 32) * 3);
  const bool staged = stage_to_smem(smem, a.pack, a.pack_bytes, bar, a.err);

  const int lane = threadIdx.x & 31;
  double* dr = dwarp + (threadIdx.x >> 5) * kMcWarpDoubles;
  double* dc = dr + 64;
  double* prod = dc + 64;
  int* pcol = reinterpret_cast<int*>(prod + 64);
  const uint64_t warp = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t nwarps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  double s = 0, s2 = 0, zeros = 0;
  if (staged) {
    for (uint64_t q = warp; q < a.trials; q += nwarps) {
      const uint64_t t = a.trial0 + q;
      dr[lane] = dr[lane + 32] = 1.0;
      dc[lane] = dc[lane + 32] = 1.0;
      __syncwarp();
      ScalingState<true> two;
      two.r0 = lane < n ? rowmask[lane] : 0ull;
      two.r1 = lane + 32 < n ? rowmask[lane + 32] : 0ull;
      two.c0 = lane < n ? colmask[lane] : 0ull;
      two.c1 = lane + 32 < n ? colmask[lane + 32] : 0ull;
      uint32_t rx = 0, ry = 0;  // this lane's step of the current 32
      WExp w;
      bool ok = true;
      int it = 0, wait = 0;  // steps until the next sweeps
      auto draw = [&]() {
        if ((it & 31) == 0) {
          const u32x4 r = philox_step(a.seed, t, (uint32_t)(it + lane), kTagScaling);
          rx = r.x;
          ry = r.y;
        }
        if (wait == 0) wait = a.y;
        wait--;
      };
      for (; it < n - 32 && ok; it++) {
        const bool sweep = wait == 0;
        draw();
        ok = scaling_step<true>(two, dr, dc, prod, pcol, a, n - it, sweep, __shfl_sync(0xffffffffu, rx, it & 31),
                                __shfl_sync(0xffffffffu, ry, it & 31), w, lane);
      }
      ScalingState<false> one;
      one.r0 = (uint32_t)two.r0;
      one.c0 = (uint32_t)two.c0;
      one.r1 = one.c1 = 0u;
      for (; it < n && ok; it++) {
        const bool sweep = wait == 0;
        draw();
        ok = scaling_step<false>(one, dr, dc, prod, pcol, a, n - it, sweep, __shfl_sync(0xffffffffu, rx, it & 31),
                                 __shfl_sync(0xffffffffu, ry, it & 31), w, lane);
      }
      const double v = ok ? w.value() : 0.0;
      if (lane == 0) {
        s += v;
        s2 += v * v;
        zeros += ok ? 0.0 : 1.0;
        if (a.trial_out) a.trial_out[q] = v;
      }
      __syncwarp();
    }
  }
  finish3(s, s2, zeros, slots, a);
}

__global__ void __launch_bounds__(kMcBlock) scaling_kernel(McArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  scaling_trials_general(a, smem);
}

__global__ void __launch_bounds__(kMcBlock, 4) scaling_kernel_binary(McArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  scaling_trials_binary(a, smem);
}

}  // namespace perm
