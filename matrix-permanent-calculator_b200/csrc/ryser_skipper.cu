// ryser_skipper.cu -- sparse exact permanent: SkipPer (skip-ahead Ryser) on
// CRS + CCS.
//
// Replaces kernel_xshared_coalescing_mshared_skipper (gpu_exact_sparse.cu:556-670)
// and its wrapper's host sum (gpu_exact_sparse.cu:1124-1190).  Per Gray index i
// the walk
//   * applies gray(i) ^ gray(previous) column by column through the CCS
//     (gpu_exact_sparse.cu:611-633),
//   * multiplies x from row n-1 downwards and stops at the first zero entry
//     (gpu_exact_sparse.cu:634-642),
//   * on a zero product jumps to the next Gray index at which some column of
//     that row flips (gpu_exact_sparse.cu:648-666).
// Differences, all B200-first: X is FP64 (the reference keeps FP32, which is
// inexact for real-valued inputs); it lives in shared memory as x[j][thread],
// so every access of a warp is bank-conflict-free; the packed CRS/CCS/value
// block is staged once per CTA with a bulk (TMA) copy; threads take Gray
// chunks from a global queue (atomic ticket) instead of one static slice, which
// balances the data-dependent skip lengths; products are accumulated with
// TwoSum and reduced in double-double; an FP64 underflow to zero without a
// zero entry is counted as a zero term instead of indexing row -1.
//
// A visited index is a chain of shared-memory latencies (a column's rows, then
// the rows of the product), with some 20 warps an SM to hide them behind; the
// start of a chunk costs ten columns more, and dense spots of visited indices
// make a few chunks take a hundred times the mean.  So
//   * both loops take four rows at a time, all loads first;
//   * a warp steps in lock step through its lanes' chunks and fetches new ones
//     by one atomic (one per thread on one address took 0.14 ms of launches
//     that visit one index a thread);
//   * when the queue is empty, lanes without work take the upper half of what
//     another lane of the warp has left;
//   * where every x is exact (integers) it is carried from chunk to chunk.
// Three nonzeros a row, binary: n = 24 0.27 -> 0.053 ms, n = 30 0.60 -> 0.45,
// n = 33 1.12 -> 0.62, n = 36 6.3 -> 2.8 (density 2.7/36: 7.2 -> 1.6).
#include "perman_common.cuh"
#include "skipper.h"

namespace perm {

constexpr uint64_t kSkipSplit = 8;  // shortest range that is shared with an idle lane

__global__ void __launch_bounds__(128) skipper_kernel(SkipArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int n = a.n;
  const int BD = blockDim.x;
  const int tid = threadIdx.x;
  double* X = reinterpret_cast<double*>(smem + a.pack_bytes);  // [n][BD]
  dd* red = reinterpret_cast<dd*>(X + (size_t)n * BD);
  uint64_t* bar = reinterpret_cast<uint64_t*>(red + 32);

  const bool staged = stage_to_smem(smem, a.pack, a.pack_bytes, bar, a.err);
  const double* x0 = reinterpret_cast<const double*>(smem);
  const double* cvals = reinterpret_cast<const double*>(smem + a.off_cvals);
  const int* rptrs = reinterpret_cast<const int*>(smem + a.off_rptrs);
  const int* cptrs = reinterpret_cast<const int*>(smem + a.off_cptrs);
  const int* cols = reinterpret_cast<const int*>(smem + a.off_cols);
  const int* rows = reinterpret_cast<const int*>(smem + a.off_rows);

  Acc acc;
  unsigned long long visited = 0;
  if (staged) {
    const unsigned lane = threadIdx.x & 31, below = (1u << lane) - 1;
    uint64_t i = 0, end = 0, prev = 0;
    bool queued = true;  // chunks may be left in the queue (the same for the warp)
    auto restart = [&] {
      if (a.exact) return;
      for (int j = 0; j < n; j++) X[j * BD + tid] = x0[j];
      prev = 0;
    };
    for (int j = 0; j < n; j++) X[j * BD + tid] = x0[j];
    for (;;) {
      const unsigned idle = __ballot_sync(0xffffffffu, i >= end);
      if (idle && queued) {
        unsigned long long c = 0;
        if (lane == 0) c = atomicAdd(a.next_chunk, (unsigned long long)__popc(idle));
        c = __shfl_sync(0xffffffffu, c, 0);
        queued = c + __popc(idle) < a.nchunks;
        c += __popc(idle & below);
        if (i >= end && c < a.nchunks) {
          i = c * a.chunk;
          end = min(i + a.chunk, a.total);
          restart();
        }
      } else if (idle) {
        // no chunks left: idle lanes take the upper halves of what others still have
        const unsigned busy = __ballot_sync(0xffffffffu, i < end && end - i >= kSkipSplit);
        if (idle == 0xffffffffu) break;
        const int pairs = min(__popc(idle), __popc(busy));
        const bool takes = ((idle >> lane) & 1) && __popc(idle & below) < pairs;
        const bool gives = ((busy >> lane) & 1) && __popc(busy & below) < pairs;
        const unsigned from = takes ? __fns(busy, 0, __popc(idle & below) + 1) : lane;
        const uint64_t mid = i + (end - i) / 2;
        const uint64_t i2 = __shfl_sync(0xffffffffu, mid, from), end2 = __shfl_sync(0xffffffffu, end, from);
        if (gives) end = mid;
        if (takes) {
          i = i2;
          end = end2;
          restart();
        }
      }
      if (i >= end) continue;
      const uint64_t g = i ^ (i >> 1);
      uint64_t diff = prev ^ g;
      while (diff) {
        const int k = __ffsll((long long)diff) - 1;
        diff &= diff - 1;
        const int p1 = cptrs[k + 1];
        const double sg = ((g >> k) & 1) ? 1.0 : -1.0;
        for (int p = cptrs[k]; p < p1; p += a.wide) {
          const int p2 = min(p1, p + a.wide);
          int at[4];
          double v[4];
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (p + u < p2) {
              at[u] = rows[p + u] * BD + tid;
              v[u] = __fma_rn(sg, cvals[p + u], X[at[u]]);
            }
#pragma unroll
          for (int u = 0; u < 4; u++)
            if (p + u < p2) X[at[u]] = v[u];
        }
      }
      prev = g;
      double prod = 1.0;
      int last_zero = -1;
      for (int j = n - 1; j >= 0 && last_zero < 0; j -= 4) {
        double v[4];
#pragma unroll
        for (int u = 0; u < 4; u++) v[u] = j >= u ? X[(j - u) * BD + tid] : 1.0;
#pragma unroll
        for (int u = 0; u < 4; u++)
          if (last_zero < 0) {
            prod *= v[u];
            if (v[u] == 0.0) last_zero = j - u;
          }
      }
      visited++;
      if (prod != 0.0 || last_zero < 0) {
        acc.add((i & 1) ? -prod : prod);
        i++;
      } else {
        uint64_t change = ~0ull;
        for (int p = rptrs[last_zero]; p < rptrs[last_zero + 1]; p++) {
          const int col = cols[p];
          const uint64_t first = 1ull << col;  // first index whose ctz is col
          uint64_t ci = first;
          if (i >= first) ci = first + (((i - first) >> (col + 1)) + 1) * (first << 1);
          if (ci < change) change = ci;
        }
        i++;
        if (change > i) i = change;
      }
    }
  }
  for (int o = 16; o; o >>= 1) visited += __shfl_down_sync(0xffffffffu, visited, o);
  if ((tid & 31) == 0) atomicAdd(a.visited, visited);
  dd bt = block_reduce_dd(acc.value(), red);
  grid_finish_dd(bt, a.partials, a.ticket, a.out, (n & 1) ? 2.0 : -2.0, red);
}

}  // namespace perm
