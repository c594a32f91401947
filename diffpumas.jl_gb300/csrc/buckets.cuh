// buckets.cuh -- how kernels deal the CSC buckets of resident ray paths (one
// bucket of entries per cell) to their warps: 32 cells per warp, their entries
// being consecutive, and a warp or a block per large bucket (the cells next to a
// detector, crossed by thousands of its rays).  Every order is fixed.
//
// The sums are FP64 and bound by that pipe (a warp instruction per 16 cycles and
// SM): a lane per cell runs as long as the fullest of 32 buckets, three times
// the mean.  So the entries of a warp's cells are cut into 32 equal runs of
// consecutive ones, a lane sums its run cell by cell, and a cell that several
// lanes hold adds up their parts.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace dp {

constexpr int kSmallBucket = 32;  // entries of a bucket that one lane takes
constexpr int kBucketWarps = 4, kBucketThreads = 32 * kBucketWarps;
constexpr int kBucketStage = 512;  // entries of 32 cells that are staged and dealt
constexpr int64_t kWarpBucket = 2048;  // entries of a bucket that one warp takes

// Blocks of a launch: the large buckets, one per warp, then the cells.
inline int bucket_blocks(long ncell, int n_big) {
  return (n_big + kBucketWarps - 1) / kBucketWarps + int((ncell + kBucketThreads - 1) / kBucketThreads);
}

// The blocks of the large buckets: sum(b, e, first, stride) is a thread's partial
// sum over entries first, first + stride, ... of [b, e); done(cell, total) stores
// the bucket's.  False for a block of cells.
template <class Sum, class Done>
__device__ __forceinline__ bool big_buckets(const int64_t* cptr, const int32_t* big, int n_big, Sum sum,
                                            Done done) {
  const int nbb = (n_big + kBucketWarps - 1) / kBucketWarps;
  if (int(blockIdx.x) >= nbb) return false;
  __shared__ double part[kBucketWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, k0 = blockIdx.x * kBucketWarps;
  auto reduce = [](double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  if (k0 + warp < n_big) {
    const int c = big[k0 + warp];
    const int64_t b = cptr[c], e = cptr[c + 1];
    if (e - b <= kWarpBucket) {
      const double s = reduce(sum(b, e, b + lane, 32));
      if (lane == 0) done(c, s);
    }
  }
  for (int k = k0; k < k0 + kBucketWarps && k < n_big; ++k) {
    const int c = big[k];
    const int64_t b = cptr[c], e = cptr[c + 1];
    if (e - b <= kWarpBucket) continue;  // the same for the whole block
    const double s = reduce(sum(b, e, b + threadIdx.x, kBucketThreads));
    if (lane == 0) part[warp] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
      double t = 0.0;
      for (int w = 0; w < kBucketWarps; ++w) t += part[w];
      done(c, t);
    }
    __syncthreads();
  }
  return true;
}

// The 32 cells of a warp of a cell block: this lane's cell (-1 past the grid), its
// entries [b, e) (none where the bucket is large), and the entries of the warp's
// cells counted off in order: n of them, this lane's from `off` on.
struct Cells {
  long cell;
  int64_t b, e;
  int off, n;
  bool big, any_big;
};
__device__ __forceinline__ Cells small_cells(const int64_t* cptr, long ncell, int n_big) {
  const int nbb = (n_big + kBucketWarps - 1) / kBucketWarps, lane = threadIdx.x & 31;
  const long c = long(blockIdx.x - nbb) * kBucketThreads + threadIdx.x;
  Cells C;
  C.cell = c < ncell ? c : -1;
  C.b = cptr[c < ncell ? c : ncell];
  C.e = cptr[c < ncell ? c + 1 : ncell];
  C.big = C.e - C.b > kSmallBucket;
  C.any_big = __any_sync(0xffffffffu, C.big);
  if (C.big) C.e = C.b;
  const int m = int(C.e - C.b);
  int sum = m;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += v;
  }
  C.off = sum - m;
  C.n = __shfl_sync(0xffffffffu, sum, 31);
  return C;
}

// A warp's share of shared memory for dealing its cells' entries.
struct Deal {
  int end[32];              // ends of the cells' entries as counted off
  int64_t at[32];           // bucket position of a cell's entries less their count
  double own[32], head[32]; // sum of a cell's part where it starts; of a lane's first part
};
// The cell that holds entry k: the first whose end is past it.
__device__ __forceinline__ int cell_of_entry(const Deal& D, int k) {
  int c = 0;
  for (int h = 16; h > 0; h >>= 1)
    if (D.end[c + h - 1] <= k) c += h;
  return c;
}
// Loads the warp's entries in order, 256 at a time and coalesced: load(k, p, ok)
// is called in a batch of eight per lane (k: the slot of the batch, p: the
// position), then keep(k, at) stores entry `at` of the batch's slot k.
template <class Load, class Keep>
__device__ __forceinline__ void stage_entries(const Cells& C, Deal& D, Load load, Keep keep) {
  const int lane = threadIdx.x & 31;
  D.end[lane] = C.off + int(C.e - C.b);
  D.at[lane] = C.b - C.off;
  D.own[lane] = 0.0;
  __syncwarp();
  const int64_t first = D.at[0];  // without large buckets the entries are consecutive
  for (int base = 0; base < C.n; base += 256) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int o = base + k * 32 + lane;
      const bool ok = o < C.n;
      load(k, (C.any_big && ok ? D.at[cell_of_entry(D, o)] : first) + o, ok);
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (base + k * 32 + lane < C.n) keep(k, base + k * 32 + lane);
  }
  __syncwarp();
}
// Sums the staged entries of the warp's cells: add(k, begin, end, s) adds entry k
// of the cell [begin, end) to s.  Returns this lane's cell's total.  All lanes
// call it after stage_entries; C.n <= kBucketStage.
template <class Add>
__device__ __forceinline__ double deal_entries(const Cells& C, Deal& D, Add add) {
  const int lane = threadIdx.x & 31, n = C.n;
  const int b = C.off, e = D.end[lane], q = (n + 31) / 32;
  const int lo = lane * q, hi = lo + q < n ? lo + q : n;
  if (lo < hi) {
    int c = cell_of_entry(D, lo);
    int begin = c ? D.end[c - 1] : 0, end = D.end[c];
    bool head = begin < lo;
    double s = 0.0;
    for (int k = lo; k < hi; ++k) {
      if (k >= end) {
        (head ? D.head[lane] : D.own[c]) = s;
        s = 0.0;
        head = false;
        do end = D.end[++c];
        while (k >= end);
        begin = k;
      }
      add(k, begin, end, s);
    }
    (head ? D.head[lane] : D.own[c]) = s;
  }
  __syncwarp();
  double s = D.own[lane];
  if (b < e)
    for (int j = b / q + 1; j * q < e; ++j) s += D.head[j];
  __syncwarp();
  return s;
}

}  // namespace dp
