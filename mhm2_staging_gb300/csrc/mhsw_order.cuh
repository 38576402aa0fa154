// mhsw_order.cuh -- the pair order of the persistent forward kernels: buckets by A length, and a
// counting sort of a batch's pairs by (bucket, B length descending) on the device.
#pragma once
#include <algorithm>
#include <climits>
#include <cstdint>

#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"
#include "mhsw_types.h"

namespace mhsw {

namespace {

// Buckets: 0..3 = A up to 64/96/128/160 rows (8-lane groups, K = 4/6/8/10),
// 4/5 = up to 192/256 rows (16-lane groups, K = 6/8), 6 = longer A (K = 8 strips),
// 7 = could exceed the int16 keys: straight to the int32 list; 8, 9 = A above long_rows rows: a
// block of its own (mhsw_long.cu), or, for bucket 8 (up to kStripRows rows, scores that fit the keys),
// strips of one lane group where the batch has many of them (strips_take_long).  The tuned row
// threshold (lane_rows, 160 or 128) moves A of 129..160 rows between bucket 3 and bucket 4.
constexpr int kBucketFirstLong = 4;
constexpr int kBucketStrip = 6;
constexpr int kBucketWide = 7;
constexpr int kBucketLongStrip = 8;
constexpr int kBucketLong = 9;
constexpr int kBuckets = 10;
constexpr int kStripRows = 1280;
__host__ __device__ constexpr int bucket_k(int b) {
  return b == 0 ? 4 : b == 1 ? 6 : b == 2 ? 8 : b == 3 ? 10 : b == 4 ? 6 : 8;
}

// min_rows: A of fewer rows go to the bucket of that many (BatchShape).
__device__ __forceinline__ int bucket_of(int M, int N, const Scoring &sc, int lane_rows, bool wide_try16,
                                         int min_rows = 0, int long_rows = INT_MAX) {
  const int R = M > min_rows ? M : min_rows;
  const int b = R <= lane_rows ? (R <= 64 ? 0 : R <= 96 ? 1 : R <= 128 ? 2 : 3)
                               : (R <= 192 ? 4 : R <= 256 ? 5 : kBucketStrip);
  // wide_try16: the int16 engine's ceiling test sends the pairs that do overflow to int32.
  // That test sees a score cross the keys' capacity only if the first cell above it still
  // fits a 16-bit key: the capacity leaves 64 values of margin and H grows by at most match
  // per step, so it holds for match <= 63; larger matches keep the bound routing.
  const long long bound = (long long)(M < N ? M : N) * sc.match;
  if (M > long_rows && bound <= kLongScore)
    return M <= kStripRows && bound <= keyed_cap(8) ? kBucketLongStrip : kBucketLong;
  if ((!wide_try16 || sc.match > 63) && bound > keyed_cap(bucket_k(b))) return kBucketWide;
  return b;
}

// Buckets of the protein kernels: A up to 128/192/256 rows (16-lane groups, K = 4/6/8), up to
// 384/512 (32-lane groups, K = 6/8), longer (strips of 512)
// -- or, for min(M, N) >= wide_from or B above kPCols, the int32 kernels (kBucketWide).
constexpr int kPCols = 65000;
__host__ __device__ constexpr int protein_bucket(int M, int N, int wide_from) {
  if ((M < N ? M : N) >= wide_from || N > kPCols) return kBucketWide;
  return M <= 128 ? 0 : M <= 192 ? 1 : M <= 256 ? 2 : M <= 384 ? 4 : M <= 512 ? 5 : kBucketStrip;
}

// ---- pair order: a counting sort over (bucket, class of len B, longest first) ---------
// Length classes are single columns below 1024 and 1/64 of an octave (1.6%) above, so the
// lane groups of a warp see equal B lengths, which is all the order is for (classes of 4
// columns cost the forward pass of 800,000 uneven pairs 0.7%).  Order within a bin is
// whatever the atomics give; no result depends on it.
constexpr int kLenBins = 1024 + 7 * 64;  // lengths up to 131071
constexpr int kOrderBins = kBuckets * kLenBins;
// Batches up to this size are ordered by one block in one launch (serving micro-batches of
// 4,000 pairs: 9 us against 26 us for the key, radix-sort and split kernels it replaced),
// larger ones by a histogram and a placement launch.
constexpr int64_t kOrderOneBlock = 4096;

__device__ __forceinline__ int len_class(int n) {  // 0 = longest
  n = n < 0 ? 0 : (n > 131071 ? 131071 : n);
  const int e = 31 - __clz(n | 1);
  const int c = n < 1024 ? n : 1024 + (e - 10) * 64 + ((n >> (e - 6)) & 63);
  return kLenBins - 1 - c;
}

constexpr int kOrderLongFirst = 7;

struct OrderArgs {
  PairSet ps;
  Scoring sc;
  int lane_rows;
  bool wide_try16;
  int64_t m, stride;  // item i < m is pair i * stride (stride 1: the whole batch; larger: the tuner's sample)
  int *queue;         // [0], [1]: claim counters of the short and long ranges; [2]: first item of the long range;
                      // [4..6]: LongCells of bucket 8; [kOrderLongFirst]: first item
                      // of the long-pair kernel
  int *first;         // first item of each bucket, then m
  int *hist, *cursor; // kOrderBins each (zeroed before the two-launch form)
  uint32_t *order;
  int max_a, max_b;   // pairs longer than these go with the empty ones
  int long_rows;      // longest A of the persistent kernels
  int min_rows;       // bucket_of's
  int protein_wide;   // above 0: buckets by protein_bucket with this wide_from (sc unused)
};

__device__ __forceinline__ int order_bin(const OrderArgs &g, int64_t p) {
  const int M = g.ps.a_len[p], N = g.ps.b_len[p];
  const int b = (M <= 0 || N <= 0 || M > g.max_a || N > g.max_b) ? (g.lane_rows > 0 ? 0 : kBucketFirstLong)
                : g.protein_wide > 0 ? protein_bucket(M, N, g.protein_wide)
                                     : bucket_of(M, N, g.sc, g.lane_rows, g.wide_try16, g.min_rows, g.long_rows);
  return b * kLenBins + len_class(N);
}

// What strips_take_long weighs for the pairs of bucket 8, in units of 1024 cells: gathered per block,
// then once per block in queue[4], [5] (64 bits) and [6].
constexpr int kLongFill = 400;  // columns' worth of the long-pair kernel's time that filling its strips takes
struct LongCells {
  unsigned long long sum;  // rows * (columns + kLongFill)
  unsigned int most;       // the longest pair's cells
};
__device__ __forceinline__ void add_long_cells(LongCells *s, const OrderArgs &g, int64_t p, int bin) {
  if (bin < kBucketLongStrip * kLenBins || bin >= (kBucketLongStrip + 1) * kLenBins) return;
  const long long M = g.ps.a_len[p], N = g.ps.b_len[p];
  atomicAdd(&s->sum, (unsigned long long)(M * (N + kLongFill) >> 10));
  atomicMax(&s->most, (unsigned int)((M * N + 1023) >> 10));
}
__device__ __forceinline__ void flush_long_cells(const LongCells &s, int *queue) {
  if (threadIdx.x != 0 || s.sum == 0) return;
  atomicAdd(reinterpret_cast<unsigned long long *>(queue + 4), s.sum);
  atomicMax(reinterpret_cast<unsigned int *>(queue + 6), s.most);
}

// Whether bucket 8 goes to the persistent kernel's lane groups, a pair a group in strips of 256
// rows, rather than to the long-pair kernel.  That kernel's strips of 512 rows are a third padding
// there, but a lane group alone sweeps only about 1 G cells/s: the groups win once what the batch
// costs the long-pair kernel is kStripShare times its longest pair's cells.  Forward pass, long-pair
// kernel / lane groups, 1,030-1,100 rows: 20,000 pairs against 300-400 columns 4.54 / 2.31 ms, against
// 1,030-1,100 9.67 / 6.68; 3,000 pairs 0.79 / 0.66 and 1.60 / 1.60, 2,000 0.57 / 0.56 and 1.14 / 1.34;
// against 4,000-6,000 columns 12,000 pairs 22.7 / 17.9, 4,000 7.8 / 9.5.  From 1,500 rows on the long-pair kernel is level or
// ahead up to 20,000 pairs (1,500-2,000 squared 18.5 / 19.4).
constexpr unsigned long long kStripShare = 3700;
__device__ __forceinline__ bool strips_take_long(const int *queue) {
  const unsigned long long sum = *reinterpret_cast<const volatile unsigned long long *>(queue + 4);
  return sum > 0 && sum >= kStripShare * *reinterpret_cast<const volatile unsigned int *>(queue + 6);
}

// Exclusive prefix sum of the kOrderBins counts in h, in place, by the whole block.
__device__ void scan_bins(int *h) {
  __shared__ int warp_sum[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int per = (kOrderBins + blockDim.x - 1) / blockDim.x;
  const int lo = threadIdx.x * per, hi = lo + per < kOrderBins ? lo + per : kOrderBins;
  int sum = 0;
  for (int b = lo; b < hi; b++) sum += h[b];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) warp_sum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int v = lane < nw ? warp_sum[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    warp_sum[lane] = v;
  }
  __syncthreads();
  int at = incl - sum + (warp > 0 ? warp_sum[warp - 1] : 0);
  for (int b = lo; b < hi; b++) {
    const int c = h[b];
    h[b] = at;
    at += c;
  }
  __syncthreads();
}

__device__ __forceinline__ void write_firsts(const OrderArgs &g, const int *base) {
  if (threadIdx.x < kBuckets) g.first[threadIdx.x] = base[threadIdx.x * kLenBins];
  if (threadIdx.x == 0) {
    g.first[kBuckets] = (int)g.m;
    g.queue[2] = base[kBucketFirstLong * kLenBins];
    g.queue[kOrderLongFirst] = base[(strips_take_long(g.queue) ? kBucketLong : kBucketLongStrip) * kLenBins];
  }
}

__global__ void __launch_bounds__(1024) k_order_one(OrderArgs g) {
  extern __shared__ int h[];
  for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) h[b] = 0;
  __shared__ LongCells cells;
  if (threadIdx.x < 7 && threadIdx.x != 2) g.queue[threadIdx.x] = 0;
  if (threadIdx.x == 0) cells = LongCells{0ull, 0u};
  __syncthreads();
  int bin[kOrderOneBlock / 1024];
#pragma unroll
  for (int k = 0; k < kOrderOneBlock / 1024; k++) {
    const int64_t i = threadIdx.x + k * 1024;
    bin[k] = i < g.m ? order_bin(g, i * g.stride) : -1;
    if (bin[k] >= 0) {
      atomicAdd(&h[bin[k]], 1);
      add_long_cells(&cells, g, i * g.stride, bin[k]);
    }
  }
  __syncthreads();
  flush_long_cells(cells, g.queue);
  scan_bins(h);
  write_firsts(g, h);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kOrderOneBlock / 1024; k++)
    if (bin[k] >= 0) g.order[atomicAdd(&h[bin[k]], 1)] = (uint32_t)((threadIdx.x + k * 1024) * g.stride);
}

__global__ void __launch_bounds__(1024) k_order_hist(OrderArgs g) {
  extern __shared__ int h[];
  __shared__ LongCells cells;
  for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) h[b] = 0;
  if (threadIdx.x == 0) cells = LongCells{0ull, 0u};
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.m; i += (int64_t)gridDim.x * blockDim.x) {
    const int bin = order_bin(g, i * g.stride);
    atomicAdd(&h[bin], 1);
    add_long_cells(&cells, g, i * g.stride, bin);
  }
  __syncthreads();
  flush_long_cells(cells, g.queue);
  for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x)
    if (h[b]) atomicAdd(&g.hist[b], h[b]);
}

// Same grid as k_order_hist: each block reserves its run of every bin with one atomic.
__global__ void __launch_bounds__(1024) k_order_place(OrderArgs g) {
  extern __shared__ int h[];
  int *base = h + kOrderBins;
  for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x) {
    base[b] = g.hist[b];
    h[b] = 0;
  }
  __syncthreads();
  scan_bins(base);
  if (blockIdx.x == 0) write_firsts(g, base);
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.m; i += step)
    atomicAdd(&h[order_bin(g, i * g.stride)], 1);
  __syncthreads();
  for (int b = threadIdx.x; b < kOrderBins; b += blockDim.x)
    if (h[b]) {
      base[b] += atomicAdd(&g.cursor[b], h[b]);
      h[b] = 0;
    }
  __syncthreads();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < g.m; i += step) {
    const int64_t p = i * g.stride;
    const int b = order_bin(g, p);
    g.order[base[b] + atomicAdd(&h[b], 1)] = (uint32_t)p;
  }
}

// The order's control block: [0..7] as OrderArgs::queue, [8..23] first item of
// each bucket and the item count, then the bin counts and cursors.
constexpr size_t kOrderHead = 24;
constexpr size_t kOrderCtl = kOrderHead + 2 * kOrderBins;

constexpr size_t kOrderSmem = sizeof(int) * kOrderBins;  // of the one-block and histogram kernels; twice of the placement
inline cudaError_t order_smem_limits() {
  cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(k_order_one), kOrderSmem);
  if (!e) e = raise_smem_limit(reinterpret_cast<const void *>(k_order_hist), kOrderSmem);
  return e ? e : raise_smem_limit(reinterpret_cast<const void *>(k_order_place), 2 * kOrderSmem);
}

// Orders m items (pair i * stride) into `order`; clears the claim counters.
inline cudaError_t order_pairs(const PairSet &ps, const Scoring &sc, int lane_rows, bool wide_try16, int64_t m,
                               int64_t stride, int *ctl, uint32_t *order, int sms, cudaStream_t st, int64_t *launches,
                               int max_a = INT_MAX, int max_b = INT_MAX, int long_rows = INT_MAX, int min_rows = 0,
                               int protein_wide = 0) {
  OrderArgs g{ps, sc, lane_rows, wide_try16, m, stride, ctl, ctl + 8, ctl + kOrderHead, ctl + kOrderHead + kOrderBins,
              order, max_a, max_b, long_rows, min_rows, protein_wide};
  cudaError_t e = order_smem_limits();
  if (e) return e;
  if (m <= kOrderOneBlock) {
    k_order_one<<<1, 1024, kOrderSmem, st>>>(g);
    if (launches) *launches += 1;
    return cudaGetLastError();
  }
  if ((e = cudaMemsetAsync(ctl, 0, sizeof(int) * kOrderCtl, st))) return e;
  // a block an SM at most: each reads and writes all bins, 53 KB
  const int grid = (int)std::min<int64_t>((m + 4095) / 4096, sms);
  k_order_hist<<<grid, 1024, kOrderSmem, st>>>(g);
  k_order_place<<<grid, 1024, 2 * kOrderSmem, st>>>(g);
  if (launches) *launches += 2;
  return cudaGetLastError();
}

}  // namespace

}  // namespace mhsw
