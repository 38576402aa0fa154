// mhsw_long.cu -- long pairs: a cluster of blocks per pair, a warp per strip of A's rows.
//
// A lane group that takes a pair of several thousand rows alone walks its strips one after
// another: 60 pairs of 1-12 kb kept 60 groups of 16 lanes busy for 0.3 s on 152 SMs.  Here the
// strips of a pair run at the same time.  Warp w takes strips w, w + W, ... (512 rows each, 16 a
// lane); strip s follows strip s - 1 by about 130 columns, reading its last row's H and E^ from a
// row in global memory that the producer publishes 32 columns at a time through a progress
// word.  While the pairs are few, a pair's strips go round the blocks of a cluster (4 SMs, 32
// warps), so a scheduler has one strip rather than four.  A strip only ever waits for an earlier one and a warp takes its
// strips in order, so the waits end; each is bounded all the same: if one gives up the pair is
// flagged, its warps go on without waiting, and the call fails.
//
// The step is the keyed int16 step of mhsw_engine16.cuh with one operation more per cell
// pair: keys are formed from H above a base kept per lane half, so scores up to
// kLongScore fit 16-bit keys.  Eight steps raise a half's maximum by at most 8 * (match + gO):
// a column's value exceeds its left neighbour's by at most that (open a gap instead of taking
// the diagonal).  So a base moved up every eight steps, once the maximum is 2048 above it,
// keeps every key in range.  A base is never above a real cell's score less one, and cells at
// or below it cannot be the best.
//
// The begin search (REV) is the same sweep over the reversed prefixes, each strip limited to
// the columns an alignment can reach (band_sides: row i's band is [i - I, i + J]); rows are
// capped as in the banded kernels and doubled until the score is reached; strips after the one
// that reached it stop.
#include <algorithm>

#include "mhsw_band.cuh"
#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"

namespace mhsw {

namespace {

constexpr int kLK = 8;                  // row pairs per lane
constexpr int kLRows = 2 * kLK * 32;    // rows per strip
constexpr int kLChunk = 32;             // columns between progress updates

constexpr int kLongWarps = 32;          // warps on one pair, at most

// Shared by the blocks of a cluster, in global memory.
struct LongShared {
  unsigned long long prog[kLongWarps];  // per warp: strip << 32 | columns published (absolute)
  unsigned long long best;
  int claim, failed;
};

__device__ __forceinline__ void cluster_barrier() {  // all threads of the cluster; orders their memory
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_fence() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ int cluster_rank() {
  int r;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ int cluster_size() {
  int r;
  asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

struct LongArgs {
  PairSet ps;
  ResultSet rs;
  Scoring sc;
  const uint32_t *order;   // forward: the pair order; long pairs are items [*first, n)
  const int *first;
  const int64_t *list;     // REV: wide list
  const int *list_n;
  int64_t list_cap;
  int *next;               // claim counter
  LongShared *shared;      // per cluster
  uint32_t *bnd;           // per cluster: one row of `cols` words per warp
  int64_t cols;
  int waits;               // polls before a wait gives up
  int *flagged;            // pairs flagged so far
};

// The keyed step with keys above a base (nbase: its negative, per half).  LAZY (gap open >= gap
// extend): the chain down the rows is one add-max per row (ShortStep in mhsw_short.cu), and the
// relu is a maximum with gO before the subtraction, which then runs on the multiply-add pipe (a
// warp has a scheduler to itself here, and the integer pipe is what it waits for).
template <bool LAZY>
__device__ __forceinline__ void long_step(int t, uint32_t zH, uint32_t zE, const uint32_t (&Wlo)[kLK],
                                          const uint32_t (&Whi)[kLK], uint32_t (&P)[kLK], uint32_t (&F)[kLK],
                                          uint32_t &Hlast, uint32_t &Ecout, uint32_t &Kl, uint32_t &Jp, uint32_t NGE,
                                          uint32_t NGO, uint32_t GO, uint32_t one, uint32_t eight, uint32_t nbase) {
  uint32_t Ev = __byte_perm(zE, Ecout, 0x5432);
  const uint32_t Htop = __byte_perm(zH, Hlast, 0x5432);
  uint32_t Q = mad_u32(P[0], one, Wlo[0]);
  P[0] = mad_u32(Htop, one, Whi[0]);
  uint32_t key[kLK];
#pragma unroll
  for (int k = 0; k < kLK; k++) {
    uint32_t Hn;
    if constexpr (LAZY) {
      const uint32_t Hp = mad_u32(__vimax3_s16x2(Q, F[k], GO), one, 0u - GO);  // (no borrow: halves >= gO)
      Hn = __viaddmax_s16x2(Ev, NGO, Hp);
      Ev = __viaddmax_s16x2(Ev, NGE, Hp);
    } else {
      const uint32_t m = __vimax3_s16x2(Q, Ev, F[k]);
      Hn = __viaddmax_s16x2_relu(m, NGO, 0u);
      Ev = __viaddmax_s16x2(Ev, NGE, Hn);
    }
    F[k] = __viaddmax_s16x2(F[k], NGE, Hn);
    if (k + 1 < kLK) {
      Q = mad_u32(P[k + 1], one, Wlo[k + 1]);
      P[k + 1] = mad_u32(Hn, one, Whi[k + 1]);
    } else {
      Hlast = Hn;
    }
    key[k] = mad_u32(__viaddmax_s16x2_relu(Hn, nbase, 0u), eight, (uint32_t)(7 - k) * 0x00010001u);
  }
  uint32_t Kn = Kl;
#pragma unroll
  for (int k = 0; k < kLK; k += 2) Kn = __vimax3_s16x2(Kn, key[k], key[k + 1]);
  Ecout = Ev;
  const uint32_t msk = sign_mask16(Kn - Kl + 0x7fff7fffu);
  const uint32_t tt = (uint32_t)t * 0x00010001u;
  Jp = (msk & tt) | (~msk & Jp);
  Kl = Kn;
}

// Sweep of rows [0, M) (a[adir * i]) over columns [0, N) (b[bdir * j]), row i limited to
// [i - I, i + J], by all W warps of the cluster (this one is number `warp`); best cell in sh.best.
// goal > 0: strips after one that reached it stop.  waits: polls before a wait gives up.
template <bool LAZY>
__device__ void long_sweep(const uint8_t *a, int adir, int M, const uint8_t *b, int bdir, int N, int I, int J, int goal,
                           const Scoring &sc, uint32_t *prof, uint32_t *bnd, int64_t cols, LongShared &sh, int warp,
                           int W, int waits) {
  using ST = Step16<kLK, 32>;
  using L = Prof16<kLK>;
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t NGE = V16::splat(-sc.gap_extend), NGO = V16::splat(-sc.gap_open);
  const uint32_t GO = V16::splat(sc.gap_open);
  const uint32_t one = (uint32_t)(sc.gap_open >> 30) + 1u, eight = one << 3;  // not folded by the compiler
  const int nstrips = (M + kLRows - 1) / kLRows;
  auto c0_of = [&](int s) { return max(0, s * kLRows - I); };
  auto c1_of = [&](int s) { return (int)min((long long)N, (long long)(s + 1) * kLRows + J); };
  volatile unsigned long long *prog = sh.prog;
  const uint4 *tab = reinterpret_cast<const uint4 *>(prof);
  for (int s = warp; s < nstrips; s += W) {
    const int c0 = c0_of(s), c1 = c1_of(s), ncols = max(c1 - c0, 0);
    const int pc1 = s > 0 ? c1_of(s - 1) : 0;  // columns the strip above computes
    const bool last = s == nstrips - 1;
    const uint32_t *top_row = bnd + (int64_t)((s + W - 1) % W) * cols;
    uint32_t *out_row = bnd + (int64_t)(s % W) * cols;
    const int row0 = s * kLRows + lane * 2 * kLK;
    __syncwarp();
    {  // profile words of the strip's rows
      int alo[kLK], ahi[kLK];
#pragma unroll
      for (int w = 0; w < kLK; w++) {
        alo[w] = row0 + w < M ? (int)a[(int64_t)adir * (row0 + w)] : kCodePad;
        ahi[w] = row0 + kLK + w < M ? (int)a[(int64_t)adir * (row0 + kLK + w)] : kCodePad;
      }
      for (int c = 0; c < L::kCodes; c++)
#pragma unroll
        for (int w = 0; w < kLK; w++) {
          prof[((c * L::kNV + L::lo_vec(w)) * 32 + lane) * 4 + L::lo_elem(w)] =
              (uint32_t)(sub_score(alo[w], c, sc, sc.gap_open) + sc.gap_open);
          prof[((c * L::kNV + L::hi_vec(w)) * 32 + lane) * 4 + L::hi_elem(w)] =
              (uint32_t)(sub_score(ahi[w], c, sc, sc.gap_open) + sc.gap_open) << 16;
        }
    }
    __syncwarp();
    // waits until the strip above has published its columns below `col` (or ended).  `seen` is
    // its progress word as loaded a chunk ago, so a strip that is not held up does not stand
    // still for the word's latency; and `fenced` says that the fence of this strip's own publishing
    // came after that load, which then orders this strip's reads as well (one fence a chunk).
    const int pw = (s + W - 1) % W;
    unsigned long long seen = 0ull;
    bool fenced = false;
    auto await = [&](int col) -> bool {
      if (s == 0) return true;
      const unsigned long long want = ((unsigned long long)(s - 1) << 32) | (unsigned)col;
      int polls = 0;
      while (seen < want) {
        if (++polls > waits || *(volatile int *)&sh.failed) return false;
        seen = prog[pw];
        fenced = false;
      }
      if (!fenced) cluster_fence();
      seen = prog[pw];
      fenced = false;
      return true;
    };
    auto load_top = [&](int t) -> uint32_t {  // boundary words of columns c0 + t + lane
      const int j = c0 + t + lane;
      return s > 0 && j < pc1 && j < c1 ? *(volatile const uint32_t *)(top_row + j) : 0u;
    };
    bool ok = __all_sync(full, await(min(c0 + kLChunk, pc1)));  // (the warp's lanes go on or give up together)
    uint32_t cur = ok ? load_top(0) : 0u;
    // H above-left of the strip's first cell, and the base of both halves: the first columns may
    // take large values from the row above at once
    uint32_t HtopPrev = 0u;
    if (s > 0 && c0 > c0_of(s - 1) && c0 - 1 < pc1 && lane == 0 && ok)
      HtopPrev = *(volatile const uint32_t *)(top_row + c0 - 1) & 0xffffu;
    const int first_top = (int)__reduce_max_sync(full, max(cur & 0xffffu, HtopPrev));
    int base_lo = max(first_top - 1024, 0), base_hi = base_lo;
    uint32_t nbase = V16::pack(-base_lo, -base_hi);
    uint32_t P[kLK], F[kLK], lo[kLK], hi[kLK];  // (P: Step16::run of mhsw_engine16.cuh)
#pragma unroll
    for (int k = 0; k < kLK; k++) P[k] = F[k] = 0u;
    P[0] = HtopPrev;  // (the high halves start a column later, at 0)
    uint32_t Hlast = 0u, Ecout = 0u, Kl = 0u, Jp = 0u;
    const int j0 = c0 - 2 * lane;
    auto code_at = [&](int j) -> int { return j >= c0 && j < c1 ? (int)b[(int64_t)bdir * j] : kCodeN; };
    // a step's words are loaded a step ahead of their use, its code three ahead
    ST::load(tab, code_at(j0), lane, lo, hi);
    int c1s = code_at(j0 + 1), c2s = code_at(j0 + 2);
    const int steps = ncols > 0 ? ncols + 63 : 0;
    for (int t0 = 0; t0 < steps && ok; t0 += kLChunk) {
      ok = __all_sync(full, await(min(c0 + t0 + 2 * kLChunk, pc1)));
      if (goal > 0 && s > 0) {
        // An earlier strip reached the score: nothing here can win.  Tested after the wait: a
        // strip that stopped this way ends its successor's wait without its columns.
        const unsigned long long bk = *(volatile unsigned long long *)&sh.best;
        if (__any_sync(full, key_value(bk) == goal && key_row(bk) < s * kLRows)) break;
      }
      const uint32_t nxt = ok ? load_top(t0 + kLChunk) : 0u;
      auto eight_steps = [&](int tb, auto guarded) {
        constexpr bool kGuard = decltype(guarded)::value;
        const uint8_t *bl = b + (int64_t)bdir * j0;
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const int t = tb + u;
          const uint32_t w = __shfl_sync(full, cur, t & 31);
          uint32_t zH = __shfl_up_sync(full, Hlast, 1), zE = __shfl_up_sync(full, Ecout, 1);
          if (lane == 0) {
            zH = w << 16;
            zE = w;
          }
          uint32_t nlo[kLK], nhi[kLK];
          ST::load(tab, c1s, lane, nlo, nhi);
          c1s = c2s;
          c2s = kGuard ? code_at(j0 + t + 3) : (int)bl[(int64_t)bdir * (t + 3)];
          long_step<LAZY>(t, zH, zE, lo, hi, P, F, Hlast, Ecout, Kl, Jp, NGE, NGO, GO, one, eight, nbase);
#pragma unroll
          for (int k = 0; k < kLK; k++) {
            lo[k] = nlo[k];
            hi[k] = nhi[k];
          }
          const int jh = c0 + t - 63;  // the last lane's high-half column
          if (!last && lane == 31 && jh >= c0 && jh < c1) out_row[jh] = __byte_perm(Hlast, Ecout, 0x7632);
        }
      };
      // every lane's look-ahead column j0 + t + 3 lies in [c0, c1)
      const bool inside = t0 >= 64 && t0 + kLChunk + 4 <= ncols;
      for (int tb = t0; tb < t0 + kLChunk; tb += 8) {
        if (inside) eight_steps(tb, std::false_type{});
        else eight_steps(tb, std::true_type{});
        if (Kl & 0x40004000u) {  // a half's maximum is 2048 above its base: move the base below it
          const int klo = (int)(Kl & 0xffffu), khi = (int)(Kl >> 16);
          const int dlo = klo & 0x4000 ? (klo >> 3) - 1 : 0, dhi = khi & 0x4000 ? (khi >> 3) - 1 : 0;
          base_lo += dlo;
          base_hi += dhi;
          Kl = (uint32_t)(klo - 8 * dlo) | ((uint32_t)(khi - 8 * dhi) << 16);
          nbase = V16::pack(-base_lo, -base_hi);
        }
      }
      cur = nxt;
      const int done = min(t0 + kLChunk - 63, ncols);
      if (!last && done > 0) {
        cluster_fence();  // by every lane: lane 31 publishes, all read the row above
        fenced = true;
        if (lane == 31) prog[warp] = ((unsigned long long)s << 32) | (unsigned)(c0 + done);
      }
    }
    if (!ok && lane == 0) sh.failed = 1;
    if (lane == 31) {
      cluster_fence();
      prog[warp] = ((unsigned long long)s << 32) | 0xffffffffu;
    }
    unsigned long long best = 0ull;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const int key = (int)(half ? (Kl >> 16) : (Kl & 0xffffu));
      if ((key >> 3) == 0) continue;  // nothing above the base
      const int v = (half ? base_hi : base_lo) + (key >> 3);
      const int r = row0 + (half ? kLK : 0) + 7 - (key & 7);
      const int col = c0 + (int)(half ? (Jp >> 16) : (Jp & 0xffffu)) - 2 * lane - half;
      if (r < M) {
        const unsigned long long kk = best_key(v, r, col);
        best = kk > best ? kk : best;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(full, best, o);
      best = other > best ? other : best;
    }
    if (lane == 0 && best) atomicMax(&sh.best, best);
    __syncwarp();
  }
}

template <bool REV, bool LAZY>
__global__ void __launch_bounds__(256, 2) k_long(LongArgs g) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int C = cluster_size(), rank = cluster_rank();
  const int W = (int)(blockDim.x >> 5) * C, warp = (int)(threadIdx.x >> 5) * C + rank;  // strips go round the blocks
  const int cluster = blockIdx.x / C;
  uint32_t *prof = reinterpret_cast<uint32_t *>(smem + (size_t)(threadIdx.x >> 5) * Prof16<kLK>::bytes(32));
  uint32_t *bnd = g.bnd + (int64_t)cluster * W * g.cols;
  LongShared &sh = g.shared[cluster];
  volatile LongShared &vs = sh;
  const bool lead = rank == 0 && threadIdx.x == 0;
  const Scoring sc = g.sc;
  const int64_t lo = REV ? 0 : *g.first;
  const int64_t hi = REV ? (*g.list_n < g.list_cap ? *g.list_n : g.list_cap) : g.ps.n;
  auto reset = [&]() {
    if (rank == 0 && threadIdx.x < kLongWarps) vs.prog[threadIdx.x] = 0ull;
    if (lead) {
      vs.best = 0ull;
      vs.failed = 0;
    }
    cluster_barrier();
  };
  for (;;) {
    cluster_barrier();
    if (lead) vs.claim = atomicAdd(g.next, 1);
    cluster_barrier();
    const int64_t item = lo + vs.claim;
    if (item >= hi) break;
    const int64_t p = REV ? g.list[item] : (int64_t)g.order[item];
    if (REV) {
      const int S = g.rs.score[p], ie = g.rs.a_end[p], je = g.rs.b_end[p];
      const int M2 = ie + 1, N2 = je + 1;
      if (!long_begin(band_first_cap(S, sc.match, M2), S)) continue;  // the wavefront kernels take it
      const uint8_t *a = g.ps.a_code + g.ps.a_off[p] + ie, *b = g.ps.b_code + g.ps.b_off[p] + je;
      int t = band_first_cap(S, sc.match, M2);
      unsigned long long best = 0ull;
      bool failed = N2 > g.cols;  // (the boundary rows hold the stated longest B)
      while (!failed) {
        int I, J;
        band_sides(t, N2, S, sc, I, J);
        reset();
        long_sweep<LAZY>(a, -1, t, b, -1, (int)min((long long)N2, (long long)t + J), I, J, S, sc, prof, bnd, g.cols, sh,
                         warp, W, g.waits);
        cluster_barrier();
        best = vs.best;
        failed = vs.failed;
        if (key_value(best) >= S || t >= M2 || failed) break;
        t = t < M2 / 2 ? 2 * t : M2;
        cluster_barrier();  // all have read the outcome before it is reset
      }
      if (lead) {
        if (key_value(best) != S || failed) {
          g.rs.flag[p] |= kFlagTooLong;  // inconsistent, or a wait gave up
          atomicAdd(g.flagged, 1);
          g.rs.a_beg[p] = -1;
          g.rs.b_beg[p] = 0;
        } else {
          g.rs.a_beg[p] = ie - key_row(best);
          g.rs.b_beg[p] = je - key_col(best);
        }
      }
    } else {
      const int M = g.ps.a_len[p], N = g.ps.b_len[p];
      const bool fits = N <= g.cols;
      reset();
      if (fits)
        long_sweep<LAZY>(g.ps.a_code + g.ps.a_off[p], 1, M, g.ps.b_code + g.ps.b_off[p], 1, N, M, N, 0, sc, prof, bnd,
                         g.cols, sh, warp, W, g.waits);
      cluster_barrier();
      if (lead) {
        const bool failed = vs.failed || !fits;
        const unsigned long long best = vs.best;
        const int S = failed ? 0 : key_value(best);
        g.rs.flag[p] = failed ? kFlagTooLong : 0u;
        if (failed) atomicAdd(g.flagged, 1);
        g.rs.score[p] = S;
        g.rs.a_end[p] = S > 0 ? key_row(best) : -1;
        g.rs.b_end[p] = S > 0 ? key_col(best) : 0;
      }
    }
  }
}

size_t long_smem(const LongPlan &pl) {
  const size_t need = (size_t)pl.warps * Prof16<kLK>::bytes(32);
  return pl.spread ? std::max(need, size_t(120) << 10) : need;  // above half an SM's
}

template <bool REV>
cudaError_t launch(LongArgs g, const LongPlan &pl, cudaStream_t st) {
  auto kern = g.sc.gap_open >= g.sc.gap_extend ? k_long<REV, true> : k_long<REV, false>;
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(kern), long_smem(pl));
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(pl.clusters * pl.cluster));
  cfg.blockDim = dim3((unsigned)(pl.warps * 32));
  cfg.dynamicSmemBytes = long_smem(pl);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)pl.cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, g);
}

}  // namespace

// While there are SMs for it, a block an SM (by its shared memory: the hardware would put a
// cluster's blocks together otherwise) in clusters of 8 blocks of 4 warps or 4 of 8, so nearly
// every strip of a pair runs at once and on a scheduler of its own; with many pairs blocks of 4
// warps, four an SM, which stay full with pairs of three strips and more.  Forward pass of 60
// pairs of 1-12 kb: clusters of 4 x 8 warps 2.55 ms, 8 x 4 3.15 (and 2.8-3.0 without the spreading),
// 2 x 8 3.97; of 20 pairs 2.51, 2.08 and 3.95.
LongPlan plan_long(int64_t n, int max_b, int sms) {
  LongPlan pl;
  pl.spread = n <= sms;
  pl.cluster = n <= sms / 8 ? 8 : n <= sms ? 4 : n <= 2 * (int64_t)sms ? 2 : 1;
  pl.warps = pl.cluster == 4 || pl.cluster == 2 ? 8 : 4;
  pl.cols = (std::max(max_b, 1) + 63) / 64 * 64;
  const int per_sm = pl.spread ? 1 : 16 / pl.warps;
  const size_t per = (size_t)pl.cluster * pl.warps * (size_t)pl.cols * sizeof(uint32_t) + sizeof(LongShared);
  pl.clusters = (int)std::min<int64_t>(n, (int64_t)sms * per_sm / pl.cluster);
  pl.clusters = (int)std::max<int64_t>(1, std::min<int64_t>(pl.clusters, (int64_t)(kLongScratch / per)));
  pl.bytes = (size_t)pl.clusters * per + 256;
  return pl;
}

// The clusters' shared words lie in front of their boundary rows.
static void carve(LongArgs &g, const LongPlan &pl, const WorkLists &wl) {
  g.shared = reinterpret_cast<LongShared *>(wl.long_bnd);
  const size_t head = ((size_t)pl.clusters * sizeof(LongShared) + 255) / 256 * 256;
  g.bnd = wl.long_bnd + head / sizeof(uint32_t);
  g.cols = pl.cols;
  g.waits = wl.long_waits;
  g.flagged = wl.failed;
}

cudaError_t launch_long_forward(const LongPlan &pl, const PairSet &ps, const ResultSet &rs, const Scoring &sc,
                                const uint32_t *order, const int *first, const WorkLists &wl, cudaStream_t st) {
  LongArgs g{};
  g.ps = ps;
  g.rs = rs;
  g.sc = sc;
  g.order = order;
  g.first = first;
  g.next = wl.long_next;
  carve(g, pl, wl);
  return launch<false>(g, pl, st);
}

cudaError_t launch_long_reverse(const LongPlan &pl, const PairSet &ps, const ResultSet &rs, const Scoring &sc,
                                const WorkLists &wl, cudaStream_t st) {
  LongArgs g{};
  g.ps = ps;
  g.rs = rs;
  g.sc = sc;
  g.list = wl.wide;
  g.list_n = wl.wide_count;
  g.list_cap = wl.cap;
  g.next = wl.long_next + 1;
  carve(g, pl, wl);
  return launch<true>(g, pl, st);
}

}  // namespace mhsw
