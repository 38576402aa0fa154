// mhsw_long.cu -- long pairs: one block per pair, a warp per strip of A's rows.
//
// A lane group that takes a pair of several thousand rows alone walks its strips one after
// another: 60 pairs of 1-12 kb kept 60 groups of 16 lanes busy for 0.3 s on 152 SMs.  Here the
// strips of a pair run at the same time.  Warp w takes strips w, w + W, ... (512 rows each, 16 a
// lane); strip s follows strip s - 1 by about 130 columns, reading its last row's H and E^ from a
// row in global memory that the producer publishes 32 columns at a time through a progress
// word in shared memory.  A strip only ever waits for an earlier one and a warp takes its
// strips in order, so the waits end; each is bounded all the same and reports the pair as
// inconsistent if it gives up.
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
constexpr int kLongWaits = 1 << 22;     // polls before a wait gives up (seconds)

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
  uint32_t *bnd;           // per block: one row of `cols` words per warp
  int64_t cols;
};

struct LongShared {
  unsigned long long prog[16];  // per warp: strip << 32 | columns published (absolute)
  unsigned long long best;
  int claim, failed;
};

// The keyed step with keys above a base (nbase: its negative, per half).
__device__ __forceinline__ void long_step(int t, uint32_t zH, uint32_t zE, const uint32_t (&Wlo)[kLK],
                                          const uint32_t (&Phi)[kLK], uint32_t (&H)[kLK], uint32_t (&F)[kLK],
                                          uint32_t &Hlast, uint32_t &Ecout, uint32_t &HtopPrev, uint32_t &Kl,
                                          uint32_t &Jp, uint32_t NGE, uint32_t NGO, uint32_t one, uint32_t eight,
                                          uint32_t nbase) {
  uint32_t Ev = __byte_perm(zE, Ecout, 0x5432);
  const uint32_t Htop = __byte_perm(zH, Hlast, 0x5432);
  uint32_t Hd = HtopPrev;
  HtopPrev = Htop;
  uint32_t key[kLK];
#pragma unroll
  for (int k = 0; k < kLK; k++) {
    const uint32_t Q = mad_u32(mad_u32(Hd, one, Wlo[k]), one, Phi[k]);
    const uint32_t m = __vimax3_s16x2(Q, Ev, F[k]);
    const uint32_t Hn = __viaddmax_s16x2_relu(m, NGO, 0u);
    Ev = __viaddmax_s16x2(Ev, NGE, Hn);
    F[k] = __viaddmax_s16x2(F[k], NGE, Hn);
    Hd = H[k];
    H[k] = Hn;
    key[k] = mad_u32(__viaddmax_s16x2_relu(Hn, nbase, 0u), eight, (uint32_t)(7 - k) * 0x00010001u);
  }
  uint32_t Kn = Kl;
#pragma unroll
  for (int k = 0; k < kLK; k += 2) Kn = __vimax3_s16x2(Kn, key[k], key[k + 1]);
  Hlast = H[kLK - 1];
  Ecout = Ev;
  const uint32_t msk = sign_mask16(Kn - Kl + 0x7fff7fffu);
  const uint32_t tt = (uint32_t)t * 0x00010001u;
  Jp = (msk & tt) | (~msk & Jp);
  Kl = Kn;
}

// Sweep of rows [0, M) (a[adir * i]) over columns [0, N) (b[bdir * j]), row i limited to
// [i - I, i + J], by all warps of the block; best cell in sh.best.  goal > 0: strips after one
// that reached it stop.
__device__ void long_sweep(const uint8_t *a, int adir, int M, const uint8_t *b, int bdir, int N, int I, int J, int goal,
                           const Scoring &sc, uint32_t *prof, uint32_t *bnd, int64_t cols, LongShared &sh) {
  using ST = Step16<kLK, 32>;
  using L = Prof16<kLK>;
  constexpr unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  const uint32_t NGE = V16::splat(-sc.gap_extend), NGO = V16::splat(-sc.gap_open);
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
    // waits until the strip above has published its columns below `col` (or ended)
    auto await = [&](int col) -> bool {
      if (s == 0) return true;
      const unsigned long long want = ((unsigned long long)(s - 1) << 32) | (unsigned)col;
      const int pw = (s - 1) % W;
      int polls = 0;
      while (prog[pw] < want) {
        if (++polls > kLongWaits || *(volatile int *)&sh.failed) return false;
        __nanosleep(64);
      }
      __threadfence_block();
      return true;
    };
    auto load_top = [&](int t) -> uint32_t {  // boundary words of columns c0 + t + lane
      const int j = c0 + t + lane;
      return s > 0 && j < pc1 && j < c1 ? *(volatile const uint32_t *)(top_row + j) : 0u;
    };
    bool ok = await(min(c0 + kLChunk, pc1));
    uint32_t cur = ok ? load_top(0) : 0u;
    // H above-left of the strip's first cell, and the base of both halves: the first columns may
    // take large values from the row above at once
    uint32_t HtopPrev = 0u;
    if (s > 0 && c0 > c0_of(s - 1) && c0 - 1 < pc1 && lane == 0 && ok)
      HtopPrev = *(volatile const uint32_t *)(top_row + c0 - 1) & 0xffffu;
    const int first_top = (int)__reduce_max_sync(full, max(cur & 0xffffu, HtopPrev));
    int base_lo = max(first_top - 1024, 0), base_hi = base_lo;
    uint32_t nbase = V16::pack(-base_lo, -base_hi);
    uint32_t H[kLK], F[kLK], Wlo[kLK], HA[kLK], HB[kLK];
#pragma unroll
    for (int k = 0; k < kLK; k++) H[k] = F[k] = HB[k] = 0u;
    uint32_t Hlast = 0u, Ecout = 0u, Kl = 0u, Jp = 0u;
    const int j0 = c0 - 2 * lane;
    auto code_at = [&](int j) -> int { return j >= c0 && j < c1 ? (int)b[(int64_t)bdir * j] : kCodeN; };
    int ceven = code_at(j0), codd = code_at(j0 + 1);
    const int steps = ncols > 0 ? ncols + 63 : 0;
    for (int t0 = 0; t0 < steps && ok; t0 += kLChunk) {
      ok = await(min(c0 + t0 + 2 * kLChunk, pc1));
      if (goal > 0 && s > 0) {
        // An earlier strip reached the score: nothing here can win.  Tested after the wait: a
        // strip that stopped this way ends its successor's wait without its columns.
        const unsigned long long bk = *(volatile unsigned long long *)&sh.best;
        if (key_value(bk) == goal && key_row(bk) < s * kLRows) break;
      }
      const uint32_t nxt = ok ? load_top(t0 + kLChunk) : 0u;
      auto eight_steps = [&](int tb, auto guarded) {
        constexpr bool kGuard = decltype(guarded)::value;
        const uint8_t *bl = b + (int64_t)bdir * j0;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
          const int t = tb + u;
          auto top = [&](int tt, uint32_t &zH, uint32_t &zE) {
            const uint32_t w = __shfl_sync(full, cur, tt & 31);
            zH = __shfl_up_sync(full, Hlast, 1);
            zE = __shfl_up_sync(full, Ecout, 1);
            if (lane == 0) {
              zH = w << 16;
              zE = w;
            }
          };
          auto put = [&](int tt) {
            const int jh = c0 + tt - 63;  // the last lane's high-half column
            if (!last && lane == 31 && jh >= c0 && jh < c1) out_row[jh] = __byte_perm(Hlast, Ecout, 0x7632);
          };
          uint32_t zH, zE;
          int c = ceven;
          ceven = kGuard ? code_at(j0 + t + 2) : (int)bl[(int64_t)bdir * (t + 2)];
          ST::load(tab, c, lane, Wlo, HA);
          top(t, zH, zE);
          long_step(t, zH, zE, Wlo, HB, H, F, Hlast, Ecout, HtopPrev, Kl, Jp, NGE, NGO, one, eight, nbase);
          put(t);
          c = codd;
          codd = kGuard ? code_at(j0 + t + 3) : (int)bl[(int64_t)bdir * (t + 3)];
          ST::load(tab, c, lane, Wlo, HB);
          top(t + 1, zH, zE);
          long_step(t + 1, zH, zE, Wlo, HA, H, F, Hlast, Ecout, HtopPrev, Kl, Jp, NGE, NGO, one, eight, nbase);
          put(t + 1);
        }
      };
      // every lane's look-ahead columns j0 + t + 2 .. + 3 lie in [c0, c1)
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
      if (!last && lane == 31) {
        const int done = min(t0 + kLChunk - 63, ncols);
        if (done > 0) {
          __threadfence_block();
          prog[warp] = ((unsigned long long)s << 32) | (unsigned)(c0 + done);
        }
      }
    }
    if (!ok && lane == 0) sh.failed = 1;
    if (lane == 31) {
      __threadfence_block();
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

template <bool REV>
__global__ void __launch_bounds__(512) k_long(LongArgs g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ LongShared sh;
  const int warp = threadIdx.x >> 5, W = blockDim.x >> 5;
  uint32_t *prof = reinterpret_cast<uint32_t *>(smem + (size_t)warp * Prof16<kLK>::bytes(32));
  uint32_t *bnd = g.bnd + (int64_t)blockIdx.x * W * g.cols;
  const Scoring sc = g.sc;
  const int64_t lo = REV ? 0 : *g.first;
  const int64_t hi = REV ? (*g.list_n < g.list_cap ? *g.list_n : g.list_cap) : g.ps.n;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) sh.claim = atomicAdd(g.next, 1);
    __syncthreads();
    const int64_t item = lo + sh.claim;
    if (item >= hi) break;
    const int64_t p = REV ? g.list[item] : (int64_t)g.order[item];
    if (REV) {
      const int S = g.rs.score[p], ie = g.rs.a_end[p], je = g.rs.b_end[p];
      const int M2 = ie + 1, N2 = je + 1;
      if (!long_begin(band_first_cap(S, sc.match, M2), S)) continue;  // the wavefront kernels take it
      const uint8_t *a = g.ps.a_code + g.ps.a_off[p] + ie, *b = g.ps.b_code + g.ps.b_off[p] + je;
      int t = band_first_cap(S, sc.match, M2);
      for (;;) {
        int I, J;
        band_sides(t, N2, S, sc, I, J);
        __syncthreads();
        if (threadIdx.x < 16) sh.prog[threadIdx.x] = 0ull;
        if (threadIdx.x == 0) {
          sh.best = 0ull;
          sh.failed = 0;
        }
        __syncthreads();
        long_sweep(a, -1, t, b, -1, (int)min((long long)N2, (long long)t + J), I, J, S, sc, prof, bnd, g.cols, sh);
        __syncthreads();
        if (key_value(sh.best) >= S || t >= M2 || sh.failed) break;
        t = t < M2 / 2 ? 2 * t : M2;
      }
      if (threadIdx.x == 0) {
        if (key_value(sh.best) != S || sh.failed) {
          g.rs.flag[p] |= kFlagTooLong;  // inconsistent
          g.rs.a_beg[p] = -1;
          g.rs.b_beg[p] = 0;
        } else {
          g.rs.a_beg[p] = ie - key_row(sh.best);
          g.rs.b_beg[p] = je - key_col(sh.best);
        }
      }
    } else {
      const int M = g.ps.a_len[p], N = g.ps.b_len[p];
      if (threadIdx.x < 16) sh.prog[threadIdx.x] = 0ull;
      if (threadIdx.x == 0) {
        sh.best = 0ull;
        sh.failed = 0;
      }
      __syncthreads();
      long_sweep(g.ps.a_code + g.ps.a_off[p], 1, M, g.ps.b_code + g.ps.b_off[p], 1, N, M, N, 0, sc, prof, bnd, g.cols, sh);
      __syncthreads();
      if (threadIdx.x == 0) {
        const int S = key_value(sh.best);
        g.rs.flag[p] = sh.failed ? kFlagTooLong : 0u;
        g.rs.score[p] = sh.failed ? 0 : S;
        g.rs.a_end[p] = S > 0 && !sh.failed ? key_row(sh.best) : -1;
        g.rs.b_end[p] = S > 0 && !sh.failed ? key_col(sh.best) : 0;
      }
    }
  }
}

constexpr size_t long_smem(int warps) { return (size_t)warps * Prof16<kLK>::bytes(32); }

template <bool REV>
cudaError_t launch(LongArgs g, const LongPlan &pl, cudaStream_t st) {
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(k_long<REV>), long_smem(pl.warps));
  if (e != cudaSuccess) return e;
  k_long<REV><<<pl.grid, pl.warps * 32, long_smem(pl.warps), st>>>(g);
  return cudaGetLastError();
}

}  // namespace

// Few pairs: 16 warps a block, so a pair's strips all run at once; many: 4, so the SMs stay
// full with pairs of three strips and more.
LongPlan plan_long(int64_t n, int max_b, int sms) {
  LongPlan pl;
  pl.warps = n <= 2 * (int64_t)sms ? 16 : 4;
  pl.cols = (std::max(max_b, 1) + 63) / 64 * 64;
  const int per_sm = 16 / pl.warps;
  pl.grid = (int)std::min<int64_t>(n, (int64_t)sms * per_sm);
  const int64_t fit = (int64_t)(kLongScratch / sizeof(uint32_t)) / (pl.warps * pl.cols);
  pl.grid = (int)std::max<int64_t>(1, std::min<int64_t>(pl.grid, fit));
  pl.bytes = (size_t)pl.grid * pl.warps * (size_t)pl.cols * sizeof(uint32_t);
  return pl;
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
  g.bnd = wl.long_bnd;
  g.cols = pl.cols;
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
  g.bnd = wl.long_bnd;
  g.cols = pl.cols;
  return launch<true>(g, pl, st);
}

}  // namespace mhsw
