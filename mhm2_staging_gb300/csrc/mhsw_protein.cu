// mhsw_protein.cu -- protein Smith-Waterman (include/mhsw.h: mhsw_align_protein).
//
// The reference declares protein kernels (src/adept-sw/kernel.cpp:510-899,
// sequence_aa_kernel / sequence_aa_reverse: score and ends, then begins, with a 24 x 24
// scoring matrix and a 91-entry ASCII encoding from the caller) that nothing in MHM2
// launches.  This path computes the same outputs with SSW's result rules, as the DNA
// path does: score = max H of the local affine recurrence (E and F opened at gap_open,
// extended at gap_extend), end = the lexicographically smallest (A row, B column) holding
// it, begin = the same rule on the reversed prefixes A[0..a_end], B[0..b_end].
//
// GB300 mapping: the keyed int16 wavefront of mhsw_engine16.cuh (k_protein16) -- a group of 16
// lanes (A up to 256 rows) or 32 takes a pair, forward and begin sweep, claiming pairs in
// length order.  The substitution scores of a lane's rows are bytes: one 128-bit shared load per
// step gives the column's scores for all of them, and one byte permute per cell pair spreads two
// of them into the halves of a word (a 24-code table of words, as the DNA engine's, would leave
// room for 4 warps an SM).  Pairs whose score could leave int16 (min(M, N) * largest score from
// 30,000 on), B above 65,000 residues, and matrices whose
// scores do not fit the bytes (below -gap open, or above 127 - gap open), take the int32
// kernels, beside the others on a side stream: one warp per pair, lanes along A (K rows a lane, 32K rows a strip), B's
// columns swept as a skewed wavefront -- lane l works on column t - l at step t and hands
// its bottom row's H and E to lane l + 1 by shuffle; strips hand their last row to the next
// through a per-warp global row.  int32 cells with DPX add-max / 3-way relu-max; the
// scoring matrix sits in shared memory, indexed by the row's code * 24 + the column's code.
// The begin pass is the same sweep on reversed views of the prefixes ending at the ends.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <vector>

#include "../../include/mhsw.h"
#include "mhsw_internal.h"
#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"
#include "mhsw_order.cuh"
#include "mhsw_types.h"

namespace mhsw {
namespace {

constexpr int kAA = 24;              // matrix dimension
constexpr int kEnc = 91;             // encoding entries (bytes 0..90)
constexpr int kPK = 8;               // rows per lane
constexpr int kPRows = 32 * kPK;     // rows per strip
constexpr int kNegBig = -(1 << 28);  // "minus infinity" for E and F at the borders

// bytes -> codes (0..23) of both arenas; any byte >= 91 or encoded outside [0, 24) sets *bad
// and gets 0.  Four bytes a step where source and destination are aligned.
__global__ void k_protein_encode(const char *__restrict__ a, uint8_t *__restrict__ ac, int64_t na,
                                 const char *__restrict__ b, uint8_t *__restrict__ bc, int64_t nb,
                                 const int16_t *__restrict__ enc, int *bad) {
  __shared__ uint8_t tab[256];
  for (int k = threadIdx.x; k < 256; k += blockDim.x) {
    const int v = k < kEnc ? enc[k] : -1;
    tab[k] = (uint8_t)(v < 0 || v >= kAA ? 0xff : v);
  }
  __syncthreads();
  bool wrong = false;
  auto one = [&](unsigned c) -> unsigned {
    const unsigned v = tab[c];
    wrong |= v == 0xff;
    return v == 0xff ? 0u : v;
  };
  const int64_t tid = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
  for (int side = 0; side < 2; side++) {
    const char *src = side ? b : a;
    uint8_t *dst = side ? bc : ac;
    const int64_t n = side ? nb : na;
    const bool vec = ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 3) == 0;
    const int64_t words = vec ? n / 4 : 0;
    for (int64_t i = tid; i < words; i += step) {
      const uint32_t w = reinterpret_cast<const uint32_t *>(src)[i];
      reinterpret_cast<uint32_t *>(dst)[i] =
          one(w & 0xff) | (one((w >> 8) & 0xff) << 8) | (one((w >> 16) & 0xff) << 16) | (one(w >> 24) << 24);
    }
    for (int64_t i = words * 4 + tid; i < n; i += step) dst[i] = (uint8_t)one((unsigned char)src[i]);
  }
  if (wrong) atomicOr(bad, 1);
}

struct PArgs {
  const uint8_t *a_code, *b_code;
  const int64_t *a_off, *b_off;
  const int32_t *a_len, *b_len;
  int64_t n;
  const int32_t *mat;  // 24 x 24
  int gO, gE;
  int32_t *score, *a_end, *b_end;  // forward: written; reverse: read (the prefixes) and
  int32_t *a_beg, *b_beg;          // begins written
  int2 *rows;                      // per warp slot: H, E of a strip's last row (max_n each)
  int64_t max_n;
  const uint32_t *list;            // int32 kernels: the pair order, from item *list_first on (null: all pairs)
  const int *list_first;
};

// ---- keyed int16 kernels ------------------------------------------------------------------

constexpr int kPadCol = kAA;                 // code of columns outside B: scores -gap open
constexpr int kPCodes = kAA + 1;
constexpr int kPWords = (kPCodes + 3) / 4;   // words of one row code's biased scores

struct P16Args {
  PArgs p;
  const uint32_t *order;
  int *ctl;                        // the order's control block
  uint32_t *bound;                 // per group: strip boundary (bound_n words; lo H, hi E^)
  int64_t bound_n;                 // longest B these kernels take, at most kPCols
};

// One step (Step16 of mhsw_engine16.cuh) with byte scores: lo words of this step's column, hi
// words of the previous one.  Bytes are below 128, so the permute's sign bytes are zeros.
// BASE: keys are formed from H above a base kept per lane half (nbase: its negative), as in
// mhsw_long.cu, so they hold scores up to int16's own limit.
template <int K, bool BASE>
struct StepP {
  static constexpr uint32_t kKeyMask = KeyBits<K>::kMask;
  __device__ static __forceinline__ void run(int t, uint32_t zH, uint32_t zE, uint32_t sel, uint32_t l0, uint32_t l1,
                                             uint32_t p0, uint32_t p1, uint32_t (&D)[K], uint32_t (&F)[K],
                                             uint32_t &Hlast, uint32_t &Ecout, uint32_t &Kl, uint32_t &Jp, uint32_t NGE,
                                             uint32_t NGO, uint32_t one, uint32_t eight, uint32_t nbase) {
    uint32_t Ev = prmt_sel(zE, Ecout, sel);
    const uint32_t Htop = prmt_sel(zH, Hlast, sel);
    auto word = [&](int k) {
      const uint32_t i = k & 3;
      return prmt_sel(k < 4 ? l0 : l1, k < 4 ? p0 : p1, i | ((8 | i) << 4) | ((4 + i) << 8) | ((12 + i) << 12));
    };
    // D[k] is row k's diagonal input (H of the row above, last column): read for Q a row ahead
    // and then replaced by the new H, so that no old H lives beside the new one
    uint32_t Q = mad_u32(D[0], one, word(0));
    D[0] = Htop;
    uint32_t key[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      const uint32_t m = __vimax3_s16x2(Q, Ev, F[k]);
      const uint32_t Hn = __viaddmax_s16x2_relu(m, NGO, 0u);
      if (k + 1 < K) {
        Q = mad_u32(D[k + 1], one, word(k + 1));
        D[k + 1] = Hn;
      } else {
        Hlast = Hn;
      }
      Ev = __viaddmax_s16x2(Ev, NGE, Hn);
      F[k] = __viaddmax_s16x2(F[k], NGE, Hn);
      const uint32_t hk = BASE ? __viaddmax_s16x2_relu(Hn, nbase, 0u) : Hn;
      key[k] = mad_u32(hk, eight, (uint32_t)(kKeyMask - k) * 0x00010001u);
    }
    uint32_t Kn = Kl;
#pragma unroll
    for (int k = 0; k < K; k += 2) Kn = __vimax3_s16x2(Kn, key[k], key[k + 1]);
    Ecout = Ev;
    const uint32_t msk = sign_mask16(Kn - Kl + 0x7fff7fffu);
    const uint32_t tt = (uint32_t)t * 0x00010001u;
    Jp = (msk & tt) | (~msk & Jp);
    Kl = Kn;
  }
};

// Sweep of A (a[adir * i], i < M) over B (b[bdir * j], j < N): the best key, and whether the
// score left the keys.  MULTI: A in strips of 2*K*G rows, the boundary row in bnd.
// BASE: the base starts at 0 and moves below a half's maximum once that is 2048 above it, looked at
// every four steps at most.  A row's H rises by at most top + gap open <= 127 a column (opening a gap
// bounds the left neighbour from below), so keys stay below 2048 + 4 * 127 < 4096; cells at or below
// the base, which is under a score already seen in the half, cannot be the best.
template <int K, int G, bool MULTI, bool BASE = false>
__device__ unsigned long long protein_sweep(const uint8_t *a, int adir, int M, const uint8_t *b, int bdir, int N,
                                            const uint32_t *rowtab, uint4 *tab, int lane, unsigned gmask, uint32_t *bnd,
                                            uint32_t NGE, uint32_t NGO, uint32_t one, int &overflow) {
  constexpr int KB = KeyBits<K>::kBits;
  constexpr uint32_t KMASK = KeyBits<K>::kMask;
  using ST = StepP<K, BASE>;
  const uint32_t scale = one << KB;
  const int nstrips = MULTI ? (M + 2 * K * G - 1) / (2 * K * G) : 1;
  const int T_end = N + 2 * G - 1;
  unsigned long long best = 0ull;
  overflow = 0;
  for (int s = 0; s < nstrips; s++) {
    const int row0 = s * 2 * K * G + lane * 2 * K;
    __syncwarp(gmask);
    // the strip's table: for four rows at a time, their scores against four codes are
    // transposed to one word per code
    {
      uint32_t *tw = reinterpret_cast<uint32_t *>(tab);
#pragma unroll
      for (int q = 0; q < 4; q++) {  // words: lo rows 0-3, 4-7, hi rows 0-3, 4-7
        if ((q & 1) * 4 >= K) continue;
        const int r0 = row0 + (q >= 2 ? K : 0) + (q & 1) * 4;
        const uint32_t *rw[4];
#pragma unroll
        for (int x = 0; x < 4; x++) rw[x] = rowtab + (r0 + x < M ? (int)a[adir * (r0 + x)] : kAA) * kPWords;
        for (int c = 0; c < kPWords; c++) {
          const uint32_t w0 = rw[0][c], w1 = rw[1][c], w2 = rw[2][c], w3 = rw[3][c];
          const uint32_t x0 = __byte_perm(w0, w1, 0x5140), x1 = __byte_perm(w2, w3, 0x5140);  // codes 0, 1
          const uint32_t y0 = __byte_perm(w0, w1, 0x7362), y1 = __byte_perm(w2, w3, 0x7362);  // codes 2, 3
          uint32_t *o = tw + ((4 * c) * G + lane) * 4 + q;
          o[0] = __byte_perm(x0, x1, 0x5410);
          if (4 * c + 1 < kPCodes) o[4 * G] = __byte_perm(x0, x1, 0x7632);
          if (4 * c + 2 < kPCodes) o[8 * G] = __byte_perm(y0, y1, 0x5410);
          if (4 * c + 3 < kPCodes) o[12 * G] = __byte_perm(y0, y1, 0x7632);
        }
      }
    }
    __syncwarp(gmask);
    const bool first = s == 0, last = s == nstrips - 1;
    uint32_t D[K], F[K];
#pragma unroll
    for (int k = 0; k < K; k++) D[k] = F[k] = 0u;
    uint32_t p0 = 0u, p1 = 0u;  // the previous column's hi scores (before column 0: -gap open)
    uint32_t Hlast = 0u, Ecout = 0u, Kl = 0u, Jp = 0u;
    int base_lo = 0, base_hi = 0;
    uint32_t nbase = 0u;
    auto move_base = [&]() {
      if constexpr (BASE) {
        static_assert(KB == 3, "keys of 12 score bits");
        if (Kl & 0x40004000u) {
          const int klo = (int)(Kl & 0xffffu), khi = (int)(Kl >> 16);
          const int dlo = klo & 0x4000 ? (klo >> 3) - 1 : 0, dhi = khi & 0x4000 ? (khi >> 3) - 1 : 0;
          base_lo += dlo;
          base_hi += dhi;
          Kl = (uint32_t)(klo - 8 * dlo) | ((uint32_t)(khi - 8 * dhi) << 16);
          nbase = V16::pack(-base_lo, -base_hi);
        }
      }
    };
    const uint32_t sel = lane == 0 && first ? 0x54BBu : 0x5432u;
    const int j0 = -2 * lane;
    auto code_at = [&](int j) -> int {  // (a load in bounds for every j: no branch around it)
      const int c = (int)b[bdir * max(0, min(j, N - 1))];
      return (unsigned)j < (unsigned)N ? c : kPadCol;
    };
    const uint8_t *ahead = b;  // the steady phase's next look-ahead code
    int ceven = code_at(j0), codd = code_at(j0 + 1);
    int t = 0;
    auto step = [&](int tt, int c) {
      const uint4 v = tab[c * G + lane];
      uint32_t zH = __shfl_up_sync(gmask, Hlast, 1, G), zE = __shfl_up_sync(gmask, Ecout, 1, G);
      if (MULTI && lane == 0 && !first) {
        const uint32_t w = tt < N ? bnd[tt] : 0u;
        zH = __byte_perm(w, 0u, 0x1000);
        zE = w;
      }
      ST::run(tt, zH, zE, sel, v.x, v.y, p0, p1, D, F, Hlast, Ecout, Kl, Jp, NGE, NGO, one, scale,
              nbase);
      p0 = v.z;
      p1 = v.w;
      if (MULTI && !last && lane == G - 1) {
        const int jh = tt - 2 * lane - 1;
        if (jh >= 0 && jh < N) bnd[jh] = __byte_perm(Hlast, Ecout, 0x7632);
      }
    };
    auto two = [&](auto guarded) {
      constexpr bool kGuard = decltype(guarded)::value;
      int c = ceven;
      ceven = kGuard ? code_at(t + 2 + j0) : (int)*ahead;
      if (!kGuard) ahead += bdir;
      step(t, c);
      c = codd;
      codd = kGuard ? code_at(t + 3 + j0) : (int)*ahead;
      if (!kGuard) ahead += bdir;
      step(t + 1, c);
    };
    // (the phases of sweep16_impl; an odd step count runs one step more over pad columns)
    for (; t < T_end && t < 2 * G - 4; t += 2) {
      two(std::true_type{});
      move_base();
    }
    ahead = b + (ptrdiff_t)bdir * (t + 2 + j0);
    // (four steps an iteration: with eight the kernel misses the instruction cache, 1.38 ms for
    // 20,000 pairs against 1.31)
    for (; t + 2 < N - 3;) {
#pragma unroll
      for (int u = 0; u < 2; u++) {
        two(std::false_type{});
        t += 2;
      }
      move_base();
    }
    for (; t < T_end; t += 2) {
      two(std::true_type{});
      move_base();
    }

    unsigned long long kbest = 0ull;
    int vmax = 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const uint32_t key = half ? (Kl >> 16) : (Kl & 0xffffu);
      if (BASE && (key >> KB) == 0) continue;  // nothing above the base
      const int v = (int)(key >> KB) + (half ? base_hi : base_lo);
      const int r = row0 + (half ? K : 0) + (int)KMASK - (int)(key & KMASK);
      const int col = (int)(half ? (Jp >> 16) : (Jp & 0xffffu)) - 2 * lane - half;
      vmax = v > vmax ? v : vmax;
      if (v > 0 && r < M) {
        const unsigned long long kk = best_key(v, r, col);
        kbest = kk > kbest ? kk : kbest;
      }
    }
    if (!BASE && vmax > KeyBits<K>::kCap) overflow = 1;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(gmask, kbest, o, G);
      kbest = other > kbest ? other : kbest;
      if (!BASE) overflow |= __shfl_xor_sync(gmask, overflow, o, G);
    }
    if (kbest > best) best = kbest;
    __syncwarp(gmask);
    if (overflow) break;  // the pair is swept again: no strip after this one matters
  }
  return best;
}

// The narrowest instantiation of the group that holds M rows.
template <int G>
__device__ __forceinline__ unsigned long long protein_rows(const uint8_t *a, int adir, int M, const uint8_t *b, int bdir,
                                                           int N, const uint32_t *rowtab, uint4 *tab, int lane,
                                                           unsigned gmask, uint32_t *bnd, uint32_t NGE, uint32_t NGO,
                                                           uint32_t one, int &over) {
  auto sweep = [&](auto k, auto multi) {
    return protein_sweep<decltype(k)::value, G, decltype(multi)::value>(a, adir, M, b, bdir, N, rowtab, tab, lane, gmask,
                                                                        bnd, NGE, NGO, one, over);
  };
  if (M <= 8 * G) return sweep(std::integral_constant<int, 4>{}, std::false_type{});
  if (M <= 12 * G) return sweep(std::integral_constant<int, 6>{}, std::false_type{});
  if (G == 16 || M <= 16 * G) return sweep(std::integral_constant<int, 8>{}, std::false_type{});
  return sweep(std::integral_constant<int, 8>{}, std::true_type{});
}

// The sweep with keys above a base, for pairs whose score left the plain keys.  (Not inlined: beside
// the plain sweeps' code it costs 20,000 ordinary pairs 2-3%.)
template <int G>
__device__ __noinline__ unsigned long long protein_based(const uint8_t *a, int adir, int M, const uint8_t *b, int bdir,
                                                            int N, const uint32_t *rowtab, uint4 *tab, int lane,
                                                            unsigned gmask, uint32_t *bnd, uint32_t NGE, uint32_t NGO,
                                                            uint32_t one) {
  int none;
  if (G == 16 || M <= 16 * G)
    return protein_sweep<8, G, false, true>(a, adir, M, b, bdir, N, rowtab, tab, lane, gmask, bnd, NGE, NGO, one, none);
  return protein_sweep<8, G, true, true>(a, adir, M, b, bdir, N, rowtab, tab, lane, gmask, bnd, NGE, NGO, one, none);
}

// Persistent: G-lane groups claim pairs of their range of the order (16 lanes: A up to 256
// rows) and run both passes.  A pair whose score leaves the keys (4032) is swept again with keys above
// a base, which costs an operation a cell pair more, not by the int32 kernels: 2,000 near-identical
// pairs of 1,400-1,600 residues 8.9 ms in int32 alone, 10.3 in int16 and then int32, 5.4 so; 4,000 of
// 600-700 2.95, 3.59 and 2.59.  The begin sweep first covers score + 32 reversed rows (an
// alignment scores at least about one a row), then the whole prefix if the score is not there.
template <int G>
__global__ void __launch_bounds__(128, 5) k_protein16(P16Args g) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ uint32_t rowtab[kPCodes * kPWords];
  const PArgs &p = g.p;
  for (int k = threadIdx.x; k < kPCodes * kPWords; k += blockDim.x) {
    const int a = k / kPWords, c0 = (k % kPWords) * 4;
    uint32_t w = 0;
    for (int x = 0; x < 4; x++)
      if (a < kAA && c0 + x < kAA) w |= (uint32_t)(p.mat[a * kAA + c0 + x] + p.gO) << (8 * x);
    rowtab[k] = w;
  }
  __syncthreads();
  const int grp = threadIdx.x / G, lane = threadIdx.x % G;
  const unsigned gmask = G == 32 ? 0xffffffffu : ((1u << (G & 31)) - 1u) << (((threadIdx.x & 31) / G) * G);
  uint4 *tab = reinterpret_cast<uint4 *>(smem) + (size_t)grp * kPCodes * G;
  uint32_t *bnd = g.bound ? g.bound + ((int64_t)blockIdx.x * (128 / G) + grp) * g.bound_n : nullptr;
  const uint32_t NGE = V16::splat(-p.gE), NGO = V16::splat(-p.gO);
  const uint32_t one = (uint32_t)(p.gO >> 30) + 1u;  // a 1 the compiler cannot fold
  const int lo = G == 16 ? 0 : g.ctl[2], hi = G == 16 ? g.ctl[2] : g.ctl[8 + kBucketWide];
  for (;;) {
    int claim = 0;
    if (lane == 0) claim = atomicAdd(g.ctl + (G == 16 ? 0 : 1), 1);
    claim = __shfl_sync(gmask, claim, 0, G);
    if (lo + claim >= hi) break;
    const uint32_t i = g.order[lo + claim];
    const int M = p.a_len[i], N = p.b_len[i];
    const uint8_t *a = p.a_code + p.a_off[i], *b = p.b_code + p.b_off[i];
    int S = 0, ie = -1, je = 0, ib = -1, jb = 0;
    if (M > 0 && N > 0) {
      // Both passes through one call: three copies of the sweeps miss the instruction cache
      // at every change of a warp's pass (20,000 pairs 1.45 -> 1.35 ms).
      const uint8_t *qa = a, *qb = b;
      int dir = 1, m = M, n = N, left_keys = 0;
      bool forward = true, based = false;
      for (;;) {
        const unsigned long long k =
            based ? protein_based<G>(qa, dir, m, qb, dir, n, rowtab, tab, lane, gmask, bnd, NGE, NGO, one)
                  : protein_rows<G>(qa, dir, m, qb, dir, n, rowtab, tab, lane, gmask, bnd, NGE, NGO, one, left_keys);
        if (forward) {
          if (!based && left_keys) {
            based = true;
            continue;
          }
          S = key_value(k);
          if (S <= 0) break;
          forward = false;
          ie = key_row(k);
          je = key_col(k);
          qa = a + ie;
          qb = b + je;
          dir = -1;
          m = min(ie + 1, S + 32);
          n = je + 1;
        } else if (key_value(k) != S && m < ie + 1) {
          m = ie + 1;
        } else {
          ib = ie - key_row(k);
          jb = je - key_col(k);
          break;
        }
      }
    }
    if (lane == 0) {
      p.score[i] = S;
      p.a_end[i] = ie;
      p.b_end[i] = je;
      p.a_beg[i] = ib;
      p.b_beg[i] = jb;
    }
  }
}

// ---- int32 kernels ------------------------------------------------------------------------

// One pass: forward (REV = false) over the whole pairs, or the begin pass (REV = true)
// over the reversed prefixes that end at each pair's end.
template <bool REV>
__global__ void __launch_bounds__(128) k_protein(PArgs g) {
  __shared__ int32_t smat[kAA * kAA];
  for (int k = threadIdx.x; k < kAA * kAA; k += blockDim.x) smat[k] = g.mat[k];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int2 *bound = g.rows + warp * g.max_n;
  const int gO = g.gO, gE = g.gE;
  for (int64_t it = (g.list ? *g.list_first : 0) + warp; it < g.n; it += nwarps) {
    const int64_t p = g.list ? (int64_t)g.list[it] : it;
    int M, N;
    const uint8_t *A = g.a_code + g.a_off[p], *B = g.b_code + g.b_off[p];
    int ie = 0, je = 0;
    if (REV) {
      if (g.score[p] <= 0) {  // score 0: begins as SSW reports them
        if (lane == 0) {
          g.a_beg[p] = -1;
          g.b_beg[p] = 0;
        }
        continue;
      }
      ie = g.a_end[p];
      je = g.b_end[p];
      M = ie + 1;
      N = je + 1;
    } else {
      M = g.a_len[p];
      N = g.b_len[p];
    }
    // codes of the pass: reversed prefixes for the begin pass
    auto acode = [&](int i) -> int { return REV ? A[ie - i] : A[i]; };
    auto bcode = [&](int j) -> int { return REV ? B[je - j] : B[j]; };
    int best = 0, bi = -1, bj = 0;  // running best over the strips done (warp-uniform)
    if (M > 0 && N > 0) {
      const int nstrips = (M + kPRows - 1) / kPRows;
      for (int s = 0; s < nstrips; s++) {
        const int row0 = s * kPRows + lane * kPK;
        int a24[kPK], Hl[kPK], Fl[kPK], rb[kPK], rj[kPK];
#pragma unroll
        for (int k = 0; k < kPK; k++) {
          const int r = row0 + k;
          a24[k] = r < M ? acode(r) * kAA : 0;
          Hl[k] = 0;
          Fl[k] = kNegBig;
          rb[k] = 0;
          rj[k] = 0;
        }
        int recvH = 0, recvE = kNegBig, prevH = 0;  // from the row above: this column, and the last
        int sendH = 0, sendE = kNegBig;
        const bool last_strip = s == nstrips - 1;
        const int steps = N + 31;
        // four steps per loop iteration (the loop's own instructions and register moves
        // are paid once per four steps: ~7% on 100-500-residue pairs)
#pragma unroll 4
        for (int t = 0; t < steps; t++) {
          // what lane l - 1 computed at t - 1 (its bottom row, column t - l)
          const int upH = __shfl_up_sync(0xffffffffu, sendH, 1);
          const int upE = __shfl_up_sync(0xffffffffu, sendE, 1);
          const int j = t - lane;
          prevH = recvH;
          if (lane == 0) {
            if (s == 0 || j >= N) {
              recvH = 0;
              recvE = kNegBig;
            } else {
              const int2 v = bound[j];
              recvH = v.x;
              recvE = v.y;
            }
          } else {
            recvH = upH;
            recvE = upE;
          }
          sendH = 0;
          sendE = kNegBig;
          if (j >= 0 && j < N) {
            const int b = bcode(j);
            int hu = recvH, eu = recvE, hd = prevH;
#pragma unroll
            for (int k = 0; k < kPK; k++) {
              const int e = __viaddmax_s32(eu, -gE, hu - gO);      // E(r, j)
              const int f = __viaddmax_s32(Fl[k], -gE, Hl[k] - gO);  // F(r, j)
              const int h = __vimax3_s32_relu(hd + smat[a24[k] + b], e, f);
              hd = Hl[k];  // H(r, j - 1): the next row's diagonal
              Hl[k] = h;
              Fl[k] = f;
              hu = h;
              eu = e;
              if (h > rb[k]) {  // first column of the row's maximum
                rb[k] = h;
                rj[k] = j;
              }
            }
            sendH = hu;
            sendE = eu;
            if (lane == 31 && !last_strip) bound[j] = make_int2(hu, eu);
          }
        }
        __syncwarp();
        // the strip's best: largest value, then smallest row (rows grow with lane and k)
        int lb = 0, li = -1, lj = 0;
#pragma unroll
        for (int k = 0; k < kPK; k++) {
          if (row0 + k < M && rb[k] > lb) {
            lb = rb[k];
            li = row0 + k;
            lj = rj[k];
          }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          const int ob = __shfl_down_sync(0xffffffffu, lb, o);
          const int oi = __shfl_down_sync(0xffffffffu, li, o);
          const int oj = __shfl_down_sync(0xffffffffu, lj, o);
          if (lane + o < 32 && (ob > lb || (ob == lb && ob > 0 && (li < 0 || oi < li)))) {
            lb = ob;
            li = oi;
            lj = oj;
          }
        }
        lb = __shfl_sync(0xffffffffu, lb, 0);
        li = __shfl_sync(0xffffffffu, li, 0);
        lj = __shfl_sync(0xffffffffu, lj, 0);
        if (lb > best) {  // a later strip replaces only with a strictly larger score
          best = lb;
          bi = li;
          bj = lj;
        }
      }
    }
    if (lane == 0) {
      if (!REV) {
        g.score[p] = best;
        g.a_end[p] = best > 0 ? bi : -1;
        g.b_end[p] = best > 0 ? bj : 0;
      } else {
        g.a_beg[p] = ie - bi;
        g.b_beg[p] = je - bj;
      }
    }
  }
}

__global__ void k_protein_pack(const int32_t *score, const int32_t *a_beg, const int32_t *a_end, const int32_t *b_beg,
                               const int32_t *b_end, int64_t n, int32_t *out5) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  out5[5 * p + 0] = score[p];
  out5[5 * p + 1] = a_beg[p];
  out5[5 * p + 2] = a_end[p];
  out5[5 * p + 3] = b_beg[p];
  out5[5 * p + 4] = b_end[p];
}

}  // namespace
}  // namespace mhsw

extern "C" {

using namespace mhsw;

int mhsw_align_protein(mhsw_driver *d, const mhsw_pairs *pairs, const int16_t *scoring_matrix,
                       const int16_t *encoding, int32_t *out5, int host_io) {
  if (!d || !pairs || !scoring_matrix || !encoding || pairs->n < 0 || (pairs->n > 0 && !out5)) return MHSW_ERR_ARG;
  const int64_t n = pairs->n;
  if (n == 0) return MHSW_OK;
  const int dev = mhsw::driver_device(d);
  if (dev < 0) return MHSW_ERR_STATE;
  for (int k = 0; k < kEnc; k++)
    if (encoding[k] < 0 || encoding[k] >= kAA) return MHSW_ERR_ARG;
  std::lock_guard<std::mutex> call_lk(mhsw::driver_call_mutex(d));
  cudaSetDevice(dev);
  cudaStream_t st = static_cast<cudaStream_t>(mhsw::driver_stream(d));
  int gO = 0, gE = 0;
  mhsw::driver_gaps(d, &gO, &gE);
  // extents: host batches are scanned in place; device batches read their lengths back
  std::vector<int32_t> dl(host_io ? 0 : 2 * (size_t)n);
  std::vector<int64_t> dof(host_io ? 0 : 2 * (size_t)n);
  const int32_t *la = pairs->a_len, *lb = pairs->b_len;
  const int64_t *oa = pairs->a_off, *ob = pairs->b_off;
  cudaError_t e = cudaSuccess;
  if (!host_io) {
    e = cudaMemcpyAsync(dl.data(), pairs->a_len, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaMemcpyAsync(dl.data() + n, pairs->b_len, sizeof(int32_t) * n, cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaMemcpyAsync(dof.data(), pairs->a_off, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaMemcpyAsync(dof.data() + n, pairs->b_off, sizeof(int64_t) * n, cudaMemcpyDeviceToHost, st);
    if (!e) e = cudaStreamSynchronize(st);
    if (e) return MHSW_ERR_CUDA;
    la = dl.data();
    lb = la + n;
    oa = dof.data();
    ob = oa + n;
  }
  int64_t ta = 0, tb = 0, max_n = 1, max_m = 1;
  for (int64_t i = 0; i < n; i++) {
    if (la[i] < 0 || lb[i] < 0 || oa[i] < 0 || ob[i] < 0) return MHSW_ERR_ARG;
    ta = std::max(ta, oa[i] + la[i]);
    tb = std::max(tb, ob[i] + lb[i]);
    max_n = std::max<int64_t>(max_n, lb[i]);
    max_m = std::max<int64_t>(max_m, la[i]);
  }
  // the keyed int16 kernels take matrices whose biased scores fit seven bits; a pair's score
  // is at most min(M, N) * top
  int top = 0, low = 0;
  for (int k = 0; k < kAA * kAA; k++) {
    top = std::max(top, (int)scoring_matrix[k]);
    low = std::min(low, (int)scoring_matrix[k]);
  }
  const bool keyed = low >= -gO && top <= 63 && top + gO <= 127 && n <= 0x7fffffff;
  const int wide_from = top > 0 ? 30000 / top : INT_MAX;  // H itself leaves int16 from there on
  const bool wide_possible = !keyed || std::min(max_m, max_n) >= wide_from || max_n > kPCols;
  char *as = nullptr, *bs = nullptr;
  int64_t *ao = nullptr, *bo = nullptr;
  int32_t *al = nullptr, *bl = nullptr;
  uint8_t *ac = nullptr, *bc = nullptr;
  int16_t *enc = nullptr;
  int32_t *mat = nullptr, *sc = nullptr, *ae = nullptr, *be = nullptr, *ab = nullptr, *bb = nullptr, *o5 = nullptr;
  int *bad = nullptr;
  int2 *rows = nullptr;
  int *ctl = nullptr;
  uint32_t *order = nullptr, *bound = nullptr;
  int sms = 152;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // one warp per pair at a time; 24 resident warps per SM (76 registers x 128 threads
  // fits 6 blocks of 4 warps) to cover the row chain's latency
  const int64_t warps = std::min<int64_t>(n, (int64_t)sms * 24);
  const size_t smem16 = 8 * (size_t)kPCodes * 16 * sizeof(uint4), smem32 = 4 * (size_t)kPCodes * 32 * sizeof(uint4);
  int occ16 = 1, occ32 = 1;
  if (keyed) {
    e = raise_smem_limit(reinterpret_cast<const void *>(k_protein16<16>), smem16);
    if (!e) e = raise_smem_limit(reinterpret_cast<const void *>(k_protein16<32>), smem32);
    if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ16, k_protein16<16>, 128, smem16);
    if (!e) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ32, k_protein16<32>, 128, smem32);
    if (e) return MHSW_ERR_CUDA;
  }
  const int64_t blocks16 = std::min<int64_t>((n + 7) / 8, (int64_t)sms * occ16);
  const int64_t blocks32 = std::min<int64_t>((n + 3) / 4, (int64_t)sms * occ32);
  const int64_t bound_n = std::min<int64_t>(max_n, kPCols);
  // the call's arrays, laid out in the handle's call arena (sized by a first pass)
  auto lay = [&](mhsw::Carve &c) {
    if (host_io) {
      c.take(&as, (size_t)ta + 16);
      c.take(&bs, (size_t)tb + 16);
      c.take(&ao, (size_t)n);
      c.take(&bo, (size_t)n);
      c.take(&al, (size_t)n);
      c.take(&bl, (size_t)n);
      c.take(&o5, (size_t)n * 5);
    }
    c.take(&ac, (size_t)ta + 16);
    c.take(&bc, (size_t)tb + 16);
    c.take(&enc, kEnc);
    c.take(&mat, kAA * kAA);
    c.take(&sc, (size_t)n);
    c.take(&ae, (size_t)n);
    c.take(&be, (size_t)n);
    c.take(&ab, (size_t)n);
    c.take(&bb, (size_t)n);
    c.take(&bad, 1);
    if (keyed) {
      c.take(&ctl, kOrderCtl);
      c.take(&order, (size_t)n);
      if (max_m > 512) c.take(&bound, (size_t)(blocks32 * 4 * bound_n));
    }
    if (wide_possible) c.take(&rows, (size_t)(warps * max_n));
  };
  mhsw::Carve sizing;
  lay(sizing);
  mhsw::Carve arena{0, mhsw::driver_call_arena(d, sizing.off)};
  if (!arena.base) return MHSW_ERR_NOMEM;
  lay(arena);
  if (host_io) {
    auto up = [&](void *dst, const void *src, size_t bytes) {
      if (!e && bytes) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    };
    up(as, pairs->a_seq, (size_t)ta);
    up(bs, pairs->b_seq, (size_t)tb);
    up(ao, pairs->a_off, sizeof(int64_t) * n);
    up(bo, pairs->b_off, sizeof(int64_t) * n);
    up(al, pairs->a_len, sizeof(int32_t) * n);
    up(bl, pairs->b_len, sizeof(int32_t) * n);
  } else {
    as = const_cast<char *>(pairs->a_seq);
    bs = const_cast<char *>(pairs->b_seq);
    ao = const_cast<int64_t *>(pairs->a_off);
    bo = const_cast<int64_t *>(pairs->b_off);
    al = const_cast<int32_t *>(pairs->a_len);
    bl = const_cast<int32_t *>(pairs->b_len);
    o5 = out5;
  }
  int32_t hmat[kAA * kAA];
  for (int k = 0; k < kAA * kAA; k++) hmat[k] = scoring_matrix[k];
  if (!e) e = cudaMemcpyAsync(mat, hmat, sizeof(hmat), cudaMemcpyHostToDevice, st);
  if (!e) e = cudaMemcpyAsync(enc, encoding, sizeof(int16_t) * kEnc, cudaMemcpyHostToDevice, st);
  if (!e) e = cudaMemsetAsync(bad, 0, sizeof(int), st);
  if (!e) {
    const int64_t steps = (std::max(ta, tb) / 4 + 255) / 256;
    k_protein_encode<<<(unsigned)std::max<int64_t>(1, std::min<int64_t>(steps, (int64_t)sms * 16)), 256, 0, st>>>(
        as, ac, ta, bs, bc, tb, enc, bad);
    e = cudaGetLastError();
  }
  PArgs g{ac, bc, ao, bo, al, bl, n, mat, gO, gE, sc, ae, be, ab, bb, rows, max_n, nullptr, nullptr};
  if (!e && keyed) {
    PairSet ps{};
    ps.a_len = al;
    ps.b_len = bl;
    ps.n = n;
    e = order_pairs(ps, Scoring{}, 1, false, n, 1, ctl, order, sms, st, nullptr, INT_MAX, INT_MAX, INT_MAX, 0,
                    wide_from);
    g.list = order;
    g.list_first = ctl + 8 + kBucketWide;
  }
  // the int32 kernels' pairs are others than the int16 kernels': side by side
  const Forks *fk = driver_forks(d);
  const bool fan = keyed && wide_possible && fk && fk->fork;
  if (!e && fan) e = fork_to(*fk, st, 1);
  if (!e && wide_possible) {
    const unsigned blocks = (unsigned)((warps * 32 + 127) / 128);
    cudaStream_t ws = fan ? fk->side[0] : st;
    k_protein<false><<<blocks, 128, 0, ws>>>(g);
    k_protein<true><<<blocks, 128, 0, ws>>>(g);
    e = cudaGetLastError();
  }
  if (!e && keyed) {
    const P16Args q{g, order, ctl, bound, bound_n};
    if (max_m > 256) k_protein16<32><<<(unsigned)blocks32, 128, smem32, st>>>(q);
    k_protein16<16><<<(unsigned)blocks16, 128, smem16, st>>>(q);
    e = cudaGetLastError();
  }
  if (fan) {
    const cudaError_t j = join_from(*fk, st, 1);  // (after a failed launch too: the arena is one call's)
    if (!e) e = j;
  }
  if (!e) {
    k_protein_pack<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(sc, ab, ae, bb, be, n, o5);
    e = cudaGetLastError();
  }
  if (!e && host_io) e = cudaMemcpyAsync(out5, o5, sizeof(int32_t) * 5 * n, cudaMemcpyDeviceToHost, st);
  int hbad = 0;
  if (!e) e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, st);
  if (!e) e = cudaStreamSynchronize(st);
  if (e) cudaStreamSynchronize(st);  // nothing of a failed call left in flight
  if (e) return e == cudaErrorMemoryAllocation ? MHSW_ERR_NOMEM : MHSW_ERR_CUDA;
  return hbad ? MHSW_ERR_ARG : MHSW_OK;
}

}  // extern "C"
