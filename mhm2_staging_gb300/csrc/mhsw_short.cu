// mhsw_short.cu -- a whole short batch in one launch: forward and begin pass of every pair.
//
// A batch of a few thousand pairs or fewer does not fill the GPU, so the general path (the
// forward kernels, a pair order for them, seven begin-pass classes on side streams, two
// wavefront launches, packing) is a chain of launches that each wait for one pair's serial
// chain.  Here one warp takes a pair end to end: B's codes staged in shared memory,
// the keyed forward sweep of mhsw_engine16.cuh over 32 lanes, then the same sweep over the
// reversed prefixes that end at the pair's end cell, then the five results.  The caller's
// bytes are translated as they are staged, so no code arena is written either.
//
// The begin sweep covers the first t = 2 * score / match + 16 reversed rows and the columns
// an alignment within them can reach (band_sides); the score is nearly always reached there,
// and the whole prefix is swept otherwise.  Both sweeps give the largest score at the
// smallest row, then column, which is SSW's rule for ends and (reversed) for begins
// (ssw_core.cpp:474-506, :1166-1178); no cell of the reversed box exceeds the score.
//
// Measured against what it replaced (whole call, resident batch): 400 mixed reads 308 -> 95 us,
// 2,000 462 -> 186, 8,100 664 -> 412; a host call of 32 pairs 207 -> 60.  short_batch draws the line to
// the general path.
//
// 32 lanes per pair give the shortest serial chain (a lane step costs its rows' chain of
// dependent maxima plus the hand-off) and no idle lanes beside a longer neighbour, at the
// price of more hand-offs per cell than the 8- and 16-lane groups of the persistent kernels.
#include <algorithm>

#include "mhsw_band.cuh"
#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"

namespace mhsw {

namespace {

constexpr int kShortPad = 72;  // N codes on both sides of B: 62 columns of lane skew plus look-ahead and unroll

__device__ __forceinline__ int base_code(unsigned char x) {  // SSW's table (c_code) by compares
  const int u = x & 0xDF;
  return u == 'A' || u == 'U' ? 0 : u == 'C' ? 1 : u == 'G' ? 2 : u == 'T' ? 3 : kCodeN;
}

// Bytes of a warp's profile table.
template <int K, bool S2>
__host__ __device__ constexpr int warp_prof(bool step) {
  constexpr int kCodes = S2 ? kCode16Zero + 1 : kCodeN + 1;
  return (int)(step ? Prof16H<K, kCodes>::bytes(32) : Prof16<K, kCodes>::bytes(32));
}

struct ShortArgs {
  PairSet ps;  // a_seq raw; b_code when the codes are resident, else b_seq raw
  Scoring sc;
  int max_a, max_b;
  int prof_bytes;
  int32_t *out5;  // n x 5, or null
  int32_t *out3;  // n x 3 (score, a_end, b_end), or null: forward pass only
  OutViews ov;    // drop-in views (null pointers: not written)
  ResultSet rs;   // the general path's result arrays (null pointers: not written)
  bool a_is_query;
};

// One step of the keyed recurrence (Step16 of mhsw_engine16.cuh) for R row pairs a lane, with
// the chain down the lane's rows shortened: E runs from H before E's own contribution,
// H' = max(max(Q, F^) - gO, 0).  Where E made H, H's update of E^ is E^ - gO <= E^ - gE (gap
// open >= gap extend, which short_batch checks), so E^' = max(E^ - gE, H') all the same.  That
// is one add-max per row on the chain instead of three operations, for one more
// instruction per cell pair: worth it where a warp has its scheduler nearly to itself.
// S2 (score2 mode) keeps each row's maximum over the valid columns in Rm, as Step16 does; STEP
// (scores up to 448: kModeStep) takes its half arithmetic, step keys and one table word a row pair.
template <int R, bool S2, bool STEP>
struct ShortStep {
  static_assert(R == 2 || R == 3 || R == 4 || R == 6 || R == 8, "row pairs per lane");
  static constexpr int kLay = R == 3 ? 4 : R;  // table layout (R = 3: that of 4, the last words unused)
  static constexpr int kCodes = S2 ? kCode16Zero + 1 : kCodeN + 1;
  using L = Prof16<kLay, kCodes>;
  using LH = Prof16H<kLay, kCodes>;
  using Eng = Step16<kLay, 32, S2, STEP ? kModeStep : kModeInt>;
  static constexpr uint32_t kKeyMask = KeyBits<R>::kMask;
  static constexpr int kStepBits = STEP ? 3 : 0;
  __device__ static __forceinline__ void load(const uint32_t *tab, int c, int lane, uint32_t (&lo)[kLay],
                                              uint32_t (&hi)[kLay]) {
    if constexpr (STEP) Eng::load_half(tab, c, lane, lo);
    else Eng::load(reinterpret_cast<const uint4 *>(tab), c, lane, lo, hi);
  }
  __device__ static __forceinline__ void put(uint32_t *tab, int c, int w, int lane, uint32_t v) {
    if constexpr (STEP) {
      tab[LH::word(c, w, lane, 32)] = v;
    } else {
      tab[((c * L::kNV + L::lo_vec(w)) * 32 + lane) * 4 + L::lo_elem(w)] = v & 0xffffu;
      tab[((c * L::kNV + L::hi_vec(w)) * 32 + lane) * 4 + L::hi_elem(w)] = v & 0xffff0000u;
    }
  }
  // P: the diagonal inputs with the high half's score added, as in Step16::run.
  __device__ static __forceinline__ void run(int t, int u, uint32_t zH, uint32_t zE, uint32_t sel,
                                             const uint32_t (&Wlo)[kLay], const uint32_t (&Whi)[kLay], uint32_t (&P)[R],
                                             uint32_t (&F)[R], uint32_t &Hlast, uint32_t &Ecout, uint32_t &Kl,
                                             uint32_t &Jp, uint32_t NGE, uint32_t NGO, uint32_t NGOh, uint32_t one,
                                             uint32_t scale, uint32_t (&Rm)[R], uint32_t vmask) {
    uint32_t Ev = prmt_sel(zE, Ecout, sel);
    const uint32_t Htop = prmt_sel(zH, Hlast, sel);
    auto add_lo = [&](uint32_t h, uint32_t w) { return STEP ? add_lo_f16x2(h, w) : mad_u32(h, one, w); };
    auto add_hi = [&](uint32_t h, uint32_t w) { return STEP ? add_hi_f16x2(h, w) : mad_u32(h, one, w); };
    uint32_t Q = add_lo(P[0], Wlo[0]), Kn = Kl;
    P[0] = add_hi(Htop, Whi[0]);
    uint32_t key[R];
#pragma unroll
    for (int k = 0; k < R; k++) {
      const uint32_t m = __vmaxs2(Q, F[k]);
      const uint32_t Hp = STEP ? add_relu_f16x2(m, NGOh) : __viaddmax_s16x2_relu(m, NGO, 0u);
      const uint32_t Hn = __viaddmax_s16x2(Ev, NGO, Hp);
      Ev = __viaddmax_s16x2(Ev, NGE, Hp);
      F[k] = __viaddmax_s16x2(F[k], NGE, Hn);
      if (k + 1 < R) {
        Q = add_lo(P[k + 1], Wlo[k + 1]);
        P[k + 1] = add_hi(Hn, Whi[k + 1]);
      } else {
        Hlast = Hn;
      }
      const uint32_t tag = (uint32_t)(kKeyMask - k) * (STEP ? 8u : 1u) + (STEP ? 7u - (uint32_t)u : 0u);
      key[k] = mad_u32(Hn, scale, tag * 0x00010001u);
      if constexpr (S2) Rm[k] = __viaddmax_s16x2(Hn, vmask, Rm[k]);
    }
#pragma unroll
    for (int k = 0; k + 1 < R; k += 2) Kn = __vimax3_s16x2(Kn, key[k], key[k + 1]);
    if constexpr (R % 2 != 0) Kn = __vmaxs2(Kn, key[R - 1]);
    Ecout = Ev;
    if constexpr (!STEP) {
      const uint32_t msk = sign_mask16(Kn - Kl + 0x7fff7fffu);
      const uint32_t tt = (uint32_t)t * 0x00010001u;
      Jp = (msk & tt) | (~msk & Jp);
    }
    Kl = Kn;
  }
};

// Keyed sweep of A rows row(0 .. M-1) (M <= 64 * R) over the columns b[0], b[dir], ...: N of
// them, with kShortPad N codes on either side.  Returns the best key (same in every lane).
// A step's profile words are loaded a step ahead of their use, its code three ahead.  S2: N
// includes SSW's zero-score padding; rowmax[row] receives each row's maximum.
template <int R, bool S2, bool STEP, class RowCode>
__device__ __forceinline__ unsigned long long sweep_warp(int M, int N, RowCode row, const uint8_t *b, int dir,
                                                         const Scoring &sc, uint32_t *prof, int lane, uint32_t one,
                                                         uint16_t *rowmax) {
  using ST = ShortStep<R, S2, STEP>;
  constexpr int K = ST::kLay;
  constexpr int KS = ST::kStepBits, KB = KeyBits<R>::kBits + KS;
  constexpr uint32_t KMASK = KeyBits<R>::kMask;
  const uint32_t NGE = V16::splat(-sc.gap_extend), NGO = V16::splat(-sc.gap_open);
  const uint32_t NGOh = (uint32_t)(0x8000 | sc.gap_open) * 0x00010001u;
  const int row0 = lane * 2 * R;
  int alo[R], ahi[R];
  uint32_t base[R];
#pragma unroll
  for (int w = 0; w < R; w++) {
    alo[w] = row0 + w < M ? row(row0 + w) : kCodePad;
    ahi[w] = row0 + R + w < M ? row(row0 + R + w) : kCodePad;
  }
  __syncwarp();
  {  // profile words, as sweep16_impl builds them
    const uint32_t miss = (uint32_t)(sc.gap_open - sc.mismatch), vn = (uint32_t)(sc.gap_open - sc.ambiguity);
    const uint32_t plus = (uint32_t)(sc.match + sc.mismatch);
    auto both = [&](int w, uint32_t v) {  // v in the halves whose row is in A
      return (alo[w] == kCodePad ? 0u : v) | (ahi[w] == kCodePad ? 0u : v << 16);
    };
#pragma unroll
    for (int w = 0; w < R; w++) {
      base[w] = (alo[w] == kCodePad ? 0u : alo[w] == kCodeN ? vn : miss) |
                (ahi[w] == kCodePad ? 0u : ahi[w] == kCodeN ? vn : miss) << 16;
      ST::put(prof, kCodeN, w, lane, both(w, vn));
      // (scores 0 against real rows)
      if constexpr (S2) ST::put(prof, kCode16Zero, w, lane, both(w, (uint32_t)sc.gap_open));
    }
#pragma unroll
    for (int c = 0; c < kCodeN; c++)
#pragma unroll
      for (int w = 0; w < R; w++)
        ST::put(prof, c, w, lane, base[w] + (alo[w] == c ? plus : 0u) + (ahi[w] == c ? plus << 16 : 0u));
  }
  __syncwarp();
  uint32_t P[R], F[R], Rm[R], lo[K], hi[K];
#pragma unroll
  for (int k = 0; k < R; k++) P[k] = F[k] = Rm[k] = 0u;
  uint32_t Hlast = 0u, Ecout = 0u, Kl = 0u, Jp = 0u;
  const uint32_t sel = lane == 0 ? 0x54BBu : 0x5432u;
  const uint32_t scale = one << KB;
  const int steps = N + 63;  // the last lane's high half ends at step N + 62
  const uint8_t *bl = b - 2 * lane * dir;
  ST::load(prof, bl[0], lane, lo, hi);
  int c1 = bl[dir], c2 = bl[2 * dir];
  for (int t = 0; t < steps; t += 4) {
    uint32_t Kb = 0u;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const uint32_t zH = __shfl_up_sync(0xffffffffu, Hlast, 1), zE = __shfl_up_sync(0xffffffffu, Ecout, 1);
      uint32_t nlo[K], nhi[K];
      ST::load(prof, c1, lane, nlo, nhi);
      c1 = c2;
      c2 = bl[(t + u + 3) * dir];
      uint32_t vmask = 0u;  // S2: -16384 in a half whose column lies outside [0, N)
      if constexpr (S2) {
        const int jl = t + u - 2 * lane;
        vmask = ((unsigned)jl < (unsigned)N ? 0u : 0x0000C000u) | ((unsigned)(jl - 1) < (unsigned)N ? 0u : 0xC0000000u);
      }
      ST::run(t + u, u, zH, zE, sel, lo, STEP ? lo : hi, P, F, Hlast, Ecout, STEP ? Kb : Kl, Jp, NGE, NGO, NGOh, one,
              scale, Rm, vmask);
#pragma unroll
      for (int k = 0; k < K; k++) {
        lo[k] = nlo[k];
        if constexpr (!STEP) hi[k] = nhi[k];
      }
    }
    if constexpr (STEP) ST::Eng::fold_block(t, Kb, Kl, Jp);
  }
  if constexpr (S2) {
#pragma unroll
    for (int k = 0; k < R; k++) {
      if (row0 + k < M) rowmax[row0 + k] = (uint16_t)(Rm[k] & 0xffffu);
      if (row0 + R + k < M) rowmax[row0 + R + k] = (uint16_t)(Rm[k] >> 16);
    }
    __syncwarp();
  }
  unsigned long long best = 0ull;
#pragma unroll
  for (int half = 0; half < 2; half++) {
    const uint32_t key = half ? (Kl >> 16) : (Kl & 0xffffu);
    const int v = (int)(key >> KB), r = row0 + (half ? R : 0) + (int)KMASK - (int)((key >> KS) & KMASK);
    const int col = (int)(half ? (Jp >> 16) : (Jp & 0xffffu)) - 2 * lane - half;
    if (v > 0 && r < M) {
      const unsigned long long kk = best_key(v, r, col);
      best = kk > best ? kk : best;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
    best = other > best ? other : best;
  }
  return best;
}

// The narrowest instantiation that holds M rows (M <= 64 * KMAX).
template <int KMAX, bool S2, bool STEP, class RowCode>
__device__ __forceinline__ unsigned long long sweep_rows(int M, int N, RowCode row, const uint8_t *b, int dir,
                                                         const Scoring &sc, uint32_t *prof, int lane, uint32_t one,
                                                         uint16_t *rowmax) {
  if (M <= 128) return sweep_warp<2, S2, STEP>(M, N, row, b, dir, sc, prof, lane, one, rowmax);
  if (M <= 192) return sweep_warp<3, S2, STEP>(M, N, row, b, dir, sc, prof, lane, one, rowmax);
  if constexpr (KMAX >= 6) {
    if (M > 384) return sweep_warp<8, S2, STEP>(M, N, row, b, dir, sc, prof, lane, one, rowmax);
    if (M > 256) return sweep_warp<6, S2, STEP>(M, N, row, b, dir, sc, prof, lane, one, rowmax);
  }
  return sweep_warp<4, S2, STEP>(M, N, row, b, dir, sc, prof, lane, one, rowmax);
}

// SSW's second-best score from the row maxima: see k_score2 in mhsw_kernels.cu.
__device__ __forceinline__ void warp_score2(const uint16_t *rm, int M, int ie, bool word, int lane, int &best, int &at) {
  const int mask = M / 2 > 15 ? M / 2 : 15;
  const int e1 = ie - mask > 0 ? ie - mask : 0;
  const int e2 = (ie + mask > M ? M : ie + mask) + (word ? 0 : 1);
  unsigned key = 0u;
  for (int i = lane; i < M; i += 32) {
    const unsigned v = rm[i];
    const unsigned k = v > 0 && (i < e1 || i >= e2) ? (v << 16) | (unsigned)(0xFFFF - i) : 0u;
    key = k > key ? k : key;
  }
  key = __reduce_max_sync(0xffffffffu, key);
  best = (int)(key >> 16);
  at = key ? 0xFFFF - (int)(key & 0xffffu) : 0;
}

__device__ __forceinline__ int16_t short_of(int v) {
  return (int16_t)(v > 32767 ? 32767 : (v < -32768 ? -32768 : v));
}

__device__ __forceinline__ void write_result(const ShortArgs &g, int64_t p, const int (&r)[5]) {
  if (g.out3) {
    g.out3[3 * p] = r[0];
    g.out3[3 * p + 1] = r[2];
    g.out3[3 * p + 2] = r[4];
    return;
  }
  if (g.out5) {
#pragma unroll
    for (int k = 0; k < 5; k++) g.out5[5 * p + k] = r[k];
  }
  if (g.rs.score) {
    g.rs.score[p] = r[0];
    g.rs.a_beg[p] = r[1];
    g.rs.a_end[p] = r[2];
    g.rs.b_beg[p] = r[3];
    g.rs.b_end[p] = r[4];
    g.rs.flag[p] = 0u;
  }
  if (g.ov.s_score) {
    const int qb = g.a_is_query ? r[1] : r[3], qe = g.a_is_query ? r[2] : r[4];
    const int rb = g.a_is_query ? r[3] : r[1], re = g.a_is_query ? r[4] : r[2];
    g.ov.s_score[p] = short_of(r[0]);
    g.ov.s_ref_beg[p] = short_of(rb);
    g.ov.s_ref_end[p] = short_of(re);
    g.ov.s_qry_beg[p] = short_of(qb);
    g.ov.s_qry_end[p] = short_of(qe);
    g.ov.w_score[p] = r[0];
    g.ov.w_ref_beg[p] = rb;
    g.ov.w_ref_end[p] = re;
    g.ov.w_qry_beg[p] = qb;
    g.ov.w_qry_end[p] = qe;
  }
}

// One warp per pair, one warp per block (so the pairs of a short batch spread over the SMs).
// Shared memory: the profile table, in score2 mode the row maxima, then B's codes between
// two pads.
template <int KMAX, bool S2, bool STEP>
__global__ void __launch_bounds__(32) k_short(ShortArgs g) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t *prof = reinterpret_cast<uint32_t *>(smem);
  uint16_t *rowmax = reinterpret_cast<uint16_t *>(smem + g.prof_bytes);
  uint8_t *bc = smem + g.prof_bytes + (S2 ? 128 * KMAX : 0) + kShortPad;  // bc[j], j in [-kShortPad, NP + kShortPad)
  const int lane = threadIdx.x;
  const Scoring sc = g.sc;
  const uint32_t one = (uint32_t)(g.max_b >> 30) + 1u;  // a 1 the compiler cannot fold
  for (int64_t p = blockIdx.x; p < g.ps.n; p += gridDim.x) {
    const int M = g.ps.a_len[p], N = g.ps.b_len[p];
    int r[5] = {0, -1, -1, 0, 0};
    int s2 = 0, s2_at = 0;
    if (M > 0 && N > 0 && M <= g.max_a && N <= g.max_b) {
      const unsigned char *a = reinterpret_cast<const unsigned char *>(g.ps.a_seq) + g.ps.a_off[p];
      const int64_t bo = g.ps.b_off[p];
      // B's codes, the columns [N, np) of score2 mode's padding, N codes around them
      auto stage = [&](int np) {
        __syncwarp();
        for (int j = lane - kShortPad; j < np + kShortPad; j += 32) {
          int c = kCodeN;
          if (j >= 0 && j < N) c = g.ps.b_code ? (int)g.ps.b_code[bo + j] : base_code((unsigned char)g.ps.b_seq[bo + j]);
          if (S2 && j >= N && j < np) c = kCode16Zero;
          bc[j] = (uint8_t)c;
        }
        __syncwarp();
      };
      auto row = [&](int i) { return base_code(a[i]); };
      int np = S2 ? ssw_pad16(N) : N;
      stage(np);
      const unsigned long long k = sweep_rows<KMAX, S2, STEP>(M, np, row, bc, 1, sc, prof, lane, one, rowmax);
      const int S = key_value(k);
      if constexpr (S2) {
        const bool word = S + ssw_bias(sc) >= 255;
        if (word && ssw_pad8(N) != np) {  // SSW's word path pads B less
          np = ssw_pad8(N);
          stage(np);
          sweep_rows<KMAX, S2, STEP>(M, np, row, bc, 1, sc, prof, lane, one, rowmax);
        }
        warp_score2(rowmax, M, S > 0 ? key_row(k) : -1, word, lane, s2, s2_at);
      }
      if (S > 0) {
        r[0] = S;
        r[2] = key_row(k);
        r[4] = key_col(k);
      }
      if (S > 0 && !g.out3) {
        const int ie = r[2], je = r[4];
        const int M2 = ie + 1, N2 = je + 1;
        // the reversed box's first t rows and the columns reachable within them, N codes
        // around them
        auto begin = [&](int t) -> unsigned long long {
          int I, J;
          band_sides(t, N2, S, sc, I, J);
          const int n2 = t + J < N2 ? t + J : N2;
          __syncwarp();
          for (int x = lane; x < kShortPad; x += 32) {
            if (je + 1 + x < np) bc[je + 1 + x] = kCodeN;
            if (je - n2 - x >= 0) bc[je - n2 - x] = kCodeN;
          }
          __syncwarp();
          return sweep_rows<KMAX, false, STEP>(t, n2, [&](int i) { return base_code(a[ie - i]); }, bc + je, -1, sc, prof,
                                         lane, one, nullptr);
        };
        const int t0 = band_first_cap(S, sc.match, M2);
        unsigned long long q = begin(t0);
        if (key_value(q) != S && t0 < M2) {
          stage(np);  // the first search overwrote codes outside its columns
          q = begin(M2);
        }
        r[1] = ie - key_row(q);
        r[3] = je - key_col(q);
      }
    }
    if (g.out3 && (M < 0 || N < 0 || M > g.max_a || N > g.max_b)) r[0] = r[2] = r[4] = -1;  // outside the stated maxima
    if (lane == 0) {
      write_result(g, p, r);
      if constexpr (S2) {
        g.rs.score2[p] = s2;
        g.rs.a_end2[p] = s2_at;
      }
    }
    __syncwarp();
  }
}

// Begin searches of the wide list, a warp each: bands wider than the banded kernels hold, those
// that outgrew theirs, and the widest of their classes while they hold few searches (warp_top_class):
// their threads walk a row pair in 0.5 us, so 250 rows took 130-160 us however few the pairs.  Same
// search as k_short's.
template <bool STEP>
__global__ void __launch_bounds__(32) k_rev_warp(PairSet ps, ResultSet rs, Scoring sc, WorkLists wl, bool longs,
                                                 bool escaped) {
  extern __shared__ __align__(16) unsigned char smem[];
  uint32_t *prof = reinterpret_cast<uint32_t *>(smem);
  uint8_t *bc = smem + warp_prof<8, false>(STEP) + kShortPad;  // reversed: bc[j] = column j of the box
  const int lane = threadIdx.x;
  const uint32_t one = (uint32_t)(sc.gap_open >> 30) + 1u;  // a 1 the compiler cannot fold
  // escaped: the searches that outgrew their band, from the end of the list
  const int64_t total = escaped ? *wl.esc_count : *wl.wide_count < wl.cap ? *wl.wide_count : wl.cap;
  for (int64_t it = blockIdx.x; it < total; it += gridDim.x) {
    const int64_t p = wl.wide[escaped ? wl.cap - 1 - it : it];
    const int S = rs.score[p], ie = rs.a_end[p], je = rs.b_end[p];
    const int M2 = ie + 1, N2 = je + 1;
    if ((longs && !escaped && long_begin(band_first_cap(S, sc.match, M2), S)) || !warp_begin(M2, N2, S, sc)) continue;
    const uint8_t *a = ps.a_code + ps.a_off[p] + ie, *b = ps.b_code + ps.b_off[p] + je;
    unsigned long long q = 0ull;
    for (int t = band_first_cap(S, sc.match, M2);; t = M2) {
      int I, J;
      band_sides(t, N2, S, sc, I, J);
      const int n2 = t + J < N2 ? t + J : N2;
      __syncwarp();
      for (int j = lane - kShortPad; j < n2 + kShortPad; j += 32)
        bc[j] = (uint8_t)((unsigned)j < (unsigned)n2 ? (int)b[-j] : kCodeN);
      __syncwarp();
      q = sweep_rows<8, false, STEP>(t, n2, [&](int i) { return (int)a[-i]; }, bc, 1, sc, prof, lane, one, nullptr);
      if (key_value(q) == S || t == M2) break;
    }
    if (lane == 0) {
      if (key_value(q) != S) {
        rs.flag[p] |= kFlagTooLong;  // inconsistent; the call fails
        atomicAdd(wl.failed, 1);
        rs.a_beg[p] = -1;
        rs.b_beg[p] = 0;
      } else {
        rs.a_beg[p] = ie - key_row(q);
        rs.b_beg[p] = je - key_col(q);
      }
    }
  }
}

}  // namespace

cudaError_t launch_rev_warp(const PairSet &ps, const ResultSet &rs, const Scoring &sc, const WorkLists &wl, int sms,
                            int max_a, int max_b, bool longs, bool escaped, cudaStream_t st) {
  const bool step = mode_for((long long)std::min(max_a, max_b) * sc.match, 8) == kModeStep;
  const size_t smem = warp_prof<8, false>(step) + 2 * kShortPad + kWarpBeginCols;
  const int64_t grid = std::min<int64_t>(ps.n, (int64_t)sms * 12);
  (step ? k_rev_warp<true> : k_rev_warp<false>)<<<(unsigned)grid, 32, smem, st>>>(ps, rs, sc, wl, longs, escaped);
  return cudaGetLastError();
}

// What the one-launch path loses on is its 32 lanes of at least four rows each (128 rows) and a sweep
// of every column by one warp.  Whole calls, resident, one launch / general path:
//   A 50-64:  2,000 pairs x 1,700 columns 189 / 208 us, 3,000 x 1,000 154 / 176, 2,500 316 / 291,
//             4,000 x 1,000 196 / 179, 1,700 295 / 230, 8,000 x 300 163 / 153, 1,000 348 / 239
//             (score2: 2,000 x 1,700 218 / 202, 8,000 x 1,000 417 / 255);
//   A 130-160: 6,500 x 1,000 382 / 362, 8,000 x 1,700 708 / 598 (score2 832 / 663);
//   A 400-512: 8,000 x 1,700 2,007 / 2,110, 3,000 x 4,600 1,696 / 2,636.
bool short_batch(const Scoring &sc, int ceiling, int64_t n, int max_a, int max_b, bool score2) {
  const int64_t columns = n * (int64_t)max_b;
  if (n > kShortPairs || columns > kShortColumns || max_a > kShortRowsMax || max_b > kShortColsMax) return false;
  if (max_a <= kShortNarrow && n > (score2 ? kNarrowPairsS2 : kNarrowPairs) && columns > kNarrowColumns) return false;
  if (max_a <= 256 && n > kMidPairs && columns > kMidColumns) return false;
  return sc.gap_open >= sc.gap_extend && keyed_scoring(sc) && !may_need_int32(sc, ceiling, max_a, max_b);
}

static cudaError_t launch(ShortArgs g, cudaStream_t st) {
  if (g.ps.n <= 0) return cudaSuccess;
  const bool small = g.max_a <= 256, s2 = g.rs.score2 != nullptr;
  const bool step = mode_for((long long)std::min(g.max_a, g.max_b) * g.sc.match, 8) == kModeStep;
  g.prof_bytes = s2 ? (small ? warp_prof<4, true>(step) : warp_prof<8, true>(step))
                    : (small ? warp_prof<4, false>(step) : warp_prof<8, false>(step));
  const size_t smem =
      ((size_t)g.prof_bytes + (s2 ? (small ? 512 : 1024) + 16 : 0) + 2 * kShortPad + (size_t)g.max_b + 15) / 16 * 16;
  auto kern = s2 ? (small ? k_short<4, true, false> : k_short<8, true, false>)
                 : (small ? k_short<4, false, false> : k_short<8, false, false>);
  if (step)
    kern = s2 ? (small ? k_short<4, true, true> : k_short<8, true, true>)
              : (small ? k_short<4, false, true> : k_short<8, false, true>);
  const cudaError_t e = raise_smem_limit(reinterpret_cast<const void *>(kern), smem);
  if (e != cudaSuccess) return e;
  kern<<<(unsigned)g.ps.n, 32, smem, st>>>(g);
  return cudaGetLastError();
}

cudaError_t launch_short(const PairSet &ps, const Scoring &sc, int max_a, int max_b, int32_t *out5, const OutViews *ov,
                         const ResultSet *rs, bool a_is_query, cudaStream_t st) {
  ShortArgs g{};
  g.ps = ps;
  g.sc = sc;
  g.max_a = max_a;
  g.max_b = max_b;
  g.out5 = out5;
  if (ov) g.ov = *ov;
  if (rs) g.rs = *rs;
  g.a_is_query = a_is_query;
  return launch(g, st);
}

cudaError_t prepare_short_forward() {
  cudaFuncAttributes a;
  cudaError_t e = cudaFuncGetAttributes(&a, k_short<4, false, false>);
  if (!e) e = cudaFuncGetAttributes(&a, k_short<8, false, false>);
  if (!e) e = cudaFuncGetAttributes(&a, k_short<4, false, true>);
  return e ? e : cudaFuncGetAttributes(&a, k_short<8, false, true>);
}

cudaError_t launch_short_forward(const PairSet &ps, const Scoring &sc, int max_a, int max_b, int32_t *out3,
                                 cudaStream_t st) {
  ShortArgs g{};
  g.ps = ps;
  g.sc = sc;
  g.max_a = max_a;
  g.max_b = max_b;
  g.out3 = out3;
  return launch(g, st);
}

}  // namespace mhsw
