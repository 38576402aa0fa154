// mhsw_engine16.cuh -- the packed-int16 wavefront engine used for the forward pass.
//
// Same wavefront as sweep_pair in mhsw_engine.cuh (lane L holds rows [2KL, 2KL+2K) of a
// strip, low halves at column j, high halves at column j-1, lane L two steps behind
// lane L-1), with these changes, which take work off the integer ALU pipe and out of the
// issue slots:
//
//  1. Gap values are kept biased by the gap-open penalty: X^ = X + gO for X in {E, F}.
//     Then X^' = max(X^ - gE, H) uses H directly, and
//       H = max(max(Hdiag + s + gO, E^, F^) - gO, 0)
//     is one 3-way max and one add-max-relu.  Hdiag + s + gO is formed with integer
//     multiply-adds (FMA pipe) of two score words, one per half, each already
//     biased by +gO (the high half's as soon as Hdiag is known, a step earlier); this
//     needs s + gO >= 0 for every score (mismatch and ambiguity not above the gap-open
//     penalty), which the driver checks before choosing this engine.  Rows past the end of
//     A score -gO (biased 0); columns outside B read as N (score -ambiguity <= 0).  Cells
//     left of column 0 then stay exactly 0, and every cell right of the last column is at most a real cell of a smaller row, so no
//     value outside the matrix can win the arg-max or raise a false overflow.
//  2. The arg-max is tracked per lane half, not per row: each cell contributes the
//     16-bit key H*2^b + (2^b-1-k) (k = row within the half, b = 3 for up to 8 rows
//     per half, else 4), so the maximum key is the
//     largest score at the smallest row; the half's running key is kept with the step
//     at which it last strictly grew.  Because steps are columns, that step is the
//     first column at which that row reached that score -- the lexicographic rule of
//     SSW (ssw_core.cpp:474-506).  Keys need H < 2^(15-b), so this engine flags pairs
//     whose score reaches the ceiling (at most KeyBits::kCap) for the int32 engine.
//  3. In integer mode the profile table holds separate low-half and high-half words for the
//     five B codes, loaded as 128-bit vectors: K/4 vectors of low words, K/4 of high words and,
//     when K is 2 mod 4, one vector holding the last two low and the last two high
//     words (every load is a full 128-bit vector, conflict-free across the groups of a
//     warp).  A step uses the words it loads: the low ones for its own low half, the high ones
//     for the next step's high half (Step16::run).
//  4. B codes are read from global memory (each loaded two steps before its use) instead
//     of being staged in shared memory, so a group's shared memory is its profile table only.
//     The sweep runs in three phases: the middle one, where every lane's look-ahead column
//     lies inside B, loads codes without the bounds test and the N substitution, eight
//     steps per loop iteration.
//  5. A lane receives its left neighbour's last-row H and E^ words by two shuffles and
//     takes their high halves with one byte permute each, whose selector is a per-lane
//     register; lane 0 of a pair's first strip, whose row above is the zero boundary,
//     holds a sign-replicate selector instead (H and E^ are never negative, so the
//     replicated sign bytes are zero).
//
// Modes of the engine, by the largest score the kernel's pairs can reach (mode_cap):
//   kModeInt   the integer step above.
//   kModeHalf  small integers as fp16 bit patterns.  A pattern n in [0, 2047] is the fp16 value
//              n * 2^-24 -- subnormal below 1024, the first normal binade above, with one
//              spacing -- so adding patterns with fp16 adds is exact integer arithmetic while
//              sums stay below 2048, and the integer maxima order them as before.  The two adds
//              forming Hdiag + s + gO and the relu(m - gO) then run on the FMA pipe at twice
//              the rate of the integer multiply-adds and off the DPX pipe.  As fused
//              multiply-adds by (1, 0) and (0, 1) the two adds also pick their half of a word,
//              so the table holds one word per row pair instead of two (Prof16H): the integer
//              form's loads kept the shared-memory pipe 70% busy next to 71% of the issue slots.
//   kModeStep  half mode with keys that also hold the step within a block of eight, below the
//              row: the largest key of a block is its largest score at the smallest row, then
//              the first step, so the running key and its step are brought up to date once a
//              block instead of once a step (four instructions of about 80).
// Forward pass, int / half / step: 800,000 uneven pairs 13.19 / 12.91 / 12.63 ms, 30,011 pairs of
// 250 bp against 2-8 kb 7.34 / 6.74 / 6.67 (12.02 and 6.47 with the diagonal of Step16::run).
// Unsigned keys (twice the cap), or a key that ages in place of step constants, give half of the
// last gain back.  With a warp a scheduler or less the integer mode is ahead (batched_forward).
//
// Score2 mode (S2) also produces what SSW's second-best score is computed from
// (ssw_core.cpp:489, :513-536): each A row's maximum of H, over B extended to P columns
// by zero-scoring positions -- SSW pads its striped query to a multiple of 16 (byte
// path) with positions that score 0 (qP_byte, ssw_core.cpp:191), and those reach its
// per-row maxima.  The extra columns lie right of the real ones, so score and end are
// unchanged.  The profile table then has a sixth code (zero score), and each row keeps a
// running maximum over the valid columns (one DPX add-max per row and step).
#pragma once
#include <type_traits>

#include "mhsw_engine.cuh"

namespace mhsw {

constexpr int kCeiling16 = 4000;  // largest score the keyed int16 engine accepts (8 or fewer rows per half)
// Lane groups of the keyed kernels: 8 lanes per pair for A up to 160 rows (K = 4, 6, 8, 10
// rows-pairs per lane), 16 lanes for longer A (K = 6, 8; strips of 256 rows beyond).
constexpr int kGKShort = 8;
constexpr int kGKLong = 16;
__host__ __device__ constexpr int keyed_cap(int K) { return K <= 8 ? (1 << 12) - 64 : (1 << 11) - 64; }

constexpr int kCode16Zero = 5;  // score2 mode: SSW's zero-scoring query padding

template <int K, int CODES = kCodeN + 1>
struct Prof16 {
  static_assert(K % 2 == 0, "row pairs per lane must be even");
  static constexpr int kCodes = CODES;        // B codes A, C, G, T, N (outside B reads as N) [, zero]
  static constexpr int kQ = K / 4;            // full vectors of low words (and of high words)
  static constexpr bool kRem = (K % 4) != 0;  // one vector: low K-2, K-1, high K-2, K-1
  static constexpr int kNV = 2 * kQ + (kRem ? 1 : 0);  // 128-bit vectors per (code, lane)
  __host__ __device__ static constexpr size_t bytes(int lanes) { return (size_t)kCodes * kNV * lanes * 16; }
  // vector and element of low word w / high word w
  __host__ __device__ static constexpr int lo_vec(int w) { return w < 4 * kQ ? w / 4 : 2 * kQ; }
  __host__ __device__ static constexpr int lo_elem(int w) { return w < 4 * kQ ? w % 4 : w - 4 * kQ; }
  __host__ __device__ static constexpr int hi_vec(int w) { return w < 4 * kQ ? kQ + w / 4 : 2 * kQ; }
  __host__ __device__ static constexpr int hi_elem(int w) { return w < 4 * kQ ? w % 4 : 2 + w - 4 * kQ; }
};

// Half mode's table: one word per row pair (low row's score in the low half, high row's in the
// high half); a step's adds take one half each of this column's and the last column's words.
template <int K, int CODES = kCodeN + 1>
struct Prof16H {
  static_assert(K % 2 == 0, "row pairs per lane must be even");
  static constexpr int kCodes = CODES;
  static constexpr int kQ = K / 4;            // 128-bit vectors per (code, lane), then
  static constexpr bool kRem = (K % 4) != 0;  // one 64-bit vector
  __host__ __device__ static constexpr size_t bytes(int lanes) { return (size_t)kCodes * K * lanes * 4; }
  // word w of (code c, lane): the 128-bit vectors of a code lie [q][lane], the 64-bit ones after them
  __host__ __device__ static constexpr int word(int c, int w, int lane, int lanes) {
    return c * K * lanes + (w < 4 * kQ ? ((w / 4) * lanes + lane) * 4 + w % 4 : 4 * kQ * lanes + lane * 2 + (w - 4 * kQ));
  }
};

template <int KMAX, int G, int CODES = kCodeN + 1, bool HALF = false>
__host__ __device__ constexpr size_t group_prof16_bytes() {
  return HALF ? Prof16H<KMAX, CODES>::bytes(G) : Prof16<KMAX, CODES>::bytes(G);
}

// Where score2 mode writes the row maxima (rowmax[row] for the pair's A rows) and the
// number of B columns it sweeps (P >= N; columns [N, P) score 0).
struct RowMaxOut {
  int32_t *rowmax;
  int P;
};

enum : int { kModeInt = 0, kModeHalf = 1, kModeStep = 2 };
// Largest score bound of a mode: half sums stay below 2048 with match and gO at most 127; step
// keys hold the score above the row and three step bits.
__host__ __device__ constexpr int mode_cap(int mode, int K) {
  return mode == kModeStep ? (1 << (K <= 8 ? 9 : 8)) - 64 : mode == kModeHalf ? 1792 : 0x7fffffff;
}
__host__ __device__ constexpr int mode_for(long long bound, int K) {
  return bound <= mode_cap(kModeStep, K) ? kModeStep : bound <= mode_cap(kModeHalf, K) ? kModeHalf : kModeInt;
}

// a + the low (high) half of w
__device__ __forceinline__ uint32_t add_lo_f16x2(uint32_t a, uint32_t w) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0x00003C00u), "r"(a));
  return r;
}
__device__ __forceinline__ uint32_t add_hi_f16x2(uint32_t a, uint32_t w) {
  uint32_t r;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(w), "r"(0x3C000000u), "r"(a));
  return r;
}
// relu(a + c) of fp16 pairs (a * 1 + c)
__device__ __forceinline__ uint32_t add_relu_f16x2(uint32_t a, uint32_t c) {
  uint32_t r;
  asm("fma.rn.relu.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(0x3C003C00u), "r"(c));
  return r;
}

__device__ __forceinline__ uint32_t mad_u32(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t r;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
  return r;
}

// PRMT with a selector held in a register; unlike __byte_perm (which reads only the low
// three bits of each selector nibble) it keeps the sign-replicate bit.
__device__ __forceinline__ uint32_t prmt_sel(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

__device__ __forceinline__ uint32_t sign_mask16(uint32_t x) {
  // each 16-bit half -> 0xffff if its bit 15 is set, else 0 (PRMT sign-replicate mode)
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, 0xBB99;" : "=r"(r) : "r"(x), "r"(0u));
  return r;
}

// One wavefront step of the keyed engine for one lane (Step16::run).
// Arg-max key of a cell: H << kKeyBits | (kKeyMask - k), k = row within the lane half.
template <int K>
struct KeyBits {
  static constexpr int kBits = K <= 8 ? 3 : 4;
  static constexpr uint32_t kMask = (1u << kBits) - 1u;
  static constexpr int kCap = (1 << (15 - kBits)) - 64;  // largest score a key holds, with margin
};

template <int K, int G, bool S2 = false, int MODE = kModeInt>
struct Step16 {
  static constexpr bool HALF = MODE != kModeInt, STEP = MODE == kModeStep;
  using L = Prof16<K, S2 ? kCode16Zero + 1 : kCodeN + 1>;
  static constexpr uint32_t kKeyMask = KeyBits<K>::kMask;
  // NGO: -gO in both halves as integers, or (HALF) as negative fp16 patterns.
  // STEP: u is the step within its block, Kl the block's largest key (fold_block).
  // inside: both halves' columns are valid in every lane (vmask unused).
  // S2: Rm[k] keeps each row's running maximum over valid columns; vmask is 0 in a half
  // whose column is valid at this step and -16384 otherwise (an add-max then ignores it).
  // P[k] is the diagonal input of row k with the high half's score already added: a step adds the
  // low half's score to it (the column's word), and once a row's H is known the high half's score
  // of the same word to that, for the next step.  So a word is used in the step that loads it, and
  // P[k] is replaced right after its only use (no word kept for the next step, no H beside it):
  // 2K registers fewer, and fewer moves at the end of the unrolled steps.  The relu of H on the
  // integer pipe for every fourth row, to even the pipes out, costs 3%; sixteen steps an
  // iteration cost 2-4%.
  __device__ static __forceinline__ void run(int t, uint32_t zH, uint32_t zE, uint32_t sel, const uint32_t (&Wlo)[K],
                                             const uint32_t (&Whi)[K], uint32_t (&P)[K], uint32_t (&F)[K],
                                             uint32_t &Hlast, uint32_t &Ecout, uint32_t &Kl, uint32_t &Jp, uint32_t NGE,
                                             uint32_t NGO, uint32_t one, uint32_t eight, uint32_t (&Rm)[K],
                                             uint32_t vmask, int u, bool inside) {
    uint32_t Ev = prmt_sel(zE, Ecout, sel);  // lo: from the left lane, hi: own lo half
    const uint32_t Htop = prmt_sel(zH, Hlast, sel);
    // halves never carry: all terms >= 0, sum < 2^15.  Written as multiply-adds by a
    // runtime 1 so they issue on the FMA pipe, not the integer ALU pipe the DP saturates.
    auto add_lo = [&](uint32_t h, uint32_t w) { return HALF ? add_lo_f16x2(h, w) : mad_u32(h, one, w); };
    auto add_hi = [&](uint32_t h, uint32_t w) { return HALF ? add_hi_f16x2(h, w) : mad_u32(h, one, w); };
    uint32_t Q = add_lo(P[0], Wlo[0]);
    P[0] = add_hi(Htop, Whi[0]);
    uint32_t key[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      uint32_t Hn;
      const uint32_t m = __vimax3_s16x2(Q, Ev, F[k]);
      if constexpr (HALF) Hn = add_relu_f16x2(m, NGO);
      else Hn = __viaddmax_s16x2_relu(m, NGO, 0u);
      if (k + 1 < K) {
        Q = add_lo(P[k + 1], Wlo[k + 1]);
        P[k + 1] = add_hi(Hn, Whi[k + 1]);
      } else {
        Hlast = Hn;
      }
      Ev = __viaddmax_s16x2(Ev, NGE, Hn);
      F[k] = __viaddmax_s16x2(F[k], NGE, Hn);
      if constexpr (STEP) key[k] = mad_u32(Hn, eight, ((uint32_t)(kKeyMask - k) * 8u + 7u - (uint32_t)u) * 0x00010001u);
      else key[k] = mad_u32(Hn, eight, (uint32_t)(kKeyMask - k) * 0x00010001u);
      if constexpr (S2) Rm[k] = inside ? __vmaxs2(Hn, Rm[k]) : __viaddmax_s16x2(Hn, vmask, Rm[k]);
    }
    Ecout = Ev;
    if constexpr (STEP) {
#pragma unroll
      for (int k = 0; k < K; k += 2) Kl = __vimax3_s16x2(Kl, key[k], key[k + 1]);
      return;
    }
    // running key per half (keys are non-negative int16): K/2 three-way maxima
    uint32_t Kn = Kl;
#pragma unroll
    for (int k = 0; k < K; k += 2) Kn = __vimax3_s16x2(Kn, key[k], key[k + 1]);
    // record the step where the running key strictly grows
    const uint32_t msk = sign_mask16(Kn - Kl + 0x7fff7fffu);
    const uint32_t tt = (uint32_t)t * 0x00010001u;
    Jp = (msk & tt) | (~msk & Jp);
    Kl = Kn;
  }
  // Step mode: the running key (score, row; step bits 0) and its step after a block of steps from
  // t on whose largest key is Kb.
  __device__ static __forceinline__ void fold_block(int t, uint32_t Kb, uint32_t &Kl, uint32_t &Jp) {
    const uint32_t n = __vmaxs2(Kb & 0xFFF8FFF8u, Kl);
    const uint32_t grown = sign_mask16(n - Kl + 0x7fff7fffu);
    const uint32_t at = (uint32_t)t * 0x00010001u + 0x00070007u - (Kb & 0x00070007u);
    Jp = (grown & at) | (~grown & Jp);
    Kl = n;
  }
  // Half mode: the words of code c.
  __device__ static __forceinline__ void load_half(const uint32_t *tab, int c, int lane, uint32_t (&W)[K]) {
    using LH = Prof16H<K, L::kCodes>;
    const uint32_t *b = tab + c * (K * G);
#pragma unroll
    for (int q = 0; q < LH::kQ; q++) {
      const uint4 v = *reinterpret_cast<const uint4 *>(b + (q * G + lane) * 4);
      W[4 * q + 0] = v.x;
      W[4 * q + 1] = v.y;
      W[4 * q + 2] = v.z;
      W[4 * q + 3] = v.w;
    }
    if constexpr (LH::kRem) {
      const uint2 v = *reinterpret_cast<const uint2 *>(b + 4 * LH::kQ * G + lane * 2);
      W[K - 2] = v.x;
      W[K - 1] = v.y;
    }
  }
  // Words of code c: low words into Wlo, high words into Whi.
  __device__ static __forceinline__ void load(const uint4 *tab, int c, int lane, uint32_t (&Wlo)[K],
                                              uint32_t (&Whi)[K]) {
    const uint4 *b = tab + c * L::kNV * G + lane;
#pragma unroll
    for (int q = 0; q < L::kQ; q++) {
      const uint4 v = b[q * G];
      Wlo[4 * q + 0] = v.x;
      Wlo[4 * q + 1] = v.y;
      Wlo[4 * q + 2] = v.z;
      Wlo[4 * q + 3] = v.w;
      const uint4 u = b[(L::kQ + q) * G];
      Whi[4 * q + 0] = u.x;
      Whi[4 * q + 1] = u.y;
      Whi[4 * q + 2] = u.z;
      Whi[4 * q + 3] = u.w;
    }
    if constexpr (L::kRem) {
      const uint4 v = b[2 * L::kQ * G];
      Wlo[K - 2] = v.x;
      Wlo[K - 1] = v.y;
      Whi[K - 2] = v.z;
      Whi[K - 1] = v.w;
    }
  }
};

// Forward sweep of one pair with the keyed engine.  B is read directly from its code
// array in global memory (one byte per lane per step, loaded two steps ahead); the
// shared memory of the group holds only the profile table.  A must be a forward view.
template <int K, int G, bool MULTI, bool S2 = false, int MODE = kModeInt>
__device__ void sweep16_impl(const SeqView &A, const SeqView &B, const Scoring &sc, const GroupSmem &gs, int lane,
                             unsigned gmask, V16::Pay *bnd, int ceiling, SweepOut &out, const RowMaxOut &rmo) {
  using ST = Step16<K, G, S2, MODE>;
  constexpr bool HALF = ST::HALF, STEP = ST::STEP;
  using L = typename ST::L;
  constexpr int RS = 2 * K * G;
  constexpr uint32_t KMASK = KeyBits<K>::kMask;
  constexpr int KS = STEP ? 3 : 0;  // step bits below the row bits
  constexpr int KB = KeyBits<K>::kBits + KS;
  const int M = A.len, N = B.len;
  const uint32_t NGE = V16::splat(-sc.gap_extend);
  const uint32_t NGO = HALF ? (uint32_t)(0x8000 | sc.gap_open) * 0x00010001u : V16::splat(-sc.gap_open);
  const uint8_t *bg = B.base;
  constexpr int kCap = STEP ? mode_cap(MODE, K) : KeyBits<K>::kCap;
  if (ceiling > kCap) ceiling = kCap;

  unsigned long long best = 0ull;
  int overflow = 0;
  const int nstrips = (M + RS - 1) / RS;
  const int NP = S2 ? rmo.P : N;  // columns swept ([N, NP) score 0 in score2 mode)
  const int T_end = NP + 2 * G - 1;
  const uint4 *tab = reinterpret_cast<const uint4 *>(gs.prof);
  // 1 and 2^KB as values the compiler cannot fold (gs.pad is a launch argument >= 0)
  const uint32_t one = (uint32_t)(gs.pad >> 30) + 1u;
  const uint32_t scale = one << KB;

  for (int s = 0; s < nstrips; s++) {
    const int row0 = s * RS + lane * 2 * K;
    __syncwarp(gmask);
    // Profile words: lo word k = s(A[row0+k], c) + gO; hi word k = (s(A[row0+K+k], c) + gO) << 16.
    // Rows past A score -gO (0 biased).  A's codes are read once, a word is its row pair's
    // mismatch word plus the match's surplus in the halves that match.
    {
      uint32_t *tw = gs.prof;
      auto put = [&](int c, int w, uint32_t v) {
        if constexpr (HALF) {
          tw[Prof16H<K, L::kCodes>::word(c, w, lane, G)] = v;
        } else {
          tw[((c * L::kNV + L::lo_vec(w)) * G + lane) * 4 + L::lo_elem(w)] = v & 0xffffu;
          tw[((c * L::kNV + L::hi_vec(w)) * G + lane) * 4 + L::hi_elem(w)] = v & 0xffff0000u;
        }
      };
      const uint32_t miss = (uint32_t)(sc.gap_open - sc.mismatch), vn = (uint32_t)(sc.gap_open - sc.ambiguity);
      const uint32_t plus = (uint32_t)(sc.match + sc.mismatch);
      int alo[K], ahi[K];
      uint32_t base[K];
#pragma unroll
      for (int w = 0; w < K; w++) {
        alo[w] = A.code(row0 + w);
        ahi[w] = A.code(row0 + K + w);
      }
      auto both = [&](int w, uint32_t v) {  // v in the halves whose row is in A
        return (alo[w] == kCodePad ? 0u : v) | (ahi[w] == kCodePad ? 0u : v << 16);
      };
#pragma unroll
      for (int w = 0; w < K; w++) {
        base[w] = (alo[w] == kCodePad ? 0u : alo[w] == kCodeN ? vn : miss) |
                  (ahi[w] == kCodePad ? 0u : ahi[w] == kCodeN ? vn : miss) << 16;
        put(kCodeN, w, both(w, vn));
        if constexpr (S2) put(kCode16Zero, w, both(w, (uint32_t)sc.gap_open));  // scores 0 against real rows
      }
#pragma unroll 1
      for (int c = 0; c < kCodeN; c++) {
#pragma unroll
        for (int w = 0; w < K; w++) put(c, w, base[w] + (alo[w] == c ? plus : 0u) + (ahi[w] == c ? plus << 16 : 0u));
      }
    }
    __syncwarp(gmask);

    const bool first_strip = (s == 0);
    const bool last_strip = (s == nstrips - 1);
    uint32_t P[K], F[K], Wlo[K], Whi[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      P[k] = 0u;  // high words before column 0 are 0 (biased)
      F[k] = 0u;  // F^ = F + gO with F = -gO before column 0
    }
    uint32_t Hlast = 0u, Ecout = 0u;
    // lane 0 of the first strip reads zeros above: the selector replicates the sign of a
    // top byte of its own (non-negative) H and E^ words; other lanes take the left lane's hi halves
    const uint32_t sel = (lane == 0 && first_strip) ? 0x54BBu : 0x5432u;
    uint32_t Kl = 0u;    // running key per half
    uint32_t Jp = 0u;    // step of the last strict increase of Kl, per half
    uint32_t Rm[K];      // score2 mode: running row maxima over valid columns
#pragma unroll
    for (int k = 0; k < K; k++) Rm[k] = 0u;
    const int j0 = -2 * lane;  // lo column at step 0
    auto code_at = [&](int j) -> int {  // (a load in bounds for every j: no branch around it)
      const int c = (int)bg[max(0, min(j, N - 1))];
      return (unsigned)j < (unsigned)N ? c : S2 && (unsigned)j < (unsigned)NP ? kCode16Zero : kCodeN;
    };
    // score2 mode: 0 in a half whose column is inside [0, NP) at step t, else -16384
    auto vmask_at = [&](int t) -> uint32_t {
      if constexpr (!S2) return 0u;
      const int jl = t + j0;
      const uint32_t lo = (unsigned)jl < (unsigned)NP ? 0u : 0x0000C000u;
      const uint32_t hi = (unsigned)(jl - 1) < (unsigned)NP ? 0u : 0xC0000000u;
      return lo | hi;
    };
    // codes of the even and odd steps, each loaded two steps before its use
    int ceven = code_at(j0), codd = code_at(j0 + 1);

    // the left lane's H of its hi-last row and E^ below it (hi halves); lane 0 of a later
    // strip reads them from the boundary row (lo: H, hi: E^), zero past column NP
    auto top = [&](int t, uint32_t &zH, uint32_t &zE) {
      zH = __shfl_up_sync(gmask, Hlast, 1, G);
      zE = __shfl_up_sync(gmask, Ecout, 1, G);
      if (MULTI && lane == 0 && !first_strip) {
        const uint32_t b = t < NP ? bnd[t] : 0u;
        zH = __byte_perm(b, 0u, 0x1000);
        zE = b;
      }
    };
    auto out_bnd = [&](int t) {
      if (MULTI && !last_strip && lane == G - 1) {
        const int jh = t - 2 * lane - 1;  // hi-half column of the last lane
        if (jh >= 0 && jh < NP) bnd[jh] = __byte_perm(Hlast, Ecout, 0x7632);
      }
    };
    int t = 0;
    const uint8_t *bl = bg + j0;
    // Two steps; `guarded` (std::true_type / std::false_type) says whether the look-ahead
    // codes need the bounds test.
    // (STEP: u is the first one's place in its block, Kb the block's largest key).
    uint32_t Kb = 0u;
    uint32_t &Kr = STEP ? Kb : Kl;
    auto step = [&](int t, int &code, auto guarded, int u) {
      constexpr bool kGuard = decltype(guarded)::value;
      const int c = code;
      code = kGuard ? code_at(t + 2 + j0) : (int)bl[t + 2];
      if constexpr (HALF) ST::load_half(gs.prof, c, lane, Wlo);
      else ST::load(tab, c, lane, Wlo, Whi);
      uint32_t zH, zE;
      top(t, zH, zE);
      ST::run(t, zH, zE, sel, Wlo, HALF ? Wlo : Whi, P, F, Hlast, Ecout, Kr, Jp, NGE, NGO, one, scale, Rm,
              kGuard ? vmask_at(t) : 0u, u, !kGuard);
      out_bnd(t);
    };
    auto two_steps = [&](auto guarded, int u) {
      step(t, ceven, guarded, u);
      step(t + 1, codd, guarded, u + 1);
    };
    // The look-ahead columns t+2+j0 and t+3+j0 lie in [0, N) for every lane of the group
    // (j0 = -2 lane, lane < G) when 2G-4 <= t <= N-4.
    // From t = 2G on the current columns do as well (the row maxima's plain form needs it).
    const int tm0 = S2 ? 2 * G : 2 * G - 4, tm1 = N - 3;
    auto fold = [&](int t0) {
      if constexpr (STEP) {
        ST::fold_block(t0, Kb, Kl, Jp);
        Kb = 0u;
      }
    };
    for (; t + 1 < T_end && t < tm0; t += 2) {
      two_steps(std::true_type{}, 0);
      fold(t);
    }
    // eight steps per iteration in the middle phase (the loop's own instructions and the
    // register moves at its back edge are paid once per eight steps); its last few steps
    // go to the guarded drain loop, which keeps one copy of the step code fewer
    for (; t + 6 < tm1;) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        two_steps(std::false_type{}, 2 * u);
        t += 2;
      }
      fold(t - 8);
    }
    for (; t + 1 < T_end; t += 2) {
      two_steps(std::true_type{}, 0);
      fold(t);
    }
    if (t < T_end) {
      step(t, ceven, std::true_type{}, 0);
      fold(t);
    }

    if constexpr (S2) {
#pragma unroll
      for (int k = 0; k < K; k++) {
        const int rl = row0 + k, rh = row0 + K + k;
        if (rl < M) rmo.rowmax[rl] = (int32_t)(Rm[k] & 0xffffu);
        if (rh < M) rmo.rowmax[rh] = (int32_t)(Rm[k] >> 16);
      }
    }
    // Decode the two halves' keys into (value, row, column) and reduce over the group.
    unsigned long long kbest = 0ull;
    int vmax_lane = 0;
#pragma unroll
    for (int half = 0; half < 2; half++) {
      const uint32_t key = half ? (Kl >> 16) : (Kl & 0xffffu);
      const int v = (int)(key >> KB);
      const int k = (int)KMASK - (int)((key >> KS) & KMASK);
      const int r = row0 + (half ? K : 0) + k;
      const int jstep = (int)(half ? (Jp >> 16) : (Jp & 0xffffu));
      const int col = jstep - 2 * lane - half;
      if (v > vmax_lane) vmax_lane = v;  // every key counts for the overflow test (PAD rows included)
      if (v > 0 && r < M) {
        const unsigned long long kk = best_key(v, r, col);
        if (kk > kbest) kbest = kk;
      }
    }
    if (vmax_lane > ceiling) overflow = 1;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
      const unsigned long long other = __shfl_xor_sync(gmask, kbest, o, G);
      kbest = other > kbest ? other : kbest;
      overflow |= __shfl_xor_sync(gmask, overflow, o, G);
    }
    if (kbest > best) best = kbest;
    __syncwarp(gmask);
  }
  out.key = best;
  out.overflow = overflow;
}

template <int K, int G, bool S2 = false, int MODE = kModeInt>
__device__ __forceinline__ void sweep16(const SeqView &A, const SeqView &B, const Scoring &sc, const GroupSmem &gs,
                                        int lane, unsigned gmask, V16::Pay *bnd, int ceiling, SweepOut &out,
                                        const RowMaxOut &rmo = RowMaxOut{nullptr, 0}) {
  if (A.len > 2 * K * G)
    sweep16_impl<K, G, true, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, out, rmo);
  else
    sweep16_impl<K, G, false, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, out, rmo);
}

}  // namespace mhsw
