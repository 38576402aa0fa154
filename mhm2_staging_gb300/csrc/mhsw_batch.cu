// mhsw_batch.cu -- the forward pass over a batch (both forms).
//
// The reference launches one block per pair with the block size fixed by the batch's
// longest sequences (src/adept-sw/driver.cpp:343-368), so uneven batches idle most
// threads.  Here the pairs are put in order of
//   (bucket(len A), len B descending)
// on the device (bucket = rows-per-lane class of the wavefront engine, so a lane group
// always runs the narrowest engine that fits; longest B first inside a bucket), and
// persistent launches of G-lane groups claim pairs from an atomic counter
// (work stealing: a group that finishes early takes the next pair).  Pairs whose
// score could exceed the int16 range (min(lenA, lenB) * match above the int16
// capacity) are sent straight to the int32 list.
#include <algorithm>
#include <chrono>

#include "mhsw_batch.h"
#include "mhsw_engine.cuh"
#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"
#include "mhsw_order.cuh"

namespace mhsw {

namespace {

constexpr int64_t kTuneSample = 256 * 1024;  // pairs the tuner's trials run on, at most

__device__ __forceinline__ unsigned group_mask_b(int G) {
  if (G == 32) return 0xffffffffu;
  const int lane32 = threadIdx.x & 31;
  return ((1u << G) - 1u) << ((lane32 / G) * G);
}

// Persistent forward kernel over one range of the sorted pair order: 8-lane groups for
// the short-read buckets (items [0, split)), 16-lane groups for the rest ([split, n)).
// A group claims its next pair from the range's atomic counter.
// MODE: the engine's (mhsw_engine16.cuh).  In the half modes the 16-lane kernel is held to 80
// registers (six blocks of 128 an SM) and the 8-lane one to 96 (five): 800,000 uneven pairs
// 12.51 -> 12.23 ms and 30,011 pairs against 2-8 kb 6.55 -> 6.47 against 96 and 128; the score2
// kernels, which keep a row maximum per row pair, lose or spill there.
template <int G, bool S2, int MODE>
__global__ void __launch_bounds__(MODE != kModeInt && !S2 ? (G == kGKLong ? 768 : 640) : 256)
    k_fwd_persist(PairSet ps, ResultSet rs, Scoring sc, const uint32_t *__restrict__ order, int *queue, int lane_rows,
                  int min_rows, bool wide_try16, int ceiling, WorkLists wl, int pad, int bcap, V16::Pay *scratch,
                  int scratch_stride) {
  constexpr bool kShort = (G == kGKShort);
  extern __shared__ __align__(16) unsigned char smem[];
  const int gpb = blockDim.x / G;
  const int grp = threadIdx.x / G;
  const int lane = threadIdx.x % G;
  const unsigned gmask = group_mask_b(G);
  constexpr int kC = S2 ? kCode16Zero + 1 : kCodeN + 1;
  constexpr size_t kProf = kShort ? group_prof16_bytes<10, G, kC, MODE != kModeInt>()
                                  : group_prof16_bytes<8, G, kC, MODE != kModeInt>();
  unsigned char *gbase = smem + (size_t)grp * kProf;  // keyed engine: profile table only
  GroupSmem gs;
  gs.prof = reinterpret_cast<uint32_t *>(gbase);
  gs.prof_lanes = G;
  gs.bcodes = nullptr;
  gs.pad = pad;
  gs.bcap = bcap;
  const int64_t gid = (int64_t)blockIdx.x * gpb + grp;
  V16::Pay *bnd = scratch ? scratch + gid * (int64_t)scratch_stride : nullptr;
  const int64_t lo = kShort ? 0 : queue[2];
  const int64_t hi = kShort ? queue[2] : queue[kOrderLongFirst];
  int *counter = queue + (kShort ? 0 : 1);

  for (;;) {
    int claim = 0;
    if (lane == 0) claim = atomicAdd(counter, 1);
    claim = __shfl_sync(gmask, claim, 0, G);
    const int64_t item = lo + claim;
    if (item >= hi) break;
    const int64_t p = order[item];
    const int M = ps.a_len[p], N = ps.b_len[p];
    const int bucket = (M <= 0 || N <= 0) ? 0 : bucket_of(M, N, sc, lane_rows, wide_try16, min_rows);
    if (bucket == kBucketWide) {
      if (lane == 0) {
        rs.flag[p] = kFlagOverflow16;
        rs.score[p] = 0;
        rs.a_end[p] = -1;
        rs.b_end[p] = 0;
        const int slot = atomicAdd(wl.ovf_count, 1);
        if (slot < wl.cap) wl.ovf[slot] = p;
      }
      continue;
    }
    const int NP = S2 ? ssw_pad16(N) : N;
    const bool too_long = (N > kMaxB) || (bucket == kBucketStrip && (bnd == nullptr || NP > scratch_stride));
    if (M <= 0 || N <= 0 || too_long) {
      if (lane == 0) {
        rs.score[p] = 0;
        rs.a_end[p] = -1;
        rs.b_end[p] = 0;
        rs.flag[p] = too_long ? kFlagTooLong : 0u;
        if (too_long) atomicAdd(wl.failed, 1);
      }
      continue;
    }
    SeqView A{ps.a_code + ps.a_off[p], 1, M};
    SeqView B{ps.b_code + ps.b_off[p], 1, N};
    SweepOut so;
    RowMaxOut rmo{nullptr, 0};
    if constexpr (S2) rmo = RowMaxOut{ps.rowmax16 + ps.a_off[p], NP};
    if constexpr (kShort) {
      switch (bucket) {
        case 0: sweep16<4, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo); break;
        case 1: sweep16<6, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo); break;
        case 2: sweep16<8, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo); break;
        default: sweep16<10, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo); break;
      }
    } else {
      if (bucket == 4) sweep16<6, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo);
      else sweep16<8, G, S2, MODE>(A, B, sc, gs, lane, gmask, bnd, ceiling, so, rmo);
    }
    if (lane == 0) {
      const int S = key_value(so.key);
      // score2 mode: the word path's padding differs from the one swept here; the int32
      // pass recomputes those row maxima
      const bool word_redo = S2 && S + ssw_bias(sc) >= 255 && ssw_pad8(N) != NP;
      if (so.overflow || word_redo) {
        rs.flag[p] = kFlagOverflow16;
        const int slot = atomicAdd(wl.ovf_count, 1);
        if (slot < wl.cap) wl.ovf[slot] = p;
        rs.score[p] = S;
        rs.a_end[p] = -1;
        rs.b_end[p] = 0;
      } else {
        rs.flag[p] = 0u;
        rs.score[p] = S;
        rs.a_end[p] = S > 0 ? key_row(so.key) : -1;
        rs.b_end[p] = S > 0 ? key_col(so.key) : 0;
      }
    }
  }
}

template <class T>
cudaError_t grow(T **p, size_t n) {
  if (*p) cudaFree(*p);
  *p = nullptr;
  return cudaMalloc(p, n * sizeof(T));
}

}  // namespace

void BatchState::release() {
  for (uint32_t **q : {&order, &s_order}) {
    if (*q) cudaFree(*q);
    *q = nullptr;
  }
  if (scratch) cudaFree(scratch);
  if (ctl) cudaFree(ctl);
  scratch = nullptr;
  ctl = nullptr;
  cap = 0;
  scratch_bytes = 0;
}

int signature_class(int a_len) {
  return a_len <= 64 ? 0 : a_len <= 96 ? 1 : a_len <= 128 ? 2 : a_len <= 160 ? 3 : a_len <= 192 ? 4 : a_len <= 256 ? 5
         : a_len <= 1024 ? 6 : 7;
}

BatchSignature batch_signature(const int32_t *a_len, int64_t n, int max_a, int max_b) {
  BatchSignature s;
  s.max_a_class = signature_class(max_a);
  s.max_a = max_a;
  s.max_b = max_b;
  s.n = n;
  if (a_len && n > 0) {
    const int64_t step = n > 4096 ? n / 4096 : 1;
    int cnt[kSigClasses] = {0};
    int64_t k = 0;
    for (int64_t i = 0; i < n; i += step, k++) cnt[signature_class(a_len[i])]++;
    for (int c = 0; c < kSigClasses; c++) s.a_mix[c] = (float)cnt[c] / (float)k;
  }
  return s;
}

static bool within(double x, double y, double factor) {
  x = x > 1 ? x : 1;
  y = y > 1 ? y : 1;
  return x <= y * factor && y <= x * factor;
}

bool BatchSignature::close_to(const BatchSignature &o) const {
  if (max_a_class != o.max_a_class || !within(max_b, o.max_b, 2.0)) return false;
  if (!(n <= 65536 && o.n <= 65536) && !within((double)n, (double)o.n, 8.0)) return false;
  if (a_mix[0] < 0 || o.a_mix[0] < 0) return true;  // a mix the host cannot see is not compared
  for (int c = 0; c < kSigClasses; c++)
    if (a_mix[c] - o.a_mix[c] > kTolerance || o.a_mix[c] - a_mix[c] > kTolerance) return false;
  return true;
}

bool may_need_int32(const Scoring &sc, int ceiling, int max_a, int max_b) {
  const long long bound = (long long)std::min(max_a, max_b) * sc.match;
  return bound > std::min(ceiling, keyed_cap(10));
}

int batched_forward(BatchState &bs, int device, const PairSet &ps, const ResultSet &rs, const WorkLists &wl,
                    const Scoring &sc, int ceiling, int max_a, int max_b, const BatchSignature &sig, bool tune,
                    cudaStream_t st, int64_t *launches, const Forks *fk) {
  auto fail = [&](cudaError_t e, const char *what) {
    bs.err = std::string(what) + ": " + cudaGetErrorString(e);
    return 1;
  };
  const int64_t n = ps.n;
  bs.tune.last_call_tuned = false;
  if (n <= 0) return 0;
  if (n > 0x7fffffff) {
    bs.err = "batch larger than 2^31 pairs";
    return 1;
  }
  cudaError_t e;
  if ((size_t)n > bs.cap) {
    const size_t c = (size_t)n + (size_t)n / 8 + 1024;
    bs.cap = 0;
    bs.moves++;
    if ((e = grow(&bs.order, c))) return fail(e, "cudaMalloc pair order");
    bs.cap = c;
  }
  if (!bs.ctl && (e = cudaMalloc(&bs.ctl, sizeof(int) * kOrderCtl))) return fail(e, "cudaMalloc order counters");
  int *queue = bs.ctl;

  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (max_b > kMaxB) {
    bs.err = "B longer than the kernel limit";
    return 1;
  }
  const bool s2 = ps.rowmax16 != nullptr;
  BatchShape plain;  // the plain form's configuration
  // A plain batch that leaves lane groups without a pair waits for the slowest warp's chain.  Its pairs
  // all take the longest one's bucket (up to 256 rows): a warp whose groups are of two buckets runs
  // their sweeps one after the other (2,000 pairs of 100-250 rows x 8,200-9,000 columns 1.79 -> 1.25 ms).
  // 16-lane groups have the shorter chain, 8-lane ones halve the warps: the lines are where the warps
  // come to two, and six, a scheduler.  Same columns, 8 / 16 lanes: 50-64 rows, 30 pairs 622 / 742 us,
  // 9,000 1,266 / 3,000; 100-128, 1,000 954 / 805, 1,500 958 / 996; 150-160, 3,600 1,469 / 1,312, 4,500
  // 1,488 / 1,703.  Beyond the outer lines the buckets' own sizes pay (7,500 of 100-250 3.29 ms).
  // (A batch of empty A only has no longer kernel to go to: any_long is max_a > lane_rows.)
  if (!tune && max_a > 0 && n <= (int64_t)sms * (max_a <= 192 ? 64 : 40)) {
    plain.min_rows = std::min(max_a, 256);
    const bool eight =
        max_a <= 64 || (max_a <= 128 && n > (int64_t)sms * 8) || (max_a <= 160 && n > (int64_t)sms * 24);
    if (!eight) plain.lane_rows = 0;
  }
  // The engine's mode by the largest score of each kernel's pairs (8-lane groups take at most
  // 160 rows).  One bucket on up to about a warp a scheduler: integers have the shorter chain.  Calls, half or
  // step keys / integers: 30 pairs of 600-1,000 rows squared 2.11 / 2.00 ms, 1,000 of 200-256 x
  // 8,200-9,000 1.01 / 0.98; 2,000 of the latter 1.25 / 1.29.  On 8 lanes only six row pairs a lane gain
  // (2,000 of 50-96 832 / 805 us; 50-64 650 / 659, 100-128 960 / 959).
  const bool few_l = plain.min_rows > 0 && plain.lane_rows == 0 && n <= (int64_t)sms * (max_a > 256 ? 13 : 8);
  const bool few_s = plain.min_rows > 64 && plain.min_rows <= 96 && n <= (int64_t)sms * 16;
  const int mode_s = few_s ? kModeInt : mode_for((long long)std::min({max_a, max_b, 160}) * sc.match, 10);
  const int mode_l = few_l ? kModeInt : mode_for((long long)std::min(max_a, max_b) * sc.match, 8);
  using Kern = decltype(&k_fwd_persist<kGKShort, false, kModeInt>);
  auto pick = [&](int mode, Kern i, Kern h, Kern t, Kern i2, Kern h2, Kern t2) -> Kern {
    return mode == kModeStep ? (s2 ? t2 : t) : mode == kModeHalf ? (s2 ? h2 : h) : (s2 ? i2 : i);
  };
  const Kern kshort = pick(mode_s, k_fwd_persist<kGKShort, false, 0>, k_fwd_persist<kGKShort, false, 1>,
                           k_fwd_persist<kGKShort, false, 2>, k_fwd_persist<kGKShort, true, 0>,
                           k_fwd_persist<kGKShort, true, 1>, k_fwd_persist<kGKShort, true, 2>);
  const Kern klong = pick(mode_l, k_fwd_persist<kGKLong, false, 0>, k_fwd_persist<kGKLong, false, 1>,
                          k_fwd_persist<kGKLong, false, 2>, k_fwd_persist<kGKLong, true, 0>,
                          k_fwd_persist<kGKLong, true, 1>, k_fwd_persist<kGKLong, true, 2>);
  // profile table of a group, one of (codes, form)
  auto prof_of = [&](bool h, size_t full, size_t full_s2, size_t half_w, size_t half_s2) -> size_t {
    return h ? (s2 ? half_s2 : half_w) : (s2 ? full_s2 : full);
  };
  constexpr int kZ = kCode16Zero + 1, kN = kCodeN + 1;
  const size_t prof_short =
      prof_of(mode_s != kModeInt, group_prof16_bytes<10, kGKShort, kN>(), group_prof16_bytes<10, kGKShort, kZ>(),
              group_prof16_bytes<10, kGKShort, kN, true>(), group_prof16_bytes<10, kGKShort, kZ, true>());
  const size_t prof_long =
      prof_of(mode_l != kModeInt, group_prof16_bytes<8, kGKLong, kN>(), group_prof16_bytes<8, kGKLong, kZ>(),
              group_prof16_bytes<8, kGKLong, kN, true>(), group_prof16_bytes<8, kGKLong, kZ, true>());
  // long pairs take blocks of their own (not in score2 mode, which needs their row maxima, nor
  // under a lowered int16 ceiling, which asks for the int32 pass)
  const bool longs = max_a > kLongRows && !s2 && wl.long_bnd && ceiling >= kCeiling16;
  const int long_rows = longs ? kLongRows : INT_MAX;
  const int pad = 2 * kGKLong;
  // strip scratch stride: B, the lane skew and score2 mode's zero-score padding (< 16)
  const int bcap = ((pad + std::max(max_b, 1) + 16 + 2 * kGKLong) + 15) / 16 * 16;

  // order of m items (pair i * stride); clears the claim counters
  auto order_items = [&](const BatchShape &sh, int64_t m, int64_t stride, uint32_t *order) -> int {
    if ((e = order_pairs(ps, sc, sh.lane_rows, sh.wide_try16, m, stride, bs.ctl, order, sms, st, launches, INT_MAX,
                         INT_MAX, long_rows, sh.min_rows)))
      return fail(e, "order launch");
    return 0;
  };

  // the two persistent launches over m ordered items
  auto run = [&](const BatchShape &sh, const uint32_t *order, int64_t m, float *ms) -> int {
    const int threads = sh.groups_per_block * 8;  // block size: 8 groups of 8 lanes or 4 of 16, etc.
    const int gpb_s = threads / kGKShort, gpb_l = threads / kGKLong;
    const size_t smem_s = (size_t)gpb_s * prof_short, smem_l = (size_t)gpb_l * prof_long;
    cudaError_t e2;
    if ((e2 = raise_smem_limit(reinterpret_cast<const void *>(kshort), smem_s))) return fail(e2, "smem attribute");
    if ((e2 = raise_smem_limit(reinterpret_cast<const void *>(klong), smem_l))) return fail(e2, "smem attribute");
    int occ_s = 0, occ_l = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_s, kshort, threads, smem_s);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ_l, klong, threads, smem_l);
    occ_s = std::max(occ_s, 1);
    occ_l = std::max(occ_l, 1);
    // no more blocks than the items fill
    auto grid_of = [&](int occ, int gpb) {
      const int64_t full = (int64_t)sms * (sh.blocks_per_sm > 0 ? std::min(sh.blocks_per_sm, occ) : occ);
      return (int)std::min<int64_t>(full, (m + gpb - 1) / gpb);
    };
    const int grid_s = grid_of(occ_s, gpb_s), grid_l = grid_of(occ_l, gpb_l);
    // every pair is in the short buckets when the longest A is and no score bound sends a
    // pair to the int32 list
    const bool any_long = max_a > sh.lane_rows || (long long)std::min(max_a, max_b) * sc.match > keyed_cap(10);
    V16::Pay *scr = nullptr;
    const int stride = bcap;
    if (max_a > 2 * 8 * kGKLong) {
      const size_t need = (size_t)grid_l * gpb_l * (size_t)stride * sizeof(V16::Pay);
      if (need > bs.scratch_bytes) {
        bs.moves++;
        if (bs.scratch) cudaFree(bs.scratch);
        bs.scratch = nullptr;
        bs.scratch_bytes = 0;
        e2 = cudaMalloc(&bs.scratch, need);
        if (e2) return fail(e2, "cudaMalloc strip scratch");
        bs.scratch_bytes = need;
      }
      scr = reinterpret_cast<V16::Pay *>(bs.scratch);
    }
    cudaEvent_t t0 = nullptr, t1 = nullptr;
    if (ms) {  // a trial: its sample is run again and again in one order
      cudaEventCreate(&t0);
      cudaEventCreate(&t1);
      cudaEventRecord(t0, st);
      cudaMemsetAsync(queue, 0, 2 * sizeof(int), st);
      cudaMemsetAsync(wl.ovf_count, 0, sizeof(int), st);
    }
    const bool any_short = sh.lane_rows > 0;
    const bool fan = any_long && any_short && fk && fk->fork;
    if (fan && (e2 = fork_to(*fk, st, 1))) return fail(e2, "fork");
    if (any_long)
      klong<<<grid_l, threads, smem_l, fan ? fk->side[0] : st>>>(ps, rs, sc, order, queue, sh.lane_rows, sh.min_rows,
                                                                 sh.wide_try16, ceiling, wl, pad, bcap, scr, stride);
    if (any_short)
      kshort<<<grid_s, threads, smem_s, st>>>(ps, rs, sc, order, queue, sh.lane_rows, sh.min_rows, sh.wide_try16, ceiling,
                                               wl, pad, bcap, nullptr, stride);
    e2 = cudaGetLastError();
    if (e2) return fail(e2, "persistent forward launch");
    if (fan && (e2 = join_from(*fk, st, 1))) return fail(e2, "join");
    if (launches) *launches += (any_long ? 1 : 0) + (any_short ? 1 : 0);
    if (ms) {
      cudaEventRecord(t1, st);
      cudaEventSynchronize(t1);
      cudaEventElapsedTime(ms, t0, t1);
      cudaEventDestroy(t0);
      cudaEventDestroy(t1);
    }
    return 0;
  };

  // a configuration tuned earlier for a signature close to this one is taken back without
  // trials (batches that alternate between workloads, such as full and partial serving
  // micro-batches, tune once each)
  if (tune && bs.autotune && (!bs.tuned || !sig.close_to(bs.tuned_for))) {
    for (int k = 0; k < bs.n_cached; k++)
      if (sig.close_to(bs.cached[k].sig)) {
        bs.shape = bs.cached[k].shape;
        bs.tuned_for = bs.cached[k].sig;
        bs.tuned = true;
        break;
      }
  }
  if (tune && bs.autotune && (!bs.tuned || !sig.close_to(bs.tuned_for))) {
    // Trials on a strided sample of the batch (every stride-th pair, so its length mix is
    // the batch's), ordered as the batch is.  Coordinate descent: the launch shape at the
    // default row threshold; then the 16-lane threshold for A of 129..160 rows; then the
    // int16/int32 split of pairs whose bound exceeds the int16 keys -- each only when the
    // sample has pairs it affects.  Trial results land in the result arrays of the sampled
    // pairs and are overwritten by the batch's own pass.
    const auto t_start = std::chrono::steady_clock::now();
    const int64_t stride = (n + kTuneSample - 1) / kTuneSample;
    const int64_t m = (n + stride - 1) / stride;
    if (!bs.s_order && (e = grow(&bs.s_order, (size_t)kTuneSample + 1024))) return fail(e, "cudaMalloc tuner sample");
    int first[kBuckets + 1] = {0};
    auto in_bucket = [&](int b) { return first[b + 1] - first[b]; };
    auto sample_order = [&](const BatchShape &sh) -> int {
      if (order_items(sh, m, stride, bs.s_order)) return 1;
      if ((e = cudaMemcpyAsync(first, bs.ctl + 8, sizeof(first), cudaMemcpyDeviceToHost, st)) ||
          (e = cudaStreamSynchronize(st)))
        return fail(e, "tuner bucket counts");
      return 0;
    };
    TuneRecord tr;
    tr.tunings = bs.tune.tunings + 1;
    tr.sample_pairs = m;
    auto trial = [&](const BatchShape &sh, float *ms) -> int {
      if (run(sh, bs.s_order, m, ms)) return 1;
      if (tr.trials < 16) tr.trial_ms[tr.trials] = *ms;
      tr.trials++;
      return 0;
    };
    BatchShape best;  // defaults: 128-thread blocks, occupancy limit, rows <= 160 in 8-lane groups
    if (sample_order(best)) return 1;
    float warm = 0.f, best_ms = 1e30f;
    if (run(best, bs.s_order, m, &warm)) return 1;  // untimed warm-up
    const BatchShape shapes[] = {{8, 0}, {16, 0}, {32, 0}, {16, 2}, {32, 1}};
    for (const BatchShape &c0 : shapes) {
      BatchShape c = best;
      c.groups_per_block = c0.groups_per_block;
      c.blocks_per_sm = c0.blocks_per_sm;
      float ms = 0.f;
      if (trial(c, &ms)) return 1;
      if (ms < best_ms) {
        best_ms = ms;
        best = c;
      }
    }
    if (in_bucket(3) > 0) {  // A of 129..160 rows present: try them in 16-lane groups
      BatchShape c = best;
      c.lane_rows = 128;
      float ms = 0.f;
      if (sample_order(c) || trial(c, &ms)) return 1;
      if (ms < best_ms) {
        best_ms = ms;
        best = c;
      }
      if (sample_order(best)) return 1;  // bucket counts of the kept threshold
    }
    if (in_bucket(kBucketWide) > 0 && sc.match <= 63) {  // bound above the int16 keys: try int16 first
      BatchShape c = best;
      c.wide_try16 = true;
      float ms = 0.f;
      if (sample_order(c) || trial(c, &ms)) return 1;
      if (ms < best_ms) best = c;
    }
    bs.shape = best;
    bs.tuned_for = sig;
    bs.tuned = true;
    bs.cached[bs.next_cached] = BatchState::Tuned{sig, best};
    bs.next_cached = (bs.next_cached + 1) % BatchState::kCached;
    if (bs.n_cached < BatchState::kCached) bs.n_cached++;
    tr.last_call_tuned = true;
    tr.wall_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t_start).count();
    bs.tune = tr;
    if ((e = cudaMemsetAsync(wl.ovf_count, 0, sizeof(int), st))) return fail(e, "memset");
    if ((e = cudaMemsetAsync(wl.failed, 0, sizeof(int), st))) return fail(e, "memset");
  }

  // the batch: ordered with the kept configuration, then the persistent launches.
  const BatchShape shape = tune ? bs.shape : plain;
  if (order_items(shape, n, 1, bs.order)) return 1;
  // The long pairs' kernel runs beside the others: 3,000 pairs of 900-1,280 rows, a third of them
  // below 1,024, take 1.58 ms, one kernel after the other 2.46.  It is launched after them: in front
  // it kept their blocks off its SMs while it had nothing to do (3,500 pairs of 1,030-1,100 rows, all of
  // them the lane groups', 1.67 -> 2.58 ms).
  const bool apart = longs && fk && fk->fork;
  if (apart && (e = fork_to(*fk, st, 2))) return fail(e, "fork");
  if (run(shape, bs.order, n, nullptr)) return 1;
  if (longs) {
    if ((e = launch_long_forward(plan_long(n, max_b, sms), ps, rs, sc, bs.order, queue + kOrderLongFirst, wl,
                                 apart ? fk->side[1] : st)))
      return fail(e, "long pair launch");
    if (launches) *launches += 1;
  }
  if (apart && (e = join_from(*fk, st, 2))) return fail(e, "join");
  return 0;
}

}  // namespace mhsw
