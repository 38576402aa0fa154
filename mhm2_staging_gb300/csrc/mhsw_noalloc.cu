// mhsw_noalloc.cu -- the allocation-free forward entry point, mhsw_forward_noalloc().
//
// Some callers cannot let a library allocate device memory while they run:
//   * a process whose device memory has been handed, up front, to its own pool or
//     caching allocator (MHM2 sizes its GPU buffers per rank from the free memory it
//     measures at start-up), where a cudaMalloc of ours may fail or squeeze the pool;
//   * a pipelined loop that cannot take the device-wide synchronisation that cudaMalloc
//     and cudaFree may imply, because other streams of the same process must keep
//     running meanwhile.
// This entry point serves them.  It computes what the forward pass of the driver
// computes -- score, A end and B end per pair, bit-exact with SSW -- with all its scratch
// memory in one file-scope device array of fixed size:
//   short batches   one launch, scratch in shared memory only (mhsw_short.cu);
//   other batches   the pair order (mhsw_order.cuh, in the array), then the keyed int16 engine
//                   in persistent kernels whose lane groups claim pairs in that order
//                   (k_fwd_noalloc16) and translate each pair's codes into their share of the
//                   array; pairs whose score bound exceeds the int16 keys, and every pair of a
//                   scoring the keyed engine cannot hold, go to the int32 engine
//                   (k_fwd_noalloc, a variant of k_fwd<V32, 4, 16>).
//
// Nothing here calls cudaMalloc, cudaFree or any library routine that allocates.
// The first call on a device does a one-time set-up with that device current: it looks
// up the scratch array's device address (cudaGetSymbolAddress, which also loads this
// module onto the device) and loads and configures the kernels of every route.  Make that
// first call before any stream capture begins.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdarg>
#include <cstdio>
#include <mutex>

#include "../../include/mhsw.h"
#include "mhsw_engine.cuh"
#include "mhsw_engine16.cuh"
#include "mhsw_launch.h"
#include "mhsw_order.cuh"

namespace mhsw {
namespace {

constexpr int kNaG = 16;  // lanes per pair
constexpr int kNaK = 4;   // row pairs per lane: strips of 2 * 4 * 16 = 128 rows
constexpr int kNaGroupsPerBlock = 8;
constexpr int kNaMaxDevices = 64;

// The scratch array: 32 MiB per device, shared by every call on that device.
constexpr size_t kNoAllocScratchBytes = size_t(32) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

__host__ __device__ constexpr size_t round_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Layout of one lane group's share of the scratch array, for a batch whose pairs
// have at most max_a A bytes and max_b B bytes:
//   [strip boundary: bcap payloads][A codes][B codes][staged B codes: bcap bytes]
struct NaLayout {
  int pad, bcap;
  size_t bnd_bytes, a_cap, b_cap, stride;
};

__host__ __device__ inline NaLayout na_layout(int max_a, int max_b) {
  NaLayout l;
  l.pad = 2 * kNaG;
  l.bcap = (int)round_up((size_t)l.pad + (size_t)max_b + 2 * kNaG, 16);
  l.bnd_bytes = round_up((size_t)l.bcap * sizeof(V32::Pay), 256);
  l.a_cap = round_up((size_t)max_a, 16);
  l.b_cap = round_up((size_t)max_b, 16);
  l.stride = round_up(l.bnd_bytes + l.a_cap + l.b_cap + (size_t)l.bcap, 256);
  return l;
}

__device__ __forceinline__ unsigned na_group_mask() {
  const int lane32 = threadIdx.x & 31;
  return ((1u << kNaG) - 1u) << ((lane32 / kNaG) * kNaG);
}

// One kNaG-lane group per pair, grid-stride over [0, n), or over the items of the pair order
// from its wide bucket on (order != null).  Group gid owns bytes
// [gid * stride, (gid + 1) * stride) of the scratch array; the host sizes the grid so
// that every group's share lies inside it.  Each pair's scratch is written (codes
// translated, B codes staged, boundary written by strip s before strip s + 1 reads it)
// before it is read, so nothing needs to start at zero.
__global__ void __launch_bounds__(kNaG * kNaGroupsPerBlock)
    k_fwd_noalloc(const char *__restrict__ a_seq, const int64_t *__restrict__ a_off,
                  const int32_t *__restrict__ a_len, const char *__restrict__ b_seq,
                  const int64_t *__restrict__ b_off, const int32_t *__restrict__ b_len, int64_t n, Scoring sc,
                  int max_a, int max_b, unsigned char *scratch, NaLayout lay, const uint32_t *order,
                  const int *wide_first, int32_t *__restrict__ out3) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr size_t kProf = group_prof_bytes<V32, kNaK, kNaG>();
  const int gpb = blockDim.x / kNaG;
  const int grp = threadIdx.x / kNaG;
  const int lane = threadIdx.x % kNaG;
  const unsigned gmask = na_group_mask();
  const int64_t gid = (int64_t)blockIdx.x * gpb + grp;
  const int64_t gstride = (int64_t)gridDim.x * gpb;

  unsigned char *mine = scratch + (size_t)gid * lay.stride;
  V32::Pay *bnd = reinterpret_cast<V32::Pay *>(mine);
  uint8_t *acodes = mine + lay.bnd_bytes;
  uint8_t *bcodes = acodes + lay.a_cap;
  GroupSmem gs;
  gs.prof = reinterpret_cast<uint32_t *>(smem + (size_t)grp * kProf);
  gs.prof_lanes = kNaG;
  gs.bcodes = bcodes + lay.b_cap;
  gs.pad = lay.pad;
  gs.bcap = lay.bcap;

  for (int64_t it = (order ? *wide_first : 0) + gid; it < n; it += gstride) {
    const int64_t i = order ? (int64_t)order[it] : it;
    const int M = a_len[i], N = b_len[i];
    if (M < 0 || N < 0 || M > max_a || N > max_b) {  // outside the stated maxima
      if (lane == 0) {
        out3[3 * i + 0] = -1;
        out3[3 * i + 1] = -1;
        out3[3 * i + 2] = -1;
      }
      continue;
    }
    if (M == 0 || N == 0) {
      if (lane == 0) {
        out3[3 * i + 0] = 0;
        out3[3 * i + 1] = -1;
        out3[3 * i + 2] = 0;
      }
      continue;
    }
    const char *as = a_seq + a_off[i];
    const char *bs = b_seq + b_off[i];
    for (int x = lane; x < M; x += kNaG) acodes[x] = c_code[(uint8_t)as[x]];
    for (int x = lane; x < N; x += kNaG) bcodes[x] = c_code[(uint8_t)bs[x]];
    __syncwarp(gmask);
    SeqView A{acodes, 1, M};
    SeqView B{bcodes, 1, N};
    SweepOut so;
    sweep_pair<V32, kNaK, kNaG>(A, B, sc, gs, lane, gmask, bnd, INT_MAX, so);
    if (lane == 0) {
      const int S = key_value(so.key);
      out3[3 * i + 0] = S;
      out3[3 * i + 1] = S > 0 ? key_row(so.key) : -1;
      out3[3 * i + 2] = S > 0 ? key_col(so.key) : 0;
    }
    __syncwarp(gmask);  // the next pair overwrites this pair's codes
  }
}

// Keyed engine over one range of the pair order: G-lane groups claim items of the short-read
// buckets (G = 8) or of the longer ones up to the wide bucket (G = 16) and translate a pair's
// A and B into their share of the scratch array.  50,000 mixed reads (5.1e9 cells): 7.05 -> 1.16 ms
// a call against the int32 engine in input order, whose shares and registers let 372 blocks run.
template <int G, int MODE>
__global__ void __launch_bounds__(128, G == kGKLong && MODE != kModeInt ? 5 : 4)
    k_fwd_noalloc16(PairSet ps, Scoring sc, int max_a, int max_b, int lane_rows, const uint32_t *__restrict__ order,
                    int *queue, const int *first, unsigned char *scratch, size_t share, size_t a_cap, size_t b_cap,
                    int32_t *__restrict__ out3) {
  constexpr bool kShort = G == kGKShort;
  constexpr int kPer = kShort ? 10 : 8;
  extern __shared__ __align__(16) unsigned char smem[];
  const int grp = threadIdx.x / G, lane = threadIdx.x % G;
  const unsigned gmask = ((1u << G) - 1u) << (((threadIdx.x & 31) / G) * G);
  GroupSmem gs;
  constexpr size_t kProf = group_prof16_bytes<kPer, G, kCodeN + 1, MODE != kModeInt>();
  gs.prof = reinterpret_cast<uint32_t *>(smem + (size_t)grp * kProf);
  gs.prof_lanes = G;
  gs.bcodes = nullptr;
  gs.pad = 0;
  gs.bcap = 0;
  unsigned char *mine = scratch + ((size_t)blockIdx.x * (128 / G) + grp) * share;
  uint8_t *ac = mine, *bc = mine + a_cap;
  V16::Pay *bnd = reinterpret_cast<V16::Pay *>(mine + a_cap + b_cap);
  const int lo = kShort ? 0 : queue[2], hi = kShort ? queue[2] : first[kBucketWide];
  auto translate = [&](uint8_t *dst, const char *src, int len) {
    int x = lane;
    for (; x + 3 * G < len; x += 4 * G) {  // four loads in flight
      const uint8_t v0 = (uint8_t)src[x], v1 = (uint8_t)src[x + G];
      const uint8_t v2 = (uint8_t)src[x + 2 * G], v3 = (uint8_t)src[x + 3 * G];
      dst[x] = c_code[v0];
      dst[x + G] = c_code[v1];
      dst[x + 2 * G] = c_code[v2];
      dst[x + 3 * G] = c_code[v3];
    }
    for (; x < len; x += G) dst[x] = c_code[(uint8_t)src[x]];
  };
  for (;;) {
    int claim = 0;
    if (lane == 0) claim = atomicAdd(queue + (kShort ? 0 : 1), 1);
    claim = __shfl_sync(gmask, claim, 0, G);
    if (lo + claim >= hi) break;
    const int64_t p = order[lo + claim];
    const int M = ps.a_len[p], N = ps.b_len[p];
    int r[3] = {0, -1, 0};
    if (M < 0 || N < 0 || M > max_a || N > max_b) {  // outside the stated maxima
      r[0] = r[2] = -1;
    } else if (M > 0 && N > 0) {
      translate(ac, ps.a_seq + ps.a_off[p], M);
      translate(bc, ps.b_seq + ps.b_off[p], N);
      __syncwarp(gmask);
      SeqView A{ac, 1, M}, B{bc, 1, N};
      SweepOut so;
      const int bucket = bucket_of(M, N, sc, lane_rows, false);
      if constexpr (kShort) {
        switch (bucket) {
          case 0: sweep16<4, G, false, MODE>(A, B, sc, gs, lane, gmask, nullptr, INT_MAX, so); break;
          case 1: sweep16<6, G, false, MODE>(A, B, sc, gs, lane, gmask, nullptr, INT_MAX, so); break;
          case 2: sweep16<8, G, false, MODE>(A, B, sc, gs, lane, gmask, nullptr, INT_MAX, so); break;
          default: sweep16<10, G, false, MODE>(A, B, sc, gs, lane, gmask, nullptr, INT_MAX, so); break;
        }
      } else {
        if (bucket == 4) sweep16<6, G, false, MODE>(A, B, sc, gs, lane, gmask, bnd, INT_MAX, so);
        else sweep16<8, G, false, MODE>(A, B, sc, gs, lane, gmask, bnd, INT_MAX, so);
      }
      r[0] = key_value(so.key);
      if (r[0] > 0) {
        r[1] = key_row(so.key);
        r[2] = key_col(so.key);
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < 3; k++) out3[3 * p + k] = r[k];
    }
    __syncwarp(gmask);  // the next pair overwrites this pair's codes
  }
}

using Na16Kern = decltype(&k_fwd_noalloc16<kGKShort, kModeInt>);
// The two kernels by mode, and the shared memory of a block.
Na16Kern na16_short(int mode) {
  return mode == kModeStep ? k_fwd_noalloc16<kGKShort, 2> : mode == kModeHalf ? k_fwd_noalloc16<kGKShort, 1>
                                                                              : k_fwd_noalloc16<kGKShort, 0>;
}
Na16Kern na16_long(int mode) {
  return mode == kModeStep ? k_fwd_noalloc16<kGKLong, 2> : mode == kModeHalf ? k_fwd_noalloc16<kGKLong, 1>
                                                                             : k_fwd_noalloc16<kGKLong, 0>;
}
size_t na16_smem_short(int mode) {
  return 16 * (mode ? group_prof16_bytes<10, kGKShort, kCodeN + 1, true>() : group_prof16_bytes<10, kGKShort>());
}
size_t na16_smem_long(int mode) {
  return 8 * (mode ? group_prof16_bytes<8, kGKLong, kCodeN + 1, true>() : group_prof16_bytes<8, kGKLong>());
}
constexpr int64_t kNaChunk = 2 << 20;  // pairs ordered at once (their order takes 8 MiB of the array)

struct NaDevice {
  int occ_short[3] = {1, 1, 1}, occ_long[3] = {1, 1, 1};  // by mode
  bool ready = false;
  unsigned char *scratch = nullptr;
  int sms = 0;
  int blocks_per_sm = 0;
};

std::mutex g_na_mu;
NaDevice g_na_dev[kNaMaxDevices];

int na_fail(char *errbuf, size_t errlen, int rc, const char *fmt, ...) {
  if (errbuf && errlen) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(errbuf, errlen, fmt, ap);
    va_end(ap);
  }
  return rc;
}

constexpr size_t na_block_smem() { return (size_t)kNaGroupsPerBlock * group_prof_bytes<V32, kNaK, kNaG>(); }

// One-time set-up for the current device: scratch address, kernel attribute, occupancy.
int na_setup(int dev, NaDevice **out, char *errbuf, size_t errlen) {
  std::lock_guard<std::mutex> lk(g_na_mu);
  NaDevice &d = g_na_dev[dev];
  if (!d.ready) {
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess)
      return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
    const size_t smem = na_block_smem();
    if (smem > 48 * 1024) {
      e = cudaFuncSetAttribute(k_fwd_noalloc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess)
        return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    }
    int sms = 0, occ = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess)
      return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "cudaDeviceGetAttribute: %s", cudaGetErrorString(e));
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_fwd_noalloc, kNaG * kNaGroupsPerBlock, smem);
    if (e != cudaSuccess)
      return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
    // limits and occupancy of the keyed kernels and the order's, so later calls only launch
    for (int m = 0; m < 3; m++)
      if ((e = raise_smem_limit(reinterpret_cast<const void *>(na16_long(m)), na16_smem_long(m))) ||
          (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.occ_long[m], na16_long(m), 128, na16_smem_long(m))) ||
          (e = raise_smem_limit(reinterpret_cast<const void *>(na16_short(m)), na16_smem_short(m))) ||
          (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&d.occ_short[m], na16_short(m), 128, na16_smem_short(m))))
        return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "keyed kernel set-up: %s", cudaGetErrorString(e));
    if ((e = prepare_short_forward()))
      return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "short batch set-up: %s", cudaGetErrorString(e));
    if ((e = order_smem_limits()))
      return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "keyed kernel set-up: %s", cudaGetErrorString(e));
    d.scratch = static_cast<unsigned char *>(p);
    d.sms = sms;
    d.blocks_per_sm = occ > 0 ? occ : 1;
    d.ready = true;
  }
  *out = &d;
  return MHSW_OK;
}

}  // namespace
}  // namespace mhsw

extern "C" int mhsw_forward_noalloc(const mhsw_pairs *pairs, short match_score, short mismatch_score,
                                    short gap_opening_score, short gap_extending_score, short ambiguity_score,
                                    int32_t *out3, void *stream, char *errbuf, size_t errlen) {
  using namespace mhsw;
  if (errbuf && errlen) errbuf[0] = '\0';
  if (!pairs) return na_fail(errbuf, errlen, MHSW_ERR_ARG, "pairs is NULL");
  const int64_t n = pairs->n;
  if (n < 0) return na_fail(errbuf, errlen, MHSW_ERR_ARG, "negative pair count");
  const Scoring sc{match_score, (short)-mismatch_score, (short)-gap_opening_score, (short)-gap_extending_score,
                   (short)-ambiguity_score};
  if (sc.match < 0 || sc.mismatch < 0 || sc.ambiguity < 0 || sc.gap_open < 1 || sc.gap_extend < 1)
    return na_fail(errbuf, errlen, MHSW_ERR_ARG,
                   "scores must be match >= 0 and mismatch/ambiguity <= 0, gap open/extend <= -1 (negated penalties)");
  if (sc.match > 127 || sc.mismatch > 127 || sc.ambiguity > 127 || sc.gap_open > 127 || sc.gap_extend > 127)
    return na_fail(errbuf, errlen, MHSW_ERR_ARG, "score magnitudes above 127 are not supported");
  if (n == 0) return MHSW_OK;
  if (!pairs->a_seq || !pairs->a_off || !pairs->a_len || !pairs->b_seq || !pairs->b_off || !pairs->b_len || !out3)
    return na_fail(errbuf, errlen, MHSW_ERR_ARG, "NULL device pointer in pairs or out3");
  const int max_a = pairs->max_a_len, max_b = pairs->max_b_len;
  if (max_a <= 0 || max_b <= 0)
    return na_fail(errbuf, errlen, MHSW_ERR_ARG, "pairs->max_a_len and pairs->max_b_len are required (> 0)");
  if (max_b > kMaxB || max_a >= (1 << 20))
    return na_fail(errbuf, errlen, MHSW_ERR_LIMIT, "max_a_len %d / max_b_len %d beyond the limits (%d / %d)", max_a,
                   max_b, (1 << 20) - 1, kMaxB);
  const NaLayout lay = na_layout(max_a, max_b);
  const int64_t fit = (int64_t)(kNoAllocScratchBytes / lay.stride);  // lane groups whose scratch fits
  if (fit < 1)
    return na_fail(errbuf, errlen, MHSW_ERR_LIMIT,
                   "one lane group needs %zu scratch bytes for max_a_len %d, max_b_len %d; the fixed scratch is %zu",
                   lay.stride, max_a, max_b, kNoAllocScratchBytes);

  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return na_fail(errbuf, errlen, MHSW_ERR_NO_GPU, "cudaGetDevice: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kNaMaxDevices) return na_fail(errbuf, errlen, MHSW_ERR_LIMIT, "device %d beyond %d", dev,
                                                      kNaMaxDevices);
  NaDevice *d = nullptr;
  int rc = na_setup(dev, &d, errbuf, errlen);
  if (rc) return rc;

  cudaStream_t st = static_cast<cudaStream_t>(stream);
  PairSet ps{};
  ps.a_seq = pairs->a_seq;
  ps.a_off = pairs->a_off;
  ps.a_len = pairs->a_len;
  ps.b_seq = pairs->b_seq;
  ps.b_off = pairs->b_off;
  ps.b_len = pairs->b_len;
  ps.n = n;
  auto launch_fail = [&](cudaError_t err) {
    return na_fail(errbuf, errlen, MHSW_ERR_CUDA, "launch: %s", cudaGetErrorString(err));
  };
  const int ceiling = kCeiling16;
  if (short_batch(sc, ceiling, n, max_a, max_b, false)) {
    if ((e = launch_short_forward(ps, sc, max_a, max_b, out3, st))) return launch_fail(e);
    return MHSW_OK;
  }
  // int32 engine over n pairs in input order (order null) or the order's wide bucket, with the
  // scratch array from `at` on
  auto run32 = [&](const PairSet &q, int64_t m, size_t at, const uint32_t *order, const int *wide_first, int32_t *out) {
    const int64_t room = (int64_t)((kNoAllocScratchBytes - at) / lay.stride);  // lane groups whose scratch fits
    // Block size: kNaGroupsPerBlock groups, or fewer when the scratch holds fewer groups.
    const int gpb = (int)std::min<int64_t>(kNaGroupsPerBlock, room);
    int64_t blocks = std::min<int64_t>(room / gpb, (int64_t)d->sms * d->blocks_per_sm);
    blocks = std::max<int64_t>(1, std::min<int64_t>(blocks, (m + gpb - 1) / gpb));
    // blocks * gpb <= room: the last group's share ends inside the scratch array.
    const size_t smem = (size_t)gpb * group_prof_bytes<V32, kNaK, kNaG>();
    k_fwd_noalloc<<<(unsigned)blocks, gpb * kNaG, smem, st>>>(q.a_seq, q.a_off, q.a_len, q.b_seq, q.b_off, q.b_len, m, sc,
                                                              max_a, max_b, d->scratch + at, lay, order, wide_first, out);
    return cudaGetLastError();
  };
  // Keyed engine: the array holds the order's control block and the order of a chunk, then the
  // shares (codes, and the strip boundary of A above 256 rows).
  const int64_t chunk = std::min<int64_t>(n, kNaChunk);
  const size_t head = round_up(kOrderCtl * sizeof(int) + (size_t)chunk * sizeof(uint32_t), 256);
  const size_t a_cap = round_up((size_t)max_a, 16), b_cap = round_up((size_t)max_b, 16);
  const size_t share = a_cap + b_cap + (max_a > 256 ? round_up((size_t)max_b * sizeof(V16::Pay), 16) : 0);
  const int64_t room = (int64_t)((kNoAllocScratchBytes - head) / share);
  const bool wide = may_need_int32(sc, ceiling, max_a, max_b);
  if (!keyed_scoring(sc) || room < 16 || (wide && kNoAllocScratchBytes - head < lay.stride)) {
    if ((e = run32(ps, n, 0, nullptr, nullptr, out3))) return launch_fail(e);
    return MHSW_OK;
  }
  int *ctl = reinterpret_cast<int *>(d->scratch);
  uint32_t *order = reinterpret_cast<uint32_t *>(ctl + kOrderCtl);
  unsigned char *shares = d->scratch + head;
  const int mode_s = mode_for((long long)std::min({max_a, max_b, 160}) * sc.match, 10);
  const int mode_l = mode_for((long long)std::min(max_a, max_b) * sc.match, 8);
  for (int64_t at = 0; at < n; at += chunk) {
    PairSet q = ps;
    q.n = std::min(chunk, n - at);
    q.a_off += at;
    q.a_len += at;
    q.b_off += at;
    q.b_len += at;
    // as in the plain form: 16-lane groups for all while a batch does not fill them
    const int lane_rows = q.n <= (int64_t)d->sms * 64 ? 0 : 160;
    if ((e = order_pairs(q, sc, lane_rows, false, q.n, 1, ctl, order, d->sms, st, nullptr, max_a,
                         max_b)))
      return launch_fail(e);
    auto grid_of = [&](int occ, int gpb) {
      const int64_t b = std::min<int64_t>((int64_t)d->sms * occ, (q.n + gpb - 1) / gpb);
      return (unsigned)std::min<int64_t>(b, room / gpb);
    };
    if (max_a > lane_rows)
      na16_long(mode_l)<<<grid_of(d->occ_long[mode_l], 8), 128, na16_smem_long(mode_l), st>>>(
          q, sc, max_a, max_b, lane_rows, order, ctl, ctl + 8, shares, share, a_cap, b_cap, out3 + 3 * at);
    if (lane_rows > 0)
      na16_short(mode_s)<<<grid_of(d->occ_short[mode_s], 16), 128, na16_smem_short(mode_s), st>>>(
          q, sc, max_a, max_b, lane_rows, order, ctl, ctl + 8, shares, share, a_cap, b_cap, out3 + 3 * at);
    if ((e = cudaGetLastError())) return launch_fail(e);
    if (wide && (e = run32(q, q.n, head, order, ctl + 8 + kBucketWide, out3 + 3 * at))) return launch_fail(e);
  }
  return MHSW_OK;
}
