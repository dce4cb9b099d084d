// scan.cu -- the per-query pruned scan (replaces KNNQuery_base,
// src/knnjoin.cu:762-858, and the small-M KNNQuery + final merge,
// src/knnjoin.cu:859-979).
//
// One warp per query, persistent blocks pulling query slots from an atomic
// counter in query-cluster order (the reference's reorder_members,
// knnjoin.cu:114-124, 768), so neighbouring warps walk the same candidate
// list.  For the surviving reference clusters Rs of the query's cluster,
// 32 at a time:
//   - each lane computes D = d(q, Rs) and drops its cluster if
//     D - radius(Rs) > theta or D + theta < smallest member distance: no
//     member can be within theta (the reference's first-member `break`,
//     knnjoin.cu:797); the survivors are visited nearest first (a warp sort
//     on D), so the running k-th distance theta falls early.
//   - Rows of more than 8 floats: members are stored contiguously, ascending
//     by d(s, Rs), in column blocks of 32 rows (the same chunk of 32 members
//     is 512 contiguous bytes; a row per lane cost 32 cache lines per load and
//     bound the scan: N = 10^6, d = 32, k = 32: 5.5 -> 3.1 ms with the list's
//     lower bounds below; N = 400,000, d = 128, k = 100: 2.5 -> 1.4).
//     Members within
//     theta of q satisfy |D - d(s,Rs)| <= theta (knnjoin.cu:796-801), a
//     contiguous band.  A warp-wide 32-ary search finds (to within 31
//     members) where the band starts; the warp walks it 32 members per step
//     with coalesced row loads and stops at the first step past its upper
//     end (re-evaluated with the current theta).
//   - Exact FP32 distances go through the warp top-k: k <= 24 a sorted
//     register list (one key per lane) merged by shuffle networks; larger k
//     an unsorted candidate set in shared memory, compacted to the keys up to
//     the FP32 band of (an upper bound of) the k-th distance when it fills,
//     sorted once at the end of the query.  This replaces the per-thread
//     insertion into an 8 KB local-memory array (knnjoin.cu:774, 813-845).
//   - The k-th boundary is then settled in FP64 (see TopKBase).
// Bounds are widened by a rounding slack (bound_tol) so that FP32 rounding
// never prunes a point that the FP32 distances would rank in the top k.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "warp_select.cuh"

namespace knnsweet {

// Shared part of the top-k variants: the append buffer, the admission
// threshold and what the FP64 re-check of the k-th boundary needs.  kShared: the
// other warps of a block lower the threshold too.
//
// The neighbour set must be the one an FP64 join gives.  Keys are FP32
// (d^2, index) words, which rank two points differently from FP64 only when
// both lie inside the FP32 rounding band of the k-th squared distance
// (band_lo / band_hi).  So the admission threshold, once k keys are in, is
// band_hi of the current k-th value (every point that may still belong to
// the final band is admitted and never pruned), compactions keep every key up
// to that value, and `lostmin` records the smallest FP32 d^2 of any key that
// had to be dropped for lack of room while it could still lie in the final
// band.  At the end of the query the band is re-decided in FP64
// (band_resolve_fp64); a query that lost a band key goes to the band kernel
// instead.
//
// Register budget: the dimension comes from the kernel parameters where it is
// needed and `lostmin` lives in a shared-memory word of the warp, so neither
// occupies a register through the scan loop.
//
// The warp's shared-memory slot holds, at fixed key offsets behind the
// buffer, `lostmin` (the smallest FP32 d^2 dropped for lack of room, +inf:
// none), the current query's statistics words (kStat*, updated by lane 0)
// and the query's slot, row and cluster (kSide*, needed only when the query
// starts and ends): kept out of registers, which the scan loop needs.
enum {
  kStatPushed = 0, kStatMerges, kStatVisited, kStatPruned, kStatChecked,
  kSideSlot, kSideQuery, kSideCluster, kSideDq, kSideKept, kStatWords
};
constexpr int kStatKeys = (kStatWords + 1) / 2;  // 64-bit words they take

template <int kLostOff, int kStatOff, bool kShared>
struct TopKBase {
  uint64_t *buf;  // append buffer (shared memory)
  int nbuf, nlist, k;
  // a candidate (d^2, index) enters iff d^2 <= thr_d2: the threshold key
  // (thr_d2, 0xffffffff) lies above every key with that distance word
  float thr_d2;
  float theta;    // distance matching thr (bound for the pruning tests)

  __device__ __forceinline__ float *lostmin() const {
    return reinterpret_cast<float *>(buf + kLostOff);
  }
  __device__ __forceinline__ unsigned *stat() const {
    return reinterpret_cast<unsigned *>(buf + kStatOff);
  }
  static constexpr int kLostAt = kLostOff, kStatAt = kStatOff;
  __device__ __forceinline__ void count(int which, unsigned v, int lane) const {
    if (lane == 0) stat()[which] += v;
  }

  // statistics: candidates pushed since the last compaction left `kept`
  __device__ __forceinline__ void settle(int now, int kept, int lane) const {
    if (lane == 0) {
      unsigned *s = stat();
      s[kStatPushed] += (unsigned)(now - (int)s[kSideKept]);
      s[kSideKept] = (unsigned)kept;
    }
  }

  __device__ __forceinline__ void reset_threshold(float th0, int lane) {
    if (lane == 0) stat()[kSideKept] = 0;
    nbuf = 0;
    nlist = 0;
    theta = th0;
    if (lane == 0) *lostmin() = __int_as_float(0x7f800000);
    // admits every d^2 <= th0^2, whatever the index
    thr_d2 = th0 * th0;
  }
  // threshold once the k-th squared distance is T: the FP32 band above it
  __device__ __forceinline__ void set_band_threshold(float T, int d) {
    float W = band_hi(T, d);
    // a threshold from the block's other warps may lie lower (elsewhere the test
    // cost the k = 200 self-join spills: 3.71 -> 3.75 ms)
    if constexpr (kShared) W = fminf(thr_d2, W);
    thr_d2 = W;
    theta = sqrtf(W);
  }
  // a dropped key's distance word (NaN from an empty key is ignored)
  __device__ __forceinline__ void note_lost(uint32_t d2bits, int lane) {
    const float v = __uint_as_float(__reduce_min_sync(kFull, d2bits));
    __syncwarp();
    if (lane == 0) *lostmin() = fminf(*lostmin(), v);
    __syncwarp();
  }
};

// Small k: the sorted list of the best keys lives in registers
// (one key per lane), with the FP32 band of the k-th kept behind it as far as
// the 32 slots allow.
template <int E, bool kShared>
struct RegTopK : TopKBase<64 * E + 2, 64 * E + 3, kShared> {
  using B = TopKBase<64 * E + 2, 64 * E + 3, kShared>;
  using B::buf, B::nbuf, B::nlist, B::k, B::count, B::note_lost, B::set_band_threshold,
      B::reset_threshold, B::settle;
  static constexpr int L = 32 * E;
  static constexpr int kCap = L;  // candidate buffer capacity
  // append buffer (L keys), L doubles for the FP64 band, 2 pivot words,
  // lostmin, statistics
  static constexpr int kSmemKeys = 2 * L + 3 + kStatKeys;
  static constexpr int kBandScratch = L, kPivot = 2 * L;
  uint64_t v[E];

  __device__ __forceinline__ int cap() const { return kCap; }

  __device__ __forceinline__ void init(uint64_t *wsm) { buf = wsm; }

  __device__ __forceinline__ void reset(float th0, int lane) {
#pragma unroll
    for (int j = 0; j < E; j++) v[j] = kKeyMax;
    reset_threshold(th0, lane);
  }

  __device__ __forceinline__ void make_room(int lane, int d) { flush(lane, d); }
  // end of the query: pending candidates merged into the list
  __device__ __forceinline__ void finish(int lane, int d) { flush(lane, d); }

  __device__ __forceinline__ void flush(int lane, int d) {
    if (nbuf == 0) return;
    __syncwarp();
    uint64_t b[E];
#pragma unroll
    for (int j = 0; j < E; j++) {
      const int p = j * 32 + lane;  // any order: the buffer gets sorted
      b[j] = p < nbuf ? buf[p] : kKeyMax;
    }
    __syncwarp();
    reg_bitonic_sort<E>(b, lane);
    // v ascending, b ascending: min(v[i], b[L-1-i]) holds the L smallest of
    // both as a bitonic sequence; the larger of each pair is dropped
    uint32_t lost = 0xffffffffu;
#pragma unroll
    for (int j = 0; j < E; j++) {
      const uint64_t o = shfl64(b[E - 1 - j], 31 - lane);
      lost = min(lost, (uint32_t)(umax64(v[j], o) >> 32));
      v[j] = umin64(v[j], o);
    }
    note_lost(lost, lane);
    reg_bitonic_merge<E>(v, lane);
    nlist = min(k, nlist + nbuf);
    settle(nbuf, 0, lane);
    count(kStatMerges, 1, lane);
    nbuf = 0;
    if (nlist == k) {
      const int kl = (k - 1) / E, kj = (k - 1) % E;
      uint64_t mine = kKeyMax;
#pragma unroll
      for (int j = 0; j < E; j++)
        if (j == kj) mine = v[j];
      const float T = key_d2(shfl64(mine, kl));
      // keys behind the k-th stay only inside its band (the ones dropped
      // here are above band_hi of a k-th that can only fall)
      const float hi = band_hi(T, d);
#pragma unroll
      for (int j = 0; j < E; j++)
        if (E * lane + j >= k && key_d2(v[j]) > hi) v[j] = kKeyMax;
      set_band_threshold(T, d);
    }
  }

  // Lane l: a d^2 word that at least l + 1 candidates do not exceed (all ones:
  // fewer).
  __device__ __forceinline__ uint32_t nearest(int lane, int d) {
    static_assert(E == 1, "one key per lane");
    flush(lane, d);
    return (uint32_t)(v[0] >> 32);
  }
  // The candidates into buf[0..n) for another warp; returns n.
  __device__ __forceinline__ int expose(int lane) { return sorted(lane, 0); }
  // The candidates, sorted, into buf[0..n); returns n.
  __device__ __forceinline__ int sorted(int lane, int) {
    __syncwarp();
    int n = 0;
#pragma unroll
    for (int j = 0; j < E; j++) {
      buf[E * lane + j] = v[j];
      n += __popc(__ballot_sync(kFull, v[j] != kKeyMax));
    }
    __syncwarp();
    return n;
  }
};

// Bitonic sort of L keys in shared memory, ascending, by one warp.
template <int L>
__device__ __forceinline__ void smem_bitonic_sort(uint64_t *s, int lane) {
#pragma unroll 1
  for (int size = 2; size <= L; size <<= 1) {
#pragma unroll 1
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
#pragma unroll
      for (int t0 = 0; t0 < (L / 2 + 31) / 32; t0++) {
        const int t = t0 * 32 + lane;
        if (t < L / 2) {
          const int i = 2 * t - (t & (stride - 1));
          const int j = i + stride;
          const bool up = (i & size) == 0;
          const uint64_t a = s[i], b = s[j];
          if ((a > b) == up) {
            s[i] = b;
            s[j] = a;
          }
        }
      }
      __syncwarp();
    }
  }
}

// Top-k as an unsorted candidate set in shared memory (capacity 2L).  When it
// fills, the k-th smallest squared distance T is found by a radix selection
// and the set keeps every key up to band_hi(T); the k results are sorted
// once, at the end of the query.
#ifndef KNN_TOPK_EARLY
#define KNN_TOPK_EARLY 160
#endif

template <int LL, bool kShared>
struct SelectTopK : TopKBase<2 * LL + 128, 2 * LL + 129, kShared> {
  using B = TopKBase<2 * LL + 128, 2 * LL + 129, kShared>;
  using B::buf, B::nbuf, B::nlist, B::k, B::count, B::note_lost, B::set_band_threshold,
      B::reset_threshold, B::settle;
  static constexpr int L = LL;          // final sort length (pow2 >= k)
  static constexpr int kCap = 2 * LL;   // candidate capacity
  // keys, 256-word histogram, lostmin, statistics
  static constexpr int kSmemKeys = 2 * LL + 129 + kStatKeys;
  // after the final sort: LL doubles for the FP64 band behind the sorted
  // keys, the pivot in the histogram's words
  static constexpr int kBandScratch = LL, kPivot = 2 * LL;
  __device__ __forceinline__ uint32_t *hist() const {
    return reinterpret_cast<uint32_t *>(buf + 2 * LL);
  }

  // A compaction once k + kEarly candidates are in (capacity permitting)
  // tightens the threshold sooner.  k = 200 self-join scan: capacity only
  // 5.06 ms; kEarly 64: 5.12, 96: 4.94, 128: 4.89, 160: 4.90, 256: 4.97
  // (with the compaction before the end-of-query selection: 96: 4.86,
  // 128 to 192: 4.76-4.78).
  static constexpr int kEarly = KNN_TOPK_EARLY;
  __device__ __forceinline__ int cap() const { return k + kEarly < kCap ? k + kEarly : kCap; }

  __device__ __forceinline__ void init(uint64_t *wsm) { buf = wsm; }

  __device__ __forceinline__ void reset(float th0, int lane) { reset_threshold(th0, lane); }

  // Reduce the set to its k smallest keys (no-op with k or fewer) when ties
  // leave no room otherwise; the keys it drops go into lostmin.
  __device__ __forceinline__ void flush(int lane, int d) {
    if (nbuf <= k) return;
    __syncwarp();
    const uint64_t kth = warp_select_kth(buf, nbuf, k, hist(), lane);
    __syncwarp();
    int w = 0;
    uint32_t lost = 0xffffffffu;
    for (int b0 = 0; b0 < nbuf; b0 += 32) {
      const int i = b0 + lane;
      const uint64_t v = i < nbuf ? buf[i] : kKeyMax;
      const bool keep = i < nbuf && v <= kth;
      if (i < nbuf && !keep) lost = min(lost, (uint32_t)(v >> 32));
      const unsigned bm = __ballot_sync(kFull, keep);
      __syncwarp();
      if (keep) buf[w + __popc(bm & ((1u << lane) - 1))] = v;
      w += __popc(bm);
    }
    __syncwarp();
    note_lost(lost, lane);
    settle(nbuf, w, lane);
    nbuf = w;  // == k
    nlist = k;
    count(kStatMerges, 1, lane);
    set_band_threshold(key_d2(kth), d);
  }

  // Room for more candidates while the query runs: keep every key whose
  // squared distance is at most band_hi of the k-th smallest one T -- at
  // least k keys, ties and the FP32 band included -- found by a 32-bit
  // selection on the keys' distance words (on data with many equal distances
  // a 64-bit selection spends most of its passes on the index bits of the
  // ties).  Falls back to the exact k-key flush when ties fill the buffer.
  __device__ __forceinline__ void make_room(int lane, int d) {
    if (nbuf <= k) return;
    __syncwarp();
#if KNN_LINEAR_SELECT
    // an upper bound of the k-th: the threshold it gives admits a little more
    const uint32_t T = warp_kth_upper_u32(reinterpret_cast<const uint32_t *>(buf) + 1, 2,
                                          nbuf, k, hist(), lane);
#else
    const uint32_t T = warp_select_kth_u32(reinterpret_cast<const uint32_t *>(buf) + 1, 2,
                                           nbuf, k, hist(), lane);
#endif
    const uint32_t W = __float_as_uint(band_hi(__uint_as_float(T), d));
    int w = 0;
    for (int b0 = 0; b0 < nbuf; b0 += 32) {
      const int i = b0 + lane;
      const uint64_t v = i < nbuf ? buf[i] : kKeyMax;
      const bool keep = i < nbuf && (uint32_t)(v >> 32) <= W;
      const unsigned bm = __ballot_sync(kFull, keep);
      __syncwarp();
      if (keep) buf[w + __popc(bm & ((1u << lane) - 1))] = v;
      w += __popc(bm);
    }
    __syncwarp();
    settle(nbuf, w, lane);
    nbuf = w;
    if (w > kCap - 32) {
      flush(lane, d);
      return;
    }
    count(kStatMerges, 1, lane);
    nlist = k;
    set_band_threshold(__uint_as_float(T), d);
  }

  // Lane l: a d^2 word that at least l + 1 candidates do not exceed (all ones:
  // fewer), the l-th of the 32 lanes' minima.
  __device__ __forceinline__ uint32_t nearest(int lane, int) {
    __syncwarp();
    uint32_t x = 0xffffffffu;
    for (int i = lane; i < nbuf; i += 32) x = min(x, (uint32_t)(buf[i] >> 32));
#pragma unroll
    for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        const uint32_t o = __shfl_xor_sync(kFull, x, stride);
        x = ((lane & stride) == 0) == ((lane & size) == 0) ? min(x, o) : max(x, o);
      }
    }
    return x;
  }
  // The candidates are in buf[0..nbuf) already.
  __device__ __forceinline__ int expose(int) { return nbuf; }
  // End of the query: nothing to do before sorted().
  __device__ __forceinline__ void finish(int lane, int) { settle(nbuf, nbuf, lane); }

  // The candidates, sorted, into buf[0..n); returns n.  Up to L keys are
  // sorted as they are; beyond that a band-inclusive compaction first, and
  // the exact k-key flush only if ties still leave more than L.
  __device__ __forceinline__ int sorted(int lane, int d) {
    if (nbuf > LL) make_room(lane, d);
    if (nbuf > LL) flush(lane, d);
    __syncwarp();
    if constexpr (LL <= 128) {
      // sorted in registers (E keys per lane; shuffles for the cross-lane
      // strides): lane l ends up with positions E*l .. E*l+E-1.  (At L = 256
      // the eight keys per lane spilled under the kernel's register cap and
      // measured slower than the shared-memory sort.)
      constexpr int E = LL / 32;
      uint64_t x[E];
#pragma unroll
      for (int j = 0; j < E; j++) {
        const int p = j * 32 + lane;  // any order: the keys get sorted
        x[j] = p < nbuf ? buf[p] : kKeyMax;
      }
      __syncwarp();
      reg_bitonic_sort<E>(x, lane);
#pragma unroll
      for (int j = 0; j < E; j++) buf[E * lane + j] = x[j];
    } else {
      // binned counting sort (k = 200 self-join scan: 4.45 ms with the
      // bitonic network alone); the network where equal distances crowd a bin
#if KNN_BIN_SORT
      if constexpr (LL <= 256)  // the bin tags of 8 keys per lane stay in registers
        if (warp_bin_sort<LL / 32>(buf, nbuf, buf + LL, hist(), lane)) return nbuf;
#endif
      for (int i = nbuf + lane; i < LL; i += 32) buf[i] = kKeyMax;
      __syncwarp();
      smem_bitonic_sort<LL>(buf, lane);
    }
    __syncwarp();
    return nbuf;
  }
};

// Offer one candidate per lane, warp-collective: the lanes with `pass` set
// (squared distance v at most the threshold's distance word, so that the key
// (v, idx) lies below the threshold key) append their keys.
template <class TK>
__device__ __forceinline__ void topk_offer(TK &tk, bool pass, float v, int32_t idx, int lane,
                                           int d) {
  unsigned b = __ballot_sync(kFull, pass);
  if (b == 0) return;
  int cnt = __popc(b);
  if (tk.nbuf + cnt > tk.cap()) {
    tk.make_room(lane, d);
    pass = pass && v <= tk.thr_d2;
    b = __ballot_sync(kFull, pass);
    cnt = __popc(b);
  }
  if (pass) tk.buf[tk.nbuf + __popc(b & ((1u << lane) - 1))] = make_key(v, idx);
  tk.nbuf += cnt;  // (counted by settle, not here: every step comes this way)
}

// Whether every FP32 squared distance of the join is exact (both sides hold
// small integers), so that FP32 keys rank exactly like FP64 ones.
__device__ __forceinline__ bool fp32_exact(const ScanArgs &a) {
  return a.inexact_r && a.inexact_q && (*a.inexact_r | *a.inexact_q) == 0;
}

// A query's starting k-th distance bound.  theta0 of its cluster is the k-th
// smallest of rq + d(Rq,Rs) + d(s,Rs) over the reference points s, rq the
// cluster's radius; the same k points lie within dq + d(Rq,Rs) + d(s,Rs) of a
// query at distance dq <= rq from the representative, so theta0 - (rq - dq),
// widened by the rounding slack, bounds that query's k-th distance too and
// starts its scan tighter.
#ifndef KNN_QUERY_THETA0
#define KNN_QUERY_THETA0 1
#endif
__device__ __forceinline__ float query_theta0(const ScanArgs &a, float dq, int qc, float tol) {
  float th = a.theta0[qc];
  if (KNN_QUERY_THETA0 && a.qrad) {
    const float rq = a.qrad[qc];
    const float cut = (rq - dq) - tol * (rq + dq + th);
    if (cut > 0.0f) th -= cut;
  }
  return th;
}

// Squared distance of a point to a block's bounding box, in the arithmetic of
// the distances: every coordinate's gap is at most the difference to any row
// of the block, and subtraction, squaring and accumulation round
// monotonically, so no row of the block has a smaller computed distance.  (A
// difference that is not a number counts as no gap.)
template <int DP4>
__device__ __forceinline__ float box_dist2(const float4 (&q)[DP4], const float4 (&lo)[DP4],
                                           const float4 (&hi)[DP4]) {
  float acc = 0.0f;
  auto one = [&](float x, float l, float h) {
    const float g = fmaxf(fmaxf(__fsub_rn(l, x), __fsub_rn(x, h)), 0.0f);
    acc = __fmaf_rn(g, g, acc);
  };
#pragma unroll
  for (int c = 0; c < DP4; c++) {
    one(q[c].x, lo[c].x, hi[c].x);
    one(q[c].y, lo[c].y, hi[c].y);
    one(q[c].z, lo[c].z, hi[c].z);
    one(q[c].w, lo[c].w, hi[c].w);
  }
  return acc;
}

// The same between two boxes: no point of one is nearer to a point of the
// other.
template <int DP4>
__device__ __forceinline__ float boxes_dist2(const float4 (&alo)[DP4], const float4 (&ahi)[DP4],
                                             const float4 (&blo)[DP4], const float4 (&bhi)[DP4]) {
  float acc = 0.0f;
  auto one = [&](float al, float ah, float bl, float bh) {
    const float g = fmaxf(fmaxf(__fsub_rn(bl, ah), __fsub_rn(al, bh)), 0.0f);
    acc = __fmaf_rn(g, g, acc);
  };
#pragma unroll
  for (int c = 0; c < DP4; c++) {
    one(alo[c].x, ahi[c].x, blo[c].x, bhi[c].x);
    one(alo[c].y, ahi[c].y, blo[c].y, bhi[c].y);
    one(alo[c].z, ahi[c].z, blo[c].z, bhi[c].z);
    one(alo[c].w, ahi[c].w, blo[c].w, bhi[c].w);
  }
  return acc;
}

// FP64 re-decision of one query's k-th boundary, by one warp.  s[0..n) holds
// the query's candidate keys sorted ascending, n > k; s[0..nlo) lie below the
// FP32 band of the k-th (band_lo(Dk) .. band_hi(Dk)), s[nlo..nhi) inside it,
// nhi > k, and every point inside the band is among them.  Keys below the
// band are in the FP64 top k, keys above it are not; the band's keys are
// ranked by (FP64 d^2, index) and the best k - nlo of them kept in place, in
// their FP32 order, so that s[0..k) is the FP64 join's neighbour set.  (The
// reference decides this boundary by a strict-less insertion of FP32
// distances, src/knnjoin.cu:815-820.)  qf: the query row; rrows: the
// reference rows in original order (keys carry original indices); dbl:
// scratch for nhi - nlo doubles; piv: 2 words.  Inlined: as an out-of-line
// call (for the few queries that need it) it cost the k = 200 self-join scan
// 8 % (5.15 against 4.82 ms), the call's register saves on every query.
__device__ __forceinline__ void band_resolve_fp64(uint64_t *s, int nlo, int nhi, int k, int d,
                                               int dp4, const float *__restrict__ qf,
                                               const float4 *__restrict__ rrows, double *dbl,
                                               uint64_t *piv, int lane) {
  const int nb = nhi - nlo, need = k - nlo;
  for (int e = lane; e < nb; e += 32) {
    const int32_t id = key_idx(s[nlo + e]);
    dbl[e] = dist2_f64(qf, reinterpret_cast<const float *>(rrows + (int64_t)id * dp4), d);
  }
  __syncwarp();
  // the need-th smallest (FP64 d^2, index) of the band (ranks are distinct)
  for (int e = lane; e < nb; e += 32) {
    const double de = dbl[e];
    const int32_t ie = key_idx(s[nlo + e]);
    int rank = 0;
    for (int f = 0; f < nb; f++) rank += f64_key_less(dbl[f], key_idx(s[nlo + f]), de, ie);
    if (rank == need - 1) {
      piv[0] = (uint64_t)__double_as_longlong(de);
      piv[1] = (uint64_t)(uint32_t)ie;
    }
  }
  __syncwarp();
  const double pd = __longlong_as_double((long long)piv[0]);
  const int32_t pi = (int32_t)piv[1];
  // keep the band's keys up to the pivot, in place, order preserved
  int w = nlo;
  for (int b0 = 0; b0 < nb; b0 += 32) {
    const int e = b0 + lane;
    const uint64_t key = e < nb ? s[nlo + e] : kKeyMax;
    const bool keep = e < nb && !f64_key_less(pd, pi, dbl[e], key_idx(key));
    const unsigned bm = __ballot_sync(kFull, keep);
    __syncwarp();
    if (keep) s[w + __popc(bm & ((1u << lane) - 1))] = key;
    w += __popc(bm);
  }
  __syncwarp();
}

// End of one query of the warp scan: sorts the candidates, settles the k-th
// boundary in FP64 unless the join's FP32 distances are exact (or, when a key of its band was dropped for lack of room,
// hands the query to the band kernel: the last output slot then carries the
// number of keys below the band and the FP32 k-th value), writes the k
// results.  Returns the FP64 distances evaluated.
template <class TK>
__device__ __forceinline__ unsigned emit_query(TK &tk, const ScanArgs &a, int32_t slot, int64_t q,
                                               int qc, int lane) {
  const int n = tk.sorted(lane, a.d);
  const bool exact32 = fp32_exact(a);
  uint64_t *s = tk.buf;
  const int k = a.k;
  bool defer = false;
  int nlo = 0;
  float Dk = 0.0f;
  unsigned checked = 0;
  if (n >= k && !exact32) {  // exact FP32 distances: the (d^2, index) order is FP64's
    Dk = key_d2(s[k - 1]);
    const float lo = band_lo(Dk, a.d), hi = band_hi(Dk, a.d);
    int nhi = 0;
    for (int b0 = 0; b0 < n; b0 += 32) {
      const int e = b0 + lane;
      const float v = e < n ? key_d2(s[e]) : __int_as_float(0x7f800000);
      nlo += __popc(__ballot_sync(kFull, v < lo));
      nhi += __popc(__ballot_sync(kFull, v <= hi));
    }
    if (*tk.lostmin() <= hi) {
      defer = true;
    } else if (nhi > k) {
      band_resolve_fp64(s, nlo, nhi, k, a.d, a.dp4,
                        reinterpret_cast<const float *>(a.qrows + q * a.dp4), a.rrows,
                        reinterpret_cast<double *>(s + TK::kBandScratch), s + TK::kPivot, lane);
      checked = (unsigned)(nhi - nlo);
    }
  }
  int32_t *oi = a.out_idx + q * k;
  float *od = a.out_dist + q * k;
  const int32_t base = a.qc_ref_base ? (int32_t)a.qc_ref_base[qc] : 0;
  for (int t = lane; t < k; t += 32) {
    const uint64_t key = t < n ? s[t] : kKeyMax;
    const bool none = key == kKeyMax;
    if (defer && t == k - 1) {
      oi[t] = nlo;
      od[t] = Dk;
    } else {
      oi[t] = none ? -1 : key_idx(key) - base;
      od[t] = none ? __int_as_float(0x7f800000) : (a.squared ? key_d2(key) : sqrtf(key_d2(key)));
    }
  }
  if (defer && lane == 0) a.unres_slot[atomicAdd(a.unres_count, 1u)] = slot;
  __syncwarp();
  return checked;
}

// ---------------------------------------------------------------------------
// Query rows.  IDXROW: the reference rows carry their original index in the
// last pad float (d < 4*DP4), which the distance then skips.
// ---------------------------------------------------------------------------
template <int DP4, bool IDXROW>
struct QueryRow {
  float4 v[DP4];
  __device__ __forceinline__ void load(const float4 *__restrict__ rows, int64_t q, int,
                                       float4 *) {
#pragma unroll
    for (int c = 0; c < DP4; c++) v[c] = rows[q * DP4 + c];
  }
  __device__ __forceinline__ float dist2(const float4 *__restrict__ r, int) const {
    return dist2_rows<DP4>(v, r);
  }
  // A row whose chunks lie `stride` float4 apart; only the first nch chunks
  // hold coordinates (the padding behind them would add exact zeros).
  __device__ __forceinline__ float dist2_chunks(const float4 *__restrict__ r, int stride,
                                                int nch) const {
    float4 row[DP4];
#pragma unroll
    for (int c = 0; c < DP4; c++)
      if (c < nch) row[c] = r[c * stride];
    float acc = 0.0f;
#pragma unroll
    for (int c = 0; c < DP4; c++)
      if (c < nch) {
        float t;
        t = __fsub_rn(v[c].x, row[c].x); acc = __fmaf_rn(t, t, acc);
        t = __fsub_rn(v[c].y, row[c].y); acc = __fmaf_rn(t, t, acc);
        t = __fsub_rn(v[c].z, row[c].z); acc = __fmaf_rn(t, t, acc);
        t = __fsub_rn(v[c].w, row[c].w); acc = __fmaf_rn(t, t, acc);
      }
    return acc;
  }
  // Member row (already in registers): distance and (IDXROW) the index
  // stored in the row's last pad float.
  __device__ __forceinline__ float dist2_member(const float4 (&row)[DP4],
                                                int32_t *idx) const {
    float acc = 0.0f;
#pragma unroll
    for (int c = 0; c < DP4; c++) {
      const float4 s = row[c];
      float t;
      t = __fsub_rn(v[c].x, s.x); acc = __fmaf_rn(t, t, acc);
      t = __fsub_rn(v[c].y, s.y); acc = __fmaf_rn(t, t, acc);
      t = __fsub_rn(v[c].z, s.z); acc = __fmaf_rn(t, t, acc);
      if (IDXROW && c == DP4 - 1) {
        *idx = __float_as_int(s.w);
      } else {
        t = __fsub_rn(v[c].w, s.w); acc = __fmaf_rn(t, t, acc);
      }
    }
    return acc;
  }
};

// Runtime width: the query row lives in the warp's shared-memory slot.
template <bool IDXROW>
struct QueryRow<0, IDXROW> {
  const float4 *v;
  __device__ __forceinline__ void load(const float4 *__restrict__ rows, int64_t q, int dp4,
                                       float4 *slot) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    for (int c = lane; c < dp4; c += 32) slot[c] = rows[q * dp4 + c];
    __syncwarp();
    v = slot;
  }
  __device__ __forceinline__ float dist2_chunks(const float4 *__restrict__ r, int stride,
                                                int nch) const {
    float acc = 0.0f;
#pragma unroll 4
    for (int c = 0; c < nch; c++) {
      const float4 u = v[c], s = r[(size_t)c * stride];
      float t;
      t = __fsub_rn(u.x, s.x); acc = __fmaf_rn(t, t, acc);
      t = __fsub_rn(u.y, s.y); acc = __fmaf_rn(t, t, acc);
      t = __fsub_rn(u.z, s.z); acc = __fmaf_rn(t, t, acc);
      t = __fsub_rn(u.w, s.w); acc = __fmaf_rn(t, t, acc);
    }
    return acc;
  }
};

// Resident warps per SM the register allocation must allow (compile-time
// tuning knobs): the scan is latency-bound, so occupancy matters; rows of
// more than 8 floats keep the query in registers and get the lower target.
#ifndef KNN_TARGET_WARPS
#define KNN_TARGET_WARPS 32
#endif
#ifndef KNN_TARGET_WARPS_WIDE
#define KNN_TARGET_WARPS_WIDE 16
#endif
// Largest k kept in a register list (one key per lane): up to 24, so that
// 8 of the 32 slots or more hold the FP32 band behind the k-th; larger k use
// the shared-memory candidate set.
#ifndef KNN_REG_TOPK_MAX_K
#define KNN_REG_TOPK_MAX_K 24
#endif

template <int L, bool kShared>
using TopKFor = std::conditional_t<(L <= 32), RegTopK<L / 32, kShared>, SelectTopK<L, kShared>>;

// Rows of more than 8 floats keep 4+ float4 of the query in registers: those
// kernels get the lower occupancy target instead of spilling.
template <int DP4, int WARPS>
constexpr int scan_min_blocks() {
  return ((DP4 == 0 || DP4 >= 4) ? KNN_TARGET_WARPS_WIDE : KNN_TARGET_WARPS) / WARPS;
}

// A query of wide rows may be left to a whole block (a launch behind the
// scan's): a few queries between distant groups of points reach a hundred
// times the members of the others, and the scan took as long as the longest
// (N = 10^6, d = 32, k = 32, six data sets: 2.9 to 5.5 ms, 2.9 to 3.3 with
// this).  The block starts it again, so a query goes only after kFarSteps steps
// of 32 members, when two thirds of the warps have no query left to take, and
// with most of a list that can be dealt out to warps before it.  Any query of
// that many steps, idle warps or not: 100,000 rows, d = 16, four clusters,
// 2,300 queries 8.2 ms; warps that keep them 2.5; 200,003 rows, d = 64, 3,000
// queries: none given up 20.0, with a third of the warps busy 15.4.
constexpr int kFarSteps = 512;
// Entries from which on a list is dealt out to a block's warps; of a shorter one
// they take parts of every cluster.  100,000 rows, d = 32 in 500 distant groups, 16
// clusters, 500 queries, k = 50: dealt out 1,017 us (a warp per query 605), in parts
// 500; one Gaussian, d = 16, 16 clusters: 992 and 1,278 (2,097).
constexpr int kShareLists = 32;

// ONE: the reference set is a single cluster of narrow rows (small joins).
template <int DP4, bool IDXROW, int L, int WARPS, bool ONE, bool SPLIT>
__global__ void __launch_bounds__(WARPS * 32, (scan_min_blocks<DP4, WARPS>()))
    scan_kernel(const ScanArgs a) {
  using TK = TopKFor<L, SPLIT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int dp4 = DP4 > 0 ? DP4 : a.dp4;
  uint64_t *keys_base = reinterpret_cast<uint64_t *>(smem_raw);
  float4 *qslot = reinterpret_cast<float4 *>(keys_base + (size_t)WARPS * TK::kSmemKeys) +
                  (size_t)w * (DP4 > 0 ? 0 : a.dp4);
  TK tk;
  tk.init(keys_base + (size_t)w * TK::kSmemKeys);
  tk.k = a.k;
  const float tol = bound_tol(a.d);
  unsigned evals = 0;
  constexpr bool kWideRows = DP4 == 0 || DP4 >= 4;
  // narrow rows: members in block order, blocks of 32 skipped by their boxes
  constexpr bool kBlocks = DP4 == 1 || DP4 == 2;
  const int nch = (a.d + 3) >> 2;  // chunks of a row that hold coordinates
  // statistics: per-lane 32-bit counts folded once per query into per-block
  // shared counters, added to the global ones at exit
  __shared__ unsigned long long blk_ctr[kScanCounters];
  if (threadIdx.x < kScanCounters) blk_ctr[threadIdx.x] = 0;
  if (lane < kStatWords) tk.stat()[lane] = 0;
  __syncthreads();

  // SPLIT: the block's warps share one query, all tighten one threshold (s_thr,
  // distance bits), and warp 0 merges their candidates.  A list of many
  // clusters is dealt out, each warp takes every WARPS-th cluster; of a list of
  // few (kShareLists) every warp walks all clusters, but takes every
  // WARPS-th block of 32 members of each.  Then one warp's k-th is far above the
  // block's: s_part[w][j] is a d^2 word that j + 1 of warp w's candidates do not
  // exceed, and the k-th smallest of all these words bounds the k-th distance
  // (words only fall, so a word read late is still true)
  __shared__ unsigned s_thr, s_part[SPLIT ? WARPS : 1][32];
  __shared__ long long s_slot;
  // (more may have been counted than there was room for in the far list)
  const int64_t listed_all =
      a.slot_list ? min((int64_t)*a.slot_count, a.m) : a.m;
  // (of a list whose length only the device knows, one of two launches returns)
  if (kWideRows && (SPLIT ? listed_all > a.split_max : listed_all <= a.split_max)) return;
  for (;;) {
    long long slot = 0;
    if constexpr (SPLIT) {
      __syncthreads();
      if (threadIdx.x == 0) {
        s_slot = (long long)atomicAdd(a.work_counter, 1ull);
        s_thr = 0x7f800000u;
      }
      s_part[w][lane] = 0xffffffffu;
      __syncthreads();
      slot = s_slot;
    } else {
      if (lane == 0) slot = (long long)atomicAdd(a.work_counter, 1ull);
      slot = __shfl_sync(kFull, slot, 0);
    }
    if (a.slot_list) {
      if (slot >= listed_all) break;
      slot = a.slot_list[slot];
    } else if (slot >= a.m) {
      break;
    } else {
      slot += a.slot_base;
    }
    // (one cluster, queries in their own order: no slot arrays)
    const int64_t q = a.qorder ? a.qorder[slot] : slot;
    const int qc = a.slot_cl ? a.slot_cl[slot] : 0;
    if (lane == 0) {
      unsigned *sw = tk.stat();
      sw[kSideSlot] = (unsigned)slot;
      sw[kSideQuery] = (unsigned)q;
      sw[kSideCluster] = (unsigned)qc;
    }
    QueryRow<DP4, IDXROW> qr;
    qr.load(a.qrows, q, dp4, qslot);
    // the query's distance to its representative: slots of narrow rows are in
    // block order, so it is computed; others carry it in their sort key
    float dq = __int_as_float(0x7f800000);
    if constexpr (kBlocks) dq = sqrtf(qr.dist2(a.qreps + (int64_t)qc * DP4, DP4));
    else if (a.qkeys) dq = __uint_as_float((uint32_t)a.qkeys[slot]);
    if (lane == 0) tk.stat()[kSideDq] = __float_as_uint(dq);  // +inf: no early exit
    tk.reset(query_theta0(a, dq, qc, tol), lane);
    __syncwarp();

    // one step: lane's member p of the cluster at `start`, if `in`.  Row
    // indices fit 32 bits (the result indices are int32): unsigned offsets make
    // every address one wide multiply-add
    int steps = 0;      // (wide rows: how far the query has come ...
    bool far = false;   // ... and whether it is left to a whole block)
    auto step = [&](int start, int p, bool in) {
      if constexpr (kWideRows && !SPLIT) steps++;
      const unsigned gp = (unsigned)(start + p);
      float v = 0.0f;
      int32_t idx = 0;
      bool pass = false;
      if (in) {
        // the index is loaded with the row, not after its distance: one
        // dependent round trip less per step
        if constexpr (kBlocks) {
          if constexpr (!IDXROW) idx = a.sidx[gp];
          float4 row[DP4];
#pragma unroll
          for (int c = 0; c < DP4; c++) row[c] = a.srows[(size_t)gp * DP4 + c];
          int32_t id = idx;
          v = qr.dist2_member(row, &id);
          if constexpr (IDXROW) idx = id;
        } else {
          idx = a.sidx[gp];
          v = qr.dist2_chunks(
              a.srows + (a.col_blocks ? col_block_at(gp, dp4) : (int64_t)gp * dp4),
              a.col_blocks ? kColStride : 1, nch);
        }
        evals++;
        pass = v <= tk.thr_d2;
      }
      topk_offer(tk, pass, v, idx, lane, a.d);
    };

    const int nr = a.rlen[qc];
    const int32_t *rl = a.rlist + (a.rl_base ? a.rl_base[qc] : (int64_t)qc * a.Rs);
    const bool share = SPLIT && nr < kShareLists;
    const int every = SPLIT && !share ? WARPS : 1, first = SPLIT && !share ? w : 0;
    const bool tally = !share || w == 0;  // list entries count once
    // the smallest threshold that some warp, or all of them together, know
    auto exchange = [&]() {
      if constexpr (SPLIT) {
        unsigned t = __float_as_uint(tk.thr_d2);
        if (share && a.k <= 32 * WARPS) {
          volatile unsigned(*part)[32] = s_part;
          part[w][lane] = min((unsigned)part[w][lane], tk.nearest(lane, a.d));
          __syncwarp();
          unsigned x[WARPS];
#pragma unroll
          for (int o = 0; o < WARPS; o++) x[o] = part[o][lane];
          // the k-th smallest, its last 10 bits rounded up
          unsigned kth = 0;
          for (int bit = 30; bit >= 10; bit--) {
            const unsigned upto = kth | ((1u << bit) - 1);
            int cnt = 0;
#pragma unroll
            for (int o = 0; o < WARPS; o++) cnt += x[o] <= upto;
            if ((int)__reduce_add_sync(kFull, (unsigned)cnt) < a.k) kth |= 1u << bit;
          }
          kth |= 1023u;
          if (kth < 0x7f800000u) t = min(t, __float_as_uint(band_hi(__uint_as_float(kth), a.d)));
        }
        if (lane == 0) t = min(atomicMin(&s_thr, t), t);
        const float tv = __uint_as_float(__shfl_sync(kFull, t, 0));
        if (tv < tk.thr_d2) {
          tk.thr_d2 = tv;
          tk.theta = sqrtf(tv);
        }
      }
    };
    for (int base = 0; base < nr; base += 32 * every) {
#if KNN_CHUNK_EXIT
      // the rest of the list is prunable when even its nearest cluster
      // (the list is ascending in d(Rq,Rs)) lies beyond theta for the
      // largest remaining radius: d(q,Rs) - cmax >= d(Rq,Rs) - d(q,Rq) -
      // max cmax; the filter's own test, with twice its rounding margin.
      // Rows of 16 floats or more (d = 32: scan 6.14 -> 5.61 ms, d = 128:
      // 14.88 -> 13.42 ms); on the k = 200, d = 3 self-join the test cost
      // more than it saved (3.82 -> 3.87 ms)
      if (kWideRows && a.clb) {
        const unsigned *sw = tk.stat();
        const float2 cb = a.clb[(size_t)sw[kSideCluster] * a.clb_stride + (base >> 5)];
        const float dqv = __uint_as_float(sw[kSideDq]), th = tk.theta;
        if (cb.x - dqv - cb.y > th + 2.0f * tol * (cb.x + dqv + cb.y + th)) {
          if (tally)
            tk.count(kStatPruned, (unsigned)(max(nr - base - first, 0) + every - 1) / every, lane);
          break;
        }
      }
#endif
      const int j = base + lane * every + first;
      const int batch = min(32, (max(nr - base - first, 0) + every - 1) / every);
      // a cluster whose d(Rq,Rs) less its radius is beyond theta + d(q,Rq) is
      // out without the distance to its representative (a gathered row per
      // lane); most batches of a long list end here, at one coalesced load
      bool listed = j < nr;
      if (a.rlb) {
        const float dqv = __uint_as_float(tk.stat()[kSideDq]), th = tk.theta;
        if (listed)
          listed = !(a.rlb[(size_t)(rl - a.rlist) + j] - dqv > th + 2.0f * tol * (dqv + th));
        if (!__any_sync(kFull, listed)) {
          if (tally) tk.count(kStatPruned, (unsigned)batch, lane);
          continue;
        }
      }
      int rs = 0;
      float D = 0.0f;
      bool alive = false;
      float cmx = 0.0f, cmn = 0.0f;
      int cst = 0, cnn = 0;
      if (listed) {
        rs = rl[j];
        if constexpr (kBlocks) D = sqrtf(qr.dist2(a.sreps + (int64_t)rs * dp4, dp4));
        else D = sqrtf(qr.dist2_chunks(a.sreps + (int64_t)rs * dp4, 1, nch));
        const float th = tk.theta;
        const float slack = tol * (2.0f * D + 2.0f * th);
        cmx = a.cmax[rs];
        cmn = a.cmin[rs];
        alive = !(D - cmx > th + slack) && !(D + th + slack < cmn);
        if (alive) {
          cst = a.soff[rs];
          cnn = a.soff[rs + 1] - cst;
        }
      }
      // visit this chunk's surviving clusters, nearest d(q, Rs) first
      unsigned amask = __ballot_sync(kFull, alive);
      if (amask == 0) {  // warp-uniform: nothing to visit in this batch
        if (tally) tk.count(kStatPruned, (unsigned)batch, lane);
        continue;
      }
      const int nalive = __popc(amask);
      int visits = 0;  // counted once per batch
      float dkey = alive ? D : __int_as_float(0x7f800000);
      // Visit order: nearest d(q, Rs) first.  Narrow rows sort the batch once
      // (bitonic network over the 32 lanes, ties to the lower lane: less work
      // per visited cluster); wider rows pick the nearest remaining cluster
      // by a warp arg-min per visit (measured faster there).
      constexpr bool kSortBatch = DP4 >= 1 && DP4 <= 2;
      float sv = dkey;
      int sl = lane;
      if (kSortBatch && nalive > 1) {  // a single survivor needs no order
#pragma unroll
        for (int size = 2; size <= 32; size <<= 1) {
#pragma unroll
          for (int stride = size >> 1; stride > 0; stride >>= 1) {
            const float ov = __shfl_xor_sync(kFull, sv, stride);
            const int ol = __shfl_xor_sync(kFull, sl, stride);
            const bool other_less = ov < sv || (ov == sv && ol < sl);
            const bool keep_min = ((lane & stride) == 0) == ((lane & size) == 0);
            if (other_less == keep_min) {
              sv = ov;
              sl = ol;
            }
          }
        }
      }
      for (int rank = 0; rank < nalive; rank++) {
        int src;
        if constexpr (kSortBatch) {
          src = nalive > 1 ? __shfl_sync(kFull, sl, rank) : __ffs(amask) - 1;
        } else {
          src = __ffs(amask) - 1;
          if (amask & (amask - 1)) {
            float mv = dkey;
            int ml = lane;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
              const float ov = __shfl_xor_sync(kFull, mv, o);
              const int ol = __shfl_xor_sync(kFull, ml, o);
              if (ov < mv || (ov == mv && ol < ml)) {
                mv = ov;
                ml = ol;
              }
            }
            src = ml;
          }
          if (lane == src) dkey = __int_as_float(0x7f800000);
          amask &= ~(1u << src);
        }
        const float Dc = __shfl_sync(kFull, D, src);
        const float cmax_c = __shfl_sync(kFull, cmx, src);
        const float cmin_c = __shfl_sync(kFull, cmn, src);
        exchange();
        float th = tk.theta;
        float slack = tol * (2.0f * Dc + 2.0f * th);
        if (Dc - cmax_c > th + slack || Dc + th + slack < cmin_c) {
          continue;
        }
        if (kWideRows && !SPLIT && steps > kFarSteps && a.far_slot && nr >= kShareLists &&
            2 * (base + rank) < nr) {
          // (every pull from the work counter past the last query is a warp that
          // has gone)
          unsigned at = kFarQueries;
          if (lane == 0) {
            const unsigned long long warps = (unsigned long long)gridDim.x * WARPS;
            const unsigned long long taken =
                *reinterpret_cast<volatile unsigned long long *>(a.work_counter);
            if (taken >= (unsigned long long)listed_all + warps - warps / 3)
              at = atomicAdd(a.far_count, 1u);
          }
          at = __shfl_sync(kFull, at, 0);
          if (at < kFarQueries) {
            if (lane == 0) a.far_slot[at] = (int32_t)slot;
            far = true;
            break;
          }
          steps = kFarSteps - 64;  // looks again after 64 steps
        }
        visits++;
        const int start = __shfl_sync(kFull, cst, src);
        const int n_c = __shfl_sync(kFull, cnn, src);
        if constexpr (kBlocks) {
          // a lane per block of 32 members: the blocks whose box comes within
          // the threshold.  In a cluster of a list they come in order (taking
          // the nearest first cost more than it saved on the k = 200 self-join:
          // 3.40 -> 3.57 ms); ONE cluster without a starting bound needs its
          // nearest first
          const int nblk = (n_c + 31) >> 5;
          const int64_t slot0 =
              a.boxes ? block_slot(start, __shfl_sync(kFull, rs, src)) : 0;
          // (distance words; all ones: no block)
          auto box_of = [&](int blk) -> uint32_t {
            if (blk >= nblk) return 0xffffffffu;
            if (!a.boxes) return 0u;
            float4 lo[DP4], hi[DP4];
            const float4 *b = a.boxes + (slot0 + blk) * 2 * DP4;
#pragma unroll
            for (int e = 0; e < DP4; e++) {
              lo[e] = b[e];
              hi[e] = b[DP4 + e];
            }
            return __float_as_uint(box_dist2<DP4>(qr.v, lo, hi));
          };
          if constexpr (ONE) {
            // the 32 blocks with the nearest one among them to begin with
            const int rounds = (nblk + 31) >> 5;
            int b0 = 0;
            uint32_t best = 0xffffffffu;
            for (int t = 0; rounds > 1 && t < rounds; t++) {
              const uint32_t m = __reduce_min_sync(kFull, box_of(32 * t + lane));
              if (m < best) {
                best = m;
                b0 = 32 * t;
              }
            }
            for (int t = 0; t < rounds; t++, b0 = b0 + 32 < 32 * rounds ? b0 + 32 : 0) {
              uint32_t bd = box_of(b0 + lane);
              for (;;) {
                const uint32_t next = __reduce_min_sync(kFull, bd);
                if (next == 0xffffffffu || __uint_as_float(next) > tk.thr_d2) break;
                const int at = __ffs((int)__ballot_sync(kFull, bd == next)) - 1;
                if (lane == at) bd = 0xffffffffu;
                const int p = 32 * (b0 + at) + lane;
                step(start, p, p < n_c);
              }
            }
          } else {
            for (int b0 = 0; b0 < nblk; b0 += 32) {
              const uint32_t bw = box_of(b0 + lane);
              const float bd = __uint_as_float(bw);
              unsigned todo = __ballot_sync(kFull, bw != 0xffffffffu && !(bd > tk.thr_d2));
              while (todo) {
                const int t = __ffs((int)todo) - 1;
                todo &= todo - 1;
                if (__shfl_sync(kFull, bd, t) > tk.thr_d2) continue;
                const int p = 32 * (b0 + t) + lane;
                step(start, p, p < n_c);
              }
            }
          }
          continue;
        }
        // one direction: from the lower band edge up (no search when the band
        // starts below the cluster's nearest member)
        const float lo_edge = Dc - th - slack;
        const int lo = lo_edge <= cmin_c ? 0 : warp_lower_bound_coarse(a.sdist + start, n_c, lo_edge, lane);
        const float inf = __int_as_float(0x7f800000);
        auto walk = [&](int from, auto stride, auto every_step) {
          float dsv = from + lane < n_c ? a.sdist[start + from + lane] : inf;
          for (int p0 = from; p0 < n_c; p0 += stride.value) {
            every_step(p0);
            th = tk.theta;
            slack = tol * (2.0f * Dc + 2.0f * th);
            const float hi_v = Dc + th + slack, lo_v = Dc - th - slack;
            const int p = p0 + lane;
            const float ds = dsv;
            // the next step's band distances come while this one's rows do
            dsv = p + stride.value < n_c ? a.sdist[start + p + stride.value] : inf;
            step(start, p, p < n_c && ds >= lo_v && ds <= hi_v);
            if (__shfl_sync(kFull, ds > hi_v, 31)) break;
          }
        };
        if (SPLIT && share) {
          // blocks at multiples of 32, wherever this warp's edge lies
          const int b = lo >> 5;
          walk(32 * (b + ((w - b) & (WARPS - 1))), std::integral_constant<int, 32 * WARPS>(),
               [&](int p0) {
                 if (((p0 / (32 * WARPS)) & 3) == 3) exchange();
               });
        } else {
          walk(lo, std::integral_constant<int, 32>(), [](int) {});
        }
      }
      if (lane == 0 && tally) {
        unsigned *st = tk.stat();
        st[kStatVisited] += (unsigned)visits;
        st[kStatPruned] += (unsigned)(batch - visits);
      }
      if (kWideRows && far) break;
    }
    tk.finish(lane, a.d);
    if constexpr (SPLIT) {
      // the other warps' candidates, into warp 0's
      if (w > 0) {
        const int cnt = tk.expose(lane);
        if (lane == 0) tk.stat()[kSideQuery] = (unsigned)cnt;
      }
      __syncthreads();
      if (w == 0) {
        for (int o = 1; o < WARPS; o++) {
          const uint64_t *ob = keys_base + (size_t)o * TK::kSmemKeys;
          const int cnt = (int)reinterpret_cast<const unsigned *>(ob + TK::kStatAt)[kSideQuery];
          const float ol = *reinterpret_cast<const float *>(ob + TK::kLostAt);
          __syncwarp();
          if (lane == 0) *tk.lostmin() = fminf(*tk.lostmin(), ol);
          for (int e = 0; e < cnt; e += 32) {
            const uint64_t key = e + lane < cnt ? ob[e + lane] : kKeyMax;
            const float v = key_d2(key);
            topk_offer(tk, e + lane < cnt && v <= tk.thr_d2, v, key_idx(key), lane, a.d);
          }
        }
        tk.finish(lane, a.d);
      }
    }
    __syncwarp();
    if ((!SPLIT || w == 0) && !far) {
      const unsigned *sw = tk.stat();
      const int32_t e_slot = (int32_t)sw[kSideSlot];
      const int64_t e_q = (int64_t)sw[kSideQuery];
      const int e_qc = (int)sw[kSideCluster];
      tk.count(kStatChecked, emit_query(tk, a, e_slot, e_q, e_qc, lane), lane);
    }
    __syncwarp();
    // (a query left to a block starts again there and is counted there)
    if (a.counters && !far) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(kFull, evals, o);
      if (lane == 0) {
        const unsigned *st = tk.stat();
        atomicAdd(&blk_ctr[0], (unsigned long long)evals);
        atomicAdd(&blk_ctr[1], (unsigned long long)st[kStatVisited]);
        atomicAdd(&blk_ctr[2], (unsigned long long)st[kStatPruned]);
        atomicAdd(&blk_ctr[3], (unsigned long long)st[kStatPushed]);
        atomicAdd(&blk_ctr[4], (unsigned long long)st[kStatMerges]);
        atomicAdd(&blk_ctr[5], (unsigned long long)st[kStatChecked]);
      }
    }
    __syncwarp();
    if (lane < kSideSlot) tk.stat()[lane] = 0;  // (warp 0 may still read the side words)
    evals = 0;
  }
  __syncthreads();
  if (a.counters && threadIdx.x < kScanCounters)
    atomicAdd(a.counters + threadIdx.x, blk_ctr[threadIdx.x]);
}

// Queries of wide rows up to this many times the resident blocks get a block
// each (scan_kernel's split): a warp per query then leaves the chip waiting
// for the query with the most clusters to visit.  200,003 reference rows,
// d = 17, k = 10, 1,013 queries: search 971 -> 289 us; 100 queries 746 -> 141.
// With more queries the chip is full either way, and every warp of a block
// starts without a threshold: eight times instead of four gave 2,000 queries
// of d = 64 1526 us for 2430, but 2,000 of d = 32 and k = 32 760 for 225.
constexpr int kSplitWaves = 4;

template <int DP4, bool IDXROW, int L, int WARPS, bool ONE>
static int launch_scan_t(const ScanArgs &a, int num_sms, cudaStream_t s) {
  using TK = TopKFor<L, false>;
  constexpr bool kWideRows = DP4 == 0 || DP4 >= 4;
  const size_t smem = (size_t)WARPS * TK::kSmemKeys * sizeof(uint64_t) +
                      (DP4 > 0 ? 0 : (size_t)WARPS * a.dp4 * sizeof(float4));
  auto resident = [&](auto kern, int64_t *blocks) -> int {
    if (smem > 48 * 1024)
      KNN_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)smem));
    int per_sm = 0;
    KNN_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, WARPS * 32, smem));
    *blocks = (int64_t)num_sms * std::max(per_sm, 1);
    return KNN_OK;
  };
  ScanArgs b = a;
  if constexpr (kWideRows) {
    auto kern = scan_kernel<DP4, IDXROW, L, WARPS, ONE, true>;
    int64_t grid = 0;
    const int rc = resident(kern, &grid);
    if (rc != KNN_OK) return rc;
    // (the queries left by a first launch are always split)
    if (a.split_max <= 0) b.split_max = (int)(kSplitWaves * grid);
    // (a list may turn out shorter than its room)
    const bool known = !a.slot_list || a.list_full;
    if (a.m <= b.split_max || !known) {
      kern<<<(int)std::min(grid, a.m), WARPS * 32, smem, s>>>(b);
      KNN_LAUNCH_CHECK();
    }
    if (a.m <= b.split_max) return KNN_OK;
  }
  auto kern = scan_kernel<DP4, IDXROW, L, WARPS, ONE, false>;
  int64_t grid = 0;
  const int rc = resident(kern, &grid);
  if (rc != KNN_OK) return rc;
  kern<<<(int)std::min<int64_t>(grid, (a.m + WARPS - 1) / WARPS), WARPS * 32, smem, s>>>(b);
  KNN_LAUNCH_CHECK();
  return KNN_OK;
}

template <int DP4, bool IDXROW, bool ONE>
static int launch_scan_l(const ScanArgs &a, int num_sms, cudaStream_t s) {
  if (a.k <= KNN_REG_TOPK_MAX_K) return launch_scan_t<DP4, IDXROW, 32, 8, ONE>(a, num_sms, s);
  if (a.k <= 64) return launch_scan_t<DP4, IDXROW, 64, 8, ONE>(a, num_sms, s);
  if (a.k <= 128) return launch_scan_t<DP4, IDXROW, 128, 8, ONE>(a, num_sms, s);
  if (a.k <= 256) return launch_scan_t<DP4, IDXROW, 256, 8, ONE>(a, num_sms, s);
  if (a.k <= 512) return launch_scan_t<DP4, IDXROW, 512, 4, ONE>(a, num_sms, s);
  return launch_scan_t<DP4, IDXROW, 1024, 4, ONE>(a, num_sms, s);
}

template <int DP4, bool IDXROW>
static int launch_scan_n(const ScanArgs &a, int num_sms, cudaStream_t s) {
  return a.Rs == 1 ? launch_scan_l<DP4, IDXROW, true>(a, num_sms, s)
                   : launch_scan_l<DP4, IDXROW, false>(a, num_sms, s);
}

// ---------------------------------------------------------------------------
// Group scan for small k (k <= 32) and narrow rows (d <= 8): one warp, up to
// 32 queries of one query cluster, a query per lane.  The queries share their
// cluster's candidate list, so the warp walks it once for all of them: a lane
// tests one listed cluster (or one block of 32 members) against the queries'
// bounding box and largest threshold, the blocks left come nearest first, and
// a block that some lane's own threshold reaches goes through shared memory:
// every lane evaluates the same member in the same instruction -- coalesced
// row loads, broadcast shared-memory reads, no divergence between lanes.
//
// A candidate (d^2 at most the lane's threshold) goes into the lane's column
// of a shared-memory buffer; when some lane's column is nearly full, all lanes
// sort theirs in registers (a fixed network, the same instructions for all)
// and merge it into their K best keys (K = pow2 >= k), which tightens the
// lane's threshold.
//
// What bounds it: instruction issue (75 % of the slots on 512 surface clouds,
// k = 16), about half of it the members and a third the merges (13 blocks and
// 7.7 merges per group).  It replaced a thread per query whose every insertion
// into a sorted list of 64-bit keys was executed by the whole warp: 4,096
// surface clouds, k = 16: search 59.4 -> 20.4 ms.  64-bit keys in the merges
// instead of distance words: 32 ms; whole clusters by their distance band
// instead of blocks by their boxes: 22.4 ms; candidates stored by predicated
// instructions instead of a branch: 22.4 ms.  At k = 8 five blocks per SM
// (96 registers) instead of six, which spilled: 64 pairs of clouds, loss and
// gradients 3.70 -> 3.41 ms.
//
// FP64 boundary: the threshold is band_hi of the k-th key, so every point
// inside the final k-th's FP32 band is evaluated and admitted; one that a merge
// drops sets `lost`.  A query whose band reaches behind its k-th (a key inside
// it was lost, or the list holds one after the k-th) goes to the band kernel,
// which re-decides the band in FP64; on data without near-ties at the k-th
// that is a small fraction of the queries, and FP64 code stays out of this
// register-bound kernel.
// ---------------------------------------------------------------------------
__device__ __forceinline__ void order_pair(uint32_t &a, uint32_t &b) {
  const uint32_t lo = min(a, b), hi = max(a, b);
  a = lo;
  b = hi;
}
// Keys as doubles: a key's upper word is a float, so no key has a double's
// exponent of all ones (kLaneEmpty is the largest finite one) and keys order
// like the doubles of their bits.  One double compare and four selects: 9.3
// cycles against 16.2 for the integer comparison of two words.
__device__ __forceinline__ void order_pair(uint64_t &a, uint64_t &b) {
  const bool sw = __longlong_as_double((long long)a) > __longlong_as_double((long long)b);
  const uint64_t lo = sw ? b : a, hi = sw ? a : b;
  a = lo;
  b = hi;
}
constexpr uint64_t kLaneEmpty = 0x7fefffffffffffffull;  // its distance word is a NaN

// Batcher's odd-even merge sort of x[LO .. LO+N) in registers (63 comparators
// for N = 16).
template <int LO, int N, int R, class T, int S>
__device__ __forceinline__ void net_merge(T (&x)[S]) {
  if constexpr (2 * R < N) {
    net_merge<LO, N, 2 * R>(x);
    net_merge<LO + R, N, 2 * R>(x);
#pragma unroll
    for (int i = LO + R; i + R < LO + N; i += 2 * R) order_pair(x[i], x[i + R]);
  } else {
    order_pair(x[LO], x[LO + R]);
  }
}
template <int LO, int N, class T, int S>
__device__ __forceinline__ void net_sort(T (&x)[S]) {
  if constexpr (N > 1) {
    net_sort<LO, N / 2>(x);
    net_sort<LO + N / 2, N / 2>(x);
    net_merge<LO, N, 1>(x);
  }
}

// One lane's candidates: a column of (distance, index) words in shared memory
// (entry j at [32 j]), every candidate up to band_hi of the k-th distance seen
// among them, and the K smallest distance words in registers, which give that
// threshold.  Entries [kept, cnt) are not merged into the registers yet.
constexpr int kLaneNew = 16;  // most entries merged at once

// Keeps the `want` smallest keys of a lane's column of n > want entries (indices
// 32 C words behind the distances), in place; returns the smallest distance
// dropped.  *ceil is the largest key that the last cut left (all ones: none yet):
// of a crowd of equal distances most new ones lie above it -- copies of a point
// come in the order of their rows -- and go in one pass; what is still too much
// goes by its largest key, a pass each.  (A rank of every entry among all, which
// this replaced, took 48 passes a cut at K = 32: 150,000 integers of 256 values,
// k = 32 8.7 -> 1.2 ms, 50,000 points in 64 places 10.8 -> 1.2.)  Out of line: only
// such crowds come here.
__device__ __noinline__ float cut_column(uint32_t *col, int C, int n, int want, uint64_t *ceil) {
  float lost = __int_as_float(0x7f800000);
  auto entry = [&](int j) { return ((uint64_t)col[32 * j] << 32) | col[32 * (C + j)]; };
  auto put = [&](int j, uint64_t x) {
    col[32 * j] = (uint32_t)(x >> 32);
    col[32 * (C + j)] = (uint32_t)x;
  };
  const uint64_t top = *ceil;
  int w = 0;
  for (int e = 0; e < n; e++) {
    const uint64_t x = entry(e);
    if (x <= top) put(w++, x);
    else lost = fminf(lost, key_d2(x));
  }
  // (w >= want: while the keys of the last cut are all here they are want, and
  // once one has gone above the threshold nothing above *ceil is left)
  if (w <= want) return lost;
  for (n = w;; n--) {
    uint64_t most = 0;
    int at = 0;
    for (int e = 0; e < n; e++) {
      const uint64_t x = entry(e);
      if (x >= most) most = x, at = e;
    }
    if (n == want) {
      *ceil = most;
      return lost;
    }
    lost = fminf(lost, key_d2(most));
    put(at, entry(n - 1));
  }
}

template <int K>
struct LaneTopK {
  static constexpr int C = K + kLaneNew;  // column entries
  uint32_t top[K];  // ascending distance words (all ones: none)
  uint32_t *col;    // distances; the indices 32 C words further on
  int kept, cnt;
  float lost;       // smallest FP32 d^2 dropped for lack of room (+inf: none)

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int j = 0; j < K; j++) top[j] = 0xffffffffu;
    kept = cnt = 0;
    lost = __int_as_float(0x7f800000);
  }
  __device__ __forceinline__ void push(float v, int32_t idx) {
    col[32 * cnt] = __float_as_uint(v);
    col[32 * (C + cnt)] = (uint32_t)idx;
    cnt++;
  }
  // whether some lane may not take four more candidates
  __device__ __forceinline__ bool crowded() const {
    return __any_sync(kFull, cnt - kept > kLaneNew - 4 || cnt > C - 4);
  }
  // the k-th distance word (selected by masks: a compare-and-select on the
  // runtime k turns the list into an indexed local-memory array)
  __device__ __forceinline__ uint32_t at(int i) const {
    uint32_t r = 0;
#pragma unroll
    for (int j = 0; j < K; j++) r |= top[j] & (0u - (uint32_t)(j == i));
    return r;
  }
  __device__ __forceinline__ uint64_t entry(int j) const {
    return ((uint64_t)col[32 * j] << 32) | col[32 * (C + j)];
  }
  // merges the new entries, updates the threshold (squared distances up to
  // thr enter) and drops the entries above it
  __device__ __forceinline__ void flush(int k, int d, float &thr, uint64_t *ceil) {
    uint32_t b[kLaneNew];
#pragma unroll
    for (int j = 0; j < kLaneNew; j++) {
      b[j] = 0xffffffffu;
      if (kept + j < cnt) b[j] = col[32 * (kept + j)];
    }
    net_sort<0, kLaneNew>(b);
    // top ascending, b descending: the minima are the K smallest of both, as
    // a bitonic sequence
    constexpr int N = K < kLaneNew ? K : kLaneNew;
#pragma unroll
    for (int j = 0; j < N; j++) top[K - 1 - j] = min(top[K - 1 - j], b[j]);
#pragma unroll
    for (int s = K / 2; s > 0; s >>= 1) {
#pragma unroll
      for (int j = 0; j < K; j++)
        if ((j & s) == 0) order_pair(top[j], top[j | s]);
    }
    const uint32_t kth = k == K ? top[K - 1] : at(k - 1);
    if (kth != 0xffffffffu) thr = band_hi(__uint_as_float(kth), d);
    int w = 0;
    const int most = (int)__reduce_max_sync(kFull, (unsigned)cnt);
    for (int j0 = 0; j0 < most; j0 += 4) {
      uint32_t dv[4], iv[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {  // C is a multiple of four
        dv[u] = col[32 * (j0 + u)];
        iv[u] = col[32 * (C + j0 + u)];
      }
#pragma unroll
      for (int u = 0; u < 4; u++)
        if (j0 + u < cnt && __uint_as_float(dv[u]) <= thr) {
          col[32 * w] = dv[u];
          col[32 * (C + w)] = iv[u];
          w++;
        }
    }
    kept = cnt = w;
    // many equal distances: the K smallest keys stay
    if (__any_sync(kFull, kept > C - 8)) cut(ceil);
  }
  // keeps the K smallest keys of the column; the others go into `lost`
  __device__ __forceinline__ void cut(uint64_t *ceil) {
    if (kept > K) lost = fminf(lost, cut_column(col, C, kept, K, ceil));
    kept = cnt = min(kept, K);
  }
};

// warps per block, each on its own group
__host__ __device__ constexpr int group_warps(int K) { return K > 16 ? 2 : 4; }

template <int DP4, bool IDXROW, int K>
__global__ void __launch_bounds__(group_warps(K) * 32, K > 16 ? 8 : (K > 1 ? 5 : 6))
    group_scan_kernel(const ScanArgs a) {
  using TK = LaneTopK<K>;
  constexpr int kGroupWarps = group_warps(K);
  __shared__ uint32_t s_col[kGroupWarps][K > 1 ? 2 * TK::C * 32 : 1];
  // the current 32 members by coordinate (negated); the last pad coordinate
  // of rows that carry their index there is the index
  __shared__ __align__(16) float s_mem[kGroupWarps][4 * DP4 + (IDXROW ? 0 : 1)][32];
  // largest key a cut left in a lane's column
  __shared__ uint64_t s_ceil[kGroupWarps][K > 1 ? 32 : 1];
  __shared__ unsigned long long blk_ctr[4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 4) blk_ctr[threadIdx.x] = 0;
  __syncthreads();
  const int d = a.d, k = a.k;
  const float tol = bound_tol(d);
  const float inf = __int_as_float(0x7f800000);
  const bool exact32 = fp32_exact(a);
  const int64_t nslots = a.slot_list ? (int64_t)*a.slot_count : a.m;
  TK tk;
  tk.col = &s_col[w][K > 1 ? lane : 0];
  unsigned evals = 0, visited = 0, listed = 0, pushed = 0;

  // Windows of 32 slots from the work counter.  Without a slot list a window
  // stands for the groups that start in it (they begin at every 32nd slot of
  // their cluster, so no list of groups is needed); with one, for the 32
  // listed slots, a group per query cluster among them.
  long long s = 0, s_end = 0, c0 = 0, c1 = 0;
  int qc = 0, listed_qc = -1;
  unsigned todo = 0;
  for (;;) {
    int64_t slot;
    bool act;
    if (a.slot_list ? todo == 0 : s >= s_end) {
      long long win = 0;
      if (lane == 0) win = (long long)atomicAdd(a.work_counter, 1ull);
      win = __shfl_sync(kFull, win, 0) * 32;
      if (win >= nslots) break;
      s = a.slot_base + win;
      s_end = min(s + 32, (long long)a.slot_base + (long long)nslots);
      if (a.slot_list) {
        const bool have = win + lane < nslots;
        s = have ? a.slot_list[win + lane] : 0;
        listed_qc = have ? a.slot_cl[s] : -1;
        todo = __ballot_sync(kFull, have);
      } else {
        qc = a.slot_cl[s];
        c0 = a.qoff[qc];
        c1 = a.qoff[qc + 1];
        s = min(c0 + ((s - c0 + 31) & ~31ll), c1);
        continue;
      }
    }
    if (a.slot_list) {
      qc = __shfl_sync(kFull, listed_qc, __ffs((int)todo) - 1);
      slot = s;
      act = listed_qc == qc;
      todo &= ~__ballot_sync(kFull, act);
    } else {
      if (s == c1) {  // the next cluster with queries
        qc = a.slot_cl[s];
        c1 = a.qoff[qc + 1];
      }
      slot = s + lane;
      act = slot < c1;
      s = min(s + 32, c1);
    }
    // one group: lane's query slot (act: it has one), all of query cluster qc
    const int64_t q = act ? a.qorder[slot] : 0;
    QueryRow<DP4, IDXROW> qr;
    qr.load(a.qrows, q, DP4, nullptr);
    constexpr int kCoords = 4 * DP4 - (IDXROW ? 1 : 0);
    float2 qq[4 * DP4];
#pragma unroll
    for (int e = 0; e < DP4; e++) {
      qq[4 * e] = make_float2(qr.v[e].x, qr.v[e].x);
      qq[4 * e + 1] = make_float2(qr.v[e].y, qr.v[e].y);
      qq[4 * e + 2] = make_float2(qr.v[e].z, qr.v[e].z);
      qq[4 * e + 3] = make_float2(qr.v[e].w, qr.v[e].w);
    }
    tk.reset();
    if constexpr (K > 1) s_ceil[w][lane] = ~0ull;
    uint64_t best = kLaneEmpty;  // the list for k = 1
    float thr = 0.0f;  // squared distances up to it enter
    if (act) {
      const float th =
          query_theta0(a, sqrtf(qr.dist2(a.qreps + (int64_t)qc * DP4, DP4)), qc, tol);
      thr = th * th;  // admits every d^2 <= theta0^2, whatever the index
    }
    // the queries' bounding box (the coordinates behind kCoords are padding)
    // and the largest threshold among them
    float4 glo[DP4], ghi[DP4];
    {
      float lo[4 * DP4], hi[4 * DP4];
#pragma unroll
      for (int c = 0; c < 4 * DP4; c++) {
        lo[c] = act ? qq[c].x : inf;
        hi[c] = act ? qq[c].x : -inf;
        if (c >= kCoords) lo[c] = hi[c] = 0.0f;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < kCoords; c++) {
          lo[c] = fminf(lo[c], __shfl_xor_sync(kFull, lo[c], o));
          hi[c] = fmaxf(hi[c], __shfl_xor_sync(kFull, hi[c], o));
        }
      }
#pragma unroll
      for (int e = 0; e < DP4; e++) {
        glo[e] = make_float4(lo[4 * e], lo[4 * e + 1], lo[4 * e + 2], lo[4 * e + 3]);
        ghi[e] = make_float4(hi[4 * e], hi[4 * e + 1], hi[4 * e + 2], hi[4 * e + 3]);
      }
    }
    auto largest = [&](float x) {  // x >= 0 (a NaN counts as the largest)
      return __uint_as_float(__reduce_max_sync(kFull, __float_as_uint(x)));
    };
    float thr_max = largest(thr);
    const int nr = a.rlen[qc];
    const int32_t *rl = a.rlist + (a.rl_base ? a.rl_base[qc] : (int64_t)qc * a.Rs);
    for (int base = 0; base < nr; base += 32) {
      // a lane per reference cluster: it can hold a member within some
      // query's threshold only if the queries' box comes within theta +
      // radius of its representative
      int c = 0, cst = 0, cnn = 0;
      float need_th = inf;  // the smallest theta that needs the cluster
      if (base + lane < nr) {
        c = rl[base + lane];
        float4 rep[DP4];
#pragma unroll
        for (int e = 0; e < DP4; e++) rep[e] = a.sreps[(int64_t)c * DP4 + e];
        const float Dg = sqrtf(box_dist2<DP4>(rep, glo, ghi));
        cst = a.soff[c];
        cnn = a.soff[c + 1] - cst;
        // D - cmax > theta + tol (2 D + 2 theta), solved for theta
        if (cnn > 0) need_th = (Dg - 2.0f * tol * Dg - a.cmax[c]) * (1.0f - 2.0f * tol);
      }
      unsigned clusters = __ballot_sync(kFull, !(need_th > sqrtf(thr_max)));
      while (clusters) {
        const int ci = __ffs((int)clusters) - 1;
        clusters &= clusters - 1;
        if (__shfl_sync(kFull, need_th, ci) > sqrtf(thr_max)) continue;
        const int start = __shfl_sync(kFull, cst, ci), n_c = __shfl_sync(kFull, cnn, ci);
        const int64_t slot0 = a.boxes ? block_slot(start, __shfl_sync(kFull, c, ci)) : 0;
        const int nblk = (n_c + 31) >> 5;
        bool hit = false;
        for (int b0 = 0; b0 < nblk; b0 += 32) {
          // a lane per block of 32 members, nearest the queries' box first
          uint32_t bd = b0 + lane < nblk ? 0u : 0xffffffffu;
          if (a.boxes && b0 + lane < nblk) {
            const float4 *b = a.boxes + (slot0 + b0 + lane) * 2 * DP4;
            float4 gap_lo[DP4], gap_hi[DP4];
#pragma unroll
            for (int e = 0; e < DP4; e++) {
              gap_lo[e] = b[e];
              gap_hi[e] = b[DP4 + e];
            }
            bd = __float_as_uint(boxes_dist2<DP4>(glo, ghi, gap_lo, gap_hi));
          }
          for (;;) {
            const uint32_t nearest = __reduce_min_sync(kFull, bd);
            if (nearest == 0xffffffffu || __uint_as_float(nearest) > thr_max) break;
            const int bi = __ffs((int)__ballot_sync(kFull, bd == nearest)) - 1;
            if (lane == bi) bd = 0xffffffffu;
            const int p = 32 * (b0 + bi) + lane;
            const bool valid = p < n_c;
            const unsigned gp = (unsigned)(start + p);
            float4 row[DP4];
#pragma unroll
            for (int e = 0; e < DP4; e++)
              // (a row past the end passes no lane: its distances are NaN)
              row[e] = valid ? a.srows[(size_t)gp * DP4 + e]
                             : make_float4(__int_as_float(0x7fffffff), 0.0f, 0.0f, 0.0f);
            bool need = act;
            if (a.boxes) {
              const float4 *b = a.boxes + (slot0 + b0 + bi) * 2 * DP4;
              float4 lo[DP4], hi[DP4];
#pragma unroll
              for (int e = 0; e < DP4; e++) {
                lo[e] = b[e];
                hi[e] = b[DP4 + e];
              }
              need = act && !(box_dist2<DP4>(qr.v, lo, hi) > thr);
            }
            if (!__any_sync(kFull, need)) continue;
            hit |= need;
            const int cnt = min(32, n_c - 32 * (b0 + bi));
            if (need) evals += (unsigned)cnt;
            float cut = need ? thr : -1.0f;  // no d^2 passes a lane that does not need the block
            __syncwarp();
#pragma unroll
            for (int e = 0; e < DP4; e++) {
              s_mem[w][4 * e][lane] = -row[e].x;
              s_mem[w][4 * e + 1][lane] = -row[e].y;
              s_mem[w][4 * e + 2][lane] = -row[e].z;
              s_mem[w][4 * e + 3][lane] = IDXROW && e == DP4 - 1 ? row[e].w : -row[e].w;
            }
            if constexpr (!IDXROW)
              s_mem[w][4 * DP4][lane] = valid ? __int_as_float(a.sidx[gp]) : 0.0f;
            __syncwarp();
            bool tightened = K == 1;  // warp-uniform
            for (int t = 0; t < cnt; t += 4) {
              // packed FP32 pairs, the scan's arithmetic for each member
              float2 v01, v23;
#pragma unroll
              for (int c = 0; c < kCoords; c++) {
                const float4 s4 = *reinterpret_cast<const float4 *>(&s_mem[w][c][t]);
                const float2 d01 = __fadd2_rn(qq[c], make_float2(s4.x, s4.y));
                const float2 d23 = __fadd2_rn(qq[c], make_float2(s4.z, s4.w));
                v01 = c == 0 ? __fmul2_rn(d01, d01) : __ffma2_rn(d01, d01, v01);
                v23 = c == 0 ? __fmul2_rn(d23, d23) : __ffma2_rn(d23, d23, v23);
              }
              const float v[4] = {v01.x, v01.y, v23.x, v23.y};
              const float4 id4 = *reinterpret_cast<const float4 *>(&s_mem[w][kCoords][t]);
              const int32_t id[4] = {__float_as_int(id4.x), __float_as_int(id4.y),
                                     __float_as_int(id4.z), __float_as_int(id4.w)};
#pragma unroll
              for (int u = 0; u < 4; u++) {
                if (v[u] <= cut) {
                  if constexpr (K > 1) {
                    tk.push(v[u], id[u]);
                  } else {
                    const uint64_t key = make_key(v[u], id[u]);
                    tk.lost = fminf(tk.lost, key_d2(umax64(best, key)));
                    best = umin64(best, key);
                    pushed++;
                  }
                }
              }
              if constexpr (K > 1) {
                if (tk.crowded()) {
                  pushed += tk.cnt - tk.kept;
                  tk.flush(k, d, thr, &s_ceil[w][lane]);
                  if (need) cut = thr;
                  tightened = true;
                }
              } else if (best != kLaneEmpty) {
                thr = band_hi(key_d2(best), d);
                if (need) cut = thr;
              }
            }
            if (tightened) thr_max = largest(thr);
          }
        }
        visited += hit;
      }
    }
    if (act) listed += nr;
    if constexpr (K > 1) {
      if (__any_sync(kFull, tk.cnt > tk.kept)) {
        pushed += tk.cnt - tk.kept;
        tk.flush(k, d, thr, &s_ceil[w][lane]);
      }
    }
    // the K best keys, ascending
    uint64_t key[K];
    if constexpr (K > 1) {
      if (__any_sync(kFull, tk.kept > K)) tk.cut(&s_ceil[w][lane]);
#pragma unroll
      for (int j = 0; j < K; j++) {
        key[j] = kLaneEmpty;
        if (j < tk.kept) key[j] = tk.entry(j);
      }
      net_sort<0, K>(key);
    } else {
      key[0] = best;
    }
    if (act) {
      // the k-th key, the key behind it, and the FP32 band around the k-th
      uint64_t kth = 0, next = 0;
#pragma unroll
      for (int j = 0; j < K; j++) {
        kth |= key[j] & (0ull - (uint64_t)(j == k - 1));
        next |= key[j] & (0ull - (uint64_t)(j == k));
      }
      if (k >= K) next = kLaneEmpty;
      bool defer = false;
      int nlo = 0;
      const float Dk = key_d2(kth);
      if (kth != kLaneEmpty && !exact32) {
        const float bhi = band_hi(Dk, d);
        // a band key was dropped, or one sits behind the k-th (NaN: none)
        defer = tk.lost <= bhi || key_d2(next) <= bhi;
        if (defer) {
          const float blo = band_lo(Dk, d);
#pragma unroll
          for (int j = 0; j < K; j++) nlo += key_d2(key[j]) < blo;
        }
      }
      int32_t *oi = a.out_idx + q * k;
      float *od = a.out_dist + q * k;
      const int32_t rbase = a.qc_ref_base ? (int32_t)a.qc_ref_base[qc] : 0;
      auto idx_of = [&](uint64_t x) {
        return x == kLaneEmpty ? -1 : key_idx(x) - rbase;
      };
      auto dist_of = [&](uint64_t x) {
        const float d2 = key_d2(x);
        return x == kLaneEmpty ? inf : (a.squared ? d2 : sqrtf(d2));
      };
      bool quads = false;
      if constexpr (K >= 4)
        quads = (k & 3) == 0 &&
                ((reinterpret_cast<uintptr_t>(a.out_idx) | reinterpret_cast<uintptr_t>(a.out_dist)) &
                 15) == 0;
      if (quads) {
        if constexpr (K >= 4) {
#pragma unroll
          for (int j = 0; j < K; j += 4)
            if (j < k) {
              *reinterpret_cast<int4 *>(oi + j) = make_int4(
                  idx_of(key[j]), idx_of(key[j + 1]), idx_of(key[j + 2]),
                  idx_of(key[j + 3]));
              *reinterpret_cast<float4 *>(od + j) = make_float4(
                  dist_of(key[j]), dist_of(key[j + 1]), dist_of(key[j + 2]),
                  dist_of(key[j + 3]));
            }
        }
      } else {
#pragma unroll
        for (int j = 0; j < K; j++)
          if (j < k) {
            oi[j] = idx_of(key[j]);
            od[j] = dist_of(key[j]);
          }
      }
      if (defer) {
        // the band kernel settles the boundary: it reads the number of keys
        // below the band and the k-th value from the last slot
        oi[k - 1] = nlo;
        od[k - 1] = Dk;
        a.unres_slot[atomicAdd(a.unres_count, 1u)] = (int32_t)slot;
      }
    }
  }
  if (a.counters) {
    unsigned pruned = listed - visited;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      evals += __shfl_xor_sync(kFull, evals, o);
      visited += __shfl_xor_sync(kFull, visited, o);
      pruned += __shfl_xor_sync(kFull, pruned, o);
      pushed += __shfl_xor_sync(kFull, pushed, o);
    }
    if (lane == 0) {
      atomicAdd(&blk_ctr[0], (unsigned long long)evals);
      atomicAdd(&blk_ctr[1], (unsigned long long)visited);
      atomicAdd(&blk_ctr[2], (unsigned long long)pruned);
      atomicAdd(&blk_ctr[3], (unsigned long long)pushed);
    }
    __syncthreads();
    if (threadIdx.x < 4) atomicAdd(a.counters + threadIdx.x, blk_ctr[threadIdx.x]);
  }
}

template <int DP4, bool IDXROW>
static int launch_group_scan(const ScanArgs &a, int num_sms, cudaStream_t s) {
  auto go = [&](auto kern, int warps) -> int {
    int per_sm = 0;
    KNN_CUDA_TRY(
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, warps * 32, 0));
    const int64_t want = (a.m + 32 * warps - 1) / (32 * warps);
    const int64_t grid = std::min<int64_t>((int64_t)num_sms * std::max(per_sm, 1), want);
    kern<<<(unsigned)std::max<int64_t>(grid, 1), warps * 32, 0, s>>>(a);
    KNN_LAUNCH_CHECK();
    return KNN_OK;
  };
  if (a.k <= 1) return go(group_scan_kernel<DP4, IDXROW, 1>, group_warps(1));
  if (a.k <= 4) return go(group_scan_kernel<DP4, IDXROW, 4>, group_warps(4));
  if (a.k <= 8) return go(group_scan_kernel<DP4, IDXROW, 8>, group_warps(8));
  if (a.k <= 16) return go(group_scan_kernel<DP4, IDXROW, 16>, group_warps(16));
  return go(group_scan_kernel<DP4, IDXROW, 32>, group_warps(32));
}

// ---------------------------------------------------------------------------
// Thread per query: the self-join's nearest point (k = 1) in short clusters of
// 5 to 8 dimensions.  The point itself or a copy of it settles a query as soon as
// its own cluster is read, so that what is left is the walk along the cluster
// list -- a hundred distances, each dropped by its test -- for which a query needs
// no more than a thread, while the box of 32 queries still reaches clusters that
// none of them does.  Members are read by their distance to the representative
// (dorder: a row of 32 bytes is one sector wherever it lies), those of the band
// |D - d(s,Rs)| <= theta only.  The start's bound, the FP32 keys and the FP64
// boundary are the other scans'.  What bounds it: the latency of a thread's
// dependent loads.  Self-joins of 30,000 uniform points, whole, group scan /
// this: d = 5 459 / 371 us, d = 8 926 / 394; 64 clouds of 2,000, d = 8 559 / 315.
// ---------------------------------------------------------------------------
template <int DP4>
__global__ void __launch_bounds__(256, 4) thread_scan_kernel(const ScanArgs a) {
  __shared__ unsigned long long blk_ctr[4];
  if (threadIdx.x < 4) blk_ctr[threadIdx.x] = 0;
  __syncthreads();
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t nslots = a.slot_list ? (int64_t)*a.slot_count : a.m;
  const float inf = __int_as_float(0x7f800000);
  unsigned evals = 0, visited = 0, pruned = 0, pushed = 0;
  if (t < nslots) {
    const int64_t slot = a.slot_list ? (int64_t)a.slot_list[t] : a.slot_base + t;
    const int64_t q = a.qorder[slot];
    const int qc = a.slot_cl[slot];
    const float tol = bound_tol(a.d);
    QueryRow<DP4, false> qr;
    qr.load(a.qrows, q, DP4, nullptr);
    float theta =
        query_theta0(a, sqrtf(qr.dist2(a.qreps + (int64_t)qc * DP4, DP4)), qc, tol);
    float thr = theta * theta;  // admits every d^2 <= theta0^2, whatever the index
    float lost = inf;           // smallest d^2 that was admitted and is not the result
    uint64_t best = kKeyMax;
    const int nr = a.rlen[qc];
    const int32_t *rl = a.rlist + (a.rl_base ? a.rl_base[qc] : (int64_t)qc * a.Rs);
    for (int j = 0; j < nr; j++) {
      const int c = rl[j];
      const float D = sqrtf(qr.dist2(a.sreps + (int64_t)c * DP4, DP4));
      float slack = tol * (2.0f * D + 2.0f * theta);
      const float cmin = a.cmin[c];
      if (D - a.cmax[c] > theta + slack || D + theta + slack < cmin) {
        pruned++;
        continue;
      }
      visited++;
      const int start = a.soff[c], n_c = a.soff[c + 1] - start;
      const float *sd = a.sdist + start;
      // first member of the band [D - theta, D + theta] (with slack)
      const float lo_edge = D - theta - slack;
      int p = 0;
      if (lo_edge > cmin) {
        int hi = n_c;
        while (p < hi) {
          const int md = (p + hi) >> 1;
          if (sd[md] < lo_edge) p = md + 1;
          else hi = md;
        }
      }
      for (; p < n_c && !(sd[p] > D + theta + slack); p++) {
        const int32_t idx = a.dorder[start + p];
        const float v = qr.dist2(a.rrows + (int64_t)idx * DP4, DP4);
        evals++;
        if (!(v <= thr)) continue;
        pushed++;
        const uint64_t key = make_key(v, idx);
        lost = fminf(lost, key_d2(umax64(best, key)));  // (of no key yet: NaN, ignored)
        if (key < best) {
          best = key;
          thr = fminf(thr, band_hi(v, a.d));
          theta = sqrtf(thr);
          slack = tol * (2.0f * D + 2.0f * theta);
        }
      }
    }
    const bool none = best == kKeyMax;
    const float d2 = key_d2(best);
    const int32_t base = a.qc_ref_base ? (int32_t)a.qc_ref_base[qc] : 0;
    const bool defer = !none && !fp32_exact(a) && lost <= band_hi(d2, a.d);
    // deferred: the band kernel settles the boundary; it reads the number of
    // keys below the band and the k-th value from the last slot
    a.out_idx[q] = defer ? 0 : (none ? -1 : key_idx(best) - base);
    a.out_dist[q] = defer ? d2 : (none ? inf : (a.squared ? d2 : sqrtf(d2)));
    if (defer) a.unres_slot[atomicAdd(a.unres_count, 1u)] = (int32_t)slot;
  }
  if (a.counters) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      evals += __shfl_xor_sync(kFull, evals, o);
      visited += __shfl_xor_sync(kFull, visited, o);
      pruned += __shfl_xor_sync(kFull, pruned, o);
      pushed += __shfl_xor_sync(kFull, pushed, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&blk_ctr[0], (unsigned long long)evals);
      atomicAdd(&blk_ctr[1], (unsigned long long)visited);
      atomicAdd(&blk_ctr[2], (unsigned long long)pruned);
      atomicAdd(&blk_ctr[3], (unsigned long long)pushed);
    }
    __syncthreads();
    if (threadIdx.x < 4) atomicAdd(a.counters + threadIdx.x, blk_ctr[threadIdx.x]);
  }
}

// ---------------------------------------------------------------------------
// Band kernel: the k-th boundary of the queries the scan kernels could not
// settle (a key of the final band was dropped for lack of room, or the
// group scan's list holds one behind the k-th).  One block per query, over
// the same candidate list: every point whose FP32 d^2 -- computed with the
// scan's own arithmetic, so the values are the same -- lies inside the band
// band_lo(Dk) .. band_hi(Dk) of the k-th is found again, and the band's
// need = k - nlo best by (FP64 d^2, index) are kept in a shared-memory set
// that is sorted and cut back to `need` whenever it fills, so any number of
// ties fits.  They are written, in FP32 key order, behind the nlo keys below
// the band that the scan already wrote.  The scan left nlo and Dk in the
// query's last output slot.
// ---------------------------------------------------------------------------
constexpr int kBandThreads = 128;
constexpr int kBandCap = 2048;  // >= KNN_MAX_K + kBandThreads: room after a cut

struct BandEntry {
  unsigned long long d64;  // FP64 d^2 bits (non-negative: they order like the values)
  unsigned long long key;  // FP32 (d^2, index) key
};

__device__ __forceinline__ bool band_entry_less(const BandEntry &x, const BandEntry &y) {
  return x.d64 < y.d64 || (x.d64 == y.d64 && (uint32_t)x.key < (uint32_t)y.key);
}

// Ascending bitonic sort of e[0..P) (P a power of two) by the block, by
// (FP64 d^2, index) or by the FP32 key.
template <bool BY_KEY>
__device__ void band_sort(BandEntry *e, int P) {
  for (int size = 2; size <= P; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = threadIdx.x; t < (P >> 1); t += blockDim.x) {
        const int i = 2 * t - (t & (stride - 1));
        const int j = i + stride;
        const bool up = (i & size) == 0;
        const BandEntry x = e[i], y = e[j];
        const bool gt = BY_KEY ? x.key > y.key : band_entry_less(y, x);
        if (gt == up) {
          e[i] = y;
          e[j] = x;
        }
      }
      __syncthreads();
    }
  }
}

// Cuts the set e[0..*cnt) back to its `need` smallest by (FP64 d^2, index);
// *thr becomes the need-th (the admission bound) once that many are in.
__device__ void band_cut(BandEntry *e, int *cnt, BandEntry *thr, int need) {
  const int c = *cnt;  // read by every thread before the barrier below
  int P = 1;
  while (P < c) P <<= 1;
  for (int i = c + threadIdx.x; i < P; i += blockDim.x) e[i] = BandEntry{~0ull, ~0ull};
  __syncthreads();
  band_sort<false>(e, P);
  if (threadIdx.x == 0) {
    const int kept = c < need ? c : need;
    *cnt = kept;
    if (kept == need) *thr = e[need - 1];
  }
  __syncthreads();
}

// FP32 squared distance over the first d coordinates, dimension order, fma:
// the scan kernels' value for the same pair (their padded coordinates add
// exact zeros).
__device__ __forceinline__ float band_dist2(const float *__restrict__ q,
                                            const float *__restrict__ r, int d, int stride = 1) {
  float acc = 0.0f;
  for (int c = 0; c < d; c++) {
    const float t = __fsub_rn(q[c], r[(size_t)(c >> 2) * (4 * stride) + (c & 3)]);
    acc = __fmaf_rn(t, t, acc);
  }
  return acc;
}

__global__ void __launch_bounds__(kBandThreads) band_resolve_kernel(const ScanArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BandEntry *ent = reinterpret_cast<BandEntry *>(smem_raw);
  float *qv = reinterpret_cast<float *>(ent + kBandCap);  // 4 * dp4 floats
  __shared__ int s_cnt, s_nvis;
  __shared__ BandEntry s_thr;
  __shared__ int s_vis[kBandThreads];
  __shared__ float s_D[kBandThreads];
  const bool narrow = a.dp4_tmpl == 1 || a.dp4_tmpl == 2;
  const int tid = threadIdx.x, k = a.k, d = a.d, dp4 = a.dp4;
  const float tol = bound_tol(d);
  const unsigned total = *a.unres_count;
  unsigned long long evals = 0;
  for (unsigned u = blockIdx.x; u < total; u += gridDim.x) {
    const int32_t slot = a.unres_slot[u];
    const int64_t q = a.qorder ? a.qorder[slot] : slot;
    const int qc = a.slot_cl ? a.slot_cl[slot] : 0;
    int32_t *oi = a.out_idx + q * k;
    float *od = a.out_dist + q * k;
    __syncthreads();  // the previous query is done with the shared state
    const int nlo = oi[k - 1];
    const float Dk = od[k - 1];
    const int need = k - nlo;
    const float lo = band_lo(Dk, d), hi = band_hi(Dk, d), th = sqrtf(hi);
    for (int c = tid; c < 4 * dp4; c += kBandThreads)
      qv[c] = reinterpret_cast<const float *>(a.qrows + q * dp4)[c];
    if (tid == 0) {
      s_cnt = 0;
      s_thr = BandEntry{~0ull, ~0ull};
    }
    __syncthreads();
    const int nr = a.rlen[qc];
    const int32_t *rl = a.rlist + (a.rl_base ? a.rl_base[qc] : (int64_t)qc * a.Rs);
    // one member (a block-uniform number of calls): into the set when its
    // FP32 distance lies in the band
    auto member = [&](bool in, int64_t gp) {
      // the set is full when one of this step's additions made it so: each
      // thread judges by its own addition's place, so that the decision is
      // the same for all (the count itself may move on while others read it)
      int full = 0;
      if (in) {
        const float v =
            a.col_blocks
                ? band_dist2(qv, reinterpret_cast<const float *>(a.srows + col_block_at(gp, dp4)),
                             d, kColStride)
                : band_dist2(qv, reinterpret_cast<const float *>(a.srows + gp * dp4), d);
        if (v >= lo && v <= hi) {
          const int32_t id = a.sidx[gp];
          const double w =
              dist2_f64(qv, reinterpret_cast<const float *>(a.rrows + (int64_t)id * dp4), d);
          evals++;
          const BandEntry e{(unsigned long long)__double_as_longlong(w), make_key(v, id)};
          if (band_entry_less(e, s_thr)) {
            const int at = atomicAdd(&s_cnt, 1);
            ent[at] = e;
            full = at + 1 > kBandCap - kBandThreads;
          }
        }
      }
      if (__syncthreads_or(full)) band_cut(ent, &s_cnt, &s_thr, need);
    };
    // a thread per listed cluster, then the block over each cluster left
    for (int j0 = 0; j0 < nr; j0 += kBandThreads) {
      __syncthreads();
      if (tid == 0) s_nvis = 0;
      __syncthreads();
      if (j0 + tid < nr) {
        const int c = rl[j0 + tid];
        const float D =
            sqrtf(band_dist2(qv, reinterpret_cast<const float *>(a.sreps + (int64_t)c * dp4), d));
        const float slack = tol * (2.0f * D + 2.0f * th);
        if (!(D - a.cmax[c] > th + slack || D + th + slack < a.cmin[c])) {
          const int v = atomicAdd(&s_nvis, 1);
          s_vis[v] = c;
          s_D[v] = D;
        }
      }
      __syncthreads();
      const int nvis = s_nvis;
      for (int v = 0; v < nvis; v++) {  // block-uniform
        const int c = s_vis[v];
        const int start = a.soff[c], n_c = a.soff[c + 1] - start;
        if (narrow) {
          // members in block order: a warp per block of 32, by its box
          for (int c0 = 0; c0 < n_c; c0 += kBandThreads) {
            const int p = c0 + tid;
            bool in = p < n_c;
            if (in && a.boxes) {
              const float *b = reinterpret_cast<const float *>(
                  a.boxes + (block_slot(start, c) + (p >> 5)) * 2 * dp4);
              float acc = 0.0f;
              for (int e = 0; e < d; e++) {
                const float g =
                    fmaxf(fmaxf(__fsub_rn(b[e], qv[e]), __fsub_rn(qv[e], b[4 * dp4 + e])), 0.0f);
                acc = __fmaf_rn(g, g, acc);
              }
              in = !(acc > hi);
            }
            member(in, (int64_t)start + p);
          }
          continue;
        }
        const float D = s_D[v], slack = tol * (2.0f * D + 2.0f * th);
        const float lo_e = D - th - slack, hi_e = D + th + slack;
        int p0 = 0, p1 = n_c;  // first member with d(s, Rc) >= lo_e
        while (p0 < p1) {
          const int md = (p0 + p1) >> 1;
          if (a.sdist[start + md] < lo_e) p0 = md + 1;
          else p1 = md;
        }
        for (int c0 = p0; c0 < n_c; c0 += kBandThreads) {  // block-uniform
          const int p = c0 + tid;
          const bool past = p >= n_c || a.sdist[start + p] > hi_e;
          const int any_past = __syncthreads_or(past);
          member(!past, (int64_t)start + p);
          if (any_past) break;
        }
      }
    }
    band_cut(ent, &s_cnt, &s_thr, need);
    // the band's share of the result, in FP32 key order
    const int got = s_cnt;  // == need: the scan's own band keys are all found again
    int P = 1;
    while (P < got) P <<= 1;
    for (int i = got + tid; i < P; i += kBandThreads) ent[i] = BandEntry{~0ull, ~0ull};
    __syncthreads();
    band_sort<true>(ent, P);
    const int32_t base = a.qc_ref_base ? (int32_t)a.qc_ref_base[qc] : 0;
    for (int t = tid; t < need; t += kBandThreads) {
      const uint64_t key = t < got ? ent[t].key : kKeyMax;
      const bool none = key == kKeyMax;
      oi[nlo + t] = none ? -1 : key_idx(key) - base;
      od[nlo + t] =
          none ? __int_as_float(0x7f800000) : (a.squared ? key_d2(key) : sqrtf(key_d2(key)));
    }
  }
  if (a.counters) {
    for (int o = 16; o > 0; o >>= 1) evals += __shfl_xor_sync(kFull, evals, o);
    if ((tid & 31) == 0 && evals) atomicAdd(a.counters + 5, evals);
    if (blockIdx.x == 0 && tid == 0) atomicAdd(a.counters + 6, (unsigned long long)total);
  }
}

static int launch_band_resolve(const ScanArgs &a, int num_sms, cudaStream_t s) {
  const size_t smem = kBandCap * sizeof(BandEntry) + (size_t)a.dp4 * sizeof(float4);
  if (smem > 48 * 1024)
    KNN_CUDA_TRY(cudaFuncSetAttribute(band_resolve_kernel,
                                      cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // a persistent grid over the list, whose length only the device knows
  // (an empty list costs one launch that returns at once)
  band_resolve_kernel<<<2 * num_sms, kBandThreads, smem, s>>>(a);
  KNN_LAUNCH_CHECK();
  return KNN_OK;
}

static int launch_scan_kernels(const ScanArgs &a, int num_sms, cudaStream_t s);

// The scan of one batch of query slots, then the band kernel for the queries
// whose k-th boundary the scan left open.
int launch_scan(const ScanArgs &a, int num_sms, cudaStream_t s) {
  if (a.m == 0) return KNN_OK;
  if (!a.rrows || !a.unres_slot || !a.unres_count) {
    set_error("scan: the FP64 boundary buffers are missing");
    return KNN_EINTERNAL;
  }
  KNN_CUDA_TRY(cudaMemsetAsync(a.unres_count, 0, sizeof(unsigned), s));
  if (a.far_slot) KNN_CUDA_TRY(cudaMemsetAsync(a.far_count, 0, sizeof(unsigned), s));
  int rc = launch_scan_kernels(a, num_sms, s);
  if (rc == KNN_OK && a.far_slot) {
    ScanArgs f = a;
    f.slot_list = a.far_slot;
    f.slot_count = a.far_count;
    f.far_slot = nullptr;
    f.m = std::min<int64_t>(a.m, kFarQueries);
    f.split_max = INT_MAX;
    KNN_CUDA_TRY(cudaMemsetAsync(a.work_counter, 0, sizeof(unsigned long long), s));
    rc = launch_scan_kernels(f, num_sms, s);
  }
  if (rc != KNN_OK) return rc;
  return launch_band_resolve(a, num_sms, s);
}

static int launch_scan_kernels(const ScanArgs &a, int num_sms, cudaStream_t s) {
  // group scan: k <= 32, rows of at most 8 floats, and enough queries that
  // groups of 32 fill the chip -- below that a warp per query has 32 times the
  // warps in flight.  Self-joins of d = 3 blobs, search in us, group / warp:
  // k = 16: 10,000 points 139 / 68, 32,000 231 / 193, 50,000 246 / 301,
  // 100,000 395 / 635, 10^6 2220 / 8271; k = 1: 10,000 61 / 51, 16,000 70 / 74,
  // 32,000 84 / 137; k = 32: 50,000 301 / 336.
  // The queries must also lie close together, against the reference points: the
  // box of 32 distant ones reaches blocks that none of them needs, the more so
  // the more dimensions there are.  Whole joins in us, group / warp, n reference
  // rows by m queries, uniform points unless said otherwise: d = 3, k = 16,
  // 150,000 by 40,000 741 / 658 (mixtures 775 to 895 / 673 to 716), 100,000 by 50,000
  // 690 / 676, k = 4 558 / 621; d = 4, k = 16, 100,000 by 50,000 1202 / 826, 60,000
  // by 60,000 1073 / 850, 150,000 by 150,000 1542 / 1751; k = 4, 60,000 by themselves d = 5 1350 / 844, d = 6 2296 / 1171,
  // d = 8 5592 / 2453 (200 mixtures 546 / 537); d = 8, k = 4, 20,000 by 200,000
  // 4817 / 5682 (8 mixtures 1388 / 2569); d = 6, k = 4, 64 clouds of 2,000 704
  // / 1017 (8 mixtures 380 / 618); d = 2, k = 4, 100,000 by 50,000 446 / 560.
  const int64_t fill = (int64_t)num_sms * 32 * (a.k == 1 ? 3 : 8);
  const int group_k = a.d <= 4 ? 32 : (a.d <= 6 ? 8 : 4);
  const bool tiny = a.n_ref <= 100 * (int64_t)a.Rs;  // clusters of a few blocks
  const bool dense = a.d <= 3   ? 2 * a.m_near >= a.n_ref
                     : a.d == 4 ? tiny || 4 * a.m_near >= (a.m >= 2 * fill ? 3 : 8) * a.n_ref
                                : tiny || a.m_near >= 4 * a.n_ref;
  // thread per query: the self-join's k = 1 in clusters of at most 128 points on
  // average, from 8,192 queries on (5,000: d = 5 to 8 232 to 273 us by warps, 238
  // to 252 by threads; 10,000, d = 8 371 and 285).  Other queries' nearest point
  // is not in hand at once: 30,000 by 25,000 group 839 us, thread 1347.
  if (a.k == 1 && a.qrows == a.rrows && a.d > 4 && a.dp4_tmpl == 2 && a.dorder &&
      a.m >= 8192 && a.n_ref <= 128 * (int64_t)a.Rs) {
    thread_scan_kernel<2><<<(unsigned)((a.m + 255) / 256), 256, 0, s>>>(a);
    KNN_LAUNCH_CHECK();
    return KNN_OK;
  }
  if (a.k <= group_k && a.m >= fill && dense && a.slot_cl && (a.dp4_tmpl == 1 || a.dp4_tmpl == 2)) {
    if (a.dp4_tmpl == 1)
      return a.idx_in_row ? launch_group_scan<1, true>(a, num_sms, s)
                          : launch_group_scan<1, false>(a, num_sms, s);
    return a.idx_in_row ? launch_group_scan<2, true>(a, num_sms, s)
                        : launch_group_scan<2, false>(a, num_sms, s);
  }
  switch (a.dp4_tmpl) {
    case 1: return a.idx_in_row ? launch_scan_n<1, true>(a, num_sms, s)
                                : launch_scan_n<1, false>(a, num_sms, s);
    case 2: return a.idx_in_row ? launch_scan_n<2, true>(a, num_sms, s)
                                : launch_scan_n<2, false>(a, num_sms, s);
    case 4: return launch_scan_l<4, false, false>(a, num_sms, s);
    case 8: return launch_scan_l<8, false, false>(a, num_sms, s);
    default: return launch_scan_l<0, false, false>(a, num_sms, s);
  }
}

}  // namespace knnsweet
