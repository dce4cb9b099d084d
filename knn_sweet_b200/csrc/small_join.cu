// small_join.cu -- joins of a few thousand narrow rows in three kernels.
//
// Clustering a small reference set costs more than it saves: some twenty
// launches (draw, scores, assignment, sort, offsets, bounds, ...) of a few
// microseconds each for a search of thirty.  Up to kSmallRows reference rows
// of at most 8 floats, the set is taken as one cluster: one kernel packs the
// rows, orders them along a Morton curve and writes the bounding boxes of the
// blocks of 32 (and packs the queries and sets the exactness flags), and the
// scan then runs a warp per query over the blocks, nearest box first, with
// the starting bound infinite.  Same arithmetic, same boundary in FP64, same
// result as the clustered join (the reference, which has no such path, spends
// its own small-M branch on splitting a query over threads,
// src/knnjoin.cu:859-979).
//
// What bounds it: launch and dependent-load latency.  1,000-point self-join,
// k = 16: 131 -> 42 us (5 launches instead of 23: the preparation 11 us, the
// scan 16); 3,001 by 1,500, k = 1: 274 -> 59; 4,000 by 16,000, k = 100: 364 ->
// 141 (clustered at the left; the gain shrinks towards the limits below).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "pipeline.cuh"

namespace knnsweet {

namespace {

constexpr int kSmallRows = 4096;       // reference rows (one block orders them)
constexpr int64_t kSmallQueries = 16384;
constexpr int kPrepThreads = 1024;

// What the scan reads of the one cluster, in one allocation.
struct SmallCtl {
  float4 rep[2];     // its representative: the origin (its radius is infinite)
  float theta0, cmin, cmax;
  int32_t soff[2], rlist, rlen;
  int inexact;
};

__device__ __forceinline__ bool not_small_integer(float v, float bound) {
  return !(v == rintf(v) && fabsf(v) <= bound);
}

// Block 0: the reference side.  The others: the queries of a cross join.
// q: null for a self-join; qp / rp: packed rows, or the input itself.
template <int DP4>
__global__ void __launch_bounds__(kPrepThreads)
    small_prep_kernel(const float *__restrict__ r, int n, int d, bool idx_in_row, float bound,
                      const float *__restrict__ q, int64_t m, float4 *rp, float4 *qp,
                      float4 *__restrict__ srows, int32_t *__restrict__ sidx,
                      float4 *__restrict__ boxes, SmallCtl *__restrict__ ctl, int *inexact_q) {
  constexpr int C = 4 * DP4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float inf = __int_as_float(0x7f800000);
  if (blockIdx.x > 0) {
    bool bad = false;
    for (int64_t i = (int64_t)(blockIdx.x - 1) * kPrepThreads + tid; i < m;
         i += (int64_t)(gridDim.x - 1) * kPrepThreads) {
      float x[C];
#pragma unroll
      for (int c = 0; c < C; c++) {
        x[c] = c < d ? q[i * d + c] : 0.0f;
        bad |= not_small_integer(x[c], bound);
      }
      if (qp) {
#pragma unroll
        for (int e = 0; e < DP4; e++)
          qp[i * DP4 + e] = make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
      }
    }
    if (__any_sync(kFull, bad) && lane == 0) atomicOr(inexact_q, 1);
    return;
  }
  __shared__ uint32_t key[kSmallRows];
  __shared__ float s_lo[C], s_hi[C];
  __shared__ float w_lo[32][C], w_hi[32][C];
  // pack, check, bounding box
  bool bad = false;
  float lo[C], hi[C];
#pragma unroll
  for (int c = 0; c < C; c++) lo[c] = inf, hi[c] = -inf;
  for (int i = tid; i < n; i += kPrepThreads) {
    float x[C];
#pragma unroll
    for (int c = 0; c < C; c++) {
      x[c] = c < d ? r[(int64_t)i * d + c] : 0.0f;
      bad |= not_small_integer(x[c], bound);
      lo[c] = fminf(lo[c], x[c]);  // ignores NaN
      hi[c] = fmaxf(hi[c], x[c]);
    }
    if (rp) {
#pragma unroll
      for (int e = 0; e < DP4; e++)
        rp[(int64_t)i * DP4 + e] = make_float4(x[4 * e], x[4 * e + 1], x[4 * e + 2], x[4 * e + 3]);
    }
  }
#pragma unroll
  for (int c = 0; c < C; c++) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lo[c] = fminf(lo[c], __shfl_xor_sync(kFull, lo[c], o));
      hi[c] = fmaxf(hi[c], __shfl_xor_sync(kFull, hi[c], o));
    }
    if (lane == 0) {
      w_lo[warp][c] = lo[c];
      w_hi[warp][c] = hi[c];
    }
  }
  const int any_bad = __syncthreads_or(bad);
  if (tid < C) {
    float l = inf, h = -inf;
    for (int w = 0; w < kPrepThreads / 32; w++) {
      l = fminf(l, w_lo[w][tid]);
      h = fmaxf(h, w_hi[w][tid]);
    }
    s_lo[tid] = l;
    s_hi[tid] = h;
  }
  if (tid == 0) {
    ctl->rep[0] = ctl->rep[1] = make_float4(0.f, 0.f, 0.f, 0.f);
    ctl->theta0 = inf;
    ctl->cmin = 0.0f;
    ctl->cmax = inf;
    ctl->soff[0] = 0;
    ctl->soff[1] = n;
    ctl->rlist = 0;
    ctl->rlen = 1;
    ctl->inexact = any_bad ? 1 : 0;
  }
  __syncthreads();
  // Morton keys (20 bits of code, the row), sorted
  const int bits = min(10, 20 / d);
  const float top = (float)((1 << bits) - 1);
  auto key_of = [&](int i) -> uint32_t {
    if (i >= n) return 0xffffffffu;
    uint32_t code = 0;
#pragma unroll
    for (int c = 0; c < C; c++)
      if (c < d) {
        const float ext = s_hi[c] - s_lo[c];
        const float x = (r[(int64_t)i * d + c] - s_lo[c]) * (ext > 0.0f ? top / ext : 0.0f);
        const int v = (int)fminf(fmaxf(x, 0.0f), top);  // (a NaN becomes 0)
        for (int b = 0; b < bits; b++) code |= (uint32_t)((v >> b) & 1) << (b * d + c);
      }
    return (code << 12) | (uint32_t)i;
  };
  auto order = [&](auto per) {
    constexpr int E = decltype(per)::value;
    uint32_t x[E];
#pragma unroll
    for (int e = 0; e < E; e++) x[e] = key_of(e * kPrepThreads + tid);
    block_sort(x, key);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < E; e++) key[E * tid + e] = x[e];
    __syncthreads();
  };
  if (n <= kPrepThreads) order(std::integral_constant<int, 1>());
  else if (n <= 2 * kPrepThreads) order(std::integral_constant<int, 2>());
  else order(std::integral_constant<int, 4>());
  // rows in that order, a warp per block of 32, and their boxes
  for (int b = warp; b < (n + 31) / 32; b += kPrepThreads / 32) {
    const int p = 32 * b + lane;
    const bool in = p < n;
    const int i = in ? (int)(key[p] & 4095u) : 0;
#pragma unroll
    for (int c = 0; c < C; c++) {
      const float x = in && c < d ? r[(int64_t)i * d + c] : 0.0f;
      lo[c] = in ? x : inf;
      hi[c] = in ? x : -inf;
    }
    if (in) {
#pragma unroll
      for (int e = 0; e < DP4; e++) {
        float4 v = make_float4(lo[4 * e], lo[4 * e + 1], lo[4 * e + 2], lo[4 * e + 3]);
        if (idx_in_row && e == DP4 - 1) v.w = __int_as_float(i);
        srows[(int64_t)p * DP4 + e] = v;
      }
      sidx[p] = i;
    }
#pragma unroll
    for (int c = 0; c < C; c++) {
      if (c < d) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          lo[c] = fminf(lo[c], __shfl_xor_sync(kFull, lo[c], o));
          hi[c] = fmaxf(hi[c], __shfl_xor_sync(kFull, hi[c], o));
        }
      } else {
        lo[c] = hi[c] = 0.0f;
      }
    }
    if (lane == 0) {
      float4 *x = boxes + (int64_t)b * 2 * DP4;
#pragma unroll
      for (int e = 0; e < DP4; e++) {
        x[e] = make_float4(lo[4 * e], lo[4 * e + 1], lo[4 * e + 2], lo[4 * e + 3]);
        x[DP4 + e] = make_float4(hi[4 * e], hi[4 * e + 1], hi[4 * e + 2], hi[4 * e + 3]);
      }
    }
  }
}

}  // namespace

// Whether a join takes this path: narrow rows, few of them, and no
// representative count asked for (then the clusters are what the caller
// wants to see in the statistics).  A warp with more than 512 results walks most
// of the blocks of a separated set without a bound to begin with, and there are
// half as many such warps: 4,096 rows of 10 distant groups, d = 8, k = 700, by
// themselves 453 us clustered, 681 here, 16,384 queries 1211 and 1961, 2,000 383
// and 450 (uniform rows 516 and 365); k = 500, 16,384 queries 1678 and 1648.
bool small_join_fits(int64_t m, int64_t n, int d, int k, const knn_options &o) {
  return d <= 8 && n >= 1 && n <= kSmallRows && m <= (k <= 512 ? kSmallQueries : 2048) &&
         o.qreps == 0 && o.sreps == 0;
}

// The join, on device pointers; `ctr` (kCtrCount counters, zeroed).  ev(i)
// records the event between the stages.
int small_join(const float *q, int64_t m, const float *r, int64_t n, int d, int k,
               int32_t *out_idx, float *out_dist, const knn_options &o, Arena &ar,
               unsigned long long *ctr, cudaStream_t s, cudaEvent_t built) {
  const bool self = q == r && m == n;
  const int dp4 = d <= 4 ? 1 : 2;
  const bool idx_in_row = 4 * dp4 > d;
  int dev = 0, num_sms = 148;
  KNN_CUDA_TRY(cudaGetDevice(&dev));
  KNN_CUDA_TRY(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
  auto in_place = [&](const float *x) {
    return 4 * dp4 == d && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
  };
  const bool pack_r = !in_place(r), pack_q = !self && !in_place(q);
  // one allocation: rows in block order, packed rows, boxes, control, indices
  const int64_t nblk = (n + 31) / 32;
  const int64_t f4 = n * dp4 + (pack_r ? n * dp4 : 0) + (pack_q ? m * dp4 : 0) + nblk * 2 * dp4;
  float4 *base;
  KNN_TRY(ar.alloc(&base, (size_t)(f4 + (sizeof(SmallCtl) + 15) / 16 + (n + m + 3) / 4 + 1)));
  float4 *srows = base, *next = base + n * dp4;
  float4 *rp = nullptr, *qp = nullptr;
  if (pack_r) rp = next, next += n * dp4;
  if (pack_q) qp = next, next += m * dp4;
  float4 *boxes = next;
  next += nblk * 2 * dp4;
  SmallCtl *ctl = reinterpret_cast<SmallCtl *>(next);
  next += (sizeof(SmallCtl) + 15) / 16;
  int32_t *sidx = reinterpret_cast<int32_t *>(next), *unres = sidx + n;

  int *inexact_q = reinterpret_cast<int *>(ctr + kCtrInexactQ);
  const float bound = floorf(sqrtf(16777216.0f / (float)d) * 0.5f);
  const int qblocks = self ? 0 : (int)std::min<int64_t>(64, (m + kPrepThreads - 1) / kPrepThreads);
  auto kern = dp4 == 1 ? small_prep_kernel<1> : small_prep_kernel<2>;
  kern<<<1 + qblocks, kPrepThreads, 0, s>>>(r, (int)n, d, idx_in_row, bound, self ? nullptr : q, m,
                                            rp, qp, srows, sidx, boxes, ctl, inexact_q);
  KNN_LAUNCH_CHECK();
  if (built) KNN_CUDA_TRY(cudaEventRecord(built, s));
  ScanArgs a{};
  const float4 *Rp = pack_r ? rp : reinterpret_cast<const float4 *>(r);
  a.qrows = self ? Rp : (pack_q ? qp : reinterpret_cast<const float4 *>(q));
  a.m = m;
  a.d = d;
  a.dp4 = a.dp4_tmpl = dp4;
  a.k = k;
  a.idx_in_row = idx_in_row;
  a.squared = (o.flags & KNN_SQUARED_DIST) != 0;
  a.qreps = a.sreps = ctl->rep;
  a.srows = srows;
  a.boxes = boxes;
  a.sidx = sidx;
  a.soff = ctl->soff;
  a.cmin = &ctl->cmin;
  a.cmax = &ctl->cmax;
  a.theta0 = &ctl->theta0;
  a.rlist = &ctl->rlist;
  a.rlen = &ctl->rlen;
  a.Rs = 1;
  a.rrows = Rp;
  a.inexact_r = &ctl->inexact;
  a.inexact_q = self ? &ctl->inexact : inexact_q;
  a.out_idx = out_idx;
  a.out_dist = out_dist;
  a.unres_slot = unres;
  a.unres_count = reinterpret_cast<unsigned *>(ctr + kCtrUnres);
  a.work_counter = ctr + kCtrWork;
  a.counters = ctr + kCtrScan;
  return launch_scan(a, num_sms, s);
}

}  // namespace knnsweet
