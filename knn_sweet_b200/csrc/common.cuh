// common.cuh -- shared device/host helpers of libknnsweet.
//
// Ordering key of a candidate neighbour: the 64-bit word
//     (float bits of the FP32 squared distance) << 32 | reference index.
// Squared distances are non-negative, so their IEEE bit patterns order like
// the values, and the word orders pairs by (distance, index): ties at equal
// distance go to the lower index.  The reference ranks by the square-rooted
// distance with strict-less insertion (src/knnjoin.cu:815-820), which keeps
// whichever tied point it visited first; the index tie-break makes the
// result deterministic.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "../../include/knnsweet.h"

namespace knnsweet {

constexpr uint64_t kKeyMax = ~0ull;
constexpr unsigned kFull = 0xffffffffu;

__host__ __device__ __forceinline__ uint64_t make_key(float d2, int32_t idx) {
#ifdef __CUDA_ARCH__
  return ((uint64_t)__float_as_uint(d2) << 32) | (uint32_t)idx;
#else
  uint32_t b;
  memcpy(&b, &d2, 4);
  return ((uint64_t)b << 32) | (uint32_t)idx;
#endif
}

__device__ __forceinline__ float key_d2(uint64_t key) {
  return __uint_as_float((uint32_t)(key >> 32));
}
__device__ __forceinline__ int32_t key_idx(uint64_t key) {
  return (int32_t)(uint32_t)(key & 0xffffffffu);
}

// Relative slack that covers FP32 rounding in the distances entering a
// triangle-inequality bound: every computed distance is within (d+4) units
// of 2^-24 of its exact value; bounds are widened by 4x that.
__host__ __device__ __forceinline__ float bound_tol(int d) {
  return (float)(4 * d + 16) * 5.9604645e-8f;
}

// FP32 rounding band of a k-th squared distance Dk.  A squared distance
// computed in FP32 (one rounding per difference, the square fused into an
// fma accumulating non-negative terms in dimension order) is within (d + 2)
// units of 2^-24 (relative) of the exact value of the same FP32 inputs.  So
// a point whose FP32 value lies above band_hi(Dk) is farther, exactly and in
// FP64, than every point at or below Dk, and a point below band_lo(Dk) is
// nearer than every point at or above Dk: only points inside the band can
// rank differently in FP32 and in FP64.  The half-width (2d + 12) units covers
// both values' errors with 8 units to spare for FP64 rounding and the band's
// own arithmetic (rounded outward).
__device__ __forceinline__ float band_hi(float D, int d) {
  return __fmul_ru(D, __fadd_ru(1.0f, (float)(2 * d + 12) * 5.9604645e-8f));
}
__device__ __forceinline__ float band_lo(float D, int d) {
  return __fmul_rd(D, __fsub_rd(1.0f, (float)(2 * d + 12) * 5.9604645e-8f));
}

// FP64 squared distance of the first d coordinates of two rows, in dimension
// order, each product and sum rounded separately -- the arithmetic of the
// FP64 brute-force join the results are checked against.
__device__ __forceinline__ double dist2_f64(const float *__restrict__ a,
                                            const float *__restrict__ b, int d) {
  double acc = 0.0;
  for (int c = 0; c < d; c++) {
    const double t = __dsub_rn((double)a[c], (double)b[c]);
    acc = __dadd_rn(acc, __dmul_rn(t, t));
  }
  return acc;
}

// (FP64 squared distance, index) order: ties go to the lower index.
__device__ __forceinline__ bool f64_key_less(double da, int32_t ia, double db, int32_t ib) {
  return da < db || (da == db && ia < ib);
}

// FP32 squared distance of two padded rows of DP4 float4 (pad lanes are 0 in
// both rows, so they add exactly 0), summed in dimension order with fma.
template <int DP4>
__device__ __forceinline__ float dist2_rows(const float4 (&a)[DP4],
                                           const float4 *__restrict__ b) {
  float acc = 0.0f;
#pragma unroll
  for (int c = 0; c < DP4; c++) {
    float4 v = b[c];
    float t;
    t = __fsub_rn(a[c].x, v.x); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(a[c].y, v.y); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(a[c].z, v.z); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(a[c].w, v.w); acc = __fmaf_rn(t, t, acc);
  }
  return acc;
}

// Same on two rows in memory with a runtime chunk count.
__device__ __forceinline__ float dist2_rows_rt(const float4 *__restrict__ a,
                                               const float4 *__restrict__ b,
                                               int dp4) {
  float acc = 0.0f;
  for (int c = 0; c < dp4; c++) {
    float4 u = a[c];
    float4 v = b[c];
    float t;
    t = __fsub_rn(u.x, v.x); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(u.y, v.y); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(u.z, v.z); acc = __fmaf_rn(t, t, acc);
    t = __fsub_rn(u.w, v.w); acc = __fmaf_rn(t, t, acc);
  }
  return acc;
}

// ---------------------------------------------------------------------------
// Nearest representative of P points per thread.  The representatives lie in
// shared memory by coordinate, negated (stage_reps), so that four of them come
// with one 16-byte broadcast read per coordinate and their distances are
// packed FP32 pairs -- each rounded as dist2_rows rounds it.  The running
// minimum moves once per four representatives (their minimum first); which of
// the four it was is found again at the end, so that a representative costs
// three packed operations (d = 3) and 1.5 others, not six and three.
// ---------------------------------------------------------------------------
// Rows reps[0..cnt) of DP4 float4 into s (4 DP4 coordinates, `stride` floats
// each, a multiple of four >= cnt); up to three rows of NaN, which are nearest
// to nothing, fill the last four.
template <int DP4>
__device__ __forceinline__ void stage_reps(const float4 *__restrict__ reps, int cnt, float *s,
                                           int stride) {
  const int full = (cnt + 3) & ~3;
  const float nan = __int_as_float(0x7fffffff);
  for (int e = threadIdx.x; e < full * DP4; e += blockDim.x) {
    const int r = e / DP4, c = e - r * DP4;
    const float4 v = r < cnt ? reps[(int64_t)r * DP4 + c] : make_float4(nan, nan, nan, nan);
    s[(4 * c) * stride + r] = -v.x;
    s[(4 * c + 1) * stride + r] = -v.y;
    s[(4 * c + 2) * stride + r] = -v.z;
    s[(4 * c + 3) * stride + r] = -v.w;
  }
}

template <int DP4, int P>
struct NearestRep {
  float q[P][4 * DP4];
  float best[P];
  int quad[P];  // first of the four representatives that hold the minimum

  __device__ __forceinline__ void load(int i, const float4 *__restrict__ row) {
#pragma unroll
    for (int c = 0; c < DP4; c++) {
      const float4 v = row ? row[c] : make_float4(0.f, 0.f, 0.f, 0.f);
      q[i][4 * c] = v.x;
      q[i][4 * c + 1] = v.y;
      q[i][4 * c + 2] = v.z;
      q[i][4 * c + 3] = v.w;
    }
    best[i] = __int_as_float(0x7f7fffff);  // FLT_MAX
    quad[i] = -1;
  }
  // squared distances to representatives j .. j+3
  __device__ __forceinline__ void four(int i, const float *s, int stride, int j,
                                       float (&v)[4]) const {
    float2 v01, v23;
#pragma unroll
    for (int c = 0; c < 4 * DP4; c++) {
      const float4 r = *reinterpret_cast<const float4 *>(s + c * stride + j);
      const float2 qc = make_float2(q[i][c], q[i][c]);
      const float2 a = __fadd2_rn(qc, make_float2(r.x, r.y));
      const float2 b = __fadd2_rn(qc, make_float2(r.z, r.w));
      v01 = c == 0 ? __fmul2_rn(a, a) : __ffma2_rn(a, a, v01);
      v23 = c == 0 ? __fmul2_rn(b, b) : __ffma2_rn(b, b, v23);
    }
    v[0] = v01.x;
    v[1] = v01.y;
    v[2] = v23.x;
    v[3] = v23.y;
  }
  // representatives base .. base + cnt - 1, staged at s
  __device__ __forceinline__ void scan(const float *s, int stride, int cnt, int base) {
    for (int j = 0; j < cnt; j += 4) {
#pragma unroll
      for (int i = 0; i < P; i++) {
        float v[4];
        four(i, s, stride, j, v);
        const float m = fminf(fminf(v[0], v[1]), fminf(v[2], v[3]));  // ignores NaN
        if (m < best[i]) {
          best[i] = m;
          quad[i] = base + j;
        }
      }
    }
  }
};

// The first of representatives quad .. quad+3 (of R) whose squared distance to
// `row` is `best`: the lowest index on ties.  quad < 0 (no distance was a
// number): representative 0, a valid cluster.
template <int DP4>
__device__ __forceinline__ int nearest_of_quad(const float4 *__restrict__ row,
                                               const float4 *__restrict__ reps, int R, int quad,
                                               float best) {
  if (quad < 0) return 0;
  float4 p[DP4];
#pragma unroll
  for (int c = 0; c < DP4; c++) p[c] = row[c];
  int b = quad;
#pragma unroll
  for (int u = 3; u >= 0; u--)
    if (quad + u < R && dist2_rows<DP4>(p, reps + (int64_t)(quad + u) * DP4) == best) b = quad + u;
  return b;
}

// A start for a walk up a sorted array towards the first a[i] >= v: a
// position lo with a[i] < v for every i < lo and that first element at most
// 31 places further on.  32-ary search: each round the lanes sample 32 evenly
// spaced positions and a ballot brackets the answer, so that a list of a few
// thousand members needs one dependent load instead of some eleven; the level
// that would find the element itself is left out (a load round trip less), as
// the walk's own range test skips the few elements below v.  Called by all 32
// lanes with the same arguments.
__device__ __forceinline__ int warp_lower_bound_coarse(const float *__restrict__ a, int n,
                                                       float v, int lane) {
  int lo = 0, hi = n;
  while (hi - lo > 32) {
    const int step = (hi - lo + 31) >> 5;
    const int p = lo + (lane + 1) * step - 1;
    const int c = __popc(__ballot_sync(kFull, (p < hi) && (a[p] < v)));
    if (step <= 32) return lo + c * step;
    const int nhi = lo + (c + 1) * step - 1;
    lo += c * step;
    hi = nhi < hi ? nhi : hi;
  }
  return lo;
}

// Ascending sort of the E * blockDim.x keys that the block's threads hold (key
// E t + e in x[e] of thread t; blockDim.x a power of two, at least 32): a
// bitonic network whose strides inside a thread and inside a warp stay in
// registers, so that only strides of 32 E keys or more go through shared
// memory (sm: E * blockDim.x keys) -- 6 of 55 stages for 1,024 keys in 256
// threads.  Every thread of the block calls it.
template <int E, class T>
__device__ __forceinline__ void block_sort(T (&x)[E], T *sm) {
  const int t = threadIdx.x, total = E * blockDim.x;
  for (int size = 2; size <= total; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride < E) {
#pragma unroll
        for (int e = 0; e < E; e++) {
#pragma unroll
          for (int f = 1; f < E; f <<= 1)
            if (stride == f && (e & f) == 0) {
              const bool up = ((E * t + e) & size) == 0;
              const T lo = min(x[e], x[e | f]), hi = max(x[e], x[e | f]);
              x[e] = up ? lo : hi;
              x[e | f] = up ? hi : lo;
            }
        }
        continue;
      }
      const bool shared = stride >= 32 * E;
      if (shared) {
        __syncthreads();
#pragma unroll
        for (int e = 0; e < E; e++) sm[E * t + e] = x[e];
        __syncthreads();
      }
#pragma unroll
      for (int e = 0; e < E; e++) {
        const int i = E * t + e;
        const T o = shared ? sm[i ^ stride] : __shfl_xor_sync(kFull, x[e], stride / E);
        const bool least = ((i & stride) == 0) == ((i & size) == 0);
        x[e] = least ? min(x[e], o) : max(x[e], o);
      }
    }
  }
}

// Per-thread last-error text (the C ABI never exits the process).
void set_error(const char *fmt, ...);
std::string &error_buffer();

// Per-thread count of kernels enqueued by the current call (reported in
// knn_stats.kernels_launched); every launch site ends in KNN_LAUNCH_CHECK.
int &launch_counter();
// The per-device stream-ordered pool the library draws its scratch from.
int scratch_pool(cudaMemPool_t *out);

}  // namespace knnsweet

#define KNN_CUDA_TRY(call)                                                   \
  do {                                                                       \
    cudaError_t e_ = (call);                                                 \
    if (e_ != cudaSuccess) {                                                 \
      ::knnsweet::set_error("%s failed: %s (%s:%d)", #call,                  \
                            cudaGetErrorString(e_), __FILE__, __LINE__);     \
      return e_ == cudaErrorMemoryAllocation ? KNN_ENOMEM : KNN_ECUDA;       \
    }                                                                        \
  } while (0)

#define KNN_LAUNCH_CHECK()                                                   \
  do {                                                                       \
    cudaError_t e_ = cudaGetLastError();                                     \
    if (e_ != cudaSuccess) {                                                 \
      ::knnsweet::set_error("kernel launch failed: %s (%s:%d)",              \
                            cudaGetErrorString(e_), __FILE__, __LINE__);     \
      return KNN_ECUDA;                                                      \
    }                                                                        \
    ++::knnsweet::launch_counter();                                          \
  } while (0)
