// pipeline.cuh -- the stages of one join shared by the entry points
// (api.cu: single device; sharded.cu: several devices): scratch arenas, the
// device counter layout, the reference and query sides and the search.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <vector>

#include "common.cuh"
#include "kernels.cuh"

namespace knnsweet {

#define KNN_TRY(expr)        \
  do {                       \
    int rc_ = (expr);        \
    if (rc_ != KNN_OK) return rc_; \
  } while (0)

// Stream-ordered scratch: every allocation is released on the same stream
// when the arena goes out of scope.  Small arrays share slabs of kSlab bytes: a
// small join asks for some forty, and each allocation and release took the
// host 1 to 2 us.
class Arena {
  static constexpr size_t kSlab = 1u << 21, kAlign = 256;

 public:
  explicit Arena(cudaStream_t s) : s_(s) {}
  ~Arena() {
    for (void *p : ptrs_) cudaFreeAsync(p, s_);
  }
  Arena(const Arena &) = delete;
  Arena &operator=(const Arena &) = delete;

  // Hands the allocations made so far to the caller: they outlive the arena.
  std::vector<void *> take() {
    std::vector<void *> out;
    out.swap(ptrs_);
    left_ = 0;  // the slab went with them
    return out;
  }

  template <class T>
  int alloc(T **out, size_t count) {
    *out = nullptr;
    if (count == 0) count = 1;
    const size_t bytes = (count * sizeof(T) + kAlign - 1) & ~(kAlign - 1);
    if (bytes > kSlab / 4) {
      void *p = nullptr;
      const int rc = take_from_pool(bytes, &p);
      *out = static_cast<T *>(p);
      return rc;
    }
    if (bytes > left_) {
      void *p = nullptr;
      const int rc = take_from_pool(kSlab, &p);
      if (rc != KNN_OK) return rc;
      slab_ = static_cast<unsigned char *>(p);
      left_ = kSlab;
    }
    *out = reinterpret_cast<T *>(slab_);
    slab_ += bytes;
    left_ -= bytes;
    return KNN_OK;
  }

 private:
  int take_from_pool(size_t bytes, void **p) {
    if (!pool_) {
      const int rc = scratch_pool(&pool_);
      if (rc != KNN_OK) return rc;
    }
    cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool_, s_);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *p = nullptr;
      set_error("device allocation of %zu bytes failed: %s", bytes, cudaGetErrorString(e));
      return e == cudaErrorMemoryAllocation ? KNN_ENOMEM : KNN_ECUDA;
    }
    ptrs_.push_back(*p);
    return KNN_OK;
  }

  unsigned char *slab_ = nullptr;
  size_t left_ = 0;
  cudaStream_t s_;
  cudaMemPool_t pool_ = nullptr;
  std::vector<void *> ptrs_;
};

// Device counters of one call, zeroed at its start.
enum CtrSlot {
  kCtrWork = 0,                         // scan work counter
  kCtrScan = 1,                         // the scan statistics (kScanCounters)
  kCtrErr = kCtrScan + kScanCounters,   // device error flag (bounded waits)
  kCtrTileWork,                         // tile-search tile counter
  kCtrTile,                             // tile-search statistics (4)
  kCtrFallback = kCtrTile + 4,          // slots the tile search leaves to the scan
  kCtrUnres,                            // queries left to the band kernel
  kCtrInexactQ,                         // the query side is not small integers
  kCtrCount
};

// One clustered point set.
struct ClusterSet {
  int R = 0;
  float4 *reps = nullptr;     // R x dp4s
  int32_t *rep_rows = nullptr;
  uint64_t *skeys = nullptr;  // n sorted (cluster, distance) keys
  int32_t *perm = nullptr;    // sorted position -> input row
  int32_t *off = nullptr;     // R + 1
};

// Host destination of the result for the host-buffer entry point: the scan
// then runs in row chunks and each chunk's rows are copied back on `copy`
// while the next chunk is computed.  `done` tells whether the copies were
// enqueued (otherwise the caller copies the whole result).
struct HostSink {
  int32_t *idx;
  float *dist;
  cudaStream_t copy;
  bool done;
};

// The reference side of a join: representatives, clusters, the
// cluster-contiguous rows and their bounds.  Depends only on the reference
// set and the options that shape its clusters.
struct RefSide {
  int64_t n = 0;
  int d = 0, dp4s = 0, tmpl = 0, Rs = 0;
  bool idx_in_row = false, col_blocks = false;
  ClusterSet sset;
  const float4 *Rp = nullptr;  // packed rows, original order
  float4 *srows = nullptr;     // cluster-contiguous rows
  // narrow rows: slot -> row in block order (the order of srows and sidx; sdist
  // stays by distance) and the blocks' bounding boxes; null otherwise
  int32_t *order = nullptr;
  float4 *boxes = nullptr;
  float *sdist = nullptr, *cmin = nullptr, *cmax = nullptr;
  int32_t *sidx = nullptr;
  int *inexact = nullptr;      // device flag: 0 when the rows are small integers
};

// The query side of a join against a built reference side: query rows,
// query clusters, representative distances, the k-th bounds and the
// surviving reference clusters of every query cluster.
struct QuerySide {
  int Rq = 0;
  const float4 *Qp = nullptr;  // query rows (packed), original order
  ClusterSet qset;             // qset.perm: slot -> query row; qset.off: slots of a cluster
  const int32_t *order = nullptr;  // slot -> query row as the scans take it
  const int *inexact = nullptr;
  float *qrad = nullptr, *drr = nullptr, *theta0 = nullptr;
  int32_t *slot_cl = nullptr, *rlist = nullptr, *rlen = nullptr;
  float *rlb = nullptr;   // per list entry: d(Rq, Rs) less the radius of Rs
  float2 *clb = nullptr;  // per list chunk: first d(Rq, Rs), largest radius from it on
};

// Argument and option ranges shared by every entry point.
int check_sizes(int64_t m, int64_t n, int32_t d, int32_t k);
int check_options(const knn_options *opt, knn_options *o);
// Representative count for n points when the caller passes 0.
int default_reps(int64_t n);
// Number of query representatives for m queries.
int query_rep_count(const knn_options &o, int64_t m, int d, int k, bool self, int Rs);
// Builds the reference side of reference rows r (device); the arrays it keeps
// come from `keep`, scratch from `tmp`.
int build_ref_side(Arena &keep, Arena &tmp, const float *r, int64_t n, int d, int Rs,
                   const knn_options &o, bool copy_rows, int *dev_err, cudaStream_t s,
                   RefSide *R);
// Builds the query side of queries q (device) against R (share: the join is a
// self-join using R's clusters).
int build_query_side(const RefSide &R, bool share, const float *q, int64_t m, int32_t k,
                     const knn_options &o, Arena &ar, unsigned long long *ctr, cudaStream_t s,
                     QuerySide *Q);
// Searches the query clusters c0 .. c1-1 (slots slot0 .. slot0+nslot-1).
int search_clusters(const RefSide &R, const QuerySide &Q, int64_t m, int32_t k, int c0, int c1,
                    int64_t slot0, int64_t nslot, int32_t *out_idx, float *out_dist,
                    const knn_options &o, cudaStream_t s, HostSink *sink, Arena &ar,
                    unsigned long long *ctr);
// Small joins of narrow rows (small_join.cu): whether a join takes that path,
// and the join itself; `built` (or null) is recorded between its stages.
bool small_join_fits(int64_t m, int64_t n, int d, int k, const knn_options &o);
int small_join(const float *q, int64_t m, const float *r, int64_t n, int d, int k,
               int32_t *out_idx, float *out_dist, const knn_options &o, Arena &ar,
               unsigned long long *ctr, cudaStream_t s, cudaEvent_t built);
// Adds the device counters of one call to `st` (synchronises `s`).
int read_stats(const unsigned long long *ctr, cudaStream_t s, knn_stats *st);

}  // namespace knnsweet
