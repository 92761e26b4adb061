// common.cuh -- shared definitions of libgpm: status/error plumbing, the
// device graph handle, a counter-based RNG usable on host and device, and
// warp helpers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>

#include "gpm.h"

namespace gpm {

// ---------------------------------------------------------------- errors
void set_error(const std::string &msg);
int fail(int status, const std::string &msg);

#define GPM_CUDA(call)                                                          \
  do {                                                                          \
    cudaError_t e_ = (call);                                                    \
    if (e_ != cudaSuccess) {                                                    \
      return ::gpm::fail(e_ == cudaErrorMemoryAllocation ? GPM_ENOMEM : GPM_ECUDA, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));   \
    }                                                                           \
  } while (0)

#define GPM_TRY(expr)            \
  do {                           \
    int s_ = (expr);             \
    if (s_ != GPM_OK) return s_; \
  } while (0)

// Checks that a launch was accepted (configuration errors); execution errors
// surface at the next synchronising call.
#define GPM_LAUNCH_CHECK() GPM_CUDA(cudaGetLastError())

int ensure_device();

// ---------------------------------------------------------------- device buffers
// A per-thread pool of device blocks kept across calls.  While an ArenaScope
// is alive on a thread, DevBuf allocations of that thread come from the pool
// and go back to it when freed, so a repeated one-shot call (upload, prepare,
// count, download) performs no cudaMalloc/cudaFree after the first.  Only
// entry points that run all their work on one stream and synchronise it
// before returning open a scope, so a block is never reused while an earlier
// kernel still reads it.
struct Arena;
Arena *current_arena();
void *arena_get(Arena *a, size_t bytes, size_t *cap);
void arena_put(Arena *a, void *p, size_t cap);
struct ArenaScope {
  ArenaScope();
  ~ArenaScope();
  Arena *prev;
};

// Every other allocation comes from a process-wide pool of idle blocks, per
// device.  A block enters it only when no work can use it any more: the
// library's own calls run on the legacy default stream, which is waited for
// first; what a caller's stream, or a graph a caller has captured, may still use
// is released inside a DirectFree scope and goes back to the driver at once.
// So a block in the pool may go to any thread and stream.  At most kPoolBytes are
// kept per device, the longest idle make room for newer ones, and all are given
// back when an allocation fails or plans are dropped.  (A first
// triangle count on R-MAT 22 made 56 cudaMalloc and 37 cudaFree calls: 27 of
// its 37 ms.)
void *pool_get(size_t bytes, size_t *cap, int *dev);  // nullptr: out of memory (cudaGetLastError not cleared)
void pool_put(void *p, size_t cap, int dev);
void pool_trim();  // the current device's cached blocks back to the driver
// While one with `on` is alive on a thread, the thread's releases bypass the pool.
struct DirectFree {
  explicit DirectFree(bool on);
  ~DirectFree();
  bool on;
};
// May work on st still run when the legacy default stream has been waited for?
inline bool foreign_stream(cudaStream_t st) { return st != nullptr && st != cudaStreamLegacy; }

// Owning device allocation; move-only.
template <typename T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0;
  Arena *arena = nullptr;  // arena the block came from (nullptr: the process-wide pool)
  size_t cap = 0;          // bytes of the block
  int dev = 0;             // its device (process-wide pool)
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  DevBuf(DevBuf &&o) noexcept : p(o.p), n(o.n), arena(o.arena), cap(o.cap), dev(o.dev) {
    o.p = nullptr;
    o.n = 0;
    o.arena = nullptr;
  }
  DevBuf &operator=(DevBuf &&o) noexcept {
    if (this != &o) {
      reset();
      p = o.p;
      n = o.n;
      arena = o.arena;
      cap = o.cap;
      dev = o.dev;
      o.p = nullptr;
      o.n = 0;
      o.arena = nullptr;
    }
    return *this;
  }
  ~DevBuf() { reset(); }
  void reset() {
    if (p) {
      if (arena) arena_put(arena, p, cap);
      else pool_put(p, cap, dev);
    }
    p = nullptr;
    n = 0;
    arena = nullptr;
  }
  // Grows to at least count elements (contents not preserved).
  int reserve(size_t count) {
    if (count <= n && p) return GPM_OK;
    reset();
    size_t bytes = (count ? count : 1) * sizeof(T);
    if (Arena *a = current_arena()) {
      p = static_cast<T *>(arena_get(a, bytes, &cap));
      if (!p) return fail(GPM_ENOMEM, "device pool allocation of " + std::to_string(bytes) + " B failed");
      arena = a;
      n = count ? count : 1;
      return GPM_OK;
    }
    p = static_cast<T *>(pool_get(bytes, &cap, &dev));
    if (!p) return fail(GPM_ENOMEM, "cudaMalloc(" + std::to_string(bytes) + " B) failed: " +
                                        cudaGetErrorString(cudaGetLastError()));
    n = count ? count : 1;
    return GPM_OK;
  }
};

// Orders the launches of one handle over all streams: scratch of its plan holds
// positions and counters that two of them must not share.  The legacy default
// stream orders its own launches (two event calls per launch cost 4 us of host
// time).  A launch inside a capture cannot wait for one outside of it and
// stays out of the order.
bool stream_capturing(cudaStream_t st);
struct LaunchOrder {
  cudaEvent_t event = nullptr;
  enum { kNone, kLegacy, kEvent } last = kNone;  // where the latest launch went: kEvent, `event` is behind it
  LaunchOrder() = default;
  LaunchOrder(const LaunchOrder &) = delete;
  LaunchOrder &operator=(const LaunchOrder &) = delete;
  ~LaunchOrder() {
    if (event) cudaEventDestroy(event);
  }
  int record(cudaStream_t st) {
    if (!event) GPM_CUDA(cudaEventCreateWithFlags(&event, cudaEventDisableTiming));
    GPM_CUDA(cudaEventRecord(event, st));
    last = kEvent;
    return GPM_OK;
  }
  int begin(cudaStream_t st) {
    const bool foreign = foreign_stream(st);
    if (last == kNone || (last == kLegacy && !foreign) || stream_capturing(st)) return GPM_OK;
    if (last == kLegacy) GPM_TRY(record(cudaStreamLegacy));
    GPM_CUDA(cudaStreamWaitEvent(st, event, 0));
    return GPM_OK;
  }
  int end(cudaStream_t st) {
    if (!foreign_stream(st)) {
      last = kLegacy;
      return GPM_OK;
    }
    return stream_capturing(st) ? GPM_OK : record(st);
  }
};

// ---------------------------------------------------------------- RNG
// splitmix64 finaliser: a counter-based generator, so edge i of a seeded
// graph is the same whichever thread (host or device) draws it.
__host__ __device__ inline uint64_t mix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}
__host__ __device__ inline uint64_t draw(uint64_t seed, uint64_t stream, uint64_t i) {
  return mix64(mix64(seed ^ (stream * 0xD1B54A32D192ED03ull)) ^ i);
}
__host__ __device__ inline double unit(uint64_t r) { return (double)(r >> 11) * (1.0 / 9007199254740992.0); }
// uniform integer in [0, n) for n < 2^32
__host__ __device__ inline uint32_t below(uint64_t r, uint64_t n) {
  return (uint32_t)(((r >> 32) * n) >> 32);
}

// R-MAT edge i: one quadrant draw per bit level, standard recursion.
__host__ __device__ inline void rmat_edge(uint64_t seed, uint64_t i, int scale, double a, double b,
                                          double c, int32_t *u, int32_t *v) {
  uint32_t x = 0, y = 0;
  const double ab = a + b, abc = a + b + c;
  for (int l = 0; l < scale; ++l) {
    double r = unit(draw(seed, 1 + l, i));
    uint32_t bx = 0, by = 0;
    if (r < a) {
    } else if (r < ab) {
      by = 1;
    } else if (r < abc) {
      bx = 1;
    } else {
      bx = 1;
      by = 1;
    }
    x = (x << 1) | bx;
    y = (y << 1) | by;
  }
  *u = (int32_t)x;
  *v = (int32_t)y;
}

__host__ __device__ inline void er_edge(uint64_t seed, uint64_t i, int64_t n, int32_t *u, int32_t *v) {
  *u = (int32_t)below(draw(seed, 101, i), (uint64_t)n);
  *v = (int32_t)below(draw(seed, 102, i), (uint64_t)n);
}

// Chung-Lu endpoint: vertex index drawn with weight (i + i0)^(-alpha) by
// inverting the continuous CDF of the weight profile.
struct ChungLu {
  double alpha, i0, lo, span, inv;  // lo = i0^(1-alpha), span = (n+i0)^(1-alpha) - lo
  int64_t n;
};
__host__ __device__ inline int32_t chung_lu_vertex(const ChungLu &p, uint64_t r) {
  double q = p.lo + unit(r) * p.span;
  double x = pow(q, p.inv) - p.i0;
  int64_t k = (int64_t)x;
  if (k < 0) k = 0;
  if (k >= p.n) k = p.n - 1;
  return (int32_t)k;
}
ChungLu chung_lu_params(int64_t n, double gamma, double mean_deg);

// ---------------------------------------------------------------- warp helpers
__device__ __forceinline__ unsigned lane_id() { return threadIdx.x & 31u; }

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Warp tasks of a queue sorted heaviest first, handed out by an atomic cursor:
// the first `lone` one at a time, the others in runs of kTaskRun.  All grabs
// meet in one word of L2, about one per clock, so a million small tasks taken
// singly cost a third of a millisecond whatever they do (Erdos-Renyi, 10^6
// vertices of mean degree 12: 588 us per triangle count, 334 us in runs;
// R-MAT 22: 4.94 -> 4.86 ms).
constexpr int kTaskRun = 8;
struct WarpTasks {
  int t = -1;
  // the next task (at or past the queue's end when there is none)
  __device__ __forceinline__ int next(int *cursor, int lone, unsigned lane) {
    if (t < lone || ((t + 1 - lone) & (kTaskRun - 1)) == 0) {
      int u = 0;
      if (lane == 0) u = atomicAdd(cursor, 1);
      u = __shfl_sync(0xffffffffu, u, 0);
      t = u < lone ? u : lone + (u - lone) * kTaskRun;
    } else {
      ++t;
    }
    return t;
  }
};

// ---------------------------------------------------------------- graph handle
struct TcPlan;
struct RankPlan;
struct RankGraph;
struct LabelCsr;
struct MotifPlan;
struct CliquePlan;
struct MotifPlan;

}  // namespace gpm

struct gpm_graph {
  int64_t n = 0;
  int64_t nnz = 0;
  int32_t max_deg = 0;
  uint64_t sum_deg2 = 0;  // sum of the squared list lengths
  bool symmetric = false; // every stored entry has its reverse (built so, not oriented since)
  gpm::DevBuf<int32_t> odeg;  // oriented from a symmetric graph: each vertex's degree there (in + out degree now)
  double hash_us = 0;     // estimated time of gpm_tc's counts with the hash kernel (tc.cu)
  int oriented = 0;
  int relabeled = 0;
  int device = 0;
  bool foreign = false;  // launched on a caller's stream: its memory is released directly (DirectFree)
  gpm::DevBuf<int64_t> off;     // n + 1
  gpm::DevBuf<int32_t> adj;     // nnz
  gpm::DevBuf<int32_t> labels;  // n (optional)
  gpm::DevBuf<int32_t> src;     // nnz, COO source of each stored entry (lazy)
  bool src_filled = false;      // src has been filled, not only recorded into a capture
  gpm::TcPlan *tc = nullptr;    // cached triangle-count schedule (HASH)
  gpm::RankPlan *rank = nullptr; // cached schedule of the BITMAP path
  gpm::RankGraph *rg = nullptr;  // cached rank-relabelled copy
  gpm::RankPlan *learned = nullptr;  // plan chosen by the attached scheduler
  gpm::LabelCsr *lcsr = nullptr;     // label-partitioned lists (matching)
  gpm::MotifPlan *motif[2] = {nullptr, nullptr};  // cached motif pipelines (3-, 4-vertex)
  gpm::CliquePlan *clique[9] = {};                // cached k-clique schedules, by k
  gpm_sched *sched = nullptr;        // learned scheduler (not owned)
  gpm::DevBuf<uint64_t> result; // small device result scratch
  ~gpm_graph();
};

namespace gpm {
// graph.cu
int build_csr_device(gpm_graph *g, int64_t n, int64_t m, const int32_t *d_src,
                     const int32_t *d_dst, int symmetrize, cudaStream_t st);
int ensure_src(gpm_graph *g, cudaStream_t st);
bool src_ready(const gpm_graph *g);  // would ensure_src launch nothing?
int compute_max_degree(gpm_graph *g, cudaStream_t st);
void free_tc_plan(TcPlan *p);
void free_rank_plan(RankPlan *p);
void free_rank_graph(RankGraph *r);
void free_label_csr(LabelCsr *p);
void free_motif_plan(MotifPlan *p);  // motif.cu
void free_clique_plan(CliquePlan *p);  // clique.cu
// Drops every cached schedule (after the stored graph changed).
void drop_plans(gpm_graph *g);
int num_sms();

// A launch parameter (a persistent grid size, after the kernel's attributes
// are set) computed by `init` the first time it is needed on each device,
// with that device current: function attributes and SM counts are per
// device.
struct PerDevice {
  static constexpr int kDevices = 64;
  std::atomic<int> v[kDevices] = {};
  template <class F>
  int get(F init) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= kDevices) return init();
    int x = v[dev].load(std::memory_order_relaxed);
    if (!x) {
      x = init();
      v[dev].store(x, std::memory_order_relaxed);
    }
    return x;
  }
};
}  // namespace gpm
