// motif.cu -- 3- and 4-vertex induced motif counts on a symmetric graph.
//
// The reference enumerates the six induced 4-vertex motifs edge by edge
// (Motif4_G2Miner, src/gpu_kernels/G2Miner_kernels.cuh:438-552); its loops
// visit every 3-star leaf triple, which costs sum over edges of d^2 on hub
// graphs.  The B200 path counts non-induced subgraphs instead and inverts the
// containment matrix (each induced 4-vertex graph contains a fixed number of
// copies of each smaller pattern):
//   S  = sum_v C(d_v,3)                          3-stars
//   P  = sum_e (d_a-1)(d_b-1) - 3T               4-paths
//   TT = sum_e t_e (d_a + d_b - 4) / 2           tailed triangles
//   C  = 4-cycles (highest-rank vertex + 2-hop counters)
//   D  = sum_e C(t_e,2)                          diamonds
//   K  = 4-cliques (clique kernel, k = 4)
//   k = K, d = D-6K, c = C-d-3K, tt = TT-4d-12K, p = P-2tt-4c-6d-12K,
//   s = S-tt-2d-4K
// where t_e is the number of triangles on edge e.  All sums are exact uint64
// (modular arithmetic, so the differences are exact whenever the induced
// counts fit in 64 bits).  3-vertex motifs: triangles T = sum t_e / 3, induced
// 2-paths = sum_v C(d_v,2) - 3T.
//
// Kernels run on the rank-relabelled graph (tc_rank.cuh); the upward part of
// each sorted list is the degree-oriented DAG.  Every kernel takes an
// optional per-vertex graph id so one launch serves a disjoint union of many
// graphs (batch.cu) with per-graph accumulators.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "motif.cuh"
#include "tc_rank.cuh"
#include "wedge.cuh"

namespace gpm {

static int grid_for(int64_t work, int block = 256) {
  int64_t g = (work + block - 1) / block;
  int64_t cap = (int64_t)num_sms() * 16;
  return (int)std::max<int64_t>(1, std::min(g, cap));
}

__device__ __forceinline__ unsigned long long choose2(unsigned long long d) {
  return d < 2 ? 0ull : (d & 1ull) ? d * ((d - 1) >> 1) : (d >> 1) * (d - 1);
}
__device__ __forceinline__ unsigned long long choose3(unsigned long long d) {
  if (d < 3) return 0ull;
  unsigned long long a = d, b = d - 1, c = d - 2;
  if (a % 2 == 0) a >>= 1; else b >>= 1;
  if (a % 3 == 0) a /= 3; else if (b % 3 == 0) b /= 3; else c /= 3;
  return a * b * c;
}

__device__ __forceinline__ int graph_of(const int32_t *gid, int64_t x) { return gid ? gid[x] : 0; }

// split[x] = first index of x's sorted list holding an id > x
__global__ void k_split(int64_t n, const int64_t *__restrict__ roff, const int32_t *__restrict__ radj,
                        int64_t *__restrict__ split) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = roff[x], hi = roff[x + 1];
    while (lo < hi) {
      int64_t mid = (lo + hi) >> 1;
      if (radj[mid] <= (int32_t)x) lo = mid + 1; else hi = mid;
    }
    split[x] = lo;
  }
}

// ------------------------------------------------------------ triangles per DAG edge
// The upward lists (doff, dadj).  Vertex task x, U = N+(x) held in a shared
// table.  For v in U (edge e1 = (x,v)) and w in N+(v) (edge e2 = (v,w)) with w
// in U (edge e3 = (x,w)): te[e1]++, te[e2]++, te[e3]++ -- every triangle once.
// e1 and e3 lie in x's own list: they are counted in shared memory by their
// position in it and added to te once per task, so a triangle costs one
// global atomic (R-MAT 18, 82 M triangles: three of four atomics of the former
// kernel's 114 M sectors).
constexpr int kTeWarpKeys = 128;  // a warp's table: tasks with |U| <= 128
constexpr int kTeCtaKeys = 8 * kTeWarpKeys;
constexpr int kTeLight = 16;      // warp tasks with at most this many neighbours are handed out in runs

// Table of up to KEYS keys of U, their positions, and the counts.
template <int KEYS>
struct TeTable {
  int32_t key[2 * KEYS];
  uint16_t pos[2 * KEYS];
  unsigned cnt[KEYS];
  static constexpr int kLog = KEYS == kTeWarpKeys ? 8 : 11;
  static_assert((1 << kLog) == 2 * KEYS, "slots are a power of two");
  __device__ __forceinline__ static uint32_t slot(int32_t k, int log) {
    return ((uint32_t)k * 2654435769u) >> (32 - log);
  }
  __device__ __forceinline__ int find(int32_t k, int log) const {
    const uint32_t mask = (1u << log) - 1u;
    uint32_t h = slot(k, log);
    while (true) {
      const int32_t s = key[h];
      if (s == k) return pos[h];
      if (s < 0) return -1;
      h = (h + 1) & mask;
    }
  }
  __device__ __forceinline__ void insert(int32_t k, int p, int log) {
    const uint32_t mask = (1u << log) - 1u;
    uint32_t h = slot(k, log);
    while (atomicCAS(&key[h], -1, k) != -1) h = (h + 1) & mask;
    pos[h] = (uint16_t)p;
  }
};
union TeShared {
  TeTable<kTeWarpKeys> warp[8];
  TeTable<kTeCtaKeys> cta;
};
__device__ __forceinline__ int ilog2ceil(int x) { return x <= 1 ? 0 : 32 - __clz(x - 1); }

// N+(v) up to kmax: where it can meet U
__device__ __forceinline__ void te_segment(const int64_t *__restrict__ doff, const int32_t *__restrict__ dadj,
                                           int32_t v, int32_t kmax, long long *st, int *len) {
  int64_t lo = doff[v], hi = doff[v + 1];
  *st = lo;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(dadj + mid) <= kmax) lo = mid + 1; else hi = mid;
  }
  *len = (int)(lo - *st);
}

__device__ __forceinline__ void te_warp_task(int32_t x, const int64_t *__restrict__ doff,
                                             const int32_t *__restrict__ dadj, unsigned *__restrict__ te,
                                             TeTable<kTeWarpKeys> &T, unsigned lane) {
  const int64_t s0 = doff[x];
  const int d = (int)(doff[x + 1] - s0);
  const int32_t kmax = dadj[s0 + d - 1];
  const int log = max(5, ilog2ceil(2 * d));
  for (int i = lane; i < (1 << log); i += 32) T.key[i] = -1;
  for (int i = lane; i < d; i += 32) T.cnt[i] = 0u;
  __syncwarp();
  for (int i = lane; i < d; i += 32) T.insert(dadj[s0 + i], i, log);
  __syncwarp();
  for (int j = 0; j < d; j += 32) {
    long long st = 0;
    int len = 0;
    if (j + (int)lane < d) te_segment(doff, dadj, dadj[s0 + j + lane], kmax, &st, &len);
    warp_segments(dadj, st, len, j, lane, [&](int32_t w, long long at, int seg) {
      const int p = T.find(w, log);
      if (p < 0) return;
      atomicAdd(&T.cnt[p], 1u);
      atomicAdd(&T.cnt[seg], 1u);
      atomicAdd(&te[at], 1u);
    });
  }
  __syncwarp();
  for (int i = lane; i < d; i += 32)
    if (T.cnt[i]) atomicAdd(&te[s0 + i], T.cnt[i]);
  __syncwarp();
}

// A task of any size by the CTA, kTeCtaKeys keys of U at a time.
__device__ __forceinline__ void te_cta_task(int32_t x, const int64_t *__restrict__ doff,
                                            const int32_t *__restrict__ dadj, unsigned *__restrict__ te,
                                            TeTable<kTeCtaKeys> &T, WedgeWalk &walk, int *turn) {
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int64_t s0 = doff[x];
  const int d = (int)(doff[x + 1] - s0);
  const int32_t kmax = dadj[s0 + d - 1];
  for (int c0 = 0; c0 < d; c0 += kTeCtaKeys) {
    const int ck = min(kTeCtaKeys, d - c0);
    const int log = max(5, ilog2ceil(2 * ck));
    for (int i = tid; i < (1 << log); i += nthr) T.key[i] = -1;
    for (int i = tid; i < ck; i += nthr) T.cnt[i] = 0u;
    __syncthreads();
    for (int i = tid; i < ck; i += nthr) T.insert(dadj[s0 + c0 + i], i, log);
    __syncthreads();
    // every v of U (all chunks) against this chunk's table
    cta_wedges(dadj, d, 64 * 512, walk, turn,
               [&](int i, long long *st, int *len) { te_segment(doff, dadj, dadj[s0 + i], kmax, st, len); },
               [&](int32_t w, long long at, int seg) {
                 const int p = T.find(w, log);
                 if (p < 0) return;
                 atomicAdd(&T.cnt[p], 1u);
                 const int q = seg - c0;
                 if (q >= 0 && q < ck) atomicAdd(&T.cnt[q], 1u);
                 else atomicAdd(&te[s0 + seg], 1u);
                 atomicAdd(&te[at], 1u);
               });
    for (int i = tid; i < ck; i += nthr)
      if (T.cnt[i]) atomicAdd(&te[s0 + c0 + i], T.cnt[i]);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(256) k_edge_tri(const int64_t *__restrict__ doff, const int32_t *__restrict__ dadj,
                                                  const int32_t *__restrict__ cta_tasks, int n_cta,
                                                  const int32_t *__restrict__ warp_tasks, int n_warp,
                                                  const int32_t *__restrict__ light_tasks, int n_light,
                                                  int *__restrict__ counters, unsigned *__restrict__ te) {
  __shared__ TeShared T;
  __shared__ WedgeWalk s_walk;
  __shared__ int s_task;
  int turn = 0;
  if (threadIdx.x == 0) s_walk.s[0].next = s_walk.s[0].nlong = 0;
  while (n_cta > 0) {
    if (threadIdx.x == 0) s_task = atomicAdd(&counters[0], 1);
    __syncthreads();
    int t = s_task;
    __syncthreads();
    if (t >= n_cta) break;
    te_cta_task(cta_tasks[t], doff, dadj, te, T.cta, s_walk, &turn);
  }
  const int wid = threadIdx.x >> 5;
  const unsigned lane = threadIdx.x & 31;
  // light tasks: dealt out in turn while a warp has few of them, else in runs
  const int warps = gridDim.x * 8;
  if (n_light <= 2 * kTaskRun * warps) {
    for (int t = blockIdx.x * 8 + wid; t < n_light; t += warps)
      te_warp_task(light_tasks[t], doff, dadj, te, T.warp[wid], lane);
    n_light = 0;
  }
  for (int light = 0; light < 2; ++light) {
    const int32_t *tasks = light ? light_tasks : warp_tasks;
    const int n = light ? n_light : n_warp;
    WarpTasks queue;
    while (n > 0) {
      const int t = queue.next(&counters[1 + light], light ? 0 : n, lane);
      if (t >= n) break;
      te_warp_task(tasks[t], doff, dadj, te, T.warp[wid], lane);
    }
  }
}

// ------------------------------------------------------------ per-edge / per-vertex sums
// acc[g*8 + 0] S, 1 A4 = sum (da-1)(db-1), 2 A1 = sum t, 3 A2 = sum C(t,2),
// 4 A3 = sum t(da+db-4), 5 K4, 6 C4, 7 sum C(d,2)
//
// A warp takes a run of consecutive blocks of up to 32 vertices, whose upward edges
// are consecutive too, keeps its sums in registers and adds them to the graph's
// totals when the run or the graph ends: one set of atomics per vertex, all on
// the same few words, took 1.87 ms for a batch of 2.2 M vertices and 35 M
// edges.
// span: vertices per block, a power of two up to 32, fewer where 32 each would
// leave SMs without a warp (complete graph of 300 vertices: 304 us in blocks of
// 32, 15 so).
__global__ void k_edge_sums(int64_t n, int span, const int64_t *__restrict__ roff, const int64_t *__restrict__ doff,
                            const int32_t *__restrict__ dadj, const unsigned *__restrict__ te,
                            const int32_t *__restrict__ gid, unsigned long long *__restrict__ acc) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = lane_id();
  const int64_t blocks = (n + span - 1) / span, run = (blocks + nw - 1) / nw;
  unsigned long long s = 0, c2 = 0, a4 = 0, a1 = 0, a2 = 0, a3 = 0;
  int g = -1;
  auto flush = [&]() {
    if (g < 0) return;
    unsigned long long *A = acc + 8 * (int64_t)g;
    unsigned long long v[6] = {s, a4, a1, a2, a3, c2};
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      const unsigned long long t = warp_sum(v[i]);
      if (lane == 0 && t) atomicAdd(&A[i == 5 ? 7 : i], t);
    }
    s = c2 = a4 = a1 = a2 = a3 = 0;
  };
  for (int64_t b = warp * run; b < min(blocks, (warp + 1) * run); ++b) {
    const int64_t x = b * span + lane;
    const bool in = (int)lane < span && x < n;
    const unsigned long long da = in ? (unsigned long long)(roff[x + 1] - roff[x]) : 0ull;
    const int64_t e0 = in ? doff[x] : 0, e1 = in ? doff[x + 1] : INT64_MAX;
    const int gx = in ? graph_of(gid, x) : -1;
    // the block's vertices graph by graph (nearly always one)
    unsigned todo = __ballot_sync(0xffffffffu, in);
    while (todo) {
      const int first = __ffs(todo) - 1, gb = __shfl_sync(0xffffffffu, gx, first);
      const unsigned mine = __ballot_sync(0xffffffffu, in && gx == gb);
      todo &= ~mine;
      if (gb != g) {
        flush();
        g = gb;
      }
      if (in && gx == gb) {
        s += choose3(da);
        c2 += choose2(da);
      }
      const int last = 31 - __clz(mine);
      const int64_t lo = __shfl_sync(0xffffffffu, e0, first), hi = __shfl_sync(0xffffffffu, e1, last);
      for (int64_t base = lo; base < hi; base += 32) {
        const int64_t e = base + lane;
        int t = 0;  // the edge's lower endpoint: the first lane whose list ends past e
#pragma unroll
        for (int r = 16; r; r >>= 1)
          if (__shfl_sync(0xffffffffu, e1, t + r - 1) <= e) t += r;
        const unsigned long long d1 = __shfl_sync(0xffffffffu, da, t & 31);
        if (e < hi) {
          const int32_t v = dadj[e];
          const unsigned long long d2 = (unsigned long long)(roff[v + 1] - roff[v]), k = te[e];
          a4 += (d1 - 1) * (d2 - 1);
          a1 += k;
          a2 += choose2(k);
          a3 += k * (d1 + d2 - 4);
        }
      }
    }
  }
  flush();
}

// ------------------------------------------------------------ 4-cycles
// Task x = highest-rank vertex of the cycle: for a in N(x) with a < x and
// y in N(a) with y < x, cnt[y]++; the task adds sum_y C(cnt[y], 2).
constexpr int kC4WarpCap = 512;  // (key, count) slots per warp -> tasks with bound <= 256
constexpr int kC4CtaSlots = 8 * kC4WarpCap;  // a hub task's shared table: the 8 warps' tables together
// Hub tasks have a 2-hop bound of at most kC4HubMax (larger ones go to
// k_c4_big), so at most that many distinct keys meet kC4CtaSlots slots: the
// table never fills and every probe sequence ends.
constexpr long long kC4HubMax = kC4CtaSlots * 3 / 4;
static_assert(kC4HubMax < kC4CtaSlots, "a hub task's keys must leave its table a free slot: c4_slot never fails");

// Slot of y in a hub task's shared table, found or newly claimed.
__device__ __forceinline__ int c4_slot(int2 *tab, int32_t y) {
  uint32_t h = ((uint32_t)y * 2654435769u) >> (32 - 12);
  for (int p = 0; p < kC4CtaSlots; ++p) {
    int cur = tab[h].x;
    if (cur == -1) {
      cur = atomicCAS(&tab[h].x, -1, y);
      if (cur == -1) cur = y;
    }
    if (cur == y) return (int)h;
    h = (h + 1) & (kC4CtaSlots - 1);
  }
  return -1;
}

// Empties a (key, count) table of `slots` entries (16-byte aligned, slots
// even) with 16-byte stores.  Counts need no scan before it: every increment
// adds the counter's old value to the task's sum (C(c+1,2) - C(c,2) = c).
__device__ __forceinline__ void c4_reset(int2 *tab, int slots, int t, int nt) {
  uint4 *v = reinterpret_cast<uint4 *>(tab);
  for (int i = t; i < slots / 2; i += nt) v[i] = make_uint4(0xffffffffu, 0u, 0xffffffffu, 0u);
}

__global__ void k_c4_tasks(int64_t n, const int64_t *__restrict__ roff, const int64_t *__restrict__ split,
                           const int32_t *__restrict__ radj, int warp_bound, long long big_min,
                           int32_t *__restrict__ cta_tasks, int32_t *__restrict__ warp_tasks,
                           int32_t *__restrict__ big_tasks, unsigned long long *__restrict__ big_b,
                           int *__restrict__ sizes) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const unsigned lane = lane_id();
  for (int64_t x = warp; x < n; x += nw) {
    unsigned long long b = 0;
    for (int64_t k = roff[x] + lane; k < split[x]; k += 32) {
      int32_t a = radj[k];
      b += (unsigned long long)(roff[a + 1] - roff[a]);
    }
    b = warp_sum(b);
    const int64_t dx = split[x] - roff[x];
    if (lane == 0 && dx >= 2) {
      if (b > (unsigned long long)big_min) {
        const int i = atomicAdd(&sizes[2], 1);
        big_tasks[i] = (int32_t)x;
        big_b[i] = b;
        atomicMax(&sizes[3], (int)dx);
      } else if (b > (unsigned long long)warp_bound) {
        cta_tasks[atomicAdd(&sizes[0], 1)] = (int32_t)x;
      } else {
        warp_tasks[atomicAdd(&sizes[1], 1)] = (int32_t)x;
      }
    }
  }
}

__global__ void __launch_bounds__(256) k_c4(const int64_t *__restrict__ roff, const int64_t *__restrict__ split,
                                            const int32_t *__restrict__ radj, const int32_t *__restrict__ gid,
                                            const int64_t *__restrict__ gbase, const int32_t *__restrict__ cta_tasks,
                                            int n_cta, const int32_t *__restrict__ warp_tasks, int n_warp,
                                            int *__restrict__ counters, unsigned long long *__restrict__ acc) {
  __shared__ __align__(16) int2 c4sm[8 * kC4WarpCap];
  __shared__ int s_task;
  const unsigned lane = threadIdx.x & 31;
  const int wid = threadIdx.x >> 5;
  // hub tasks: counters in a shared-memory hash table over the 8 warps' tables
  static_assert(kC4CtaSlots == 4096, "c4_slot hashes to 12 bits");
  while (true) {
    if (threadIdx.x == 0) s_task = atomicAdd(&counters[0], 1);
    __syncthreads();
    int t = s_task;
    __syncthreads();
    if (t >= n_cta) break;
    const int32_t x = cta_tasks[t];
    const int g = graph_of(gid, x);
    const int64_t a0 = roff[x], a1 = split[x];
    c4_reset(c4sm, kC4CtaSlots, threadIdx.x, blockDim.x);
    __syncthreads();
    unsigned long long c = 0;
    for (int64_t k = a0 + wid; k < a1; k += 8) {
      int32_t a = radj[k];
      for (int64_t j = roff[a] + lane; j < roff[a + 1]; j += 32) {
        int32_t y = __ldg(radj + j);
        if (y >= x) break;
        const int h = c4_slot(c4sm, y);
        if (h >= 0) c += (unsigned long long)atomicAdd(&c4sm[h].y, 1);
      }
    }
    c = warp_sum(c);
    if (lane == 0 && c) atomicAdd(&acc[8 * g + 6], c);
    __syncthreads();
  }
  // tail tasks: shared-memory (key, count) table per warp
  int2 *tab = c4sm + wid * kC4WarpCap;
  c4_reset(tab, kC4WarpCap, lane, 32);
  __syncwarp();
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&counters[1], 1);
    t = __shfl_sync(0xffffffffu, t, 0);
    if (t >= n_warp) break;
    const int32_t x = warp_tasks[t];
    unsigned long long c = 0;
    for (int64_t k = roff[x]; k < split[x]; ++k) {
      int32_t a = radj[k];
      for (int64_t j = roff[a] + lane; j < roff[a + 1]; j += 32) {
        int32_t y = __ldg(radj + j);
        if (y >= x) break;
        uint32_t h = ((uint32_t)y * 2654435769u) >> (32 - 9);
        while (true) {
          int prev = atomicCAS(&tab[h].x, -1, y);
          if (prev == -1 || prev == y) break;
          h = (h + 1) & (kC4WarpCap - 1);
        }
        c += (unsigned long long)atomicAdd(&tab[h].y, 1);
      }
    }
    __syncwarp();
    c4_reset(tab, kC4WarpCap, lane, 32);
    __syncwarp();
    c = warp_sum(c);
    if (lane == 0 && c) atomicAdd(&acc[8 * graph_of(gid, x) + 6], c);
  }
}

// ------------------------------------------------------------ giant 4-cycle tasks
// A task whose 2-hop bound passes big_min has far more distinct y than a hash
// table of k_c4's holds (nearly every wedge ends at its own y).  Its counters
// are indexed by y directly, a window of keys at a time, in shared memory --
// 16-bit halves of 32-bit words while x has fewer than 65536 neighbours below
// it, so no count can carry into the next key.  Every increment adds the
// counter's old value to the sum (C(c+1,2) - C(c,2) = c), so no scan is needed.
// The windows go down from x; a walk (wedge.cuh) leaves in `cursor` where each
// list's part began, the next window's ends there and its start is near, so a
// list is searched in full once per task.  Ranks ascend with degree and y lies
// below x, so the window just below x takes most wedges (R-MAT 18: 91 % end
// within 50,000 of x, Chung-Lu 200,000: 61 %), but the rest may span many: with
// two full searches per list and window, and counters in global memory from
// the ninth window on, motifs of R-MAT 18 / R-MAT 20 / the 256 Chung-Lu graphs
// took 7.2 / 101 / 1320 ms, with cursors 6.2 / 39.6 / 698 ms (lane groups with
// a cursor per list, 1024 threads and 200 KB: 11.8 / 70.7 / 806 ms, whole
// pipelines).  It is bound by the latency of the lists and of the counters' old
// values at 32 to 48 warps per SM.  Two CTAs per SM and windows of 51,200 keys
// while every member has at most kC4WideMin vertices, one CTA and windows of
// 102,400 keys beyond: members that span many windows pay for each with a walk
// over all lists (two searches each).  ms narrow / wide, Chung-Lu of exponent 2.8 and
// mean degree 64: 150,001 vertices 3.38 / 3.84, 250,001 6.48 / 6.87, 400,001 12.25 /
// 11.97, 600,001 22.1 / 20.5, 10^6 47.8 / 40.7; R-MAT 18 6.1 / 6.4, R-MAT 20 39.4 /
// 39.1.  (2 x 1024 threads with 100 KB each: R-MAT 20 41.6, 10^6 vertices 52.0.)
template <int THREADS, int PER_SM, int WORDS>
struct C4Shape {
  static constexpr int kThreads = THREADS, kPerSm = PER_SM, kWords = WORDS, kSmem = 4 * WORDS;
  // Tasks whose bound is at most kHashMax count in an open-addressing table
  // over the same shared memory, slots of (key + 1, count) with 0 = empty.  The
  // bound caps the distinct keys below the slot count, so every probe ends.
  static constexpr unsigned kHashSlots = WORDS / 2;
  static constexpr unsigned long long kHashMax = kHashSlots * 6 / 10;
};
using C4Narrow = C4Shape<768, 2, 25600>;
using C4Wide = C4Shape<1024, 1, 51200>;
constexpr int64_t kC4WideMin = 400000;
constexpr int64_t kC4CursorBytes = 4ll << 30;  // most global memory for cursors

template <unsigned SLOTS>
__device__ __forceinline__ unsigned c4_hash_add(unsigned *cw, unsigned key1) {
  unsigned h = (unsigned)(((unsigned long long)(key1 * 2654435761u) * SLOTS) >> 32);
  for (unsigned p = 0; p < SLOTS; ++p) {
    unsigned cur = cw[2 * h];
    if (cur == 0u) {
      cur = atomicCAS(&cw[2 * h], 0u, key1);
      if (cur == 0u) cur = key1;
    }
    if (cur == key1) return atomicAdd(&cw[2 * h + 1], 1u);
    if (++h == SLOTS) h = 0;
  }
  return 0u;
}

__device__ __forceinline__ int64_t first_at_least(const int32_t *__restrict__ a, int64_t lo, int64_t hi, int64_t key) {
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (__ldg(a + mid) < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// hash_max: at most S::kHashMax
template <class S>
__global__ void __launch_bounds__(S::kThreads, S::kPerSm)
    k_c4_big(const int64_t *__restrict__ roff, const int64_t *__restrict__ split, const int32_t *__restrict__ radj,
             const int32_t *__restrict__ gid, const int64_t *__restrict__ gbase, const int32_t *__restrict__ tasks,
             const unsigned long long *__restrict__ task_b, int n_tasks, int *__restrict__ counters,
             int *__restrict__ cursors, int cursor_len, unsigned long long hash_max,
             unsigned long long *__restrict__ acc) {
  extern __shared__ __align__(16) unsigned hot[];
  __shared__ int s_task;
  __shared__ WedgeWalk s_walk;
  int *cursor = cursors + (int64_t)blockIdx.x * cursor_len;
  const unsigned lane = threadIdx.x & 31;
  int turn = 0;
  if (threadIdx.x == 0) s_walk.s[0].next = s_walk.s[0].nlong = 0;
  for (int i = threadIdx.x; i < S::kWords; i += blockDim.x) hot[i] = 0u;
  while (true) {
    if (threadIdx.x == 0) s_task = atomicAdd(&counters[2], 1);
    __syncthreads();
    const int t = s_task;
    __syncthreads();
    if (t >= n_tasks) break;
    const int32_t x = tasks[t];
    const unsigned long long W = task_b[t];
    const int g = graph_of(gid, x);
    const int32_t base = gbase ? (int32_t)gbase[g] : 0;
    const int64_t a0 = roff[x];
    const int dx = (int)(split[x] - a0);
    const int sh = dx < 65536 ? 1 : 0;
    const unsigned mask = sh ? 0xffffu : 0xffffffffu;
    unsigned long long c = 0;
    if (W <= hash_max) {
      cta_wedges(radj, dx, W, s_walk, &turn,
                 [&](int i, long long *st, int *len) {
                   const int32_t a = radj[a0 + i];
                   *st = roff[a];
                   *len = (int)(first_at_least(radj, *st, roff[a + 1], x) - *st);
                 },
                 [&](int32_t y, long long, int) { c += c4_hash_add<S::kHashSlots>(hot, (unsigned)(y - base) + 1u); });
      uint4 *v = reinterpret_cast<uint4 *>(hot);
      for (int i = threadIdx.x; i < S::kWords / 4; i += blockDim.x) v[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
    }
    for (int32_t hi = W <= hash_max ? base : x; hi > base;) {
      const int32_t lo = (int32_t)max((int64_t)base, (int64_t)hi - ((int64_t)S::kWords << sh));
      cta_wedges(radj, dx, W, s_walk, &turn,
                 [&](int i, long long *st, int *len) {  // entries of N(a) in [lo, hi), a the i-th neighbour of x
                   const int64_t s0 = roff[radj[a0 + i]];
                   int64_t s = s0, e;
                   if (hi < x && i < cursor_len) e = s0 + cursor[i];
                   else e = first_at_least(radj, s0, roff[radj[a0 + i] + 1], hi);
                   if (lo > base) {
                     if (i < cursor_len) {  // back from e in doubling steps
                       int64_t top = e, step = 1;
                       while (s0 < top && __ldg(radj + max(s0, top - step)) >= lo) {
                         top = max(s0, top - step);
                         step *= 2;
                       }
                       s = first_at_least(radj, max(s0, top - step), top, lo);
                       cursor[i] = (int)(s - s0);
                     } else {
                       s = first_at_least(radj, s0, e, lo);
                     }
                   }
                   *st = s;
                   *len = (int)(e - s);
                 },
                 [&](int32_t y, long long, int) {
                   const unsigned o = (unsigned)(y - lo), s = (o & (unsigned)sh) << 4;
                   c += (atomicAdd(&hot[o >> sh], 1u << s) >> s) & mask;
                 });
      const int words = ((hi - lo) >> sh) + 1;
      uint4 *v = reinterpret_cast<uint4 *>(hot);
      for (int i = threadIdx.x; 4 * i < words; i += blockDim.x)
        if (i < S::kWords / 4) v[i] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      hi = lo;
    }
    c = warp_sum(c);
    if (lane == 0 && c) atomicAdd(&acc[8 * g + 6], c);
  }
}

// ------------------------------------------------------------ combine
__global__ void k_motif_combine(int ngraphs, const unsigned long long *__restrict__ acc,
                                unsigned long long *__restrict__ out /* ngraphs x 8 */) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ngraphs; g += gridDim.x * blockDim.x) {
    const unsigned long long *A = acc + 8 * g;
    unsigned long long T = A[2] / 3, S = A[0], P = A[1] - 3 * T, TT = A[4] / 2, D = A[3], C = A[6], K = A[5];
    unsigned long long k = K, d = D - 6 * K, c = C - d - 3 * K, tt = TT - 4 * d - 12 * K;
    unsigned long long p = P - 2 * tt - 4 * c - 6 * d - 12 * K, s = S - tt - 2 * d - 4 * K;
    unsigned long long *o = out + 8 * g;
    o[0] = A[7] - 3 * T;  // induced 2-paths
    o[1] = T;
    o[2] = s;
    o[3] = p;
    o[4] = tt;
    o[5] = c;
    o[6] = d;
    o[7] = k;
  }
}

// ------------------------------------------------------------ pipeline
__global__ void k_up_len(int64_t n, const int64_t *__restrict__ roff, const int64_t *__restrict__ split,
                         int64_t *__restrict__ len) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x)
    len[x] = roff[x + 1] - split[x];
}
__global__ void k_up_copy(int64_t n, const int64_t *__restrict__ roff, const int64_t *__restrict__ split,
                          const int32_t *__restrict__ radj, const int64_t *__restrict__ doff,
                          int32_t *__restrict__ dadj) {
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t x = warp; x < n; x += nw)
    for (int64_t k = split[x] + lane_id(); k < roff[x + 1]; k += 32) dadj[doff[x] + (k - split[x])] = radj[k];
}
// tasks of the per-edge triangle pass: vertices with >= 2 upward neighbours.
// sizes: [0] CTA tasks, [1] warp tasks of more than kTeLight neighbours, filled
// from the front of warp_tasks, [2] the others, from the back
__global__ void k_te_tasks(int64_t n, const int64_t *__restrict__ doff, int cta_min, int32_t *__restrict__ cta_tasks,
                           int32_t *__restrict__ warp_tasks, int *__restrict__ sizes) {
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
    const int64_t d = doff[x + 1] - doff[x];
    if (d < 2) continue;
    if (d > cta_min) cta_tasks[atomicAdd(&sizes[0], 1)] = (int32_t)x;
    else if (d > kTeLight) warp_tasks[atomicAdd(&sizes[1], 1)] = (int32_t)x;
    else warp_tasks[n - 1 - atomicAdd(&sizes[2], 1)] = (int32_t)x;
  }
}

// The upward parts of a rank-ordered symmetric graph as a CSR of its own
// (the degree-oriented DAG, every list pointing to larger ids).
static int dag_from_split(int64_t n, const int64_t *roff, const int64_t *split, const int32_t *radj,
                          DevBuf<int64_t> &doff, DevBuf<int32_t> &dadj, int *max_deg, cudaStream_t st) {
  DevBuf<int64_t> len;
  GPM_TRY(len.reserve(n));
  GPM_TRY(doff.reserve(n + 1));
  if (n > 0) k_up_len<<<grid_for(n), 256, 0, st>>>(n, roff, split, len.p);
  size_t tmp = 0;
  GPM_CUDA(cub::DeviceScan::InclusiveSum(nullptr, tmp, len.p, doff.p + 1, (int)n, st));
  DevBuf<char> t;
  GPM_TRY(t.reserve(tmp));
  GPM_CUDA(cudaMemsetAsync(doff.p, 0, sizeof(int64_t), st));
  if (n > 0) GPM_CUDA(cub::DeviceScan::InclusiveSum(t.p, tmp, len.p, doff.p + 1, (int)n, st));
  int64_t m = 0;
  GPM_CUDA(cudaMemcpyAsync(&m, doff.p + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  DevBuf<int64_t> mx;
  GPM_TRY(mx.reserve(1));
  size_t tmp2 = 0;
  GPM_CUDA(cub::DeviceReduce::Max(nullptr, tmp2, len.p, mx.p, (int)std::max<int64_t>(n, 1), st));
  DevBuf<char> t2;
  GPM_TRY(t2.reserve(tmp2));
  int64_t hmx = 0;
  if (n > 0) {
    GPM_CUDA(cub::DeviceReduce::Max(t2.p, tmp2, len.p, mx.p, (int)n, st));
    GPM_CUDA(cudaMemcpyAsync(&hmx, mx.p, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
  }
  GPM_CUDA(cudaStreamSynchronize(st));
  GPM_TRY(dadj.reserve(std::max<int64_t>(m, 1)));
  if (n > 0) k_up_copy<<<grid_for(n * 32), 256, 0, st>>>(n, roff, split, radj, doff.p, dadj.p);
  *max_deg = (int)hmx;
  return GPM_OK;
}

// Work cursors behind the sums, zeroed with them: the triangle pass's (3), the
// 4-cycle stage's (3) and the clique stage's (3), each in two words of acc.
constexpr int kMotifCursors = 6;
static int *te_cursors(MotifPlan *p) { return reinterpret_cast<int *>(p->acc.p + 8 * (size_t)p->in.ngraphs); }
static int *c4_cursors(MotifPlan *p) { return te_cursors(p) + 4; }
static int *k4_cursors(MotifPlan *p) { return te_cursors(p) + 8; }

// f(C4Narrow{}) or f(C4Wide{})
template <class F>
static int c4_shape(int64_t max_graph_n, F f) {
  return max_graph_n > kC4WideMin ? f(C4Wide{}) : f(C4Narrow{});
}

static int te_grid() {
  static PerDevice grid;
  return grid.get([] {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_edge_tri, 256, 0);
    return std::max(1, per_sm) * num_sms();
  });
}

// Builds every schedule and scratch buffer of the pipeline (host syncs and
// allocations happen here, never in motif_plan_run).
int motif_plan_build(const MotifInput &in, MotifPlan *p, cudaStream_t st) {
  p->in = in;
  const int64_t n = in.n;
  const int64_t *roff = in.roff;
  const int32_t *radj = in.radj;
  GPM_TRY(p->acc.reserve(8 * (size_t)in.ngraphs + kMotifCursors));
  GPM_TRY(p->out.reserve(8 * (size_t)in.ngraphs));
  GPM_TRY(p->split.reserve(n));
  if (n > 0) k_split<<<grid_for(n), 256, 0, st>>>(n, roff, radj, p->split.p);
  GPM_TRY(dag_from_split(n, roff, p->split.p, radj, p->doff, p->dadj, &p->dag_max, st));
  GPM_TRY(p->te.reserve(p->dadj.n));
  // queues of the per-edge triangle pass and of the 4-cycle pass
  DevBuf<int> sizes;
  GPM_TRY(sizes.reserve(7));
  GPM_TRY(p->te_ct.reserve(n));
  GPM_TRY(p->te_wt.reserve(n));
  GPM_TRY(p->c4_ct.reserve(n));
  GPM_TRY(p->c4_wt.reserve(n));
  DevBuf<int32_t> bt;
  DevBuf<unsigned long long> bb;
  GPM_TRY(bt.reserve(n));
  GPM_TRY(bb.reserve(n));
  GPM_CUDA(cudaMemsetAsync(sizes.p, 0, 7 * sizeof(int), st));
  if (n > 0) {
    k_te_tasks<<<grid_for(n), 256, 0, st>>>(n, p->doff.p, std::min(in.te_cta_min, kTeWarpKeys), p->te_ct.p, p->te_wt.p, sizes.p);
    if (in.size == 4) {
      const int wb = std::min(in.c4_warp_bound, kC4WarpCap / 2);
      long long big_min = in.c4_big_min;
      if (const char *e = getenv("GPM_C4_BIG_MIN")) big_min = atoll(e);
      big_min = std::min(std::max<long long>(big_min, (long long)wb), kC4HubMax);
      // hub tasks (bound <= big_min) must fit c4_slot's table, or they would drop wedges
      if (big_min > kC4HubMax) return fail(GPM_EINVAL, "4-cycle hub bound above the hub table");
      k_c4_tasks<<<grid_for(n * 32), 256, 0, st>>>(n, roff, p->split.p, radj, wb, big_min,
                                                   p->c4_ct.p, p->c4_wt.p, bt.p, bb.p, sizes.p + 3);
    }
  }
  int h[7];
  GPM_CUDA(cudaMemcpyAsync(h, sizes.p, sizeof h, cudaMemcpyDeviceToHost, st));
  GPM_CUDA(cudaStreamSynchronize(st));
  p->te_nc = h[0];
  p->te_nw = h[1];
  p->te_nl = h[2];
  p->c4_nc = h[3];
  p->c4_nw = h[4];
  p->c4_nb = h[5];
  p->te_grid = te_grid();
  if (in.size == 3) {
    GPM_CUDA(cudaStreamSynchronize(st));
    return GPM_OK;
  }
  // giant tasks, largest bound first
  GPM_TRY(p->c4_bt.reserve(std::max(p->c4_nb, 1)));
  GPM_TRY(p->c4_bb.reserve(std::max(p->c4_nb, 1)));
  if (p->c4_nb > 0) {
    size_t tmp = 0;
    GPM_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, bb.p, p->c4_bb.p, bt.p, p->c4_bt.p, p->c4_nb, 0,
                                                       64, st));
    DevBuf<char> t;
    GPM_TRY(t.reserve(tmp));
    GPM_CUDA(cub::DeviceRadixSort::SortPairsDescending(t.p, tmp, bb.p, p->c4_bb.p, bt.p, p->c4_bt.p, p->c4_nb, 0,
                                                       64, st));
    int words = 0;
    GPM_TRY(c4_shape(in.max_graph_n, [&](auto shape) -> int {
      using S = decltype(shape);
      words = S::kWords;
      p->c4_hash_max = S::kHashMax;
      GPM_CUDA(cudaFuncSetAttribute(k_c4_big<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem));
      int per_sm = 0;
      GPM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_c4_big<S>, S::kThreads, S::kSmem));
      p->c4_big_grid = std::max(1, per_sm) * num_sms();
      return GPM_OK;
    }));
    // tests send small tasks through the windows
    if (const char *e = getenv("GPM_C4_HASH_MAX"))
      p->c4_hash_max = std::min<unsigned long long>(p->c4_hash_max, std::max(0ll, atoll(e)));
    p->c4_big_grid = std::min(p->c4_big_grid, p->c4_nb);
    // cursors for the longest task's neighbours, where some member spans two
    // windows, as far as memory goes (the others search their whole list again)
    int64_t len = in.max_graph_n <= words ? 0 : h[6];
    if (const char *e = getenv("GPM_C4_CURSORS")) len = std::min<int64_t>(len, std::max(0ll, atoll(e)));
    len = std::min(len, kC4CursorBytes / 4 / p->c4_big_grid);
    while (p->c4_cursor.reserve((size_t)len * p->c4_big_grid) != GPM_OK) {
      if (len == 0) return GPM_ENOMEM;
      len = len < 4096 ? 0 : len / 2;
    }
    p->c4_cursor_len = (int)len;
    GPM_CUDA(cudaStreamSynchronize(st));
  }
  {
    int per_sm = 0;
    GPM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_c4, 256, 0));
    p->c4_grid = std::max(1, per_sm) * num_sms();
  }
  GPM_TRY(clique_plan_build(&p->k4, n, p->doff.p, p->dadj.p, p->dag_max, 4, in.gid, p->acc.p, 8, 5, st,
                            in.cq_warp_max, k4_cursors(p)));
  GPM_CUDA(cudaStreamSynchronize(st));
  return GPM_OK;
}

// Triangles per edge, counted from zero.
static int te_launch(MotifPlan *p, cudaStream_t st) {
  GPM_CUDA(cudaMemsetAsync(p->te.p, 0, sizeof(unsigned) * p->dadj.n, st));
  if (p->te_nc + p->te_nw + p->te_nl > 0)
    k_edge_tri<<<p->te_grid, 256, 0, st>>>(p->doff.p, p->dadj.p, p->te_ct.p, p->te_nc, p->te_wt.p, p->te_nw,
                                           p->te_wt.p + (p->in.n - p->te_nl), p->te_nl, te_cursors(p), p->te.p);
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

// The 4-cycle launches: giant tasks first (largest bound first), then hub and tail tasks.
static int c4_launch(MotifPlan *p, cudaStream_t st) {
  const MotifInput &in = p->in;
  if (p->c4_nb > 0)
    GPM_TRY(c4_shape(in.max_graph_n, [&](auto shape) -> int {
      using S = decltype(shape);
      k_c4_big<S><<<p->c4_big_grid, S::kThreads, S::kSmem, st>>>(
          in.roff, p->split.p, in.radj, in.gid, in.gbase, p->c4_bt.p, p->c4_bb.p, p->c4_nb, c4_cursors(p),
          p->c4_cursor.p, p->c4_cursor_len, p->c4_hash_max, p->acc.p);
      return GPM_OK;
    }));
  if (p->c4_nc + p->c4_nw > 0)
    k_c4<<<p->c4_grid, 256, 0, st>>>(in.roff, p->split.p, in.radj, in.gid, in.gbase, p->c4_ct.p, p->c4_nc,
                                     p->c4_wt.p, p->c4_nw, c4_cursors(p), p->acc.p);
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

// Launches only (capturable): zero the sums, triangles per edge, per-edge
// and per-vertex sums, 4-cycles, 4-cliques, inversion.
int motif_plan_run(MotifPlan *p, cudaStream_t st) {
  const MotifInput &in = p->in;
  const int64_t n = in.n;
  // the sums, and behind them the cursors of all stages
  GPM_CUDA(cudaMemsetAsync(p->acc.p, 0, sizeof(unsigned long long) * (8 * in.ngraphs + kMotifCursors), st));
  GPM_TRY(te_launch(p, st));
  int span = 1;
  while (span < 32 && n / span > (int64_t)num_sms() * 32) span *= 2;
  if (n > 0)
    k_edge_sums<<<grid_for((n + span - 1) / span * 32), 256, 0, st>>>(n, span, in.roff, p->doff.p, p->dadj.p, p->te.p, in.gid, p->acc.p);
  if (in.size == 4) {
    GPM_TRY(c4_launch(p, st));
    GPM_TRY(clique_plan_run(&p->k4, st, false));
  }
  k_motif_combine<<<std::max(1, (in.ngraphs + 255) / 256), 256, 0, st>>>(in.ngraphs, p->acc.p, p->out.p);
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

int motif_plan_run_stage(MotifPlan *p, int stage, cudaStream_t st) {
  if (stage == 0) {
    GPM_CUDA(cudaMemsetAsync(te_cursors(p), 0, 4 * sizeof(int), st));
    GPM_TRY(te_launch(p, st));
  } else if (stage == 1) {
    GPM_CUDA(cudaMemsetAsync(c4_cursors(p), 0, 4 * sizeof(int), st));
    GPM_TRY(c4_launch(p, st));
  } else {
    GPM_TRY(clique_plan_run(&p->k4, st));
  }
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

}  // namespace gpm

namespace gpm {
void free_motif_plan(MotifPlan *p) { delete p; }
}  // namespace gpm

using namespace gpm;

extern "C" int gpm_motif(gpm_graph *g, int k, uint64_t *out) {
  if (!g || !out) return fail(GPM_EINVAL, "gpm_motif: NULL argument");
  if (k != 3 && k != 4) return fail(GPM_EUNSUPPORTED, "motif size must be 3 or 4");
  if (g->oriented) return fail(GPM_EINVAL, "motif counting needs the symmetric (unoriented) graph");
  GPM_TRY(ensure_rank_graph(g, 0));
  // the pipeline (task queues, scratch) is built on the first call of each
  // size and kept with the graph, so later calls only launch
  MotifPlan *&plan = g->motif[k - 3];
  if (!plan) {
    MotifInput in;
    in.n = g->n;
    in.nnz = g->nnz;
    in.roff = g->rg->roff.p;
    in.radj = g->rg->radj.p;
    in.max_graph_n = g->n;
    in.size = k;
    MotifPlan *p = new MotifPlan();
    const int s = motif_plan_build(in, p, 0);
    if (s != GPM_OK) {
      delete p;
      return s;
    }
    plan = p;
  }
  GPM_TRY(motif_plan_run(plan, 0));
  unsigned long long h[8];
  GPM_CUDA(cudaMemcpy(h, plan->out.p, sizeof h, cudaMemcpyDeviceToHost));
  if (k == 3) {
    out[0] = h[0];
    out[1] = h[1];
  } else {
    for (int i = 0; i < 6; ++i) out[i] = h[2 + i];
  }
  return GPM_OK;
}
