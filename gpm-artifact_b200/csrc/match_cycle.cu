// match_cycle.cu -- counted 4-cycle queries (sub_ceci semantics) without
// walking their embeddings.
//
// For opposite query vertices a, c and the two between them, b and d, the
// count is the sum over pairs (a, c) of images of B(a, c) * D(a, c), where
// B and D are the numbers of label-b and label-d common neighbours (for equal
// labels b = d, of B (B - 1): b and d take different images).  One task per
// image of a: the 2-hop walk a - b - c counts B(a, .) into one counter per
// vertex of c's label class, the walk a - d - c adds up the counters it meets.
// The work is the wedges, not the embeddings (R-MAT 19, labels 0 0 3 1: 0.6 G
// wedges; 145-178 ms by the depth-first walk, which tests every wedge for its
// closing edge, 3.3 ms here, 2.7 of it in k_cycle_big: 0.8 G increments, loads
// and clears, bound by the latency of lists and counters at 32 warps per SM).
//
// Counters are indexed by the rank inside the label class in descending degree
// order.  A walk ends at a vertex in proportion to its degree, so the ranks
// below kHot, kept in shared memory, take most of the increments; the others
// are a CTA's own array in global memory (mostly L2 resident).  Tasks whose
// smaller side has at most kSmallBound wedges count in a hash table per warp
// instead.
#include <cub/cub.cuh>

#include <algorithm>

#include "match.cuh"
#include "wedge.cuh"

namespace gpm {

constexpr int kSmallWarps = 8, kSmallSlots = 512;
constexpr unsigned long long kSmallBound = kSmallSlots / 2;
constexpr int kBigThreads = 512, kBigPerSm = 2;
constexpr int kHot = 24576;                 // shared counters of a CTA (96 KB, two CTAs per SM)
constexpr int64_t kTailBytes = 4ll << 30;   // most global memory for the counters of ranks >= kHot

struct CycleSpace {
  DevBuf<int2> small;           // tasks: (vertex, 1 when the d side is counted first)
  DevBuf<int4> big;             // the same, then the wedges of the counted and of the other side (capped)
  DevBuf<int> sizes;            // [0] small tasks, [1] big tasks, [2], [3] their cursors
  DevBuf<unsigned> tail;        // grid x (class size - kHot), all zero between launches
  int64_t tail_len = 0;         // counters per CTA
  int grid = 0;                 // CTAs of k_cycle_big
};
void free_cycle_space(CycleSpace *s) { delete s; }

struct CycleArgs {
  const int64_t *off;
  const int32_t *ladj, *loff, *lrk, *lrank;
  int L, lb, lc, ld;
  bool skip_root;  // a and c carry the same label: c must not be a
};

// sum over all vertices v of label `lm` of d_l0(v) * d_l1(v): the wedges of
// the opposite pair (l0, l1) through lm
__global__ void k_cycle_wedges(int64_t n, const int32_t *__restrict__ vs, const int32_t *__restrict__ loff, int L,
                               int l0, int l1, unsigned long long *__restrict__ out) {
  unsigned long long c = 0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t *o = loff + (int64_t)vs[i] * (L + 1);
    c += (unsigned long long)(o[l0 + 1] - o[l0]) * (unsigned long long)(o[l1 + 1] - o[l1]);
  }
  c = warp_sum(c);
  if (lane_id() == 0 && c) atomicAdd(out, c);
}

// The middles of v with label l: their first entry in ladj and their number.
__device__ __forceinline__ void middles(const CycleArgs &A, int32_t v, int l, int64_t *s, int *m) {
  const int32_t *o = A.loff + (int64_t)v * (A.L + 1) + l;
  *s = A.off[v] + o[0];
  *m = o[1] - o[0];
}
// label-lc segment of middle b: first entry and length
__device__ __forceinline__ void ends(const CycleArgs &A, int32_t b, long long *st, int *len) {
  const int32_t *o = A.loff + (int64_t)b * (A.L + 1) + A.lc;
  const int32_t s = o[0];
  *st = A.off[b] + s;
  *len = o[1] - s;
}

__device__ __forceinline__ unsigned long long wedge_bound(const CycleArgs &A, int32_t v, int l, unsigned lane) {
  int64_t s;
  int m;
  middles(A, v, l, &s, &m);
  unsigned long long w = 0;
  for (int i = lane; i < m; i += 32) {
    const int32_t *o = A.loff + (int64_t)__ldg(A.ladj + s + i) * (A.L + 1) + A.lc;
    w += (unsigned long long)(o[1] - o[0]);
  }
  return warp_sum(w);
}

// Roots with wedges on both sides into the queue of their size; a warp takes
// up to 32 roots and queues them with one atomic per queue -- fewer where there
// are too few for all SMs, since it takes them one after another (a query with
// 3,671 roots, ER 10,007 x 64: 128 us with 32 each, 79 so).  Roots come in
// descending degree order, so a warp takes every (nroots / per)-th of them: neighbours
// would give all hubs to a few warps (R-MAT 19, labels 0 0 3 1: 1.3-2.1 ms; the
// whole call 5.6 ms then, 3.4 ms now).  The side with fewer
// wedges is the one that is counted (its counters are written and cleared).
__global__ void k_cycle_split(CycleArgs A, const int32_t *__restrict__ roots, int64_t nroots, int per, int2 *__restrict__ small,
                              int4 *__restrict__ big, int *__restrict__ sizes) {
  const unsigned lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const bool same = A.lb == A.ld;
  const int64_t groups = (nroots + per - 1) / per;
  for (int64_t r0 = warp; r0 < groups; r0 += nw) {
    int4 mine = make_int4(0, 0, 0, 0);
    int which = 0;  // 1 small, 2 big
    for (int j = 0; j < per && r0 + j * groups < nroots; ++j) {
      const int32_t v = roots[r0 + j * groups];
      const unsigned long long wb = wedge_bound(A, v, A.lb, lane), wd = same ? wb : wedge_bound(A, v, A.ld, lane);
      if ((int)lane == j && min(wb, wd) > 0) {
        const unsigned long long cap = 0x7fffffffull;
        mine = make_int4(v, wd < wb, (int)min(min(wb, wd), cap), (int)min(max(wb, wd), cap));
        which = min(wb, wd) <= kSmallBound ? 1 : 2;
      }
    }
#pragma unroll
    for (int q = 1; q <= 2; ++q) {
      const unsigned m = __ballot_sync(0xffffffffu, which == q);
      if (!m) continue;
      int at = 0;
      if (lane == 0) at = atomicAdd(&sizes[q - 1], __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      at += __popc(m & ((1u << lane) - 1u));
      if (which == q && q == 1) small[at] = make_int2(mine.x, mine.y);
      if (which == q && q == 2) big[at] = mine;
    }
  }
}

// f(rank of c) for every wedge v - b - c of up to 32 middles b = ladj[s .. s + m)
template <class F>
__device__ __forceinline__ void walk_wedges(const CycleArgs &A, int64_t s, int m, unsigned lane, F f) {
  long long st = 0;
  int len = 0;
  if ((int)lane < m) ends(A, __ldg(A.ladj + s + lane), &st, &len);
  warp_segments(A.lrk, st, len, 0, lane, [&](int32_t x, long long, int) { f(x); });
}

__device__ __forceinline__ uint32_t small_slot(int32_t key) { return ((uint32_t)key * 2654435769u) >> (32 - 9); }
static_assert(kSmallSlots == 512, "small_slot hashes to 9 bits");

__global__ void __launch_bounds__(kSmallWarps * 32)
    k_cycle_small(CycleArgs A, const int2 *__restrict__ tasks, int *__restrict__ sizes,
                  const int32_t *__restrict__ member, unsigned long long *__restrict__ out) {
  __shared__ int2 stab[kSmallWarps][kSmallSlots];
  int2 *tab = stab[threadIdx.x >> 5];
  const unsigned lane = lane_id();
  const int n = sizes[0];
  const bool same = A.lb == A.ld;
  unsigned long long c = 0;
  for (int i = lane; i < kSmallSlots; i += 32) tab[i] = make_int2(-1, 0);
  __syncwarp();
  WarpTasks queue;
  // runs only where the warps have many tasks each: the first are the heaviest
  // (the same query 79 us in runs, 42 so; R-MAT 14, labels 0 1 2 3 202, 91)
  const int lone = n <= 2 * kTaskRun * (int)gridDim.x * kSmallWarps ? n : 0;
  while (true) {
    const int t = queue.next(&sizes[2], lone, lane);
    if (t >= n) break;
    const int2 task = tasks[t];
    const int32_t self = A.skip_root ? A.lrank[task.x] : -1;
    int64_t s;
    int m;
    middles(A, task.x, task.y ? A.ld : A.lb, &s, &m);
    for (int i = 0; i < m; i += 32)
      walk_wedges(A, s + i, min(32, m - i), lane, [&](int32_t x) {
        if (x == self) return;
        uint32_t h = small_slot(x);
        while (true) {  // at most kSmallBound keys in twice as many slots
          const int prev = atomicCAS(&tab[h].x, -1, x);
          if (prev == -1 || prev == x) break;
          h = (h + 1) & (kSmallSlots - 1);
        }
        const int old = atomicAdd(&tab[h].y, 1);
        if (same) c += 2ull * (unsigned)old;  // B (B - 1) = sum of twice the old values
      });
    __syncwarp();
    if (!same) {
      middles(A, task.x, task.y ? A.lb : A.ld, &s, &m);
      for (int i = 0; i < m; i += 32)
        walk_wedges(A, s + i, min(32, m - i), lane, [&](int32_t x) {
          uint32_t h = small_slot(x);
          while (true) {
            const int2 e = tab[h];
            if (e.x == x) c += (unsigned)e.y;
            if (e.x == x || e.x == -1) break;
            h = (h + 1) & (kSmallSlots - 1);
          }
        });
      __syncwarp();
    }
    for (int i = lane; i < kSmallSlots; i += 32) tab[i] = make_int2(-1, 0);
    __syncwarp();
    if (member) {
      c = warp_sum(c);
      if (lane == 0 && c) atomicAdd(&out[member[task.x]], c);
      c = 0;
    }
  }
  c = warp_sum(c);
  if (lane == 0 && c) atomicAdd(out, c);
}

__global__ void __launch_bounds__(kBigThreads, kBigPerSm)
    k_cycle_big(CycleArgs A, const int4 *__restrict__ tasks, int *__restrict__ sizes, unsigned *__restrict__ tails,
                int64_t tail_len, const int32_t *__restrict__ member, unsigned long long *__restrict__ out) {
  extern __shared__ __align__(16) unsigned hot[];
  __shared__ int s_task;
  __shared__ WedgeWalk s_walk;
  unsigned *tail = tails + (int64_t)blockIdx.x * tail_len;
  const unsigned lane = lane_id();
  int turn = 0;
  if (threadIdx.x == 0) s_walk.s[0].next = s_walk.s[0].nlong = 0;
  const int n = sizes[1];
  const bool same = A.lb == A.ld;
  unsigned long long c = 0;
  for (int i = threadIdx.x; i < kHot; i += kBigThreads) hot[i] = 0u;
  while (true) {
    if (threadIdx.x == 0) s_task = atomicAdd(&sizes[3], 1);
    __syncthreads();
    const int t = s_task;
    __syncthreads();
    if (t >= n) break;
    const int4 task = tasks[t];
    const int32_t self = A.skip_root ? A.lrank[task.x] : -1;
    // f over the wedges of side l
    auto side = [&](int l, int wedges, auto f) {
      int64_t s;
      int m;
      middles(A, task.x, l, &s, &m);
      cta_wedges(A.lrk, m, (unsigned long long)wedges, s_walk, &turn,
                 [&](int i, long long *st, int *len) { ends(A, __ldg(A.ladj + s + i), st, len); },
                 [&](int32_t x, long long, int) { f(x); });
    };
    const int first = task.y ? A.ld : A.lb;
    if (same) {
      side(first, task.z, [&](int32_t x) {
        if (x == self) return;
        c += 2ull * (x < kHot ? atomicAdd(&hot[x], 1u) : atomicAdd(&tail[x - kHot], 1u));
      });
    } else {
      side(first, task.z, [&](int32_t x) {
        if (x == self) return;
        if (x < kHot) atomicAdd(&hot[x], 1u);
        else atomicAdd(&tail[x - kHot], 1u);
      });
      side(task.y ? A.lb : A.ld, task.w, [&](int32_t x) { c += x < kHot ? hot[x] : __ldcg(&tail[x - kHot]); });
    }
    // back to zero: the same walk again
    side(first, task.z, [&](int32_t x) {
      if (x < kHot) hot[x] = 0u;
      else tail[x - kHot] = 0u;
    });
    if (member) {
      c = warp_sum(c);
      if (lane == 0 && c) atomicAdd(&out[member[task.x]], c);
      c = 0;
    }
  }
  c = warp_sum(c);
  if (lane == 0 && c) atomicAdd(out, c);
}

// ------------------------------------------------------------ label classes
__global__ void k_class_keys(int64_t n, const int64_t *__restrict__ off, const int32_t *__restrict__ labels,
                             uint64_t *__restrict__ key, int32_t *__restrict__ val) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    key[v] = ((uint64_t)(uint32_t)labels[v] << 32) | (uint32_t)~(uint32_t)(off[v + 1] - off[v]);
    val[v] = (int32_t)v;
  }
}
// lstart[l] = first position of lorder with a label of at least l (l = 0 .. L)
__global__ void k_class_starts(int64_t n, const uint64_t *__restrict__ key, int L, int64_t *__restrict__ lstart) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l > L) return;
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if ((int64_t)(key[mid] >> 32) < l) lo = mid + 1; else hi = mid;
  }
  lstart[l] = lo;
}
__global__ void k_class_ranks(int64_t n, const int32_t *__restrict__ lorder, const int32_t *__restrict__ labels,
                              const int64_t *__restrict__ lstart, int32_t *__restrict__ lrank) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v = lorder[i];
    lrank[v] = (int32_t)(i - lstart[labels[v]]);
  }
}
__global__ void k_entry_ranks(int64_t nnz, const int32_t *__restrict__ ladj, const int32_t *__restrict__ lrank,
                              int32_t *__restrict__ lrk) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nnz; i += (int64_t)gridDim.x * blockDim.x)
    lrk[i] = lrank[ladj[i]];
}

static int blocks_for(int64_t work, int per_sm = 16) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((work + 255) / 256, (int64_t)num_sms() * per_sm));
}

static int ensure_label_classes(gpm_graph *g, LabelCsr *lc) {
  if (!lc->lstart.empty()) return GPM_OK;
  const int64_t n = g->n, nnz = g->nnz;
  DevBuf<uint64_t> key, key2;
  DevBuf<int32_t> val;
  DevBuf<int64_t> ds;
  GPM_TRY(key.reserve(n));
  GPM_TRY(key2.reserve(n));
  GPM_TRY(val.reserve(n));
  GPM_TRY(ds.reserve(lc->L + 1));
  GPM_TRY(lc->lorder.reserve(n));
  GPM_TRY(lc->lrank.reserve(n));
  GPM_TRY(lc->lrk.reserve(nnz));
  k_class_keys<<<blocks_for(n), 256>>>(n, g->off.p, g->labels.p, key.p, val.p);
  size_t tmp = 0;
  GPM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, key.p, key2.p, val.p, lc->lorder.p, (int)n, 0, 38));
  DevBuf<char> t;
  GPM_TRY(t.reserve(tmp));
  GPM_CUDA(cub::DeviceRadixSort::SortPairs(t.p, tmp, key.p, key2.p, val.p, lc->lorder.p, (int)n, 0, 38));
  k_class_starts<<<1, 128>>>(n, key2.p, lc->L, ds.p);
  k_class_ranks<<<blocks_for(n), 256>>>(n, lc->lorder.p, g->labels.p, ds.p, lc->lrank.p);
  k_entry_ranks<<<blocks_for(nnz), 256>>>(nnz, lc->ladj.p, lc->lrank.p, lc->lrk.p);
  GPM_LAUNCH_CHECK();
  std::vector<int64_t> h(lc->L + 1);
  GPM_CUDA(cudaMemcpy(h.data(), ds.p, sizeof(int64_t) * (lc->L + 1), cudaMemcpyDeviceToHost));
  lc->lstart = h;
  return GPM_OK;
}

LabelCsr::~LabelCsr() { free_cycle_space(cycle); }

// ------------------------------------------------------------ host
bool is_cycle4(const gpm_query *q, const LabelCsr *lc) {
  if (q->n != 4) return false;
  for (int i = 0; i < 4; ++i)
    if (q->deg[i] != 2 || q->labels[i] < 0 || q->labels[i] >= lc->L) return false;
  return true;
}

int cycle_plan(gpm_graph *g, LabelCsr *lc, const gpm_query *q, unsigned long long min_wedges, CyclePlan *p,
               CycleSpace **space, bool *fits) {
  *fits = false;
  const int classes = ensure_label_classes(g, lc);
  if (classes == GPM_ENOMEM) return GPM_OK;
  GPM_TRY(classes);
  // the vertices around the cycle: 0, x, opposite, y
  const int x = __builtin_ctzll(q->adjmask[0]), y = 63 - __builtin_clzll(q->adjmask[0]), o = 6 - x - y;
  const int32_t l[4] = {q->labels[0], q->labels[x], q->labels[o], q->labels[y]};
  auto size = [&](int lab) { return lc->lstart[lab + 1] - lc->lstart[lab]; };
  // wedges of the pairs (0, opposite) and (x, y), both through two labels
  DevBuf<unsigned long long> w;
  GPM_TRY(w.reserve(2));
  GPM_CUDA(cudaMemset(w.p, 0, 16));
  for (int pair = 0; pair < 2; ++pair)
    for (int side = 1; side < 4; side += 2) {
      const int lm = l[(pair + side) & 3];
      if (size(lm) > 0)
        k_cycle_wedges<<<blocks_for(size(lm)), 256>>>(size(lm), lc->lorder.p + lc->lstart[lm], lc->loff.p, lc->L,
                                                      l[pair], l[pair + 2], w.p + pair);
    }
  GPM_LAUNCH_CHECK();
  unsigned long long h[2];
  GPM_CUDA(cudaMemcpy(h, w.p, sizeof h, cudaMemcpyDeviceToHost));
  const int pair = h[1] < h[0];
  if (h[pair] < min_wedges) return GPM_OK;
  // the rarer label is the one with counters: fewer of them, most in shared memory
  const bool flip = size(l[pair]) < size(l[pair + 2]);
  p->la = flip ? l[pair + 2] : l[pair];
  p->lc = flip ? l[pair] : l[pair + 2];
  p->lb = l[pair + 1];
  p->ld = l[(pair + 3) & 3];
  const int64_t tail_len = std::max<int64_t>(0, size(p->lc) - kHot);
  const int64_t nroots = size(p->la);
  if (!*space) *space = new CycleSpace();
  CycleSpace *s = *space;
  static PerDevice set;
  set.get([] {
    cudaFuncSetAttribute(k_cycle_big, cudaFuncAttributeMaxDynamicSharedMemorySize, kHot * (int)sizeof(unsigned));
    return 1;
  });
  if (s->grid == 0 || tail_len > s->tail_len) {
    size_t free_b = 0, total_b = 0;
    GPM_CUDA(cudaMemGetInfo(&free_b, &total_b));
    const int64_t room = std::min<int64_t>(kTailBytes, (int64_t)(free_b / 4)) / 4;
    int grid = num_sms() * kBigPerSm;
    if (tail_len > 0) grid = (int)std::min<int64_t>(grid, room / tail_len);
    if (grid < num_sms() / 2) return GPM_OK;
    // the old array stays until the new one is there: other plans share the scratch
    DevBuf<unsigned> tail;
    if (tail.reserve((size_t)(grid * std::max<int64_t>(tail_len, 1))) != GPM_OK) return GPM_OK;
    GPM_CUDA(cudaMemset(tail.p, 0, sizeof(unsigned) * grid * std::max<int64_t>(tail_len, 1)));
    s->tail = std::move(tail);
    s->grid = grid;
    s->tail_len = tail_len;
  }
  if ((int64_t)s->big.n < nroots) {
    DevBuf<int2> small;
    DevBuf<int4> big;
    if (small.reserve(nroots) != GPM_OK || big.reserve(nroots) != GPM_OK) return GPM_OK;
    s->small = std::move(small);
    s->big = std::move(big);
  }
  GPM_TRY(s->sizes.reserve(4));
  *fits = true;
  return GPM_OK;
}

int cycle_launch(const gpm_graph *g, const LabelCsr *lc, const CyclePlan &p, const CycleSpace *s,
                 const int32_t *member, unsigned long long *out, cudaStream_t st) {
  const int64_t nroots = lc->lstart[p.la + 1] - lc->lstart[p.la];
  if (nroots == 0) return GPM_OK;
  const CycleArgs A{g->off.p, lc->ladj.p, lc->loff.p, lc->lrk.p, lc->lrank.p, lc->L, p.lb, p.lc, p.ld, p.la == p.lc};
  GPM_CUDA(cudaMemsetAsync(s->sizes.p, 0, 4 * sizeof(int), st));
  const int per = (int)std::min<int64_t>(32, std::max<int64_t>(1, nroots / ((int64_t)num_sms() * 32)));
  k_cycle_split<<<blocks_for((nroots + per - 1) / per * 32), 256, 0, st>>>(A, lc->lorder.p + lc->lstart[p.la], nroots,
                                                                           per, s->small.p, s->big.p, s->sizes.p);
  k_cycle_big<<<s->grid, kBigThreads, kHot * sizeof(unsigned), st>>>(A, s->big.p, s->sizes.p, s->tail.p, s->tail_len,
                                                                     member, out);
  k_cycle_small<<<num_sms() * 6, kSmallWarps * 32, 0, st>>>(A, s->small.p, s->sizes.p, member, out);
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

}  // namespace gpm
