// match.cuh -- the label-partitioned lists of a data graph, shared by the
// labelled-matching kernels (match.cu, match_cycle.cu).
#pragma once
#include <vector>

#include "common.cuh"

constexpr int kMaxQ = 64;  // query vertices (sub_ceci/configuration/config.h:12)

struct gpm_query {
  int n = 0;
  int32_t labels[kMaxQ];
  unsigned long long adjmask[kMaxQ];  // bit j set iff query edge (i, j)
  int deg[kMaxQ];
};

namespace gpm {

// Label-partitioned copy of a labelled graph's lists (cached per graph).
struct LabelCsr {
  int L = 0;  // partitions (max label + 1); 0: labels too wide, lists copied as they are
  DevBuf<int32_t> ladj, loff;
  // adjacency bitmaps of the vertices with at least hub_min neighbours
  DevBuf<int32_t> hub_slot;
  DevBuf<uint32_t> hub_bm;
  int64_t hub_words = 0;
  int hubs = 0, hub_min = 0;
  // Label classes (built by the first 4-cycle query): the vertices by (label,
  // degree descending), a vertex's rank inside its class, and that rank of
  // every entry of ladj.  Class l is lorder[lstart[l] .. lstart[l + 1]).
  DevBuf<int32_t> lorder, lrank, lrk;
  std::vector<int64_t> lstart;
  struct CycleSpace *cycle = nullptr;  // 4-cycle scratch of single calls
  LabelCsr() = default;
  LabelCsr(const LabelCsr &) = delete;
  LabelCsr &operator=(const LabelCsr &) = delete;
  ~LabelCsr();
};

// [s, e): v's neighbours with label l inside its label-partitioned list,
// relative to off[v].  L == 0: the lists are not partitioned (labels >= 64),
// the whole list is scanned and the label test filters.
__device__ __forceinline__ void seg_range(const int64_t *__restrict__ off, const int32_t *__restrict__ loff, int L,
                                          int32_t v, int l, int64_t *s, int64_t *e) {
  if (L == 0) {
    *s = 0;
    *e = off[v + 1] - off[v];
  } else if (l < 0 || l >= L) {
    *s = *e = 0;
  } else {
    *s = loff[(int64_t)v * (L + 1) + l];
    *e = loff[(int64_t)v * (L + 1) + l + 1];
  }
}

// The lanes' segments of ladj (st, len) laid end to end, every lane taking
// one entry of the concatenation per round: f(t, valid, x) with x the entry
// and t the lane whose segment it lies in (called by all 32 lanes; valid is
// false past the end).
template <class F>
__device__ __forceinline__ void flat_segments(const int32_t *__restrict__ ladj, long long st, long long len, F f) {
  const unsigned lane = lane_id();
  long long inc = len;  // inclusive prefix over the lanes
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long v = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)lane >= o) inc += v;
  }
  const long long total = __shfl_sync(0xffffffffu, inc, 31);
  const long long first = st - (inc - len);  // entry idx of lane t's segment is ladj[first of t + idx]
  for (long long base = 0; base < total; base += 32) {
    const long long idx = base + lane;
    // t = first lane whose inclusive prefix exceeds idx
    int lo = 0, hi = 31;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      const int mid = (lo + hi) >> 1;
      const long long pm = __shfl_sync(0xffffffffu, inc, mid);
      if (pm > idx) hi = mid; else lo = mid + 1;
    }
    const long long ft = __shfl_sync(0xffffffffu, first, lo);
    const bool valid = idx < total;
    f(lo, valid, valid ? __ldg(ladj + ft + idx) : 0);
  }
}

// ---------------------------------------------------------------- 4-cycles (match_cycle.cu)
struct CycleSpace;  // device scratch; one per stream of work (a batch, or the graph's single calls)
void free_cycle_space(CycleSpace *s);

// A counted 4-cycle query on one data graph: opposite labels (la, lc), with
// the labels lb and ld between them.
struct CyclePlan {
  int la = 0, lb = 0, lc = 0, ld = 0;
};
// Is q a 4-cycle whose labels all occur as partitions of lc?
bool is_cycle4(const gpm_query *q, const LabelCsr *lc);
// Chooses the opposite pair and makes room for the launch (*space grows, or is
// created).  *fits = false: fewer than min_wedges wedges, or the counters would
// take too much memory; the query has to be walked.
int cycle_plan(gpm_graph *g, LabelCsr *lc, const gpm_query *q, unsigned long long min_wedges, CyclePlan *p,
               CycleSpace **space, bool *fits);
// Launches only: the count is added to out[member ? member[root] : 0].
int cycle_launch(const gpm_graph *g, const LabelCsr *lc, const CyclePlan &p, const CycleSpace *space,
                 const int32_t *member, unsigned long long *out, cudaStream_t st);

}  // namespace gpm
