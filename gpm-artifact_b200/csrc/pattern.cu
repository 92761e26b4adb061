// pattern.cu -- named patterns P1..P8 and Motif4 (G2MinerSolver,
// src/G2MinerSolver.cuh:17-176, and PatternSolver, src/PatternSolver.cuh:16-265).
//
// Both reference families compute, per stored edge (v0, v1) of the symmetric
// graph, the same nested set algebra (G2Miner with materialised lists,
// PatternSolver with frequency products minus corrections); on sorted
// duplicate-free lists they give the same counts:
//   P1, Motif4[0]  induced 3-stars            (motif pipeline, motif.cu)
//   P4, Motif4[1]  induced 4-paths            (motif pipeline)
//   Motif4[2..5]   tailed triangle, 4-cycle, diamond, 4-clique (motif pipeline)
//   P2 P3 P5 P6 P7 P8  enumerated here: one warp per stored edge, lists
//   materialised in per-warp global scratch with ballot compaction (order
//   preserved), membership by binary search in the longer list.
// The per-edge programs restate G2Miner_kernels.cuh:52-435.
#include <algorithm>
#include <string>

#include "common.cuh"
#include "motif.cuh"
#include "tc_rank.cuh"

namespace gpm {

constexpr int32_t kNoUb = 0x7fffffff;

__device__ __forceinline__ bool member(const int32_t *__restrict__ b, int nb, int32_t key) {
  int lo = 0, hi = nb - 1;
  while (lo <= hi) {
    int mid = (lo + hi) >> 1;
    int32_t x = __ldg(b + mid);
    if (x == key) return true;
    if (x < key) lo = mid + 1; else hi = mid - 1;
  }
  return false;
}

// out = {x in a : x < ub, (x in b) == keep_in}; returns |out| (warp-uniform).
// out == nullptr: count only.
__device__ int wset(const int32_t *a, int na, const int32_t *b, int nb, int32_t ub, bool keep_in, int32_t *out,
                    unsigned lane) {
  int cnt = 0;
  for (int base = 0; base < na; base += 32) {
    int i = base + lane;
    bool below = false, take = false;
    int32_t key = 0;
    if (i < na) {
      key = a[i];
      below = key < ub;
      take = below && (member(b, nb, key) == keep_in);
    }
    unsigned m = __ballot_sync(0xffffffffu, take);
    if (out && take) out[cnt + __popc(m & ((1u << lane) - 1u))] = key;
    cnt += __popc(m);
    if (__ballot_sync(0xffffffffu, i < na && !below)) break;  // sorted: the rest is >= ub
  }
  __syncwarp();
  return cnt;
}

__device__ __forceinline__ int wdiff(const int32_t *a, int na, const int32_t *b, int nb, int32_t ub, int32_t *out,
                                     unsigned lane) {
  return wset(a, na, b, nb, ub, false, out, lane);
}
__device__ __forceinline__ int wisect(const int32_t *a, int na, const int32_t *b, int nb, int32_t ub, int32_t *out,
                                      unsigned lane) {
  return wset(a, na, b, nb, ub, true, out, lane);
}
// NBR(v) expands to the (pointer, length) pair of v's sorted list
#define NBR(v) (adj + off[v]), (int)(off[(v) + 1] - off[v])
#define DIFF(...) wdiff(__VA_ARGS__, lane)
#define ISECT(...) wisect(__VA_ARGS__, lane)

// Heavy edges: both endpoints' lists together longer than `degree`.  Their
// outer loop is shared out over `parts` warps, each of which builds the lists
// for itself: an edge's cost grows with the cube of its degrees and more, and
// one warp on the heaviest edge held up the whole count.  P7 walks common
// neighbours alone, which are few, so its lists are what costs.  us per call,
// one warp per edge / (degree, parts) = (48, 16) / (96, 16) / (192, 16), Chung-
// Lu graphs: P5, 2,001 vertices 2918, 617, 715, 1764; P2, 801: 1745, 536, 1287,
// 1868; P3, 801: 1556, 780, 1750, 1631; P6, 2,001: 859, 242, 265, 502; P8, 20,001:
// 10164, 4681, 4464, 4646; P7, 4,099: 271, 324, 227, 179.  P7 at 192 with 1 / 4 / 8 / 16
// parts: Chung-Lu 4,099 x 9 203, 129, 120, 115, 20,001 x 9 612, 377, 457, 715, 3,001 x 30
// 893, 503, 524, 677.
struct HeavyRule {
  int64_t degree;
  int parts;
};
// And longer than kHeavyMean times the edges' mean: where all edges are alike, the
// parts build the same lists for nothing.  us, start of the sharing / without /
// with that bound: complete graph of 300, P2 1145, 7010, 559, P5 15051, 22810, 14832; ER
// 3,000 x 30, P6 781, 1079, 187; R-MAT 10 P6 57798, 4208, 5093 (bounds of 1.5 and 2
// times the mean: 5444, 10714).
constexpr double kHeavyMean = 1.25;
static HeavyRule heavy_rule(int p) { return p == 7 ? HeavyRule{192, 4} : HeavyRule{48, 16}; }
__global__ void k_heavy_edges(HeavyRule rule, int64_t nnz, const int64_t *__restrict__ off, const int32_t *__restrict__ adj,
                              const int32_t *__restrict__ src, uint32_t *__restrict__ heavy,
                              unsigned long long *__restrict__ nheavy) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < nnz; e += (int64_t)gridDim.x * blockDim.x) {
    const int32_t v0 = src[e], v1 = adj[e];
    if (off[v0 + 1] - off[v0] + off[v1 + 1] - off[v1] > rule.degree) heavy[atomicAdd(nheavy, 1ull)] = (uint32_t)e;
  }
}

// Pattern p on all edges that are not heavy (heavy == nullptr), or on the
// heavy ones, whose (edge, part) pairs come from the cursor *next.
__global__ void __launch_bounds__(256) k_pattern(int p, HeavyRule rule, int64_t nnz, const int64_t *__restrict__ off,
                                                 const int32_t *__restrict__ adj, const int32_t *__restrict__ src,
                                                 int32_t *__restrict__ scratch, int64_t maxd,
                                                 const uint32_t *__restrict__ heavy,
                                                 const unsigned long long *__restrict__ nheavy,
                                                 unsigned long long *__restrict__ next,
                                                 unsigned long long *__restrict__ out) {
  const unsigned lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int32_t *A = scratch + warp * maxd * 5, *B = A + maxd, *C = B + maxd, *D = C + maxd, *E = D + maxd;
  unsigned long long c = 0;
  const int step = heavy ? rule.parts : 1;
  const int64_t tasks = heavy ? (int64_t)*nheavy * rule.parts : nnz;
  for (int64_t t = warp; t < tasks; t += nw) {
    int64_t e = t;
    int part = 0;
    if (heavy) {  // t counts the warp's own rounds here; the task comes from the cursor
      unsigned long long q = 0;
      if (lane == 0) q = atomicAdd(next, 1ull);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= (unsigned long long)tasks) break;
      e = heavy[q / rule.parts];
      part = (int)(q % rule.parts);
      t = warp - nw;  // the cursor alone ends the loop
    }
    const int32_t v0 = src[e], v1 = adj[e];
    if (!heavy && off[v0 + 1] - off[v0] + off[v1 + 1] - off[v1] > rule.degree) continue;
    int nA, nB, nC, nD, nE;
    switch (p) {
      case 2:  // G2Miner_kernels.cuh:68-103
        nA = DIFF(NBR(v0), NBR(v1), kNoUb, A);
        nB = DIFF(NBR(v1), NBR(v0), kNoUb, B);
        for (int i = part; i < nB; i += step) {
          nC = DIFF(A, nA, NBR(B[i]), kNoUb, C);
          for (int j = 0; j < nC; ++j) c += DIFF(C, nC, NBR(C[j]), C[j], nullptr);
        }
        break;
      case 3:  // :126-157
        nA = DIFF(NBR(v0), NBR(v1), kNoUb, A);
        for (int i = part; i < nA; i += step) {
          nB = DIFF(A, nA, NBR(A[i]), A[i], B);
          for (int j = 0; j < nB; ++j) c += DIFF(B, nB, NBR(B[j]), B[j], nullptr);
        }
        break;
      case 5:  // :219-261
        nA = DIFF(NBR(v0), NBR(v1), kNoUb, A);
        nB = DIFF(NBR(v1), NBR(v0), kNoUb, B);
        nC = ISECT(NBR(v0), NBR(v1), kNoUb, C);
        for (int i = part; i < nC; i += step) {
          nD = DIFF(A, nA, NBR(C[i]), kNoUb, D);
          nE = DIFF(B, nB, NBR(C[i]), kNoUb, E);
          for (int j = 0; j < nD; ++j) c += DIFF(E, nE, NBR(D[j]), kNoUb, nullptr);
        }
        break;
      case 6:  // :281-318
        nC = ISECT(NBR(v0), NBR(v1), kNoUb, C);
        nB = DIFF(NBR(v1), NBR(v0), kNoUb, B);
        for (int i = part; i < nC; i += step) {
          nD = DIFF(C, nC, NBR(C[i]), kNoUb, D);
          nE = DIFF(B, nB, NBR(C[i]), kNoUb, E);
          for (int j = 0; j < nD; ++j) c += DIFF(E, nE, NBR(D[j]), kNoUb, nullptr);
        }
        break;
      case 7:  // :339-371
        nC = ISECT(NBR(v0), NBR(v1), kNoUb, C);
        for (int i = part; i < nC; i += step) {
          nD = DIFF(C, nC, NBR(C[i]), C[i], D);
          for (int j = 0; j < nD; ++j) c += DIFF(D, nD, NBR(D[j]), D[j], nullptr);
        }
        break;
      case 8:  // :394-430
        nC = ISECT(NBR(v0), NBR(v1), kNoUb, C);
        nB = DIFF(NBR(v1), NBR(v0), kNoUb, B);
        for (int i = part; i < nB; i += step) {
          nD = DIFF(C, nC, NBR(B[i]), kNoUb, D);
          for (int j = 0; j < nD; ++j) c += ISECT(D, nD, NBR(D[j]), D[j], nullptr);
        }
        break;
      default:
        break;
    }
  }
  if (lane == 0 && c) atomicAdd(out, c);
}

// Enumerated count of pattern p in {2,3,5,6,7,8} on the symmetric graph.
int pattern_enumerate(gpm_graph *g, int p, cudaStream_t st, uint64_t *result) {
  GPM_TRY(ensure_src(g, st));
  DevBuf<unsigned long long> d;
  GPM_TRY(d.reserve(3));  // the count, the heavy edges, their cursor
  GPM_CUDA(cudaMemsetAsync(d.p, 0, 24, st));
  const int64_t maxd = std::max(1, g->max_deg);
  // scratch: 5 lists of max degree per warp, capped at ~8 GB
  int64_t warps = (int64_t)num_sms() * 4 * 8;
  const int64_t cap_words = (int64_t)2 << 30;
  while (warps > 32 && warps * maxd * 5 > cap_words) warps >>= 1;
  DevBuf<int32_t> scratch;
  GPM_TRY(scratch.reserve((size_t)(warps * maxd * 5)));
  if (g->nnz > 0) {
    DevBuf<uint32_t> heavy;
    HeavyRule rule = heavy_rule(p);
    // nor are edges heavy that are like most others: the graph's heavy ones
    // are what holds up the count
    const double mean = 2.0 * (double)g->sum_deg2 / (double)g->nnz;  // of an edge's two list lengths
    rule.degree = std::max<int64_t>(rule.degree, (int64_t)(kHeavyMean * mean));
    if (g->nnz >= (1ll << 32)) rule.degree = INT64_MAX;  // edges are listed by 32-bit numbers
    bool some = 2 * maxd > rule.degree;
    if (some) {
      const int s = heavy.reserve(g->nnz);
      if (s != GPM_OK && s != GPM_ENOMEM) return s;
      if (s == GPM_ENOMEM) {  // no room for the list: a warp per edge, heavy or not
        some = false;
        rule.degree = INT64_MAX;
      }
    }
    if (some) {
      k_heavy_edges<<<(int)std::min<int64_t>((g->nnz + 255) / 256, num_sms() * 8), 256, 0, st>>>(
          rule, g->nnz, g->off.p, g->adj.p, g->src.p, heavy.p, d.p + 1);
      k_pattern<<<(int)(warps / 8), 256, 0, st>>>(p, rule, g->nnz, g->off.p, g->adj.p, g->src.p, scratch.p, maxd, heavy.p,
                                                  d.p + 1, d.p + 2, d.p);
    }
    k_pattern<<<(int)(warps / 8), 256, 0, st>>>(p, rule, g->nnz, g->off.p, g->adj.p, g->src.p, scratch.p, maxd, nullptr,
                                                nullptr, nullptr, d.p);
    GPM_LAUNCH_CHECK();
    GPM_CUDA(cudaStreamSynchronize(st));  // heavy is released here
  }
  unsigned long long h = 0;
  GPM_CUDA(cudaMemcpyAsync(&h, d.p, 8, cudaMemcpyDeviceToHost, st));
  GPM_CUDA(cudaStreamSynchronize(st));
  *result = h;
  return GPM_OK;
}

}  // namespace gpm

using namespace gpm;

extern "C" int gpm_pattern(gpm_graph *g, const char *name, int family, uint64_t *counters, uint64_t *result) {
  if (!g || !name || !result) return fail(GPM_EINVAL, "gpm_pattern: NULL argument");
  if (family != GPM_G2MINER && family != GPM_PATTERN_SOLVER) return fail(GPM_EINVAL, "unknown pattern family");
  if (g->oriented) return fail(GPM_EINVAL, "pattern counting runs on the symmetric (unoriented) graph");
  const std::string nm(name);
  uint64_t h[6] = {0, 0, 0, 0, 0, 0};
  uint64_t res = 0;
  int p = -1;
  if (nm == "Motif4") p = 0;
  else if (nm.size() == 2 && nm[0] == 'P' && nm[1] >= '1' && nm[1] <= '8') p = nm[1] - '0';
  if (p < 0) return fail(GPM_EINVAL, nm + " not support!");  // G2MinerSolver.cuh:157
  uint64_t m4[6];
  if (p == 0 || p == 1 || p == 4) {
    GPM_TRY(gpm_motif(g, 4, m4));
  }
  if (p == 0) {
    for (int i = 0; i < 6; ++i) h[i] = m4[i];
    // G2MinerSolver returns h_total[0]; PatternSolver h_total[1] - h_total[2]
    res = family == GPM_G2MINER ? h[0] : h[1] - h[2];
  } else {
    uint64_t cnt = 0;
    if (p == 1) cnt = m4[0];
    else if (p == 4) cnt = m4[1];
    else GPM_TRY(pattern_enumerate(g, p, 0, &cnt));
    res = cnt;
    // G2Miner accumulates into counters[0]; PatternSolver reports counters[1]
    // (minus the correction it keeps in counters[2], folded in here).
    if (family == GPM_G2MINER) h[0] = cnt;
    else h[1] = cnt;
  }
  if (counters)
    for (int i = 0; i < 6; ++i) counters[i] = h[i];
  *result = res;
  return GPM_OK;
}
