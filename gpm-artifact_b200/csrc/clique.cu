// clique.cu -- k-clique counting (CFSolver, src/CFSolver.cuh:15-158).
//
// The reference counts, for every stored edge (v0,v1), the cliques grown by
// nested materialised intersections W1 = N(v0) & N(v1), W2 = W1 & N(v2), ...
// (clique_4_edge_warp / clique_5_edge_warp).  On a degree-oriented DAG that
// is the number of k-cliques.
//
// B200 path (upward rank graph, see tc_rank.cuh): a vertex task u turns its
// out-list L = N+(u) into a local DAG whose adjacency rows are bitsets
// (row_i = {j : L[j] in N+(L[i])}).  Because the rank graph points upward,
// row_i only has bits j > i, so the (k-1)-cliques of the local DAG are found
// by consuming bits in increasing order and AND-ing rows -- popcounts instead
// of list intersections.
//   * tasks with |L| <= 64: one warp, rows are uint64 held in shared memory,
//     one lane per starting row;
//   * tasks with 64 < |L| <= 2048: one CTA, rows of W = ceil(|L|/32) words
//     in shared memory (or a per-CTA global slab when they do not fit).
// Building the rows is most of the work of a 4-clique count (R-MAT 20: 4.2 G
// list entries looked up in L, 1.4 G row words ANDed afterwards), so an entry
// is looked up in a hash table of L's positions, a row whose list is much
// longer than the rest of L looks that rest up in the list instead, and hubs
// answer for the top ranks from a bitmap.  R-MAT 20, 4-cliques: 24.1 ms with a
// binary search of L per entry, 13.2 ms with table and search, 7.6 ms with the
// bitmaps too, 5.8 ms with the rows ANDed strip by strip (cq_pairs; a row word
// per thread kept 11 of 32 lanes active): 4.7 ms CTA tasks, 75 % issue-active,
// and 1.1 ms warp tasks.
// Graphs whose stored edges do not all point upward in rank order, or with
// an out-list longer than 2048, use an edge-centric kernel shaped like the
// reference (materialised lists in per-warp global scratch).
#include <cub/cub.cuh>

#include <algorithm>

#include "common.cuh"
#include "motif.cuh"
#include "tc_rank.cuh"

namespace gpm {

constexpr int kCqWarpMax = 64;      // warp tasks: |L| <= 64
constexpr int kCqCtaMax = 2048;     // CTA tasks: |L| <= 2048 (W <= 64)
constexpr int kCqMaxK = 8;
// A row's list is searched for the rest of L when it is more than this many
// times longer: a search is some ten dependent loads, a lookup one or two
// shared-memory reads.
constexpr int kCqSearch = 6;
// Vertices with at least kCqCoreMin neighbours above them among the top kCqCore ranks
// keep those as a bitmap (2 KB): whether they are adjacent to the rest of L
// is then one bit test per member.
constexpr int64_t kCqCore = 16384;
constexpr int kCqCoreMin = 64;
struct CqCore {
  const int32_t *rowid;  // nullptr: no bitmaps
  const uint32_t *rows;
  int32_t base;
  int words;
};
// CTA tasks whose layout (cq_layout) fits in kCqSmemSmall run in 256-thread CTAs, several per SM; larger ones in
// 512-thread CTAs with kCqSmemBig, two per SM, and beyond that in a slab.
constexpr size_t kCqSmemSmall = 44 * 1024, kCqSmemBig = 112 * 1024;
constexpr int kCqSmallThreads = 256, kCqBigThreads = 512;
// Cliques of other sizes than 4 and 5 walk a row's set in one warp while the
// others of its CTA wait at the end of the task, so they run in 256-thread
// CTAs (k_clique_any), rows past kCqSmemAny in the slab.  The heaviest tasks end
// the count: few CTAs per SM finish each of them sooner, and the warp tasks run
// beside them on the caller's stream and fill what they leave.  ms with 5 / 4 / 3 / 2
// CTAs per SM (the warp tasks inside the same kernel), in brackets 3 as it is:
// R-MAT 16, k = 6: 117 / 116 / 108 / 130 (108), R-MAT 17, k = 6: 300 / 292 / 301 / 372 (300),
// R-MAT 14, k = 7: 300 / 302 / 289 / 280 (289), Chung-Lu 300,001, k = 6: 0.58 / 0.66 /
// 0.81 / - (0.53).  (4 and 5 CTAs, the warp tasks after them: R-MAT 16 119, R-MAT 14
// 360; 5 CTAs on rows from a binary search: 108, 294, 328, 0.83.)
constexpr size_t kCqSmemAny = 40 * 1024;
constexpr int kCqAnyThreads = 256, kCqAnyPerSm = 3;
constexpr int kCqFewPerSm = 5;  // CTAs of k_clique_warp per SM where each warp gets few tasks
__host__ __device__ constexpr bool cq_any(int k) { return k != 4 && k != 5; }

static int grid_for(int64_t work, int block = 256) {
  int64_t g = (work + block - 1) / block;
  int64_t cap = (int64_t)num_sms() * 16;
  return (int)std::max<int64_t>(1, std::min(g, cap));
}

// Positions of L's keys in an open-addressing table of 2^logcap slots (P =
// uint8_t or uint16_t, all ones = empty); the key itself is read from L.
template <class P>
__device__ __forceinline__ int find_pos(const P *tab, int logcap, const int32_t *L, int32_t key) {
  const uint32_t mask = (1u << logcap) - 1u;
  uint32_t h = ((uint32_t)key * 2654435769u) >> (32 - logcap);
  while (true) {
    const int p = tab[h];
    if (p == (int)(P)~(P)0) return -1;
    if (L[p] == key) return p;
    h = (h + 1) & mask;
  }
}

// Is key in the sorted list a[0 .. n)?
__device__ __forceinline__ bool in_list(const int32_t *__restrict__ a, int64_t n, int32_t key) {
  int64_t lo = 0, hi = n - 1;
  while (lo <= hi) {
    const int64_t mid = (lo + hi) >> 1;
    const int32_t x = __ldg(a + mid);
    if (x == key) return true;
    if (x < key) lo = mid + 1; else hi = mid - 1;
  }
  return false;
}

// first index in sorted a[0..n) with a[i] > key
__device__ __forceinline__ int64_t upper_bound_g(const int32_t *__restrict__ a, int64_t n, int32_t key) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if (__ldg(a + mid) <= key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// ------------------------------------------------------------ warp tasks (|L| <= 64)
// number of q-cliques inside bitset X of the local DAG (q >= 1)
__device__ unsigned long long local_count64(const unsigned long long *rows, unsigned long long X, int q) {
  if (q == 1) return __popcll(X);
  if (q == 2) {
    unsigned long long c = 0;
    while (X) {
      int l = __ffsll(X) - 1;
      X &= X - 1;
      c += __popcll(X & rows[l]);
    }
    return c;
  }
  unsigned long long stk[kCqMaxK];
  int depth = 0;
  stk[0] = X;
  unsigned long long c = 0;
  // stk[depth] holds the candidates still to extend at level depth; a set
  // at level depth needs q - depth more vertices.
  while (depth >= 0) {
    unsigned long long &S = stk[depth];
    if (!S) { --depth; continue; }
    int l = __ffsll(S) - 1;
    S &= S - 1;
    unsigned long long Y = S & rows[l];
    int left = q - depth - 1;  // vertices still needed after picking l
    if (left == 1) c += __popcll(Y);
    else if (left == 2) {
      while (Y) {
        int m = __ffsll(Y) - 1;
        Y &= Y - 1;
        c += __popcll(Y & rows[m]);
      }
    } else if (Y) stk[++depth] = Y;
  }
  return c;
}

// Shared memory of a warp task.  Row i's list part that can meet L is radj[st[i]
// .. st[i] + len[i]); scan[i] / pair[i]: inclusive prefixes of the entries to
// look up in L, and of the pairs (i, j > i) to search in row i's list.
struct CqWarp {
  unsigned long long rows[kCqWarpMax];
  int64_t st[kCqWarpMax];
  int32_t L[kCqWarpMax], len[kCqWarpMax], scan[kCqWarpMax], pair[kCqWarpMax];
  uint8_t tab[256];
};

// first i of 32 or (two) 64 with pre[i] > x (pre inclusive, x < its last)
__device__ __forceinline__ int segment_of(const int32_t *pre, bool two, int x) {
  int lo = two && pre[31] <= x ? 32 : 0;
#pragma unroll
  for (int s = 16; s; s >>= 1)
    if (pre[lo + s - 1] <= x) lo += s;
  return lo;
}

__device__ unsigned long long clique_warp_task(int32_t u, int k, const int64_t *__restrict__ roff,
                                               const int32_t *__restrict__ radj, CqWarp &sm) {
  const unsigned lane = lane_id();
  const int64_t s0 = roff[u];
  const int d = (int)(roff[u + 1] - s0);
  reinterpret_cast<uint2 *>(sm.tab)[lane] = make_uint2(~0u, ~0u);
  const int halves = d > 32 ? 2 : 1;
  for (int h = 0; h < halves; ++h) {
    const int i = (int)lane + 32 * h;
    if (i < d) sm.L[i] = radj[s0 + i];
    sm.rows[i] = 0ull;
  }
  __syncwarp();
  const int32_t kmax = sm.L[d - 1];
  int carry_s = 0, carry_p = 0;
  for (int h = 0; h < halves; ++h) {
    const int i = (int)lane + 32 * h;
    int ns = 0, np = 0;
    if (i < d) {
      const int32_t v = sm.L[i];
      // position i under v's hash; bytes are claimed through their word
      uint32_t slot = ((uint32_t)v * 2654435769u) >> 24;
      while (true) {
        unsigned *word = reinterpret_cast<unsigned *>(sm.tab) + (slot >> 2);
        const unsigned sh = (slot & 3) * 8, old = *(volatile unsigned *)word;
        if (((old >> sh) & 255u) == 255u) {
          if (atomicCAS(word, old, (old & ~(255u << sh)) | ((unsigned)i << sh)) == old) break;
        } else {
          slot = (slot + 1) & 255u;
        }
      }
      const int64_t s = roff[v];
      const int len = (int)upper_bound_g(radj + s, roff[v + 1] - s, kmax), rest = d - 1 - i;
      sm.st[i] = s;
      sm.len[i] = len;
      if (rest * kCqSearch < len) np = rest;
      else ns = len;
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int vs = __shfl_up_sync(0xffffffffu, ns, o), vp = __shfl_up_sync(0xffffffffu, np, o);
      if ((int)lane >= o) {
        ns += vs;
        np += vp;
      }
    }
    ns += carry_s;
    np += carry_p;
    sm.scan[i] = ns;
    sm.pair[i] = np;
    carry_s = __shfl_sync(0xffffffffu, ns, 31);
    carry_p = __shfl_sync(0xffffffffu, np, 31);
  }
  __syncwarp();
  // both kinds of work laid end to end, so short lists leave no lanes idle
  for (int x = lane; x < carry_s; x += 32) {
    const int i = segment_of(sm.scan, d > 32, x);
    const int p = find_pos(sm.tab, 8, sm.L, __ldg(radj + sm.st[i] + (x - (sm.scan[i] - sm.len[i]))));
    if (p >= 0) atomicOr(&sm.rows[i], 1ull << p);
  }
  for (int x = lane; x < carry_p; x += 32) {
    const int i = segment_of(sm.pair, d > 32, x);
    const int j = d - (sm.pair[i] - x);
    if (in_list(radj + sm.st[i], sm.len[i], sm.L[j])) atomicOr(&sm.rows[i], 1ull << j);
  }
  __syncwarp();
  unsigned long long c = 0;
  for (int i = lane; i < d; i += 32) c += local_count64(sm.rows, sm.rows[i], k - 2);
  __syncwarp();
  return c;
}

// ------------------------------------------------------------ CTA tasks (64 < |L| <= 2048)
// Bitsets of W <= 64 words spread over a warp: lane w holds words w, w + 32.
struct WarpSet {
  uint32_t a, b;
};
__device__ __forceinline__ int wpop(WarpSet s) { return __popc(s.a) + __popc(s.b); }

// Lowest set bit of a warp-spread set, cleared in place; -1 if empty.
__device__ __forceinline__ int wtake(WarpSet &s, unsigned lane) {
  unsigned m = __ballot_sync(0xffffffffu, s.a != 0);
  int base = 0;
  uint32_t word;
  int f;
  if (m) {
    f = __ffs(m) - 1;
    word = __shfl_sync(0xffffffffu, s.a, f);
  } else {
    m = __ballot_sync(0xffffffffu, s.b != 0);
    if (!m) return -1;
    f = __ffs(m) - 1;
    word = __shfl_sync(0xffffffffu, s.b, f);
    base = 1024;
  }
  int bit = __ffs(word) - 1;
  if ((int)lane == f) {
    if (base) s.b &= s.b - 1; else s.a &= s.a - 1;
  }
  return base + f * 32 + bit;
}

__device__ __forceinline__ WarpSet wrow(const uint32_t *rows, int W, int j, unsigned lane) {
  const uint32_t *r = rows + (size_t)j * W;
  WarpSet s;
  s.a = (int)lane < W ? r[lane] : 0u;
  s.b = (int)lane + 32 < W ? r[lane + 32] : 0u;
  return s;
}

// index of the k-th (0-based) set bit of w (k < popc(w))
__device__ __forceinline__ int kth_bit(uint32_t w, int k) {
  int pos = 0;
#pragma unroll
  for (int s = 16; s; s >>= 1) {
    const int c = __popc(w & ((1u << s) - 1u));
    if (k >= c) {
      k -= c;
      w >>= s;
      pos += s;
    }
  }
  return pos;
}

// Sum over l in X of |X & row_l| -- the 2-cliques inside warp-spread X --
// with the members l of X spread over the lanes: lane t takes the t-th
// member of each round of 32 and ANDs X (staged in the warp's shared words
// xs) with its row word by word from l's own word on (row_l has no bits
// below l).  Each lane returns its partial sum.
__device__ unsigned long long wsum_pairs(const uint32_t *rows, int W, WarpSet X, uint32_t *xs, unsigned lane) {
  __syncwarp();
  xs[lane] = X.a;
  xs[lane + 32] = X.b;
  __syncwarp();
  // members are numbered word by word: words 0..31 (X.a of lanes 0..31), then 32..63
  int inc = __popc(X.a), incb = __popc(X.b);
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int va = __shfl_up_sync(0xffffffffu, inc, o), vb = __shfl_up_sync(0xffffffffu, incb, o);
    if ((int)lane >= o) {
      inc += va;
      incb += vb;
    }
  }
  const int ta = __shfl_sync(0xffffffffu, inc, 31), total = ta + __shfl_sync(0xffffffffu, incb, 31);
  unsigned long long c = 0;
  for (int base = 0; base < total; base += 32) {
    const int idx = base + (int)lane;
    // word holding member idx: first word whose inclusive prefix exceeds it
    const bool hi = idx >= ta;
    const int key = hi ? idx - ta : idx;
    int lo = 0, up = 31;
#pragma unroll
    for (int r = 0; r < 5; ++r) {
      const int mid = (lo + up) >> 1;
      const int pa = __shfl_sync(0xffffffffu, inc, mid), pb = __shfl_sync(0xffffffffu, incb, mid);
      if ((hi ? pb : pa) > key) up = mid; else lo = mid + 1;
    }
    const int pa_lo = __shfl_sync(0xffffffffu, inc, lo), pb_lo = __shfl_sync(0xffffffffu, incb, lo);
    if (idx < total) {
      const int w = lo + (hi ? 32 : 0);
      const uint32_t word = xs[w];
      const int excl = (hi ? pb_lo : pa_lo) - __popc(word);
      const int l = w * 32 + kth_bit(word, key - excl);
      const uint32_t *rl = rows + (size_t)l * W;
      unsigned s = 0;
      for (int ww = l >> 5; ww < W; ++ww) s += __popc(xs[ww] & rl[ww]);
      c += s;
    }
  }
  return c;
}

// q-cliques inside warp-spread X; stk holds (q) levels of W words per warp
__device__ unsigned long long warp_count_set(const uint32_t *rows, int W, WarpSet X, int q, uint32_t *xs,
                                             unsigned lane) {
  if (q == 1) return (unsigned long long)wpop(X);
  if (q == 2) return wsum_pairs(rows, W, X, xs, lane);
  WarpSet stk[kCqMaxK];
  int depth = 0;
  stk[0] = X;
  unsigned long long c = 0;
  while (depth >= 0) {
    int l = wtake(stk[depth], lane);
    if (l < 0) { --depth; continue; }
    WarpSet r = wrow(rows, W, l, lane);
    WarpSet Y{stk[depth].a & r.a, stk[depth].b & r.b};
    int left = q - depth - 1;
    if (left == 1) c += (unsigned long long)wpop(Y);
    else if (left == 2) c += wsum_pairs(rows, W, Y, xs, lane);
    else stk[++depth] = Y;
  }
  return c;
}

// ------------------------------------------------------------ compaction (5-cliques)
// The bits of y selected by a mask moved together to the low end, the mask
// given by its five move words (compress by parallel suffix: H. S. Warren,
// Hacker's Delight, section 7-4).
__device__ __forceinline__ void compact_moves(uint32_t m, uint32_t *mv) {
  uint32_t mk = ~m << 1;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    uint32_t mp = mk ^ (mk << 1);
    mp ^= mp << 2;
    mp ^= mp << 4;
    mp ^= mp << 8;
    mp ^= mp << 16;
    const uint32_t v = mp & m;
    mv[i] = v;
    m = (m ^ v) | (v >> (1 << i));
    mk &= ~mp;
  }
}
__device__ __forceinline__ uint32_t compact_bits(uint32_t y, const uint32_t *mv) {
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const uint32_t t = y & mv[i];
    y = (y ^ t) | (t >> (1 << i));
  }
  return y;
}

// Rows of up to kCqWarpX members are compacted and counted by one warp.
// Words of its buffer: move words and bit offsets of W row words, then
// kCqWarpX rows of kCqWarpX bits and their members.
constexpr int kCqWarpX = 128;
__host__ __device__ constexpr size_t cq_warp_words(int W) {
  return ((size_t)6 * W + 3) / 4 * 4 + kCqWarpX * (kCqWarpX / 32) + kCqWarpX / 2;
}

// Shared-memory layout of a CTA task in words (16-byte aligned parts).  comp:
// the warps' buffers, and the CTA's own compacted rows when those are done.
struct CqLayout {
  size_t tab, xl, heavy, moves, comp, comp_words, rows, total;
  int logcap;
};
// Words from one row to the next: cq_pairs reads 4-cliques' rows 16 bytes at a time.
__host__ __device__ constexpr int cq_stride(int W, int k) { return k == 4 ? (W + 3) & ~3 : W; }
__host__ __device__ inline CqLayout cq_layout(int d, int k, int nwarps, bool rows_in) {
  CqLayout l;
  const int W = (d + 31) >> 5;
  l.logcap = 8;
  while ((1 << l.logcap) < 4 * d && l.logcap < 12) ++l.logcap;
  l.tab = ((size_t)d + 3) & ~(size_t)3;
  l.xl = l.tab + ((size_t)1 << l.logcap) / 2;
  const size_t list = k == 5 ? (((size_t)d + 1) / 2 + 3) & ~(size_t)3 : 0;
  l.heavy = l.xl + list;
  l.moves = l.heavy + list;
  l.comp = l.moves + (k == 5 ? (6 * (size_t)W + 3) & ~(size_t)3 : 0);
  l.comp_words = k == 5 ? nwarps * cq_warp_words(W) : 0;
  l.rows = l.comp + l.comp_words;
  l.total = l.rows + (rows_in ? (size_t)d * cq_stride(W, k) : 0);
  return l;
}

// Members of X = a row of W <= 64 words (lane: words lane, lane + 32), their
// number, and per word the compaction moves and first position: mem[0 .. m),
// mv[6 w ..].  One warp; mem == nullptr: the number alone.
__device__ __forceinline__ int cq_members(const uint32_t *ri, int W, unsigned lane, uint16_t *mem, uint32_t *mv) {
  int run = 0;
  for (int w0 = 0; w0 < W; w0 += 32) {
    const int w = w0 + (int)lane;
    uint32_t word = w < W ? ri[w] : 0u;
    const int nb = __popc(word);
    int inc = nb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, inc, o);
      if ((int)lane >= o) inc += v;
    }
    if (mem && w < W) {
      int at = run + inc - nb;
      mv[6 * w + 5] = at;
      compact_moves(word, mv + 6 * w);
      for (; word; word &= word - 1) mem[at++] = (uint16_t)(w * 32 + __ffs(word) - 1);
    }
    run += __shfl_sync(0xffffffffu, inc, 31);
  }
  return run;
}

// Rows of the members x0 .. x0 + 31 (lane: x0 + lane) compacted to X's
// columns: comp + x * stride, stride words of which the last are zero.  The
// columns fill up word by word at the same pace in every lane.
__device__ __forceinline__ void cq_compact(const uint32_t *rows, const uint32_t *ri, int W, const uint16_t *mem, int m,
                                           int x0, const uint32_t *mv, uint32_t *comp, int stride, unsigned lane) {
  const int x = x0 + (int)lane;
  if (x >= m) return;
  const uint32_t *rl = rows + (int)mem[x] * W;
  uint32_t *cx = comp + x * stride;
  unsigned long long acc = 0;
  int at = 0, fill = 0;  // words written, bits pending
  for (int w = 0; w < W; ++w) {
    const uint32_t mask = ri[w];
    if (!mask) continue;
    acc |= (unsigned long long)compact_bits(rl[w] & mask, mv + 6 * w) << fill;
    fill += __popc(mask);
    if (fill >= 32) {
      cx[at++] = (uint32_t)acc;
      acc >>= 32;
      fill -= 32;
    }
  }
  for (; at < stride; ++at) {
    cx[at] = (uint32_t)acc;
    acc = 0;
  }
}

// Pairs (a, b) of the compacted rows, a in 32 r + lane, b a member of word w
// of row a: the common members of both in the NW words from column word q on.
// All lanes walk the same word and the same columns, so they differ only in
// how many members their word has.
template <int NW>
__device__ __forceinline__ unsigned cq_pairs(const uint32_t *comp, int stride, int m, int r, int w, int q,
                                             unsigned lane) {
  const int a = 32 * r + (int)lane;
  uint32_t own[NW], oth[NW];
  uint32_t word = 0;
  if (a < m) {
    word = comp[a * stride + w];
#pragma unroll
    for (int i = 0; i < NW; ++i) own[i] = comp[a * stride + q + i];
  }
  unsigned s = 0;
  for (; word; word &= word - 1) {
    const uint32_t *cb = comp + (w * 32 + __ffs(word) - 1) * stride + q;
    if (NW == 4) {
      const uint4 t = *reinterpret_cast<const uint4 *>(cb);
      oth[0] = t.x, oth[1] = t.y, oth[2 % NW] = t.z, oth[3 % NW] = t.w;
    } else {
      const uint2 t = *reinterpret_cast<const uint2 *>(cb);
      oth[0] = t.x, oth[1] = t.y;
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) s += __popc(own[i] & oth[i]);
  }
  return s;
}

// One vertex task on a CTA.  SM: the rows are in shared memory (smem), else in
// the CTA's slab (two halves of slab_half words: rows, compacted rows; without rows the
// first half holds the compacted ones).  Each
// thread returns its part of the count.
template <int KM, bool SM>
__device__ unsigned long long clique_cta_task(int32_t u, int k, const int64_t *__restrict__ roff,
                                              const int32_t *__restrict__ radj, uint32_t *smem, uint32_t *slab, size_t slab_half,
                                              const CqCore &core, uint32_t *xs) {
  const int tid = threadIdx.x, nthr = blockDim.x, wid = tid >> 5, nw = nthr >> 5;
  const unsigned lane = tid & 31;
  const int64_t s0 = roff[u];
  const int d = (int)(roff[u + 1] - s0);
  const int W = (d + 31) >> 5, RS = KM == 4 ? cq_stride(W, 4) : W;
  const CqLayout lay = cq_layout(d, k, nw, SM);
  int32_t *L = reinterpret_cast<int32_t *>(smem);
  uint16_t *tab = reinterpret_cast<uint16_t *>(smem + lay.tab);
  uint32_t *rows = SM ? smem + lay.rows : slab;
  for (int i = tid; i < d; i += nthr) L[i] = radj[s0 + i];
  for (int i = tid; i < (1 << lay.logcap) / 2; i += nthr) smem[lay.tab + i] = ~0u;
  for (int i = tid; i < d * RS; i += nthr) rows[i] = 0u;
  __syncthreads();
  for (int i = tid; i < d; i += nthr) {
    uint32_t h = ((uint32_t)L[i] * 2654435769u) >> (32 - lay.logcap);
    while (atomicCAS(reinterpret_cast<unsigned short *>(tab) + h, (unsigned short)0xffff, (unsigned short)i) != 0xffff)
      h = (h + 1) & ((1u << lay.logcap) - 1u);
  }
  __syncthreads();
  const int32_t kmax = L[d - 1];
  int jc = d;  // first position in the core
  if (core.rowid) {
    int lo = 0;
    while (lo < jc) {
      const int mid = (lo + jc) >> 1;
      if (L[mid] < core.base) lo = mid + 1; else jc = mid;
    }
  }
  // warp wid builds rows wid, wid + nw, ...; the scan ranges of 32 of them at
  // a time are found in parallel, one lane per row.  With a bitmap row, only
  // the keys below the core are looked up.
  for (int i0 = wid; i0 < d; i0 += nw * 32) {
    const int mine = i0 + (int)lane * nw;
    long long ms = 0;
    int mlen = 0, mrow = -1;
    if (mine < d) {
      const int32_t v = L[mine];
      if (core.rowid && jc < d) mrow = core.rowid[v];
      if (mrow < 0 || mine + 1 < jc) {
        ms = roff[v];
        mlen = (int)upper_bound_g(radj + ms, roff[v + 1] - ms, mrow < 0 ? kmax : core.base - 1);
      }
    }
    for (int j = 0; j < 32 && i0 + j * nw < d; ++j) {
      const int i = i0 + j * nw, len = __shfl_sync(0xffffffffu, mlen, j), row = __shfl_sync(0xffffffffu, mrow, j);
      const int32_t *__restrict__ list = radj + __shfl_sync(0xffffffffu, ms, j);
      uint32_t *ri = rows + i * RS;
      const int jend = row < 0 ? d : jc;  // positions from jend on by the bitmap
      if (row >= 0) {
        const uint32_t *__restrict__ bits = core.rows + (size_t)row * core.words;
        const int first = max(i + 1, jc);
        for (int b = first & ~31; b < d; b += 32) {
          const int q = b + (int)lane;
          bool in = false;
          if (q >= first && q < d) {
            const unsigned o = (unsigned)(L[q] - core.base);
            in = (__ldg(bits + (o >> 5)) >> (o & 31)) & 1u;
          }
          const unsigned m = __ballot_sync(0xffffffffu, in);
          if (lane == 0 && m) ri[b >> 5] = m;
        }
        __syncwarp();
        if (i + 1 >= jc) continue;
      }
      if ((jend - 1 - i) * kCqSearch < len) {  // the rest of L searched in the list, a word of the row at a time
        for (int b = (i + 1) & ~31; b < jend; b += 32) {
          const int q = b + (int)lane;
          const unsigned m = __ballot_sync(0xffffffffu, q > i && q < jend && in_list(list, len, L[q]));
          if (lane == 0 && m) ri[b >> 5] |= m;
        }
        continue;
      }
      int t = lane;
      for (; t + 32 < len; t += 64) {
        const int32_t x0 = __ldg(list + t), x1 = __ldg(list + t + 32);
        const int p0 = find_pos(tab, lay.logcap, L, x0);
        if (p0 >= 0) atomicOr(&ri[p0 >> 5], 1u << (p0 & 31));
        const int p1 = find_pos(tab, lay.logcap, L, x1);
        if (p1 >= 0) atomicOr(&ri[p1 >> 5], 1u << (p1 & 31));
      }
      if (t < len) {
        const int p = find_pos(tab, lay.logcap, L, __ldg(list + t));
        if (p >= 0) atomicOr(&ri[p >> 5], 1u << (p & 31));
      }
    }
  }
  __syncthreads();
  unsigned long long c = 0;
  if (KM == 4) {
    // (strip r, word w >= r, columns from 4 (w / 4) on; row_l has no bits below l)
    const int strips = W;
    unsigned s = 0;
    int t = 0;
    for (int w = 0; w < strips; ++w)
      for (int q = w & ~3; q < strips; q += 4)
        for (int r = 0; r <= w; ++r, ++t)
          if (t % nw == wid) s += cq_pairs<4>(rows, RS, d, r, w, q, lane);
    c += s;
  } else if (KM == 5) {
    // For each row i, the triangles of the local DAG inside X = row_i: the
    // rows of X's members are compacted to X's columns (|X| bits in place of
    // |L|, R-MAT 20: 91 of 350 for |L| in 257 .. 512), then every member pair
    // ANDs compacted rows.  Rows of up to kCqWarpX members by one warp each;
    // the others are listed and taken by the whole CTA afterwards.  R-MAT 19 /
    // 20: 71 / 188 ms on full-width rows, 22.3 / 66 ms compacted.
    uint16_t *xl = reinterpret_cast<uint16_t *>(smem + lay.xl);
    uint16_t *heavy = reinterpret_cast<uint16_t *>(smem + lay.heavy);
    __shared__ int s_heavy;
    if (tid == 0) s_heavy = 0;
    __syncthreads();
    {
      uint32_t *wmv = smem + lay.comp + wid * cq_warp_words(W);
      uint32_t *cr = wmv + (6 * W + 3) / 4 * 4;
      uint16_t *mem = reinterpret_cast<uint16_t *>(cr + kCqWarpX * (kCqWarpX / 32));
      for (int i = wid; i < d; i += nw) {
        const uint32_t *ri = rows + i * W;
        int m = cq_members(ri, W, lane, nullptr, nullptr);
        if (m < 3) continue;
        if (m > kCqWarpX) {
          if (lane == 0) heavy[atomicAdd(&s_heavy, 1)] = (uint16_t)i;
          continue;
        }
        cq_members(ri, W, lane, mem, wmv);
        __syncwarp();
        const int stride = m <= 64 ? 2 : 4, strips = (m + 31) >> 5;
        for (int x0 = 0; x0 < m; x0 += 32) cq_compact(rows, ri, W, mem, m, x0, wmv, cr, stride, lane);
        __syncwarp();
        unsigned s = 0;
        for (int w = 0; w < strips; ++w)
          for (int r = 0; r <= w; ++r)
            s += m <= 64 ? cq_pairs<2>(cr, 2, m, r, w, 0, lane) : cq_pairs<4>(cr, 4, m, r, w, 0, lane);
        c += s;
        __syncwarp();
      }
    }
    __syncthreads();
    const int nh = s_heavy;
    __syncthreads();  // s_heavy becomes |X| below
    uint32_t *mv = smem + lay.moves;
    for (int hi = 0; hi < nh; ++hi) {
      const uint32_t *ri = rows + heavy[hi] * W;
      if (wid == 0) {
        const int m = cq_members(ri, W, lane, xl, mv);
        if (lane == 0) s_heavy = m;
      }
      __syncthreads();
      const int m = s_heavy, strips = (m + 31) >> 5, stride = (strips + 3) & ~3;
      // the slab holds what the warps' buffers have no room for
      uint32_t *comp = (size_t)m * stride <= lay.comp_words ? smem + lay.comp : slab + (SM ? 0 : slab_half);
      for (int r = wid; r < strips; r += nw) cq_compact(rows, ri, W, xl, m, 32 * r, mv, comp, stride, lane);
      __syncthreads();
      // (r <= w, four column words from 4 (w / 4) on): small w first, they have most columns
      unsigned s = 0;
      int t = 0;
      for (int w = 0; w < strips; ++w)
        for (int q = w & ~3; q < strips; q += 4)
          for (int r = 0; r <= w; ++r, ++t)
            if (t % nw == wid) s += cq_pairs<4>(comp, stride, m, r, w, q, lane);
      c += s;
      __syncthreads();
    }
  } else {
    // each lane accumulates the popcounts of its own words; the warp sum is the
    // count.  Rows differ far in their work and the first hold most: taken one
    // by one
    __shared__ int s_row;
    if (tid == 0) s_row = 0;
    __syncthreads();
    while (true) {
      int i = 0;
      if (lane == 0) i = atomicAdd(&s_row, 1);
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i >= d) break;
      c += warp_count_set(rows, W, wrow(rows, W, i, lane), k - 2, xs, lane);
    }
  }
  __syncthreads();
  return c;
}

// The CTA tasks of a queue, heaviest first, in WORDS words of shared memory.
// KM: 4, 5, or 0 for the other clique sizes.  SLAB: rows that do not fit are in
// the CTA's slab.
template <int KM, bool SLAB, size_t WORDS>
__device__ __forceinline__ void clique_cta(int k, const int64_t *__restrict__ roff, const int32_t *__restrict__ radj,
                                           const int32_t *__restrict__ tasks, int ntasks, int *__restrict__ cursor,
                                           uint32_t *smem, uint32_t *slab, size_t slab_half, const CqCore &core,
                                           uint32_t *xs, const int32_t *__restrict__ gid,
                                           unsigned long long *__restrict__ acc, int stride, int slot) {
  __shared__ int s_task;
  const unsigned lane = threadIdx.x & 31;
  while (true) {
    if (threadIdx.x == 0) s_task = atomicAdd(cursor, 1);
    __syncthreads();
    int t = s_task;
    __syncthreads();
    if (t >= ntasks) break;
    const int32_t u = tasks[t];
    unsigned long long c;
    if (SLAB && cq_layout((int)(roff[u + 1] - roff[u]), k, blockDim.x / 32, true).total > WORDS)
      c = clique_cta_task<KM, false>(u, k, roff, radj, smem, slab, slab_half, core, xs);
    else
      c = clique_cta_task<KM, true>(u, k, roff, radj, smem, slab, slab_half, core, xs);
    c = warp_sum(c);
    if (lane == 0 && c) atomicAdd(&acc[(size_t)stride * (gid ? gid[u] : 0) + slot], c);
  }
}

template <int KM, bool BIG>
__global__ void __launch_bounds__(BIG ? kCqBigThreads : kCqSmallThreads)
    k_clique_cta(int k, const int64_t *__restrict__ roff, const int32_t *__restrict__ radj,
                 const int32_t *__restrict__ tasks, int ntasks, int *__restrict__ cursor, uint32_t *__restrict__ slabs,
                 size_t slab_half, CqCore core, const int32_t *__restrict__ gid, unsigned long long *__restrict__ acc,
                 int stride, int slot) {
  extern __shared__ __align__(16) uint32_t csm[];
  clique_cta<KM, BIG, (BIG ? kCqSmemBig : kCqSmemSmall) / 4>(k, roff, radj, tasks, ntasks, cursor, csm,
                                                             slabs + (size_t)blockIdx.x * (BIG ? 2 : 1) * slab_half, slab_half,
                                                             core, nullptr, gid, acc, stride, slot);
}

__global__ void __launch_bounds__(256) k_clique_warp(int k, const int64_t *__restrict__ roff,
                                                     const int32_t *__restrict__ radj,
                                                     const int32_t *__restrict__ tasks, int ntasks,
                                                     int *__restrict__ cursor, const int32_t *__restrict__ gid,
                                                     unsigned long long *__restrict__ acc, int stride, int slot) {
  __shared__ CqWarp sm[8];
  const unsigned lane = threadIdx.x & 31;
  WarpTasks queue;
  // runs only where the warps have many tasks each (ER, 38,647 vertices: 41 us
  // with runs past the first two per warp, 31 us without)
  const int lone = ntasks <= 16 * kTaskRun * (int)gridDim.x ? ntasks : gridDim.x * 16;
  while (true) {
    const int t = queue.next(cursor, lone, lane);
    if (t >= ntasks) break;
    const int32_t u = tasks[t];
    unsigned long long c = warp_sum(clique_warp_task(u, k, roff, radj, sm[threadIdx.x >> 5]));
    if (lane == 0 && c) atomicAdd(&acc[(size_t)stride * (gid ? gid[u] : 0) + slot], c);
  }
}

// CTA tasks of cliques of other sizes than 4 and 5.
__global__ void __launch_bounds__(kCqAnyThreads, 4)  // 48 registers, no spills
    k_clique_any(int k, const int64_t *__restrict__ roff, const int32_t *__restrict__ radj,
                 const int32_t *__restrict__ tasks, int ntasks, int *__restrict__ cursor, uint32_t *__restrict__ slabs,
                 size_t slab_words, CqCore core, const int32_t *__restrict__ gid, unsigned long long *__restrict__ acc,
                 int stride, int slot) {
  extern __shared__ __align__(16) uint32_t csm[];
  __shared__ uint32_t sxs[kCqAnyThreads / 32][64];  // staged sets (wsum_pairs)
  clique_cta<0, true, kCqSmemAny / 4>(k, roff, radj, tasks, ntasks, cursor, csm,
                                      slabs + (size_t)blockIdx.x * slab_words, 0, core, sxs[threadIdx.x >> 5], gid, acc,
                                      stride, slot);
}

__global__ void k_clique_tasks(int64_t n, const int64_t *__restrict__ roff, int k, int warp_max, int small_max,
                               uint32_t *__restrict__ ckey,
                               int32_t *__restrict__ cval, uint32_t *__restrict__ wkey, int32_t *__restrict__ wval,
                               int *__restrict__ sizes) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
    int64_t d = roff[u + 1] - roff[u];
    if (d < k - 1) continue;
    if (d > warp_max) {
      int i = atomicAdd(&sizes[0], 1);
      ckey[i] = ~(uint32_t)d;
      cval[i] = (int32_t)u;
      if (d > small_max) atomicAdd(&sizes[2], 1);
    } else {
      int i = atomicAdd(&sizes[1], 1);
      wkey[i] = ~(uint32_t)d;
      wval[i] = (int32_t)u;
    }
  }
}

// ------------------------------------------------------------ edge-centric (reference-shaped)
// Warp-cooperative c = a & b by binary search of the shorter list's keys in
// the longer one, compacted in order with ballots; returns |c|.
__device__ int warp_isect_store(const int32_t *a, int na, const int32_t *b, int nb, int32_t *c, unsigned lane) {
  const int32_t *look = a, *srch = b;
  int nl = na, ns = nb;
  if (na > nb) { look = b; srch = a; nl = nb; ns = na; }
  int cnt = 0;
  for (int base = 0; base < nl; base += 32) {
    int i = base + lane;
    bool f = false;
    int32_t key = 0;
    if (i < nl) {
      key = look[i];
      int lo = 0, hi = ns - 1;
      while (lo <= hi) {
        int mid = (lo + hi) >> 1;
        int32_t x = srch[mid];
        if (x == key) { f = true; break; }
        if (x < key) lo = mid + 1; else hi = mid - 1;
      }
    }
    unsigned m = __ballot_sync(0xffffffffu, f);
    if (f) c[cnt + __popc(m & ((1u << lane) - 1u))] = key;
    cnt += __popc(m);
  }
  __syncwarp();
  return cnt;
}

__device__ unsigned long long warp_isect_count(const int32_t *a, int na, const int32_t *b, int nb, unsigned lane) {
  const int32_t *look = a, *srch = b;
  int nl = na, ns = nb;
  if (na > nb) { look = b; srch = a; nl = nb; ns = na; }
  unsigned long long c = 0;
  for (int i = lane; i < nl; i += 32) {
    int32_t key = look[i];
    int lo = 0, hi = ns - 1;
    while (lo <= hi) {
      int mid = (lo + hi) >> 1;
      int32_t x = srch[mid];
      if (x == key) { ++c; break; }
      if (x < key) lo = mid + 1; else hi = mid - 1;
    }
  }
  return c;
}

__global__ void __launch_bounds__(256) k_clique_edge(int64_t nnz, int k, const int64_t *__restrict__ off,
                                                     const int32_t *__restrict__ adj, const int32_t *__restrict__ src,
                                                     int32_t *__restrict__ scratch, int maxd,
                                                     unsigned long long *__restrict__ out) {
  const unsigned lane = lane_id();
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  int32_t *lists = scratch + warp * (int64_t)maxd * (kCqMaxK - 2);
  int sizes[kCqMaxK], cursor[kCqMaxK];
  unsigned long long c = 0;
  for (int64_t e = warp; e < nnz; e += nw) {
    int32_t v0 = src[e], v1 = adj[e];
    int n1 = warp_isect_store(adj + off[v0], (int)(off[v0 + 1] - off[v0]), adj + off[v1],
                              (int)(off[v1 + 1] - off[v1]), lists, lane);
    // lists[l] holds the candidates after l+2 clique vertices
    if (k == 3) { c += lane == 0 ? (unsigned long long)n1 : 0ull; continue; }
    sizes[0] = n1;
    cursor[0] = 0;
    int depth = 0;
    while (depth >= 0) {
      if (cursor[depth] >= sizes[depth]) { --depth; continue; }
      int32_t *cur = lists + (int64_t)depth * maxd;
      int32_t x = cur[cursor[depth]++];
      const int32_t *nx = adj + off[x];
      int dx = (int)(off[x + 1] - off[x]);
      if (depth + 3 == k - 1) {
        c += warp_isect_count(cur, sizes[depth], nx, dx, lane);
      } else {
        int32_t *nxt = lists + (int64_t)(depth + 1) * maxd;
        sizes[depth + 1] = warp_isect_store(cur, sizes[depth], nx, dx, nxt, lane);
        cursor[depth + 1] = 0;
        ++depth;
      }
    }
  }
  c = warp_sum(c);
  if (lane == 0 && c) atomicAdd(out, c);
}

// ------------------------------------------------------------ host
template <class K>
static int cq_grid(K kernel, int threads, size_t smem) {
  if (smem) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
  return std::max(1, per_sm) * num_sms();
}

// The kernels of clique size 4 or 5: f(small CTA kernel, big CTA kernel).
template <class F>
static void cq_kernels(int k, F f) {
  if (k == 4) f(k_clique_cta<4, false>, k_clique_cta<4, true>);
  else f(k_clique_cta<5, false>, k_clique_cta<5, true>);
}

struct CqGrids {
  int small, big, warp;  // of the other sizes: small = 0, big = k_clique_any's
};
static CqGrids cq_grids(int k) {
  static PerDevice small[2], big[2], warp, any;
  CqGrids g;
  if (cq_any(k)) {
    g.small = 0;
    g.big = any.get([] { return std::min(cq_grid(k_clique_any, kCqAnyThreads, kCqSmemAny), kCqAnyPerSm * num_sms()); });
  } else {
    cq_kernels(k, [&](auto s, auto b) {
      g.small = small[k - 4].get([&] { return cq_grid(s, kCqSmallThreads, kCqSmemSmall); });
      g.big = big[k - 4].get([&] { return cq_grid(b, kCqBigThreads, kCqSmemBig); });
    });
  }
  g.warp = warp.get([] { return cq_grid(k_clique_warp, 256, 0); });
  return g;
}

// Largest |L| whose layout fits the small CTAs.
static int cq_small_max(int k) {
  int d = kCqWarpMax;
  while (d < kCqCtaMax && cq_layout(d + 1, k, kCqSmallThreads / 32, true).total * 4 <= kCqSmemSmall) ++d;
  return d;
}

// Plan: task queues (heaviest first) and row slabs; the run is launches only.
int clique_plan_build(CliquePlan *p, int64_t n, const int64_t *roff, const int32_t *radj, int max_deg, int k,
                      const int32_t *gid, unsigned long long *acc, int stride, int slot, cudaStream_t st,
                      int warp_max, int *cursors) {
  warp_max = std::max(1, std::min(warp_max, kCqWarpMax));
  p->n = n;
  p->roff = roff;
  p->radj = radj;
  p->k = k;
  p->gid = gid;
  p->acc = acc;
  p->stride = stride;
  p->slot = slot;
  p->n_cta = p->n_warp = 0;
  if (n == 0) return GPM_OK;
  if (max_deg > kCqCtaMax) return fail(GPM_EUNSUPPORTED, "out-list longer than 2048 on the bitset clique path");
  DevBuf<uint32_t> ckey, wkey;
  DevBuf<int32_t> cval, wval;
  DevBuf<int> sizes;
  GPM_TRY(ckey.reserve(n));
  GPM_TRY(wkey.reserve(n));
  GPM_TRY(cval.reserve(n));
  GPM_TRY(wval.reserve(n));
  GPM_TRY(p->ctasks.reserve(n));
  GPM_TRY(p->wtasks.reserve(n));
  GPM_TRY(sizes.reserve(3));
  p->cursors = cursors;
  if (!cursors) {
    GPM_TRY(p->counters.reserve(3));
    p->cursors = p->counters.p;
  }
  GPM_CUDA(cudaMemsetAsync(sizes.p, 0, 3 * sizeof(int), st));
  k_clique_tasks<<<grid_for(n), 256, 0, st>>>(n, roff, k, warp_max, cq_small_max(k), ckey.p, cval.p, wkey.p, wval.p,
                                              sizes.p);
  int h[3];
  GPM_CUDA(cudaMemcpyAsync(h, sizes.p, sizeof h, cudaMemcpyDeviceToHost, st));
  GPM_CUDA(cudaStreamSynchronize(st));
  for (int which = 0; which < 2; ++which) {
    int cnt = h[which];
    if (cnt <= 0) continue;
    DevBuf<uint32_t> k2;
    GPM_TRY(k2.reserve(cnt));
    size_t tmp = 0;
    uint32_t *kin = which ? wkey.p : ckey.p;
    int32_t *vin = which ? wval.p : cval.p, *vout = which ? p->wtasks.p : p->ctasks.p;
    GPM_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp, kin, k2.p, vin, vout, cnt, 0, 32, st));
    DevBuf<char> t;
    GPM_TRY(t.reserve(tmp));
    GPM_CUDA(cub::DeviceRadixSort::SortPairs(t.p, tmp, kin, k2.p, vin, vout, cnt, 0, 32, st));
  }
  p->n_cta = h[0];
  p->n_warp = h[1];
  p->n_big = h[2];
  // per-CTA slabs: rows, and for the big CTAs compacted rows, that do not fit
  // in shared memory
  const size_t W = (size_t)(max_deg + 31) / 32;
  const CqGrids grids = cq_grids(k);
  if (cq_any(k)) p->n_big = p->n_cta;
  p->big_grid = std::max(1, std::min(grids.big, p->n_big));
  if (p->n_big > 0 && p->n_big < p->n_cta + p->n_warp && !p->side &&
      (cudaStreamCreateWithFlags(&p->side, cudaStreamNonBlocking) != cudaSuccess ||
       cudaEventCreateWithFlags(&p->fork, cudaEventDisableTiming) != cudaSuccess ||
       cudaEventCreateWithFlags(&p->join, cudaEventDisableTiming) != cudaSuccess)) {
    cudaGetLastError();
    return fail(GPM_ECUDA, "clique plan: side stream");
  }
  const CqLayout big = cq_layout(max_deg, k, (cq_any(k) ? kCqAnyThreads : kCqBigThreads) / 32, true);
  const size_t comp_max = (size_t)max_deg * ((W + 3) & ~(size_t)3);
  const bool spill = p->n_big && (big.total * 4 > (cq_any(k) ? kCqSmemAny : kCqSmemBig) ||
                                  (k == 5 && comp_max > kCqBigThreads / 32 * cq_warp_words(1)));
  p->slab_words = comp_max;
  // a grid of half the CTAs where their slabs find no memory
  auto reserve = [](DevBuf<uint32_t> &buf, size_t per_cta, int *grid) -> int {
    while (true) {
      const int s = buf.reserve(std::max<size_t>(1, per_cta * *grid));
      if (s != GPM_ENOMEM || *grid == 1) return s;
      *grid /= 2;
    }
  };
  GPM_TRY(reserve(p->slabs, spill ? (cq_any(k) ? 1 : 2) * p->slab_words : 0, &p->big_grid));
  p->small_grid = std::max(1, std::min(grids.small, p->n_cta - p->n_big));
  // small CTAs: compacted rows beyond the warps' buffers
  const int sd = std::min(max_deg, cq_small_max(k)), sw = (sd + 31) / 32;
  p->small_slab = (size_t)sd * ((sw + 3) & ~3);
  const bool small_spill = p->n_cta > p->n_big && k == 5 && p->small_slab > kCqSmallThreads / 32 * cq_warp_words(1);
  GPM_TRY(reserve(p->small_slabs, small_spill ? p->small_slab : 0, &p->small_grid));
  // the bitmaps last: what cannot do without memory comes first
  if (p->n_cta > 0) {
    int64_t nkeys = 0;
    GPM_CUDA(cudaMemcpyAsync(&nkeys, roff + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st));
    GPM_CUDA(cudaStreamSynchronize(st));
    const int s = core_rows_build(n, roff, radj, nkeys, kCqCore, kCqCoreMin, p->rowid, &p->core, st);
    if (s == GPM_ENOMEM) {  // counted without them
      p->core = CoreRows();
      p->rowid.reset();
    } else {
      GPM_TRY(s);
    }
  }
  GPM_CUDA(cudaStreamSynchronize(st));
  return GPM_OK;
}

int clique_plan_run(CliquePlan *p, cudaStream_t st, bool zero) {
  if (p->n_cta + p->n_warp == 0) return GPM_OK;
  if (zero) GPM_CUDA(cudaMemsetAsync(p->cursors, 0, 3 * sizeof(int), st));
  const CqGrids grids = cq_grids(p->k);
  const int nsmall = p->n_cta - p->n_big;
  const CqCore core{p->core.n_rows ? p->rowid.p : nullptr, p->core.rows.p, p->core.base, p->core.words};
  // the large tasks may be few: they run beside the others
  cudaStream_t bst = st;
  if (p->side) {
    bst = p->side;
    GPM_CUDA(cudaEventRecord(p->fork, st));
    GPM_CUDA(cudaStreamWaitEvent(bst, p->fork, 0));
  }
  if (cq_any(p->k)) {
    if (p->n_big > 0)
      k_clique_any<<<p->big_grid, kCqAnyThreads, kCqSmemAny, bst>>>(p->k, p->roff, p->radj, p->ctasks.p, p->n_big,
                                                                    p->cursors, p->slabs.p, p->slab_words, core,
                                                                    p->gid, p->acc, p->stride, p->slot);
  } else {
    cq_kernels(p->k, [&](auto small, auto big) {
      if (p->n_big > 0)
        big<<<p->big_grid, kCqBigThreads, kCqSmemBig, bst>>>(p->k, p->roff, p->radj, p->ctasks.p, p->n_big, p->cursors,
                                                             p->slabs.p, p->slab_words, core, p->gid, p->acc,
                                                             p->stride, p->slot);
      if (nsmall > 0)
        small<<<p->small_grid, kCqSmallThreads, kCqSmemSmall, st>>>(
            p->k, p->roff, p->radj, p->ctasks.p + p->n_big, nsmall, p->cursors + 1, p->small_slabs.p, p->small_slab,
            core, p->gid, p->acc, p->stride, p->slot);
    });
  }
  if (bst != st) GPM_CUDA(cudaEventRecord(p->join, bst));
  // few tasks per warp: fewer warps meet less often at the cursor (us at eight /
  // five CTAs per SM, k = 4: ER 100,003 x 4, 24,000 tasks 54 / 46, ER 10,007 x 16
  // 36 / 33; but ER 100,003 x 32, 100,000 tasks 118 / 142)
  const int warp_grid = p->n_warp <= 4 * 8 * grids.warp ? std::min(grids.warp, kCqFewPerSm * num_sms()) : grids.warp;
  if (p->n_warp > 0)
    k_clique_warp<<<std::min(warp_grid, (p->n_warp + 7) / 8), 256, 0, st>>>(
        p->k, p->roff, p->radj, p->wtasks.p, p->n_warp, p->cursors + 2, p->gid, p->acc, p->stride, p->slot);
  if (bst != st) GPM_CUDA(cudaStreamWaitEvent(st, p->join, 0));  // joined whether or not the launches were accepted
  GPM_LAUNCH_CHECK();
  return GPM_OK;
}

int clique_run_upward(int64_t n, const int64_t *roff, const int32_t *radj, int max_deg, int k, const int32_t *gid,
                      unsigned long long *acc, int stride, int slot, cudaStream_t st) {
  CliquePlan p;
  GPM_TRY(clique_plan_build(&p, n, roff, radj, max_deg, k, gid, acc, stride, slot, st));
  GPM_TRY(clique_plan_run(&p, st));
  GPM_CUDA(cudaStreamSynchronize(st));  // the plan's scratch is released on return
  return GPM_OK;
}

void free_clique_plan(CliquePlan *p) { delete p; }

int clique_launch(gpm_graph *g, int k, cudaStream_t st, unsigned long long *d_out, bool edge_centric = false) {
  GPM_CUDA(cudaMemsetAsync(d_out, 0, sizeof(unsigned long long), st));
  if (g->nnz == 0) return GPM_OK;
  GPM_TRY(ensure_rank_graph(g, st));
  if (!edge_centric && g->rg->upward && g->max_deg <= kCqCtaMax) {
    // the schedule (task queues, per-CTA bitset slabs) is built on the first
    // call for this k and kept with the graph
    CliquePlan *&p = g->clique[k];
    if (!p) {
      CliquePlan *q = new CliquePlan();
      const int s = clique_plan_build(q, g->n, g->rg->roff.p, g->rg->radj.p, g->max_deg, k, nullptr, d_out, 0, 0, st);
      if (s != GPM_OK) {
        delete q;
        return s;
      }
      p = q;
    }
    p->acc = d_out;
    return clique_plan_run(p, st);
  }
  // edge-centric path on the stored graph
  GPM_TRY(ensure_src(g, st));
  int grid = num_sms() * 8;
  int64_t warps = (int64_t)grid * 8;
  int maxd = std::max(1, g->max_deg);
  DevBuf<int32_t> scratch;
  GPM_TRY(scratch.reserve((size_t)warps * maxd * (kCqMaxK - 2)));
  k_clique_edge<<<grid, 256, 0, st>>>(g->nnz, k, g->off.p, g->adj.p, g->src.p, scratch.p, maxd, d_out);
  GPM_LAUNCH_CHECK();
  GPM_CUDA(cudaStreamSynchronize(st));
  return GPM_OK;
}

}  // namespace gpm

using namespace gpm;

extern "C" int gpm_clique_ex(gpm_graph *g, int k, int variant, uint64_t *out) {
  if (!g || !out) return fail(GPM_EINVAL, "gpm_clique: NULL argument");
  if (k < 3 || k > kCqMaxK) return fail(GPM_EUNSUPPORTED, "k-clique supports 3 <= k <= 8");
  if (variant != GPM_CLIQUE_AUTO && variant != GPM_CLIQUE_EDGE) return fail(GPM_EINVAL, "unknown clique variant");
  GPM_TRY(g->result.reserve(8));
  GPM_TRY(clique_launch(g, k, 0, (unsigned long long *)g->result.p, variant == GPM_CLIQUE_EDGE));
  GPM_CUDA(cudaMemcpy(out, g->result.p, sizeof(uint64_t), cudaMemcpyDeviceToHost));
  return GPM_OK;
}

extern "C" int gpm_clique(gpm_graph *g, int k, uint64_t *out) { return gpm_clique_ex(g, k, GPM_CLIQUE_AUTO, out); }
