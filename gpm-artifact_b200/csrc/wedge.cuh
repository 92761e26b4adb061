// wedge.cuh -- 2-hop walks: every entry of the lists of a vertex's neighbours
// (its "middles"), by one warp or one CTA.  Shared by the 4-cycle counters of
// the motif pipeline (motif.cu) and of labelled matching (match_cycle.cu).
#pragma once
#include "common.cuh"

namespace gpm {

constexpr int kWedgeLong = 64;    // segments of at least this many entries are streamed by the whole warp
constexpr int kWedgePiece = 256;  // and, shared by the CTA, in pieces of this many

// Below, f(entry, position, segment) is called for entries data[position] of a
// numbered segment.

// data[s .. e) of segment `seg`, the warp's lanes side by side
template <class F>
__device__ __forceinline__ void warp_stream(const int32_t *__restrict__ data, long long s, long long e, int seg,
                                            unsigned lane, F f) {
  long long i = s + lane;
  for (; i + 96 < e; i += 128) {
    const int32_t x0 = __ldg(data + i), x1 = __ldg(data + i + 32), x2 = __ldg(data + i + 64),
                  x3 = __ldg(data + i + 96);
    f(x0, i, seg);
    f(x1, i + 32, seg);
    f(x2, i + 64, seg);
    f(x3, i + 96, seg);
  }
  for (; i < e; i += 32) f(__ldg(data + i), i, seg);
}

// Every entry of the lanes' segments data[st .. st + len), lane t's numbered seg0
// + t: long ones one after another, the others laid end to end over the lanes.
template <class F>
__device__ __forceinline__ void warp_segments(const int32_t *__restrict__ data, long long st, int len, int seg0,
                                              unsigned lane, F f) {
  for (unsigned lm = __ballot_sync(0xffffffffu, len >= kWedgeLong); lm; lm &= lm - 1) {
    const int t = __ffs(lm) - 1;
    const long long ts = __shfl_sync(0xffffffffu, st, t);
    warp_stream(data, ts, ts + __shfl_sync(0xffffffffu, len, t), seg0 + t, lane, f);
  }
  const int n = len >= kWedgeLong ? 0 : len;
  int inc = n;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if ((int)lane >= o) inc += v;
  }
  const int total = __shfl_sync(0xffffffffu, inc, 31);
  const long long first = st - (inc - n);  // entry idx of lane t's segment is data[first of t + idx]
  for (int base = 0; base < total; base += 32) {
    const int idx = base + (int)lane;
    int lo = 0;  // first lane whose inclusive prefix exceeds idx
#pragma unroll
    for (int r = 16; r; r >>= 1)
      if (__shfl_sync(0xffffffffu, inc, lo + r - 1) <= idx) lo += r;
    const long long ft = __shfl_sync(0xffffffffu, first, lo & 31);
    if (idx < total) f(__ldg(data + ft + idx), ft + idx, seg0 + lo);
  }
}

// Shared state of a CTA's walks: two sets, used in turn, the idle one zeroed.
struct WedgeWalk {
  static constexpr int kLong = 64;
  struct {
    int next, nlong;
    long long st[kLong];
    int len[kLong], seg[kLong];
  } s[2];
};

// Every entry of the segments seg(i) -> (start, length), i < m, of m middles, W
// entries in all (an estimate will do), by the CTA.  Runs of
// middles go to the warps through a shared counter; a segment that holds more
// than 1/64 of the work would keep one warp busy while the others wait at the
// barrier, so those are listed and shared out in pieces.  (Dealt out in fixed
// runs, with long segments left to their warp, k_cycle_big waited at barriers
// two thirds of the time: 3.5 ms at R-MAT 19, 2.7 ms so.)  Ends with a
// barrier; *turn alternates between the two sets of S.
template <class Seg, class F>
__device__ __forceinline__ void cta_wedges(const int32_t *__restrict__ data, int m, unsigned long long W, WedgeWalk &S,
                                           int *turn, Seg seg, F f) {
  const unsigned lane = lane_id();
  const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  auto &q = S.s[*turn];
  *turn ^= 1;
  if (threadIdx.x == 0) S.s[*turn].next = S.s[*turn].nlong = 0;
  const int thr = (int)min(max(W / 64, (unsigned long long)kWedgePiece), (unsigned long long)1 << 30);
  const int run = max(1, min(32, m / (2 * nw)));
  while (true) {
    int i = 0;
    if (lane == 0) i = atomicAdd(&q.next, run);
    i = __shfl_sync(0xffffffffu, i, 0);
    if (i >= m) break;
    long long st = 0;
    int len = 0;
    if ((int)lane < run && i + (int)lane < m) seg(i + (int)lane, &st, &len);
    if (len > thr) {
      const int at = atomicAdd(&q.nlong, 1);
      if (at < WedgeWalk::kLong) {
        q.st[at] = st;
        q.len[at] = len;
        q.seg[at] = i + (int)lane;
        len = 0;
      }
    }
    __syncwarp();
    warp_segments(data, st, len, i, lane, f);
  }
  __syncthreads();
  const int nlong = min(q.nlong, WedgeWalk::kLong);
  int piece = wid;  // this warp's next piece, counted from the current segment's first
  for (int j = 0; j < nlong; ++j) {
    const long long st = q.st[j];
    const int len = q.len[j], pieces = (len + kWedgePiece - 1) / kWedgePiece;
    for (; piece < pieces; piece += nw) {
      const int b = piece * kWedgePiece;
      warp_stream(data, st + b, st + min(len, b + kWedgePiece), q.seg[j], lane, f);
    }
    piece -= pieces;
  }
  __syncthreads();
}

}  // namespace gpm
