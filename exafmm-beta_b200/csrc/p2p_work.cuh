// Work items of the P2P kernels (FP64 and mixed).
//
// A warp evaluates one target leaf against the bodies of its P2P list.  Leaves
// differ in cost by orders of magnitude: in a 100,000-body cube the average
// leaf meets 1,770 sources, a sparse leaf at the edge of the root box 21,900,
// and one warp working through that list alone took 1.5 ms (mixed) or 5.1 ms
// (FP64) of a P2P phase whose arithmetic fills the GPU for 0.2 or 0.3 ms.  So
//   * every leaf's source stream (the bodies of its list's leaves, one after
//     another) is cut into segments by a fixed rule on the leaf alone: a
//     multiple of kSegAlign sources, in units c of the kernel's segment cost
//     (target slots x sources) half the leaf within c to 8 c, 4 c for leaves
//     above 32 c, at most kMaxSeg segments; a leaf's result is the sum of its
//     segments' sums in order.  8 c above 32 c too would take the mixed P2P of 4M
//     bodies from 17.38 to 17.34 ms and of a 1M-charge water box from 4.47 to
//     4.41, but of 30,000 bodies on a sphere at ncrit 128 from 250 to 297 us and
//     of a 90,000-charge box from 291 to 334: their costly leaves need their
//     segments shared out (100,000-body cube: 0.36 ms; with quarters of such
//     leaves 0.55, with whole leaves 0.83);
//   * a leaf may be divided into items of whole segments, taken by different
//     warps; these leave each segment's sums in scratch and the last warp to
//     finish adds them in order.  A leaf taken whole adds its segments in the
//     same order, so how leaves are divided (which depends on what else is in
//     the solve) does not change a bit of the result.  Divided are the leaves
//     that cost more than a quarter of a resident warp's share (FP64 P2P of the
//     100,000-body cube 0.46 ms, 0.52 with half a share), and every
//     eighth of the others above 1/16 into items of 1/64 of a share, for the end
//     of the queue (mixed P2P of a 7,019-body sphere 82 us, 87 without; the same
//     time from 100,000 bodies on);
//   * items are queued in four classes, those above 1/2, 1/8 and 1/32 of a
//     share first, so that the persistent warps finish together.
// Building the queue is two launches (costs, then one scan that emits the
// items), where sorting the leaves by cost took 10 or more (3 radix passes).
#pragma once
#include <algorithm>

#include "fmm.h"
#include "scan.cuh"

namespace exafmm_b200 {

constexpr int kMaxSeg = 64;     // segments of a stream at most
constexpr int kSegAlign = 256;  // sources: whole chunks of every group width
constexpr int kHeavyPerWarp = 4, kSmallPerWarp = 64;  // items of a warp's share: divided above 1/4, small ones 1/64

// Lanes (log2) of the narrowest group that holds the targets still left, `tpl` per lane.
__host__ __device__ __forceinline__ int pass_log_lanes(int left, int tpl) {
  return left <= 4 * tpl ? 2 : left <= 8 * tpl ? 3 : left <= 16 * tpl ? 4 : 5;
}
// Target slots of a leaf of n bodies in passes of varying width, plus `charge` per pass.
__host__ __device__ __forceinline__ int pass_slots(int n, int tpl, int charge) {
  int cost = 0;
  const int full = n / (32 * tpl);
  cost += full * (32 * tpl + charge);
  for (int tb = full * 32 * tpl; tb < n;) {
    const int w = tpl << pass_log_lanes(n - tb, tpl);
    cost += w + charge;
    tb += w;
  }
  return cost;
}

struct Count4 {
  unsigned long long a, b, c, d;
  __host__ __device__ Count4 operator+(const Count4 &o) const { return {a + o.a, b + o.b, c + o.c, d + o.d}; }
};
__device__ __forceinline__ Count4 shfl_up_any(Count4 v, int o) {
  return {__shfl_up_sync(0xffffffffu, v.a, o), __shfl_up_sync(0xffffffffu, v.b, o),
          __shfl_up_sync(0xffffffffu, v.c, o), __shfl_up_sync(0xffffffffu, v.d, o)};
}
__device__ __forceinline__ Count4 shfl_any(Count4 v, int src) {
  return {__shfl_sync(0xffffffffu, v.a, src), __shfl_sync(0xffffffffu, v.b, src),
          __shfl_sync(0xffffffffu, v.c, src), __shfl_sync(0xffffffffu, v.d, src)};
}

// Device view of the queue.
constexpr int kItemClasses = 4;
struct P2PItems {
  // item: (leaf, first source, end source, its leaf's scratch base or -1 when the leaf is whole; leaf -1: none)
  const int4 *items;         // kItemClasses regions of cap items
  const int *count;          // items of each class
  const int4 *leaf;          // per leaf: sources of a segment, items, segments, targets per lane
  double4 *scratch;          // segment sums of divided leaves: [segment][target]
  int *done;                 // per leaf: items finished
  unsigned long long *next;  // work counter
  long long cap, ncells;
};

// The next item (warp-uniform); false when the queue is empty.
__device__ __forceinline__ bool p2p_next(const P2PItems &w, int4 &item) {
  for (;;) {
    unsigned long long t = 0;
    if ((threadIdx.x & 31) == 0) t = atomicAdd(w.next, 1ull);
    long long k = (long long)__shfl_sync(0xffffffffu, t, 0);
    const int4 *at = w.items;
    int cls = 0;
    for (; cls < kItemClasses; cls++) {
      const int n = w.count[cls];
      if (k < n) break;
      k -= n;
      at += w.cap;
    }
    if (cls == kItemClasses) return false;
    item = at[k];
    if (item.x >= 0) return true;
  }
}

// A target's sums over its sources, added to its result.
__device__ __forceinline__ void p2p_add(double4 *trg, const double (&v)[4]) {
  double4 r = *trg;
  r.x += v[0];
  r.y -= v[1];
  r.z -= v[2];
  r.w -= v[3];
  *trg = r;
}

// What a warp keeps of its item while it streams: in shared memory, read again
// where it is needed, so that it takes no registers from the pair loops.
// The place in the leaf's source stream (list entry q, body o of it) and a window
// of 32 list entries from qw on stay from segment to segment, so that only the
// first of an item waits for the list.
struct P2PState {
  int4 item, cb;      // item; the target leaf's cell
  int seg, tpl;       // sources of a segment, targets per lane
  int b, end;         // its P2P list
  int at, tb;         // first source of this segment, first target of this pass
  int4 pos;           // place in the stream (q, o, qw), sources left of this segment
  int4 win[32];       // the window's entries: first body, bodies, image
};

// The window of list entries from q on.
__device__ __forceinline__ void p2p_window(P2PState &st, int q, const int *src, const int4 *cell_b) {
  const int lane = threadIdx.x & 31;
  const int qq = q + lane;
  int4 v = make_int4(0, 0, 13, 0);
  if (qq < st.end) {
    const int packed = src[qq];
    const int4 cb = cell_b[packed & 0x3ffffff];
    v = make_int4(cb.x, cb.y, packed >> 26, 0);
  }
  __syncwarp();
  st.win[lane] = v;
  __syncwarp();
}

// To source `skip` of the stream; `left` sources follow.
__device__ __forceinline__ void p2p_seek(P2PState &st, int skip, const int *src, const int4 *cell_b) {
  int q = st.b, qw = q - 64, o = 0;
  while (skip > 0 && q < st.end) {
    p2p_window(st, q, src, cell_b);
    qw = q;
    const int size = st.win[threadIdx.x & 31].y;
    const int incl = warp_inclusive_scan(size);
    const unsigned past = __ballot_sync(0xffffffffu, incl > skip);
    if (!past) {  // the whole window lies before it
      skip -= __shfl_sync(0xffffffffu, incl, 31);
      q += 32;
      continue;
    }
    const int l = __ffs((int)past) - 1;
    q += l;
    o = skip - __shfl_sync(0xffffffffu, incl - size, l);
    skip = 0;
  }
  __syncwarp();
  if ((threadIdx.x & 31) == 0) st.pos = make_int4(q, o, qw, 0);
  __syncwarp();
}

// Stages up to `room` of the segment's next sources: stage(k, body, img) puts
// body `body` seen through image img at place k, one call per lane and body.
// Returns the bodies staged (0: the segment is done).
template <typename Stage>
__device__ __forceinline__ int p2p_fill(P2PState &st, int room, const int *src, const int4 *cell_b, Stage &&stage) {
  const int lane = threadIdx.x & 31;
  int4 p = st.pos;
  int filled = 0;
  while (filled < room && p.w > 0) {
    if (p.x - p.z >= 32) {
      if (p.x >= st.end) break;
      p2p_window(st, p.x, src, cell_b);
      p.z = p.x;
    }
    const int4 e = st.win[p.x - p.z];
    const int m = min(min(room - filled, e.y - p.y), p.w);
    // one or two rounds; unrolled, the hot code outgrows the instruction cache
    // (mixed P2P of 4M bodies 17.73 against 17.54 ms)
#pragma unroll 1
    for (int k = lane; k < m; k += 32) stage(filled + k, (long long)e.x + p.y + k, e.z);
    filled += m;
    p.w -= m;
    p.y += m;
    if (p.y == e.y) {
      p.x++;
      p.y = 0;
    }
  }
  __syncwarp();
  if (lane == 0) st.pos = p;
  return filled;
}

// Finishing an item of a divided leaf: the warp that finishes its last item
// adds the segments' sums to the targets in order (lane-strided).
__device__ __forceinline__ void p2p_finish(const P2PItems &w, P2PState &st, double4 *trg) {
  const int c = st.item.x, base = st.item.w, first = st.cb.x, n = st.cb.y;
  const int4 lf = w.leaf[c];
  __threadfence();
  __syncwarp();
  int old = 0;
  if ((threadIdx.x & 31) == 0) old = atomicAdd(&w.done[c], 1);
  old = __shfl_sync(0xffffffffu, old, 0);
  if (old != lf.y - 1) return;
  __threadfence();
  for (int i = threadIdx.x & 31; i < n; i += 32) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int s = 0; s < lf.z; s++) {
      const double *v = reinterpret_cast<const double *>(w.scratch + base + (long long)s * n + i);
#pragma unroll
      for (int k = 0; k < 4; k++) t[k] += __ldcg(v + k);
    }
    p2p_add(trg + first + i, t);
  }
}

// The sums of the pass's target j (lane-group member and slot) over one
// segment: kept for p2p_finish, or added to the result at once (either way
// segment by segment, in order: the results of a solve start from zero).  Added
// up in shared memory instead, they took 3 KB of a warp's 12 and the L1 that
// this leaves (mixed P2P of 4M bodies 17.54 against 17.38 ms).
__device__ __forceinline__ void p2p_store(const P2PItems &w, P2PState &st, int j, const double (&v)[4],
                                          double4 *trg) {
  const int i = st.tb + j;
  if (i >= st.cb.y) return;
  if (st.item.w >= 0) {
    w.scratch[st.item.w + (long long)(st.at / st.seg) * st.cb.y + i] = make_double4(v[0], v[1], v[2], v[3]);
    return;
  }
  p2p_add(trg + st.cb.x + i, v);
}

// The item's leaf and list into st.
__device__ __forceinline__ void p2p_begin(P2PState &st, const int4 &item, int seg, int tpl, const int *off,
                                          const int4 *cell_b) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    const int4 cb = cell_b[item.x];
    st.item.x = item.x;
    st.item.y = item.y;
    st.item.z = item.z;
    st.item.w = item.w;
    st.cb.x = cb.x;
    st.cb.y = cb.y;
    st.seg = seg;
    st.tpl = tpl;
    st.b = off[item.x];
    st.end = off[item.x + 1];
    st.tb = 0;
  }
  __syncwarp();
}

// One item: `pass(log2 lanes)` evaluates one pass over it for the targets from
// st.tb on.
template <typename Pass>
__device__ __forceinline__ void p2p_passes(P2PState &st, int tpl, Pass &&pass) {
  for (;;) {
    const int left = st.cb.y - st.tb;
    if (left <= 0) break;
    const int lS = pass_log_lanes(left, tpl);
    pass(lS);
    __syncwarp();
    if ((threadIdx.x & 31) == 0) st.tb += tpl << lS;
    __syncwarp();
  }
}

// Targets per lane of a leaf of n bodies: tpl 2 or 3, or (0) the one that
// costs fewer target slots, with kPassCharge more per pass over the sources.
constexpr int kPassCharge = 4;
__host__ __device__ __forceinline__ int targets_per_lane(int n, int tpl) {
  if (tpl) return tpl;
  return pass_slots(n, 3, kPassCharge) < pass_slots(n, 2, kPassCharge) ? 3 : 2;
}

// Builds the queue on a.stream.  tpl: targets per lane (targets_per_lane);
// warps: resident warps of the kernel that takes it; seg_cost: slots x sources
// of the smallest segment.
P2PItems p2p_plan(Context &C, const FmmArgs &a, P2PWork &w, int tpl, int warps, int seg_cost);

}  // namespace exafmm_b200
