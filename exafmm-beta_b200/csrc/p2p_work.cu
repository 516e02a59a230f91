// Builds the P2P kernels' work queue (p2p_work.cuh).
#include "p2p_work.cuh"

namespace exafmm_b200 {
namespace {

// Sources of every leaf with a P2P list (0: none); the total cost, target
// slots x sources, in *total.  A warp per cell, its lanes over the list.
__global__ void __launch_bounds__(256)
k_p2p_cost(const int *off, const int *src, long long ncells, const int4 *cell_b, const int4 *cell_bj, int tpl,
           int *nsrc, unsigned long long *total) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  unsigned long long sum = 0;
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    int s = 0;
    for (int q = b + lane; q < e; q += 32) s += cell_bj[src[q] & 0x3ffffff].y;
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) {
      const int nb = cell_b[c].y;
      nsrc[c] = s;
      if (s > 0) sum += (unsigned long long)s * (unsigned)pass_slots(nb, targets_per_lane(nb, tpl), 0);
    }
  }
  __shared__ unsigned long long part[8];
  if (lane == 0) part[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) t += part[i];
    if (t) atomicAdd(total, t);
  }
}

// Counts per cell: items of classes 0 | 1 << 32, 2 | 3 << 32, and scratch slots
// of heavy and of other divided leaves.
struct P2PScan {
  using T = Count4;
  const int4 *cell_b;
  const int *nsrc;
  const unsigned long long *total_cost;
  int4 *items, *leaf;
  int *count;
  long long cap, scratch_heavy, scratch_small;  // capacities: items of a class, scratch slots
  int tpl, warps, seg_cost;

  struct Leaf {
    int tpl, seg, nseg, k, cls;
    bool heavy;
  };
  __device__ Leaf leaf_of(long long c) const {
    Leaf l{2, 0, 0, 0, -1, false};
    const int ns = nsrc[c];
    if (ns <= 0) return l;
    const int nb = cell_b[c].y;
    l.tpl = targets_per_lane(nb, tpl);
    const int slots = pass_slots(nb, l.tpl, 0);
    const unsigned long long x = (unsigned long long)ns * (unsigned)slots;
    // segments: a rule on this leaf alone
    const unsigned long long c1 = (unsigned)seg_cost;
    const unsigned long long sc = x > 32 * c1 ? 4 * c1 : min(max(x / 2, c1), 8 * c1);
    const int want = max(1, max((int)(sc / slots), ns / kMaxSeg));
    l.seg = (want + kSegAlign - 1) / kSegAlign * kSegAlign;
    l.nseg = (int)(((long long)ns + l.seg - 1) / l.seg);
    // items: whole segments, by the leaf's share of the total
    const unsigned long long share = *total_cost / (unsigned)warps;
    const unsigned long long t = share / kHeavyPerWarp + 1, u = share / kSmallPerWarp + 1;
    l.heavy = x > t;
    unsigned long long k = 1;
    if (l.heavy) k = (x + t - 1) / t;
    else if ((c & 7) == 0 && 16 * x >= share) k = (x + u - 1) / u;
    l.k = (int)min(k, (unsigned long long)l.nseg);
    const unsigned long long per = x / l.k;
    l.cls = 2 * per >= share ? 0 : 8 * per >= share ? 1 : 32 * per >= share ? 2 : 3;
    return l;
  }
  __device__ T value(long long c) const {
    const Leaf l = leaf_of(c);
    T v{0, 0, 0, 0};
    const unsigned long long n = (unsigned long long)l.k << (l.cls & 1 ? 32 : 0);
    if (l.cls >= 0) (l.cls < 2 ? v.a : v.b) = n;
    if (l.k > 1) (l.heavy ? v.c : v.d) = (unsigned long long)l.nseg * (unsigned)cell_b[c].y;
    return v;
  }
  __device__ void emit(long long c, const T &, const T &excl) const {
    const Leaf l = leaf_of(c);
    if (l.cls < 0) return;
    leaf[c] = make_int4(l.seg, l.k, l.nseg, l.tpl);
    const unsigned long long at = (l.cls < 2 ? excl.a : excl.b) >> (l.cls & 1 ? 32 : 0) & 0xffffffffull;
    int4 *dst = items + l.cls * cap + at;
    // a divided leaf without room in its scratch area is taken whole by its
    // first item (the same sums in the same order)
    const long long used = (long long)(l.heavy ? excl.c : excl.d);
    const bool room = l.k > 1 && used + (long long)l.nseg * cell_b[c].y <= (l.heavy ? scratch_heavy : scratch_small);
    const int ns = nsrc[c];
    if (!room) {
      dst[0] = make_int4((int)c, 0, ns, -1);
      for (int i = 1; i < l.k; i++) dst[i] = make_int4(-1, 0, 0, -1);
    } else {
      const int base = (int)(used + (l.heavy ? 0 : scratch_heavy));
      for (int i = 0; i < l.k; i++) {
        const long long s0 = (long long)l.nseg * i / l.k, s1 = (long long)l.nseg * (i + 1) / l.k;
        dst[i] = make_int4((int)c, (int)(s0 * l.seg), (int)min(s1 * l.seg, (long long)ns), base);
      }
    }
  }
  __device__ void total(const T &t) const {
    count[0] = (int)(t.a & 0xffffffffull);
    count[1] = (int)(t.a >> 32);
    count[2] = (int)(t.b & 0xffffffffull);
    count[3] = (int)(t.b >> 32);
  }
};

}  // namespace

P2PItems p2p_plan(Context &C, const FmmArgs &a, P2PWork &w, int tpl, int warps, int seg_cost) {
  cudaStream_t st = a.stream;
  const long long nc = a.ncells;
  P2PItems v;
  // a leaf of cost x is divided into at most x / (the item size) + 1 items
  v.cap = nc + (long long)warps * kSmallPerWarp + 1;
  v.ncells = nc;
  // scratch of divided leaves: every segment of every leaf for the heavy ones,
  // up to 2^23 slots (256 MB).  In small trees of large leaves most are heavy:
  // with eight segments a body many found no room and went whole (FP64 P2P of
  // a 30,000-body Plummer sphere at ncrit 128 1.34 ms, 0.29 with it).  Two
  // segments a body, up to 2^21 slots, for the others.
  P2PScan s;
  s.scratch_heavy = std::min(kMaxSeg * a.n, 1LL << 23);
  s.scratch_small = std::min(2 * a.n, 1LL << 21);
  w.items.ensure(kItemClasses * v.cap);
  w.leaf.ensure(nc);
  w.nsrc.ensure(nc);
  w.count.ensure(kItemClasses);
  w.scratch.ensure(s.scratch_heavy + s.scratch_small);
  w.zero.ensure(2 * sizeof(unsigned long long) + nc * sizeof(int));  // total cost, work counter, done[nc]
  unsigned long long *total = reinterpret_cast<unsigned long long *>(w.zero.p);
  EXA_CUDA(cudaMemsetAsync(w.zero.p, 0, 2 * sizeof(unsigned long long) + nc * sizeof(int), st));
  v.items = w.items.p;
  v.count = w.count.p;
  v.leaf = w.leaf.p;
  v.scratch = w.scratch.p;
  v.done = reinterpret_cast<int *>(total + 2);
  v.next = total + 1;
  const int4 *cell_bj = a.src_cell_b ? a.src_cell_b : a.cell_b;
  const int grid = (int)std::max<long long>(1, std::min<long long>(kNumSMs * 8, (nc + 7) / 8));
  k_p2p_cost<<<grid, 256, 0, st>>>(a.p2p_off, a.p2p_src, nc, a.cell_b, cell_bj, tpl, w.nsrc.p, total);
  EXA_CHECK_LAUNCH();
  s.cell_b = a.cell_b;
  s.nsrc = w.nsrc.p;
  s.total_cost = total;
  s.items = w.items.p;
  s.leaf = w.leaf.p;
  s.count = w.count.p;
  s.cap = v.cap;
  s.tpl = tpl;
  s.warps = warps;
  s.seg_cost = seg_cost;
  launch_scan<256, 2>(s, nullptr, nc, nc, C.scan, C.err.p, st);
  return v;
}

}  // namespace exafmm_b200
