// FP64 P2P (kernels/laplace.h:150-235): pot += q/r, grad += q (x_j - x_i)/r^3,
// r = 0 pairs skipped.
//
// Bound: the FP64 pipe (64 multiply-adds per SM and clock on B200), 18 FP64
// operations a pair (3 separations, 3 for r^2, 5 for 1/r from the hardware's
// approximation, 3 for q/r and q/r^3, 4 sums).  One warp takes an item of a
// target leaf (p2p_work.cuh); its lanes form G = 32 / S groups of S lanes, two
// targets a lane, S the narrowest that holds the leaf's targets, and the
// groups take interleaved sources of the leaf's stream, staged through shared
// memory in chunks of 32 G.  Every lane so holds targets in leaves of 8 to 64
// bodies (the previous form, 32 lanes x 2 targets of one leaf, used 30-50 % of
// its slots at the usual ncrit 64, called rsqrt(double) per pair, and one warp
// served the longest list alone).  1M-body Plummer sphere at ncrit 64 15.4 -> 4.57
// ms, 100K-body cube 5.06 -> 0.46; the pipe 69 % busy.
#include "p2p_work.cuh"
#include "pair64.cuh"

namespace exafmm_b200 {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kTpl = 2;        // targets per lane
constexpr int kWarps64 = 16;   // resident warps per SM (one-warp blocks, at most 128 registers)
constexpr int kSegCost64 = 4096;  // slots x sources of a segment: about 10 us of a warp

// One chunk of staged sources: (x, y) and (z, q) apart, so that the groups,
// which read G consecutive sources at once, hit distinct banks.
struct Stage64 {
  double2 xy[256], zq[256];
};

// Streams the segment's bodies through the warp and adds their action on the
// lane's targets to acc.
template <bool PERIODIC>
__device__ __forceinline__ void stream64(int lS, Stage64 &sm, P2PState &st, const int *src,
                                         const int4 *cell_b, const double4 *xs, double cycle, const double (&x)[kTpl],
                                         const double (&y)[kTpl], const double (&z)[kTpl], double (&acc)[kTpl][4]) {
  const int lane = threadIdx.x & 31, G = 32 >> lS;
  for (;;) {
    const int filled = p2p_fill(st, 32 * G, src, cell_b, [&](int k, long long body, int img) {
      double4 b = xs[body];
      if (PERIODIC) {
        b.x += (double)(img / 9 - 1) * cycle;
        b.y += (double)((img / 3) % 3 - 1) * cycle;
        b.z += (double)(img % 3 - 1) * cycle;
      }
      sm.xy[k] = make_double2(b.x, b.y);
      sm.zq[k] = make_double2(b.z, b.w);
    });
    if (filled == 0) break;
    const int n = ((filled + 2 * G - 1) >> (6 - lS)) << (6 - lS);  // two sources per group and step
    // padding: far away with zero charge, adds exactly zero
    for (int k = filled + lane; k < n; k += 32) {
      sm.xy[k] = make_double2(1e18, 1e18);
      sm.zq[k] = make_double2(1e18, 0.0);
    }
    __syncwarp();
#pragma unroll 1
    for (int k = lane >> lS; k < n; k += 2 * G) {
      const double2 a0 = sm.xy[k], b0 = sm.zq[k], a1 = sm.xy[k + G], b1 = sm.zq[k + G];
      double dx[2 * kTpl], dy[2 * kTpl], dz[2 * kTpl], qq[2 * kTpl];
#pragma unroll
      for (int u = 0; u < kTpl; u++) {
        dx[2 * u] = x[u] - a0.x;
        dy[2 * u] = y[u] - a0.y;
        dz[2 * u] = z[u] - b0.x;
        qq[2 * u] = b0.y;
        dx[2 * u + 1] = x[u] - a1.x;
        dy[2 * u + 1] = y[u] - a1.y;
        dz[2 * u + 1] = z[u] - b1.x;
        qq[2 * u + 1] = b1.y;
      }
      pairs64<2 * kTpl, 2>(dx, dy, dz, qq, acc);
    }
    __syncwarp();
  }
}

// One pass over the item's segments for the leaf's targets from st.tb on.
template <bool PERIODIC>
__device__ __forceinline__ void pass64(int lS, Stage64 &sm, P2PState &st, const P2PItems &w, const int *src,
                                       const int4 *cell_bj, const double4 *xt, const double4 *xs, double4 *trg,
                                       double cycle) {
  const int lane = threadIdx.x & 31;
  double x[kTpl], y[kTpl], z[kTpl];
#pragma unroll
  for (int u = 0; u < kTpl; u++) {
    const int i = st.tb + (lane & ((1 << lS) - 1)) + (u << lS);
    double4 v = make_double4(0, 0, 0, 0);
    if (i < st.cb.y) v = xt[(long long)st.cb.x + i];
    x[u] = v.x;
    y[u] = v.y;
    z[u] = v.z;
  }
  p2p_seek(st, st.item.y, src, cell_bj);
  if (lane == 0) st.at = st.item.y;
  __syncwarp();
  while (st.at < st.item.z) {
    if (lane == 0) st.pos.w = min(st.seg, st.item.z - st.at);
    __syncwarp();
    double acc[kTpl][4];
#pragma unroll
    for (int u = 0; u < kTpl; u++)
#pragma unroll
      for (int k = 0; k < 4; k++) acc[u][k] = 0.0;
    stream64<PERIODIC>(lS, sm, st, src, cell_bj, xs, cycle, x, y, z, acc);
#pragma unroll
    for (int u = 0; u < kTpl; u++) {
#pragma unroll 1
      for (int off = 1 << lS; off < 32; off <<= 1)
#pragma unroll
        for (int k = 0; k < 4; k++) acc[u][k] += __shfl_xor_sync(kFull, acc[u][k], off);
      if (lane < (1 << lS)) p2p_store(w, st, lane + (u << lS), acc[u], trg);
    }
    __syncwarp();
    if (lane == 0) st.at += st.seg;
    __syncwarp();
  }
}

template <bool PERIODIC>
__global__ void __launch_bounds__(32, kWarps64)
k_p2p64(P2PItems w, const int *off, const int *src, const int4 *cell_b, const int4 *cell_bj, const double4 *xt,
        const double4 *xs, double4 *trg, double cycle) {
  __shared__ Stage64 sm;
  __shared__ P2PState state;
  P2PState &st = state;
  // without a queue (one operator call): every cell whole, in turn
  for (long long c0 = blockIdx.x;; c0 += gridDim.x) {
    int4 item;
    int seg = 0x40000000;
    if (w.items) {
      if (!p2p_next(w, item)) return;
      seg = w.leaf[item.x].x;
    } else {
      if (c0 >= w.ncells) return;
      item = make_int4((int)c0, 0, 0x40000000, -1);
      if (off[c0] == off[c0 + 1]) continue;
    }
    p2p_begin(st, item, seg, kTpl, off, cell_b);
    p2p_passes(st, kTpl, [&](int lS) { pass64<PERIODIC>(lS, sm, st, w, src, cell_bj, xt, xs, trg, cycle); });
    if (st.item.w >= 0) p2p_finish(w, st, trg);
  }
}

void launch64(const FmmArgs &a, const P2PItems &w, bool periodic) {
  const int4 *bj = a.src_cell_b ? a.src_cell_b : a.cell_b;
  const double4 *xs = a.src_xt ? a.src_xt : a.xt;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(
      w.items ? w.cap : w.ncells, (long long)kNumSMs * kWarps64));
  if (periodic)
    k_p2p64<true><<<grid, 32, 0, a.stream>>>(w, a.p2p_off, a.p2p_src, a.cell_b, bj, a.xt, xs, a.trg64, a.cycle);
  else
    k_p2p64<false><<<grid, 32, 0, a.stream>>>(w, a.p2p_off, a.p2p_src, a.cell_b, bj, a.xt, xs, a.trg64, a.cycle);
  EXA_CHECK_LAUNCH();
}

}  // namespace

void p2p_fp64(Context &C, const FmmArgs &a, bool periodic, P2PWork &w) {
  if (a.ncells <= 0) return;
  launch64(a, p2p_plan(C, a, w, kTpl, kNumSMs * kWarps64, kSegCost64), periodic);
}

void p2p_fp64(const FmmArgs &a) {
  P2PItems w{};
  w.ncells = a.ncells;
  if (a.ncells > 0) launch64(a, w, true);
}

}  // namespace exafmm_b200
