// M2L as dense products per offset class (the mixed form's FP32 M2L for regular
// pairs).
//
// Between scaled expansions the M2L (kernels/laplace.h:292-322; the scaled form
// of m2l_fast.cuh) is a linear map that depends only on the offset of the two
// cell centers in units of the target radius and on the level difference:
//   acc_j^k = sum_{n,m} s(k,m) (R_s/R_t)^n Ms_n^m S'_{j+n}^{m-k}(d / R_t),
//   L_j^k  += (-1)^j A_j^k R_t^{-(j+1)} acc_j^k,        Ms = A_n^m M_n^m / R_s^n.
// Every center is the root center plus dyadic multiples of the radii, to
// rounding, so d / min(R_s, R_t) is an integer vector: (level difference, that
// vector) is a class key.  Written over real degrees of freedom (Re of every coefficient,
// Im of those with m > 0: 2 NTERM - P of them, 64 at P = 8), a class's map is
// one ND x ND real matrix K (built once per solve from FP64 harmonics).
//
// The pairs of each class are sorted together; one block takes up to
// 128 of them and forms Y = K x [Ms of their sources] as a dense product in
// FP32 (the operator loaded once per block, 8 x 8 outputs per thread), writing
// each pair's column of Y at the pair's position in the target-grouped list.
// A second pass sums, per target, its pairs' columns in list order in FP64 and
// adds them to L: deterministic, no atomics.  The 4,096 multiply-adds per pair
// (at P = 8) replace the 9,216 of the pair-by-pair complex contraction.
//
// Pairs through periodic images form classes of their own (the image and the
// target level join the key, since the shift is not a multiple of the radii).
// Every class gets its operator, even one used by a single pair: leaving the
// classes of fewer than 8, 16, 32 or 64 pairs to the pair-by-pair kernel
// measured slower on a 4M-body solve, the 512-system batch and the periodic
// water box alike (the build of one more operator costs less than a pair
// through the pair-by-pair kernel's launches).  Pairs whose class found no
// hash slot stay with the pair-by-pair FP32 kernel, which then runs on a
// compacted list of just those pairs (left_off / left_src); pairs outside the
// mixed policy stay with the FP64 kernel as before.
//
// Two engines form the products.  The tensor-core one (k_m2l_class_mma) splits
// every operand entry into three bf16 pieces, x = hi + mid + lo (24 significant
// bits, the FP32 mantissa), and accumulates the six products of pieces whose
// weights reach 2^-16 (hi.hi, hi.mid, mid.hi, hi.lo, lo.hi, mid.mid) with
// tcgen05.mma into an FP32 accumulator in tensor memory: the terms left out
// weigh about 2^-24, FP32 rounding.  The CUDA-core one (k_m2l_class_gemm) is a
// plain FP32 product.
//
// The plain method takes the same route in FP64 (k_m2l_class_gemm64): operators,
// multipoles, products and contributions in FP64, for the pairs whose centers
// are at the class's offset to FP64 precision (on_lattice).
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "fmm.h"
#include "harmonics.cuh"
#include "scan.cuh"

namespace exafmm_b200 {
namespace {

constexpr unsigned long long kEmpty = ~0ull;
constexpr int kClsBits = 20;      // class id field of the pair key
constexpr int kMaxSlabs = 100;    // k_slabs: at most twice this and one
constexpr int kProbe = 64;        // hash probe limit (a pair that finds no slot stays per-pair)

__host__ __device__ inline int nd_of(int P) { return P * (P + 1) - P; }
__host__ __device__ inline int ndp_of(int P) { return (nd_of(P) + 15) / 16 * 16; }

__device__ __forceinline__ unsigned long long mix64(unsigned long long k) {
  // MurmurHash3's 64-bit finalizer
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  k ^= k >> 33;
  return k;
}

// Real degree of freedom d -> (n, m, part): d < NT is Re of coefficient d,
// d >= NT the Im parts of the m > 0 coefficients in (n, m) order.
__device__ __forceinline__ void dof_decode(int d, int NT, int &n, int &m, int &part) {
  if (d < NT) {
    tri_decode(d, n, m);
    part = 0;
  } else {
    int e = d - NT;
    n = 1;
    while (e >= n) {
      e -= n;
      n++;
    }
    m = e + 1;
    part = 1;
  }
}

// Three bf16 pieces of x (hi, mid, lo; each the rounding of what the previous
// ones leave), as raw bits.
__device__ __forceinline__ void split_bf16x3(double x, unsigned short out[3]) {
#pragma unroll
  for (int p = 0; p < 3; p++) {
    const __nv_bfloat16 h = __double2bfloat16(x);
    out[p] = __bfloat16_as_ushort(h);
    x -= (double)__bfloat162float(h);
  }
}

// Offset, in bf16 elements, of entry (row, k) of a K-major tensor-core operand
// with NDP entries per row, in the canonical layout without swizzle: core
// matrices of 8 rows x 16 bytes (8 entries) stored as 128 contiguous bytes, the
// NDP / 8 core matrices of an 8-row group side by side along k (leading byte
// offset 128), row groups NDP / 8 x 128 bytes apart (stride byte offset).
__host__ __device__ __forceinline__ int core_off(int row, int k, int NDP) {
  return ((row >> 3) * (NDP >> 3) + (k >> 3)) * 64 + (row & 7) * 8 + (k & 7);
}

__device__ __forceinline__ unsigned long long class_key(int dl, long long dx, long long dy, long long dz) {
  return ((unsigned long long)(dl + 16) << 48) | ((unsigned long long)(dx + 32768) << 32) |
         ((unsigned long long)(dy + 32768) << 16) | (unsigned long long)(dz + 32768);
}

// A pair through a periodic image: the source sits at its cell's center plus
// the image shift (a multiple of the cycle, not of the radii), so the offset
// in units of the target radius is the integer offset of the two cells minus
// shift / R_t, which depends on the target level too.  Key: bit 63 set, the
// target level at bits 58-62, dl + 16 at 53-57, the image at 48-52, then the
// cells' integer offset as in class_key (whose keys keep bit 63 clear).
__device__ __forceinline__ unsigned long long class_key_image(int lt, int dl, int img, long long dx, long long dy,
                                                              long long dz) {
  return (1ull << 63) | ((unsigned long long)lt << 58) | ((unsigned long long)(dl + 16) << 53) |
         ((unsigned long long)img << 48) | ((unsigned long long)(dx + 32768) << 32) |
         ((unsigned long long)(dy + 32768) << 16) | (unsigned long long)(dz + 32768);
}

// Whether the centers' separation d is k radii (of rmin), k the rounded offset
// of its class, to within 2^-48 (3.6e-15) of its length.  The tree rounds every
// center, so it is not exactly: by a few ulp of the coordinates, up to 4e-15 of
// a cell at the origin but 1e-12 at level 4 of a unit box centered at 1,000.  The
// bodies' expansions are about the rounded centers, so in FP64 a pair further
// off than that stays with the pair-by-pair kernel, which takes d itself.
__device__ __forceinline__ bool on_lattice(const double (&d)[3], const double (&k)[3], double rmin) {
  const double len = (fabs(k[0]) + fabs(k[1]) + fabs(k[2])) * rmin;
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (fabs(fma(-k[i], rmin, d[i])) > len * 0x1p-48) return false;
  return true;
}

// 1. Per pair of the target-grouped list: its class's hash slot, or -1.
__global__ void k_pair_class(const int *off, const int *src, long long ncells, const double4 *cell_x,
                             const int2 *cell_pl, int min_level, int max_dl, unsigned long long *hk,
                             long long hmask, int *pair_slot) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    if (b == e) continue;
    const double4 Xt = cell_x[c];
    const int lt = cell_pl[c].y;
    for (int q = b + lane; q < e; q += 32) {
      const int packed = src[q];
      const int cj = packed & 0x3ffffff, img = packed >> 26;
      const int ls = cell_pl[cj].y;
      const int dl = ls - lt;
      int slot = -1;
      if (lt >= min_level && lt < 32 && dl <= max_dl && dl >= -max_dl) {
        const double4 Xs = cell_x[cj];
        const double rmin = fmin(Xt.w, Xs.w);
        const double fx = rint((Xt.x - Xs.x) / rmin), fy = rint((Xt.y - Xs.y) / rmin), fz = rint((Xt.z - Xs.z) / rmin);
        if (fabs(fx) < 32767 && fabs(fy) < 32767 && fabs(fz) < 32767) {
          const unsigned long long key =
              img == 13 ? class_key(dl, (long long)fx, (long long)fy, (long long)fz)
                        : class_key_image(lt, dl, img, (long long)fx, (long long)fy, (long long)fz);
          long long h = (long long)(mix64(key) & (unsigned long long)hmask);
          for (int p = 0; p < kProbe; p++) {
            // a slot's key, once set, never changes: read it at L2 and CAS only
            // while the slot is still empty
            unsigned long long old = __ldcg(&hk[h]);
            if (old == kEmpty) old = atomicCAS(&hk[h], kEmpty, key);
            if (old == kEmpty || old == key) {
              slot = (int)h;
              break;
            }
            h = (h + 1) & hmask;
          }
        }
      }
      pair_slot[q] = slot;
    }
  }
}

// 2. The classes (every occupied slot), in arbitrary order (sorted by key next).
__global__ void k_class_compact(const unsigned long long *hk, long long hcap,
                                unsigned long long *ck, int *cs, int *ncls, int cap) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < hcap; h += (long long)gridDim.x * blockDim.x) {
    if (hk[h] != kEmpty) {
      const int i = atomicAdd(ncls, 1);
      if (i < cap) {
        ck[i] = hk[h];
        cs[i] = (int)h;
      }
    }
  }
}

__global__ void k_class_ids(const int *cs_sorted, int ncls, int *hid) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < ncls; i += gridDim.x * blockDim.x) hid[cs_sorted[i]] = i;
}

// 1'. and 2'. of the plain method, for one system's targets [c0, c1) (pairs from
// qb on): the class's hash slot per pair (or -1), the number of classes in
// cnt[0], of pairs that have one in cnt[1] and of the pair-by-pair kernel's
// steps for these (32 pairs of a target or what is left) in cnt[2].  The table has at least eight slots
// per class the caller takes (limit): past the limit no class is added, and
// cnt[0] says so; up to it every class has its slot, whatever the timing.
__global__ void k_pair_class64(const int *off, const int *src, long long c0, long long c1, int qb,
                               const double4 *cell_x, const int2 *cell_pl, unsigned long long *hk, long long hmask,
                               int limit, int *pair_slot, int *cnt) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  int taken = 0, steps = 0;
  for (long long c = c0 + (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < c1; c += warps) {
    const int b = off[c], e = off[c + 1];
    if (b == e) continue;
    const double4 Xt = cell_x[c];
    const int lt = cell_pl[c].y;
    int here = 0;
    for (int q = b + lane; q < e; q += 32) {
      const int cj = src[q] & 0x3ffffff;
      const int dl = cell_pl[cj].y - lt;
      int slot = -1;
      if (dl <= 15 && dl >= -15) {  // what a key holds
        const double4 Xs = cell_x[cj];
        const double rmin = fmin(Xt.w, Xs.w);
        const double d[3] = {Xt.x - Xs.x, Xt.y - Xs.y, Xt.z - Xs.z};
        const double f[3] = {rint(d[0] / rmin), rint(d[1] / rmin), rint(d[2] / rmin)};
        if (fabs(f[0]) < 32767 && fabs(f[1]) < 32767 && fabs(f[2]) < 32767 && on_lattice(d, f, rmin)) {
          here++;
          const unsigned long long key = class_key(dl, (long long)f[0], (long long)f[1], (long long)f[2]);
          long long h = (long long)(mix64(key) & (unsigned long long)hmask);
          for (long long p = 0; p <= hmask; p++) {
            unsigned long long old = __ldcg(&hk[h]);
            if (old == kEmpty || (p & 63) == 63) {
              if (__ldcg(&cnt[0]) > limit) break;
              if (old == kEmpty) old = atomicCAS(&hk[h], kEmpty, key);
              if (old == kEmpty) atomicAdd(&cnt[0], 1);
            }
            if (old == kEmpty || old == key) {
              slot = (int)h;
              break;
            }
            h = (h + 1) & hmask;
          }
        }
      }
      pair_slot[q - qb] = slot;
    }
    for (int o = 16; o > 0; o >>= 1) here += __shfl_xor_sync(0xffffffffu, here, o);
    taken += here;
    steps += (here + 31) / 32;
  }
  if (lane == 0 && taken) {
    atomicAdd(&cnt[1], taken);
    atomicAdd(&cnt[2], steps);
  }
}

__global__ void k_class_ids64(const unsigned long long *hk, long long hcap, unsigned long long *ck, int *hid, int *n) {
  for (long long h = blockIdx.x * (long long)blockDim.x + threadIdx.x; h < hcap; h += (long long)gridDim.x * blockDim.x)
    if (hk[h] != kEmpty) {
      const int i = atomicAdd(n, 1);
      ck[i] = hk[h];
      hid[h] = i;
    }
}

// The systems of a forest with at least min_pairs pairs: first and end cell, first and end pair.
__global__ void k_sys_ranges(const int *off, const int *sys_cell, int nsys, int min_pairs, int4 *out, int *n) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nsys; s += gridDim.x * blockDim.x) {
    const int c0 = sys_cell[s], c1 = sys_cell[s + 1];
    if (off[c1] - off[c0] >= min_pairs) out[atomicAdd(n, 1)] = make_int4(c0, c1, off[c0], off[c1]);
  }
}

// Cuts targets [c0, c1) into slabs of at most `rows` pairs (or one target): out[i]
// = (first cell, first pair) of slab i and, after the last, (c1, off[c1]).  One warp.
__global__ void k_slabs(const int *off, int c0, int c1, long long rows, int2 *out, int *n) {
  const int lane = threadIdx.x;
  int k = 0;
  for (int c = c0; c < c1; k++) {
    const int first = off[c];
    if (lane == 0) out[k] = make_int2(c, first);
    int lo = c + 1, hi = c1;  // the last end with at most `rows` pairs, 32 probes a step
    while (lo < hi) {
      const int step = (hi - lo + 31) / 32;
      const int at = (int)min((long long)lo + (long long)(lane + 1) * step, (long long)hi);
      const int in = __popc(__ballot_sync(0xffffffffu, (long long)off[at] - first <= rows));
      const int top = in == 32 ? hi : (int)min((long long)lo + (long long)(in + 1) * step, (long long)hi) - 1;
      lo = (int)min((long long)lo + (long long)in * step, (long long)hi);
      hi = top;
    }
    c = lo;
  }
  if (lane == 0) {
    out[k] = make_int2(c1, off[c1]);
    *n = k;
  }
}

// 3. Operator of each class: FP32 k-major, Kt[class][input dof][output dof]
// (CUDA-core engine), or three bf16 pieces of it per class, each an operand
// image of NDP output rows x NDP inputs in the core_off layout (tensor cores).
// cell_x[0].w (the root radius) and cycle place the image shifts of
// class_key_image keys (one system, never a forest, has image pairs).
// Operand layouts of k_build_K: FP32 k-major Kt[class][input][output] (CUDA
// cores), three bf16 pieces in the core_off image, or in the 128-byte-swizzled
// image (TMA).  NDP and the layout are template parameters so that mapping an
// entry's position to its (output, input) pair is shifts and constant
// divisions, not runtime divisions (the build was bound by integer work).
enum KLayout : int { kKFp32 = 0, kKCore = 1, kKSwizzled = 2, kKFp64 = 3 };

// With cstart (FP64), classes without a pair in it are left out.
template <int NDP, int LAYOUT>
__global__ void __launch_bounds__(256)
k_build_K(DevTables t, const unsigned long long *ck, int P, float *Kt, unsigned short *Kb, double *Kd,
          const double4 *cell_x, double cycle, const int *cstart) {
  if (LAYOUT == kKFp64 && cstart && cstart[blockIdx.x] == cstart[blockIdx.x + 1]) return;
  extern __shared__ double2 S[];  // S'_p^q, q >= 0, at d / R_t
  constexpr int KB = (NDP + 63) / 64;  // 128-byte K-blocks of the swizzled image
  constexpr int IMG = LAYOUT == kKSwizzled ? KB * NDP * 64 : NDP * NDP;
  const int NT = t.nterm, ND = nd_of(P);
  const unsigned long long key = ck[blockIdx.x];
  const bool image = (key >> 63) != 0;
  const int dl = image ? (int)((key >> 53) & 31) - 16 : (int)((key >> 48) & 0xffff) - 16;
  const double ux = (double)(long long)((key >> 32) & 0xffff) - 32768.0;
  const double uy = (double)(long long)((key >> 16) & 0xffff) - 32768.0;
  const double uz = (double)(long long)(key & 0xffff) - 32768.0;
  const double to_rt = dl > 0 ? ldexp(1.0, -dl) : 1.0;  // min(R_s, R_t) / R_t
  double sx = 0.0, sy = 0.0, sz = 0.0;                    // image shift / R_t
  if (image) {
    const int lt = (int)((key >> 58) & 31), img = (int)((key >> 48) & 31);
    const double inv_rt = 1.0 / ldexp(cell_x[0].w, -lt);
    sx = (double)(img / 9 - 1) * cycle * inv_rt;
    sy = (double)((img / 3) % 3 - 1) * cycle * inv_rt;
    sz = (double)(img % 3 - 1) * cycle * inv_rt;
  }
  if ((int)threadIdx.x < 2 * P - 1)
    singular_column(t, threadIdx.x, 2 * P - 1, ux * to_rt - sx, uy * to_rt - sy, uz * to_rt - sz, t.ainv, S);
  // (n, m, part) of every real degree of freedom, decoded once per block, and
  // (R_s / R_t)^n for every source degree n
  __shared__ int dof_nmp[128];
  __shared__ double fn_of[32];
  for (int d = threadIdx.x; d < ND && d < 128; d += blockDim.x) {
    int n, m, part;
    dof_decode(d, NT, n, m, part);
    dof_nmp[d] = n | (m << 8) | (part << 16);
  }
  if ((int)threadIdx.x < P) fn_of[threadIdx.x] = ldexp(1.0, -dl * (int)threadIdx.x);
  __syncthreads();
  for (int e = threadIdx.x; e < IMG; e += blockDim.x) {
    int c, r;  // input and output dof; with Kb, e walks the operand image so the stores are contiguous
    if constexpr (LAYOUT == kKSwizzled) {  // K-block c / 64, row r, 16-byte chunk ((c % 64) / 8) ^ (r % 8)
      const int kb = e / (NDP * 64), w = e - kb * NDP * 64;
      r = w >> 6;
      c = kb * 64 + (((((w >> 3) & 7) ^ (r & 7))) << 3) + (w & 7);
    } else if constexpr (LAYOUT == kKCore) {
      const int ci = e >> 6, w = e & 63;
      r = (ci / (NDP >> 3)) * 8 + (w >> 3);
      c = (ci % (NDP >> 3)) * 8 + (w & 7);
    } else {
      c = e / NDP;
      r = e - c * NDP;
    }
    double val = 0.0;
    if (r < ND && c < ND) {
      const int er = dof_nmp[r], ec = dof_nmp[c];
      const int j = er & 0xff, k = (er >> 8) & 0xff, rp = er >> 16;
      const int n = ec & 0xff, mp = (ec >> 8) & 0xff, cp = ec >> 16;
      const double fn = fn_of[n];  // (R_s / R_t)^n
      double sr = 0.0, si = 0.0;
      for (int side = 0; side < (mp > 0 ? 2 : 1); side++) {
        const int m = side == 0 ? mp : -mp;
        const int q = m - k, p = j + n;
        double2 Sv = q >= 0 ? S[tri(p) + q] : cconj(S[tri(p) - q]);
        const double s = (m < 0) ? 1.0 : (m <= k ? (double)sgn_pow(m) : (double)sgn_pow(k));
        // the input's contribution to M_n^m: Re part -> 1, Im part -> +i (m > 0) or -i (m < 0)
        double tr = s * Sv.x, ti = s * Sv.y;
        if (cp == 1) {
          const double a = tr;
          if (m > 0) {
            tr = -ti;
            ti = a;
          } else {
            tr = ti;
            ti = -a;
          }
        }
        sr += tr;
        si += ti;
      }
      val = fn * (rp == 0 ? sr : si);
    }
    if constexpr (LAYOUT == kKFp64) {
      Kd[(long long)blockIdx.x * NDP * NDP + c * NDP + r] = val;
    } else if constexpr (LAYOUT == kKFp32) {
      Kt[(long long)blockIdx.x * NDP * NDP + c * NDP + r] = (float)val;
    } else {
      unsigned short h[3];
      split_bf16x3(val, h);
      unsigned short *dst = Kb + (long long)blockIdx.x * 3 * IMG + e;  // e == the operand offset of (r, c)
#pragma unroll
      for (int p = 0; p < 3; p++) dst[p * IMG] = h[p];
    }
  }
}

// Scaled multipoles over real degrees of freedom, padded to NDP: FP32 rows
// (Msr[cell][dof]), or three bf16 pieces per cell (Msb[cell][piece][dof]).
__global__ void k_scale_M_real(DevTables t, const double2 *M, const double4 *cell_x, long long ncells, int P,
                               float *Msr, unsigned short *Msb, double *Msd) {
  const int NT = t.nterm, ND = nd_of(P), NDP = ndp_of(P);
  const long long total = ncells * NDP;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long c = i / NDP;
    const int d = (int)(i - c * NDP);
    double v = 0.0;
    if (d < ND) {
      int n, m, part;
      dof_decode(d, NT, n, m, part);
      const int o = tri(n) + m;
      const double s = t.anm[o] * pow(cell_x[c].w, -(double)n);
      const double2 mv = M[c * NT + o];
      v = (part == 0 ? mv.x : mv.y) * s;
    }
    if (Msr) Msr[i] = (float)v;
    if (Msd) Msd[i] = v;
    if (Msb) {
      unsigned short h[3];
      split_bf16x3(v, h);
#pragma unroll
      for (int p = 0; p < 3; p++) Msb[(c * 3 + p) * NDP + d] = h[p];
    }
  }
}

// 4. Per target: flag the pairs of classes with an operator (taken) and count the
// leftover pairs of the mixed policy (for the pair-by-pair kernel).
__device__ __forceinline__ bool policy_pair(int lt, int ls, int min_level, int max_dl) {
  const int dl = lt - ls;
  return lt >= min_level && dl <= max_dl && dl >= -max_dl;
}

__global__ void k_gemm_flags(const int *off, const int *src, long long ncells, const int *pair_slot, const int *hid,
                             const int2 *cell_pl, int min_level, int max_dl, unsigned char *taken, int *left_cnt,
                             unsigned *pkey, int *pval) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    const int lt = cell_pl[c].y;
    int left = 0;
    for (int q = b + lane; q < e; q += 32) {
      const int s = pair_slot[q];
      const int cls = s >= 0 ? hid[s] : -1;
      taken[q] = cls >= 0 ? 1 : 0;
      pkey[q] = cls >= 0 ? (unsigned)cls : 0xffffffffu;  // sort key: class, the rest last
      pval[q] = q;
      if (cls < 0 && policy_pair(lt, cell_pl[src[q] & 0x3ffffff].y, min_level, max_dl)) left++;
    }
    for (int o = 16; o > 0; o >>= 1) left += __shfl_xor_sync(0xffffffffu, left, o);
    if (lane == 0) left_cnt[c] = left;
  }
}

// The plain method's flags, for pairs [qb, qb + n).
__global__ void k_gemm_flags64(const int *pair_slot, const int *hid, long long n, unsigned char *taken, unsigned *pkey,
                               int *pval) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
    const int s = pair_slot[q];
    taken[q] = s >= 0;
    pkey[q] = s >= 0 ? (unsigned)hid[s] : 0xffffffffu;
    pval[q] = (int)q;
  }
}
__global__ void k_left_count(const int *off, long long ncells, const unsigned char *taken, int *left_cnt) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    int left = 0;
    for (int q = off[c] + lane; q < off[c + 1]; q += 32) left += !taken[q];
    for (int o = 16; o > 0; o >>= 1) left += __shfl_xor_sync(0xffffffffu, left, o);
    if (lane == 0) left_cnt[c] = left;
  }
}

// Offsets of the leftover pairs per target (exclusive scan of the counts).
struct LeftScan {
  using T = int;
  const int *cnt;
  int *off2;
  long long n;
  __device__ T value(long long i) const { return cnt[i]; }
  __device__ void emit(long long i, const T &, const T &excl) const { off2[i] = excl; }
  __device__ void total(const T &t) const { off2[n] = t; }
};

// The leftover pairs (not taken, inside the mixed policy) in list order.
__global__ void k_left_fill(const int *off, const int *src, long long ncells, const unsigned char *taken,
                            const int2 *cell_pl, int min_level, int max_dl, const int *off2, int *src2) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    const int lt = cell_pl[c].y;
    int at = off2[c];
    for (int base = b; base < e; base += 32) {
      const int q = base + lane;
      bool keep = false;
      int v = 0;
      if (q < e) {
        v = src[q];
        keep = !taken[q] && policy_pair(lt, cell_pl[v & 0x3ffffff].y, min_level, max_dl);
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) src2[at + __popc(m & ((1u << lane) - 1u))] = v;
      at += __popc(m);
    }
  }
}

// The pairs outside the mixed policy (root levels, large size ratios), which
// stay FP64: counted per target, then compacted in list order.
__global__ void k_complement_count(const int *off, const int *src, long long ncells, const int2 *cell_pl,
                                   int min_level, int max_dl, int *cnt) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    const int lt = cell_pl[c].y;
    int k = 0;
    if (lt < min_level) {
      k = e - b;  // every pair of a root-level target
    } else {
      for (int q = b + lane; q < e; q += 32)
        if (!policy_pair(lt, cell_pl[src[q] & 0x3ffffff].y, min_level, max_dl)) k++;
      for (int o = 16; o > 0; o >>= 1) k += __shfl_xor_sync(0xffffffffu, k, o);
    }
    if (lane == 0) cnt[c] = k;
  }
}

__global__ void k_complement_fill(const int *off, const int *src, long long ncells, const int2 *cell_pl,
                                  int min_level, int max_dl, const int *off2, int *src2) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long c = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < ncells; c += warps) {
    const int b = off[c], e = off[c + 1];
    const int lt = cell_pl[c].y;
    int at = off2[c];
    if (off2[c + 1] == at) continue;
    for (int base = b; base < e; base += 32) {
      const int q = base + lane;
      bool keep = false;
      int v = 0;
      if (q < e) {
        v = src[q];
        keep = lt < min_level || !policy_pair(lt, cell_pl[v & 0x3ffffff].y, min_level, max_dl);
      }
      const unsigned m = __ballot_sync(0xffffffffu, keep);
      if (keep) src2[at + __popc(m & ((1u << lane) - 1u))] = v;
      at += __popc(m);
    }
  }
}

// 5. Class ranges in the class-sorted pairs, and chunks of kChunk pairs.
constexpr int kChunk = 128;

__global__ void k_class_ranges(const unsigned *skey, long long n, int ncls, int *cstart) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c <= ncls; c += gridDim.x * blockDim.x) {
    long long lo = 0, hi = n;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (skey[mid] < (unsigned)c) lo = mid + 1;
      else hi = mid;
    }
    cstart[c] = (int)lo;
  }
}

struct ChunkScan {
  using T = int;
  const int *cstart;
  int *cbase;
  int n;
  __device__ T value(long long i) const { return (cstart[i + 1] - cstart[i] + kChunk - 1) / kChunk; }
  __device__ void emit(long long i, const T &, const T &excl) const { cbase[i] = excl; }
  __device__ void total(const T &t) const { cbase[n] = t; }
};

// Per chunk: (class, first sorted position, pairs); and per sorted position of
// a taken pair, its source cell (so a product block starts from two
// independent loads rather than a search and a chain of dependent ones).
__global__ void k_chunk_table(const int *cstart, const int *cbase, int ncls, int4 *chunks) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncls; c += gridDim.x * blockDim.x) {
    const int b = cstart[c], e = cstart[c + 1];
    for (int j = cbase[c], p = b; p < e; j++, p += kChunk) chunks[j] = make_int4(c, p, min(kChunk, e - p), 0);
  }
}

__global__ void k_sorted_sources(const int *sval, const int *src, const int *ntaken, int *ssrc) {
  const int n = *ntaken;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    ssrc[i] = src[sval[i]] & 0x3ffffff;
}

__device__ __forceinline__ void cp_async16(void *sdst, const void *gsrc) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(sdst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 6. One block per chunk (one class, up to kChunk pairs): Y[pair] = K_class x Ms[source].
// The operator ([input][output]) and the sources' columns ([pair][input], row
// stride BSTR) are copied into shared memory with cp.async.  Thread (tx, ty)
// holds rows 4ty..4ty+3 and H+4ty..H+4ty+3 (H = NDP / 2) of columns tx + 4j,
// j < 8: both operand reads are conflict-free (rows: consecutive threads take
// consecutive 16-byte groups; columns: the four tx read four distinct banks),
// and every 16-byte column read feeds 32 multiply-adds over four inputs.
template <int NDP>
__global__ void __launch_bounds__(128)
k_m2l_class_gemm(const unsigned *skey, const int *sval, const int *cstart, const int *cbase, int ncls,
                 const int *src, const float *Kt, const float *Msr, float *Y) {
  constexpr int H = NDP / 2;
  constexpr int RG = H / 4;                      // row groups: 8 at NDP = 64
  constexpr int CG = 128 / RG;                   // column groups: 16 at NDP = 64
  constexpr int NC = CG * 8;                     // columns per pass
  constexpr int BSTR = NDP + 4;                  // floats per staged column
  extern __shared__ float4 smem4[];
  float *sK = reinterpret_cast<float *>(smem4);  // [NDP input][NDP output]
  float *sB = sK + NDP * NDP;                    // [kChunk pair][BSTR]
  __shared__ int s_q[kChunk], s_src[kChunk];
  const int chunk = blockIdx.x;
  if (chunk >= cbase[ncls]) return;
  int lo = 0, hi = ncls;  // class of this chunk: last c with cbase[c] <= chunk
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (cbase[mid] <= chunk) lo = mid;
    else hi = mid;
  }
  const int cls = lo;
  const int p0 = cstart[cls] + (chunk - cbase[cls]) * kChunk;
  const int cnt = min(kChunk, cstart[cls + 1] - p0);
  const float *Kg = Kt + (long long)cls * NDP * NDP;
  for (int i = threadIdx.x; i < NDP * NDP / 4; i += 128) cp_async16(sK + 4 * i, Kg + 4 * i);
  if (threadIdx.x < kChunk) {
    const int q = threadIdx.x < cnt ? sval[p0 + threadIdx.x] : -1;
    s_q[threadIdx.x] = q;
    s_src[threadIdx.x] = q >= 0 ? (src[q] & 0x3ffffff) : -1;
  }
  __syncthreads();
  for (int w = threadIdx.x; w < kChunk * (NDP / 4); w += 128) {
    const int i = w / (NDP / 4), q4 = w % (NDP / 4);
    float *dst = sB + i * BSTR + 4 * q4;
    if (i < cnt) cp_async16(dst, Msr + (long long)s_src[i] * NDP + 4 * q4);
    else *reinterpret_cast<float4 *>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  cp_async_commit();
  cp_async_wait_all();
  __syncthreads();
  const int ty = threadIdx.x % RG, tx = threadIdx.x / RG;
  if (tx >= CG) return;  // 128 threads need not split evenly (no barrier follows)
  for (int c0 = 0; c0 < cnt; c0 += NC) {
    if (c0 + tx >= cnt) continue;
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    for (int k4 = 0; k4 < NDP; k4 += 4) {
      float4 b[8];
#pragma unroll
      for (int j = 0; j < 8; j++)  // columns past the chunk (discarded below) read its last column
        b[j] = *reinterpret_cast<const float4 *>(sB + min(c0 + tx + CG * j, kChunk - 1) * BSTR + k4);
#pragma unroll
      for (int kq = 0; kq < 4; kq++) {
        const float4 a0 = *reinterpret_cast<const float4 *>(sK + (k4 + kq) * NDP + 4 * ty);
        const float4 a1 = *reinterpret_cast<const float4 *>(sK + (k4 + kq) * NDP + H + 4 * ty);
        const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const float bv = kq == 0 ? b[j].x : kq == 1 ? b[j].y : kq == 2 ? b[j].z : b[j].w;
#pragma unroll
          for (int i = 0; i < 8; i++) acc[i][j] = fmaf(av[i], bv, acc[i][j]);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int i = c0 + tx + CG * j;
      if (i < cnt) {
        float *y = Y + (long long)s_q[i] * NDP;
        *reinterpret_cast<float4 *>(y + 4 * ty) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
        *reinterpret_cast<float4 *>(y + H + 4 * ty) = make_float4(acc[4][j], acc[5][j], acc[6][j], acc[7][j]);
      }
    }
  }
}

// ---- tensor-core engine (tcgen05, sm_100a)
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor of a K-major operand without swizzle:
// start address, leading byte offset (between the two core matrices along k
// that one instruction reads) and stride byte offset (between 8-row groups),
// all in 16-byte units; descriptor version 1 at bit 46; layout 0 = no swizzle.
__device__ __forceinline__ unsigned long long umma_desc(unsigned addr, unsigned lbo, unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | ((unsigned long long)((lbo >> 4) & 0x3fffu) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void umma_bf16(unsigned tmem_d, unsigned long long da, unsigned long long db, unsigned idesc,
                                          unsigned accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Waits for phase `parity` of the mbarrier at bar for at most about 2^31 clocks
// (about a second); false if it did not complete.
__device__ __forceinline__ bool mbar_wait_bounded(unsigned bar, unsigned parity) {
  const long long t0 = clock64();
  while (true) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > (1ll << 31)) return false;
  }
}

// TMEM columns: two accumulators of NDP FP32 columns each (hi.hi, and the
// five smaller products), at column 0 and NCOLS / 2; a power of two >= 32.
__host__ __device__ constexpr int mma_cols(int NDP) {
  return 2 * NDP <= 32 ? 32 : 2 * NDP <= 64 ? 64 : 2 * NDP <= 128 ? 128 : 256;
}

// Dynamic shared memory of k_m2l_class_mma<NDP>: the three pieces of the
// gathered source tile and of the operator, raised where needed to at least
// 456 bytes per TMEM column claimed.  An SM has 233,472 bytes of shared memory
// and 512 TMEM columns, so the CTAs that fit on one SM by shared memory never
// ask for more columns than it has and tcgen05.alloc never waits.
__host__ __device__ constexpr size_t mma_smem_bytes(int NDP) {
  return (size_t)3 * (kChunk * NDP + NDP * NDP) * 2 > (size_t)mma_cols(NDP) * 456
             ? (size_t)3 * (kChunk * NDP + NDP * NDP) * 2
             : (size_t)mma_cols(NDP) * 456;
}

// CTAs of k_m2l_class_mma<NDP> that fit on one SM (by shared memory).
__host__ __device__ constexpr int mma_ctas_per_sm(int NDP) {
  return (int)(233472 / (mma_smem_bytes(NDP) + 1152 + 1024));
}

// 6'. The per-class products on the tensor cores.  Persistent: each CTA takes a
// contiguous range of chunks (one class, up to kChunk pairs each; consecutive
// chunks mostly share a class, whose operator then stays in shared memory).
// Per chunk: D[pair][output] = sum_k Ms[source][k] K[k][output] with M = 128
// pairs, N = NDP outputs, K = NDP inputs, both operands K-major bf16 in shared
// memory (core_off layout), the accumulators (128 lanes x NDP FP32 columns) in
// tensor memory.  The tensor cores' FP32 sums are not round-to-nearest, so the
// hi.hi product gets its own accumulator and the five smaller products
// (2^-8 and 2^-16 of it) another: the large one sees NDP / 16 additions, and
// the epilogue adds the two in FP32.
// Per chunk j: thread 0 issues the 6 x NDP / 16 MMAs and commits them to an
// mbarrier; every thread loads chunk j+2's indices meanwhile (those of j+1
// were loaded during chunk j-1's products); once the
// products are done, all threads start the cp.async gather of chunk j+1's
// source pieces (lane pairs fetch whole 32-byte sectors) and, while it is in
// flight, read chunk j's accumulators (warp w: TMEM lanes 32w..32w+31) and
// write each pair's column of Y with 32-byte stores.
template <int NDP>
__device__ __forceinline__ void mma_gather(unsigned short *sA, unsigned short *sB, const int *s_src, int cnt,
                                           int cls, int &cur_cls, const unsigned short *Kb,
                                           const unsigned short *Msb) {
  constexpr int NG = NDP / 8, A_ELEMS = kChunk * NDP, B_ELEMS = NDP * NDP;
  if (cls != cur_cls) {  // a new class: its operator pieces
    const unsigned short *Kg = Kb + (long long)cls * 3 * B_ELEMS;
    for (int i = threadIdx.x; i < 3 * B_ELEMS / 8; i += 128) cp_async16(sB + 8 * i, Kg + 8 * i);
    cur_cls = cls;
  }
  // unit u: bit 0 = group parity, bits 1-4 = row within 16, then (row block of
  // 16, group pair, piece): a warp fetches 16 rows x 32 bytes (16 whole
  // sectors) and writes four whole core matrices (conflict-free)
  for (int u = threadIdx.x; u < kChunk * 3 * NG; u += 128) {
    const int i = ((u >> 5) & 7) * 16 + ((u >> 1) & 15);
    const int r2 = u >> 8;  // (group pair, piece)
    const int gp = r2 % (NG / 2), p = r2 / (NG / 2);
    const int g = 2 * gp + (u & 1);
    unsigned short *dst = sA + p * A_ELEMS + core_off(i, 8 * g, NDP);
    if (i < cnt) cp_async16(dst, Msb + ((long long)s_src[i] * 3 + p) * NDP + 8 * g);
    else *reinterpret_cast<uint4 *>(dst) = make_uint4(0u, 0u, 0u, 0u);
  }
  cp_async_commit();
}

// The gathered tiles complete and visible to the tensor cores; the previous
// TMEM reads ordered before the next MMAs.
__device__ __forceinline__ void mma_tiles_ready() {
  cp_async_wait_all();
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
      "%14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

__device__ __forceinline__ void st_global_v8(float *p, const float (&v)[8]) {
  asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(v[0]), "f"(v[1]), "f"(v[2]),
               "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7])
               : "memory");
}

template <int NDP>
__global__ void __launch_bounds__(128)
k_m2l_class_mma(const int4 *chunks, const int *nchunks, const int *sval, const int *ssrc,
                const unsigned short *Kb, const unsigned short *Msb, float *Y, int *err) {
  constexpr int NG = NDP / 8;                // 16-byte groups per operand row
  constexpr int A_ELEMS = kChunk * NDP;      // one piece of the source tile
  constexpr int B_ELEMS = NDP * NDP;         // one piece of the operator
  constexpr int NCOLS = mma_cols(NDP);
  constexpr unsigned D1 = NCOLS / 2;         // column of the small products' accumulator
  constexpr unsigned SBO = NG * 128;         // bytes between 8-row groups
  // kind::f16 instruction descriptor: D FP32 (bits 4-5 = 1), A and B bf16
  // (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
  constexpr unsigned IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NDP >> 3) << 17) |
                             ((unsigned)(kChunk >> 4) << 24);
  static_assert(NDP % 16 == 0 && NDP >= 16 && NDP <= 256, "N of an M = 128 MMA: multiple of 16 in [16, 256]");
  static_assert(2 * NDP <= NCOLS, "two accumulators");
  static_assert(kChunk == 128, "one TMEM lane and one thread per pair");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned short *sA = reinterpret_cast<unsigned short *>(smem_raw);
  unsigned short *sB = sA + 3 * A_ELEMS;
  __shared__ int s_src[kChunk];
  __shared__ __align__(8) unsigned long long s_bar;
  __shared__ unsigned s_tmem;
  const int total = *nchunks;
  const int j0 = (int)((long long)total * blockIdx.x / gridDim.x);
  const int j1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
  if (j0 >= j1) return;
  const unsigned bar = smem_u32(&s_bar);
  if (threadIdx.x < 32) {  // warp 0 owns the accumulators' columns
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                 "r"(NCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  int4 ch = chunks[j0];  // this thread's pair of the first chunk
  int q = (int)threadIdx.x < ch.z ? sval[ch.y + threadIdx.x] : -1;
  s_src[threadIdx.x] = q >= 0 ? ssrc[ch.y + threadIdx.x] : -1;
  int cur_cls = -1;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = s_tmem;
  mma_gather<NDP>(sA, sB, s_src, ch.z, ch.x, cur_cls, Kb, Msb);
  // the next chunk's descriptor, list positions and sources, loaded one chunk
  // ahead of their use
  int4 chn = ch;
  int qn = -1, scn = -1;
  if (j0 + 1 < j1) {
    chn = chunks[j0 + 1];
    qn = (int)threadIdx.x < chn.z ? sval[chn.y + threadIdx.x] : -1;
    scn = (int)threadIdx.x < chn.z ? ssrc[chn.y + threadIdx.x] : -1;
  }
  mma_tiles_ready();
  for (int j = j0; j < j1; j++) {
    const int cnt = ch.z, qc = q;
    if (threadIdx.x == 0) {
      const unsigned a0 = smem_u32(sA), b0 = smem_u32(sB);
      // pieces (of the sources, of the operator): hi.hi into D0, the rest into D1
      const int pa[6] = {0, 0, 2, 1, 0, 1}, pb[6] = {0, 2, 0, 1, 1, 0};
#pragma unroll
      for (int t = 0; t < 6; t++)
#pragma unroll
        for (int k = 0; k < NDP / 16; k++) {  // 16 inputs = two core matrices = 256 bytes per step
          const unsigned long long da = umma_desc(a0 + (unsigned)(pa[t] * A_ELEMS * 2 + k * 256), 128, SBO);
          const unsigned long long db = umma_desc(b0 + (unsigned)(pb[t] * B_ELEMS * 2 + k * 256), 128, SBO);
          umma_bf16(tmem + (t == 0 ? 0u : D1), da, db, IDESC, (t > 1 || k > 0) ? 1u : 0u);
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                   : "memory");
    }
    int sc = -1;
    if (j + 1 < j1) {
      ch = chn;
      q = qn;
      sc = scn;
    }
    if (j + 2 < j1) {  // the chunk after, while the products run
      chn = chunks[j + 2];
      qn = (int)threadIdx.x < chn.z ? sval[chn.y + threadIdx.x] : -1;
      scn = (int)threadIdx.x < chn.z ? ssrc[chn.y + threadIdx.x] : -1;
    }
    bool done = true;  // one poller per warp
    if ((threadIdx.x & 31) == 0) done = mbar_wait_bounded(bar, (unsigned)((j - j0) & 1));
    done = __shfl_sync(0xffffffffu, done, 0);
    tc_fence_after();
    if (!__syncthreads_and(done)) {  // products done: the tiles and s_src are free
      if (threadIdx.x == 0) atomicOr(err, kErrMmaTimeout);
      break;
    }
    if (j + 1 < j1) {
      s_src[threadIdx.x] = sc;
      __syncthreads();
      mma_gather<NDP>(sA, sB, s_src, ch.z, ch.x, cur_cls, Kb, Msb);
    }
    {  // chunk j's accumulators -> Y, while the gather is in flight
      const int warp = threadIdx.x >> 5;  // row threadIdx.x = TMEM lane threadIdx.x
      const unsigned taddr = tmem + ((unsigned)(warp * 32) << 16);
      float *y = (int)threadIdx.x < cnt ? Y + (long long)qc * NDP : nullptr;
#pragma unroll
      for (int c0 = 0; c0 < NDP; c0 += 16) {
        unsigned r[16], v[16];
        tmem_ld16(taddr + (unsigned)c0, r);
        tmem_ld16(taddr + D1 + (unsigned)c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (y) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; e++) o[e] = __uint_as_float(r[8 * h + e]) + __uint_as_float(v[8 * h + e]);
            st_global_v8(y + c0 + 8 * h, o);
          }
        }
      }
    }
    mma_tiles_ready();
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS) : "memory");
  }
}

// ---- the P = 8 products with the source pieces gathered by TMA
// The operands in the canonical 128-byte-swizzle K-major layout: NDP = 64
// inputs per row = 128 bytes, row r at r * 128, its 16-byte chunk c stored at
// chunk position c ^ (r % 8), 8-row atoms of 1024 bytes (1024-byte aligned).
// TMA writes the source rows in this layout itself (tensor map swizzle 128B);
// the operator image is written so by k_build_K: entry (row, k) at bf16 offset
// row * 64 + (((k / 8) ^ (row % 8)) * 8) + k % 8.

// Shared-memory matrix descriptor of a K-major, 128-byte-swizzled operand:
// start address, stride byte offset 1024 (8-row atoms), leading byte offset
// unused (1), version 1, layout SWIZZLE_128B (2 at bit 61).
__device__ __forceinline__ unsigned long long umma_desc_sw128(unsigned addr) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | (1ull << 16) | ((unsigned long long)(1024 >> 4) << 32) |
         (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

// Four source rows (cells y0..y3, 64 bf16 from column x) into 4 x 128 bytes at dst.
__device__ __forceinline__ void tma_gather4(unsigned dst, const CUtensorMap *map, unsigned bar, int x, int y0, int y1,
                                            int y2, int y3) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%3, %4, %5, %6, %7}], [%2];" ::"r"(dst),
      "l"(reinterpret_cast<unsigned long long>(map)), "r"(bar), "r"(x), "r"(y0), "r"(y1), "r"(y2), "r"(y3)
      : "memory");
}

// 128-byte K-blocks per operand row, and the kernel's shared memory (A and B
// pieces in K-blocks, plus alignment slack).
__host__ __device__ constexpr int tma_kblocks(int NDP) { return (NDP + 63) / 64; }
__host__ __device__ constexpr size_t tma_smem_bytes(int NDP) {
  return (size_t)3 * tma_kblocks(NDP) * (kChunk + NDP) * 128 + 1024;
}

// As k_m2l_class_mma<NDP>, with the chunk's source pieces (3 x KB x 128 rows
// x 128 bytes, KB = 1 at P = 8, 2 at P = 10) brought in by 96 KB
// tile::gather4 loads (3 KB per lane of warp 0) completing on an mbarrier,
// instead of cp.async of all threads.  At NDP = 112 the second K-block holds
// inputs 64-127 of a row: past 112 it reads the next piece (or zeros past the
// row's end), which no MMA step reaches (the last one ends at input 112).
template <int NDP>
__global__ void __launch_bounds__(128)
k_m2l_class_mma_tma(const __grid_constant__ CUtensorMap msb_map, const int4 *chunks, const int *nchunks,
                    const int *sval, const int *ssrc, const unsigned short *Kb, float *Y, int *err) {
  constexpr int KB = tma_kblocks(NDP);
  constexpr int A_ELEMS = KB * kChunk * 64, B_ELEMS = KB * NDP * 64;  // one piece of each, in K-blocks
  constexpr int NCOLS = mma_cols(NDP);
  constexpr unsigned D1 = NCOLS / 2;
  constexpr unsigned IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(NDP >> 3) << 17) |
                             ((unsigned)(kChunk >> 4) << 24);
  constexpr unsigned A_BYTES = 3 * A_ELEMS * 2;
  static_assert(NDP % 16 == 0 && NDP <= 128, "one or two 128-byte K-blocks");
  extern __shared__ unsigned char smem_raw[];
  unsigned short *sA = reinterpret_cast<unsigned short *>(
      (reinterpret_cast<unsigned long long>(smem_raw) + 1023) & ~1023ull);
  unsigned short *sB = sA + 3 * A_ELEMS;
  __shared__ int s_src[kChunk];
  __shared__ __align__(8) unsigned long long s_bar, s_tbar;
  __shared__ unsigned s_tmem;
  const int total = *nchunks;
  const int j0 = (int)((long long)total * blockIdx.x / gridDim.x);
  const int j1 = (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
  if (j0 >= j1) return;
  const unsigned bar = smem_u32(&s_bar), tbar = smem_u32(&s_tbar);
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s_tmem)),
                 "r"(NCOLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  int4 ch = chunks[j0];
  int q = (int)threadIdx.x < ch.z ? sval[ch.y + threadIdx.x] : -1;
  s_src[threadIdx.x] = q >= 0 ? ssrc[ch.y + threadIdx.x] : -1;
  int cur_cls = -1;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const unsigned tmem = s_tmem;
  const unsigned a0 = smem_u32(sA), b0 = smem_u32(sB);
  // one chunk's loads: the operator pieces if the class changed (cp.async, all
  // threads), the source pieces by TMA (thread 0); rows past the chunk repeat
  // its first source (their products are not stored)
  auto issue_loads = [&](int cls, int cnt) {
    if (cls != cur_cls) {
      const unsigned short *Kg = Kb + (long long)cls * 3 * B_ELEMS;
      for (int i = threadIdx.x; i < 3 * B_ELEMS / 8; i += 128) cp_async16(sB + 8 * i, Kg + 8 * i);
      cur_cls = cls;
    }
    cp_async_commit();
    if (threadIdx.x < 32) {  // warp 0: lane g issues row group g of every piece and K-block
      if (threadIdx.x == 0) mbar_expect_tx(tbar, A_BYTES);
      __syncwarp();
      const int g = threadIdx.x, f = s_src[0];
      int y[4];
#pragma unroll
      for (int u = 0; u < 4; u++) y[u] = 4 * g + u < cnt ? s_src[4 * g + u] : f;
#pragma unroll
      for (int p = 0; p < 3; p++)
#pragma unroll
        for (int kb = 0; kb < KB; kb++)
          tma_gather4(a0 + (unsigned)(p * A_ELEMS * 2 + kb * kChunk * 128 + g * 512), &msb_map, tbar,
                      p * NDP + 64 * kb, y[0], y[1], y[2], y[3]);
    }
  };
  issue_loads(ch.x, ch.z);
  // the next chunk's descriptor, list positions and sources, loaded one chunk
  // ahead of their use (so the three dependent loads are not waited for
  // between the products and the next gather)
  int4 chn = ch;
  int qn = -1, scn = -1;
  if (j0 + 1 < j1) {
    chn = chunks[j0 + 1];
    qn = (int)threadIdx.x < chn.z ? sval[chn.y + threadIdx.x] : -1;
    scn = (int)threadIdx.x < chn.z ? ssrc[chn.y + threadIdx.x] : -1;
  }
  bool ok = true;
  for (int j = j0; j < j1; j++) {
    const int cnt = ch.z, qc = q, it = j - j0;
    // this chunk's tiles: the source pieces (TMA) and the operator (cp.async)
    bool got = true;
    if ((threadIdx.x & 31) == 0) got = mbar_wait_bounded(tbar, (unsigned)(it & 1));
    got = __shfl_sync(0xffffffffu, got, 0);
    cp_async_wait_all();
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    if (!__syncthreads_and(got)) {
      ok = false;
      break;
    }
    tc_fence_after();
    if (threadIdx.x == 0) {
      const int pa[6] = {0, 0, 2, 1, 0, 1}, pb[6] = {0, 2, 0, 1, 1, 0};
#pragma unroll
      for (int t = 0; t < 6; t++)
#pragma unroll
        for (int k = 0; k < NDP / 16; k++) {  // 16 inputs = 32 bytes along the swizzled rows of K-block k / 4
          const int kb = k >> 2, kk = k & 3;
          const unsigned long long da =
              umma_desc_sw128(a0 + (unsigned)(pa[t] * A_ELEMS * 2 + kb * kChunk * 128 + kk * 32));
          const unsigned long long db =
              umma_desc_sw128(b0 + (unsigned)(pb[t] * B_ELEMS * 2 + kb * NDP * 128 + kk * 32));
          umma_bf16(tmem + (t == 0 ? 0u : D1), da, db, IDESC, (t > 1 || k > 0) ? 1u : 0u);
        }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                   : "memory");
    }
    int sc = -1;
    if (j + 1 < j1) {
      ch = chn;
      q = qn;
      sc = scn;
    }
    if (j + 2 < j1) {  // the chunk after, while the products run
      chn = chunks[j + 2];
      qn = (int)threadIdx.x < chn.z ? sval[chn.y + threadIdx.x] : -1;
      scn = (int)threadIdx.x < chn.z ? ssrc[chn.y + threadIdx.x] : -1;
    }
    bool done = true;
    if ((threadIdx.x & 31) == 0) done = mbar_wait_bounded(bar, (unsigned)(it & 1));
    done = __shfl_sync(0xffffffffu, done, 0);
    tc_fence_after();
    if (!__syncthreads_and(done)) {  // products done: the tiles and s_src are free
      ok = false;
      break;
    }
    if (j + 1 < j1) {
      s_src[threadIdx.x] = sc;
      __syncthreads();
      issue_loads(ch.x, ch.z);
    }
    {  // chunk j's accumulators -> Y, while the next loads are in flight
      const int warp = threadIdx.x >> 5;
      const unsigned taddr = tmem + ((unsigned)(warp * 32) << 16);
      float *yrow = (int)threadIdx.x < cnt ? Y + (long long)qc * NDP : nullptr;
#pragma unroll
      for (int c0 = 0; c0 < NDP; c0 += 16) {
        unsigned r[16], v[16];
        tmem_ld16(taddr + (unsigned)c0, r);
        tmem_ld16(taddr + D1 + (unsigned)c0, v);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (yrow) {
#pragma unroll
          for (int h = 0; h < 2; h++) {
            float o[8];
#pragma unroll
            for (int e = 0; e < 8; e++) o[e] = __uint_as_float(r[8 * h + e]) + __uint_as_float(v[8 * h + e]);
            st_global_v8(yrow + c0 + 8 * h, o);
          }
        }
      }
    }
  }
  if (!ok && (threadIdx.x & 31) == 0) atomicOr(err, kErrMmaTimeout);
  cp_async_wait_all();
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(NCOLS) : "memory");
  }
}

// 6''. The plain method's products, FP64.  Bound: the FP64 pipe (ND^2
// multiply-adds a pair: 4,096 at P = 8, where the pair-by-pair contraction
// takes 9,216 and its recurrences).  Persistent blocks of 256 threads take
// contiguous ranges of chunks, so the operator (ND x NDP, at most 90 KB) stays
// in shared memory across a class's chunks.  Up to P = 8 a tile is a chunk of
// 128 pairs and two blocks share an SM, one gathering (cp.async) while the
// other multiplies; at P = 10 one block holds the operator and two tiles of 64
// pairs, the next one gathered ahead.  Thread (tx, ty) holds outputs tx + 16 j
// of pairs ty + 16 v: two inputs of a pair come in one 16-byte read, an operator
// row is read by 16 consecutive threads, and a pair's outputs are stored in
// 128-byte runs.  Each output is
// one FP64 sum over the inputs in order, whatever the chunk, so a pair's
// contribution does not depend on the pairs beside it.  M2L phase, pair by pair
// against products: 1M-body Plummer sphere at P = 8 (15.1M pairs, 550 a class)
// 31.4 -> 11.7 ms; 100K-body cube at P = 10 (0.6M pairs, 90 a class) 3.25 -> 2.35.
// FP64 pipe 47 % of active cycles at P = 8 (5.6M pairs of a 400K-body Plummer
// sphere), 40 % on that cube, where the SMs are active 68 % of the launch.
__host__ __device__ constexpr int gemm64_rows(int NDP) { return NDP > 64 ? 64 : 128; }
__host__ __device__ constexpr int gemm64_bufs(int NDP) { return NDP > 64 ? 2 : 1; }
__host__ __device__ constexpr size_t gemm64_smem_bytes(int NDP, int ND) {
  return ((size_t)ND * NDP + (size_t)gemm64_bufs(NDP) * gemm64_rows(NDP) * (NDP + 2)) * sizeof(double);
}

// NV x NJ outputs a thread (pairs ty + 16 v, outputs tx + 16 j) over ND inputs.
template <int NDP, int NV>
__device__ __forceinline__ void gemm64_tile(const double *a, const double *b, int ND, const int *q, double *Y, int tx) {
  constexpr int NJ = NDP / 16, ASTR = NDP + 2;
  double acc[NV][NJ];
#pragma unroll
  for (int v = 0; v < NV; v++)
#pragma unroll
    for (int j = 0; j < NJ; j++) acc[v][j] = 0.0;
#pragma unroll 2
  for (int k = 0; k < ND; k += 2) {
    double2 x[NV];
#pragma unroll
    for (int v = 0; v < NV; v++) x[v] = *reinterpret_cast<const double2 *>(a + 16 * v * ASTR + k);
    const double *bk = b + k * NDP + tx;
#pragma unroll
    for (int j = 0; j < NJ; j++) {
      const double b0 = bk[16 * j], b1 = bk[NDP + 16 * j];
#pragma unroll
      for (int v = 0; v < NV; v++) acc[v][j] = fma(x[v].y, b1, fma(x[v].x, b0, acc[v][j]));
    }
  }
#pragma unroll
  for (int v = 0; v < NV; v++) {
    const int at = q[16 * v];
    if (at >= 0) {
#pragma unroll
      for (int j = 0; j < NJ; j++) Y[(long long)at * NDP + tx + 16 * j] = acc[v][j];
    }
  }
}

template <int NDP>
__global__ void __launch_bounds__(256, NDP > 64 ? 1 : 2)
k_m2l_class_gemm64(const int4 *chunks, const int *first, const int *last, int cls0, const int *sval, const int *ssrc,
                   const double *K, const double *Ms, double *Y, int ND) {
  constexpr int ASTR = NDP + 2, ROWS = gemm64_rows(NDP), BUFS = gemm64_bufs(NDP), PARTS = kChunk / ROWS;
  constexpr int TPR = 256 / ROWS;  // threads that gather one row
  extern __shared__ __align__(16) double smem_d[];
  __shared__ int s_q[2][ROWS];
  double *sK = smem_d;                      // [input][output]
  double *sA = smem_d + (size_t)ND * NDP;   // [buffer][pair][input]
  const int total = *last - *first;
  const int j0 = *first + (int)((long long)total * blockIdx.x / gridDim.x);
  const int j1 = *first + (int)((long long)total * (blockIdx.x + 1) / gridDim.x);
  if (j0 >= j1) return;
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int row = threadIdx.x / TPR, part = threadIdx.x % TPR;  // this thread's share of a gather
  // tile i of the range: chunk j0 + i / PARTS, its pairs from (i % PARTS) * ROWS on (perhaps none)
  const int tiles = PARTS * (j1 - j0);
  auto source = [&](int i, int &q) {
    q = -1;
    if (i >= tiles) return -1;
    const int4 ch = chunks[j0 + i / PARTS];
    const int at = (i % PARTS) * ROWS + row;
    if (at >= ch.z) return -1;
    q = sval[ch.y + at];
    return ssrc[ch.y + at];
  };
  auto gather = [&](int i, int src, int q) {
    if (part == 0) s_q[i & 1][row] = q;
    if (src >= 0) {
      const double *from = Ms + (long long)src * NDP;
      double *to = sA + (i % BUFS) * ROWS * ASTR + row * ASTR;
      for (int u = part; u < ND / 2; u += TPR) cp_async16(to + 2 * u, from + 2 * u);
    }
    cp_async_commit();
  };
  int cur = -1, nq;
  int next = source(0, nq);
  if (BUFS == 2) {
    gather(0, next, nq);
    next = source(1, nq);
  }
  for (int i = 0; i < tiles; i++) {
    const int4 ch = chunks[j0 + i / PARTS];
    const int cnt = min(ROWS, ch.z - (i % PARTS) * ROWS);
    gather(i + BUFS - 1, next, nq);  // its buffer was read before the last barrier
    next = source(i + BUFS, nq);
    if (ch.x != cur) {  // a new class: its operator (inputs from ND on are padding)
      const double *Kg = K + (long long)(ch.x - cls0) * NDP * NDP;
      for (int u = threadIdx.x; u < ND * NDP / 2; u += 256) cp_async16(sK + 2 * u, Kg + 2 * u);
      cp_async_commit();
      cur = ch.x;
      cp_async_wait_all();
    } else if (BUFS == 2) {
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      cp_async_wait_all();
    }
    __syncthreads();
    const double *a = sA + (i % BUFS) * ROWS * ASTR + ty * ASTR;
    const int *q = s_q[i & 1] + ty;
    // whole 16-pair rows of the tile only: classes often end in a short one
    if (cnt > ROWS / 2) gemm64_tile<NDP, ROWS / 16>(a, sK, ND, q, Y, tx);
    else if (cnt > ROWS / 4) gemm64_tile<NDP, ROWS / 32>(a, sK, ND, q, Y, tx);
    else if (cnt > 0) gemm64_tile<NDP, ROWS / 64>(a, sK, ND, q, Y, tx);
    __syncthreads();
  }
  cp_async_wait_all();
}

// 7. Per target cell of [c0, c1), in list order: the sum of its taken pairs'
// columns of Y (FP64), scaled by (-1)^j A_j^k R_t^{-(j+1)}, added to L.  Lane l holds
// entries VEC l .. VEC l + VEC - 1 of a column (VEC = 4 floats, one 16-byte
// load per lane and pair, for NDP > 64; else 2).  A group's rows are loaded
// together with its taken flags (the rows of pairs not taken hold whatever is
// there and are dropped by a select, so the loads do not wait for the flags),
// and the next group's loads are in flight while this one is added.
template <int NDP, typename T>
__global__ void k_m2l_class_reduce(const int *off, long long c0, long long c1, const unsigned char *taken, const T *Y,
                                   const double4 *cell_x, DevTables t, int P, double2 *L) {
  constexpr int VEC = NDP > 64 ? 4 : 2;
  constexpr int LANES = NDP / VEC;  // lanes that hold entries
  static_assert(NDP % VEC == 0 && LANES <= 32, "one row per warp-wide load");
  constexpr int G = sizeof(T) * VEC > 16 ? 4 : 8;  // rows in flight
  struct alignas(VEC * sizeof(T) < 16 ? VEC * sizeof(T) : 16) V {
    T f[VEC];
  };
  const int lane = threadIdx.x & 31;
  const bool active = lane < LANES;
  const int NT = t.nterm, ND = nd_of(P);
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  auto load = [&](int q, int e, bool &tk, V &v) {
    tk = false;
    v = V{};
    if (q < e) {
      tk = taken[q] != 0;
      if (active) v = *reinterpret_cast<const V *>(Y + (long long)q * NDP + VEC * lane);
    }
  };
  for (long long c = c0 + (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < c1; c += warps) {
    const int b = off[c], e = off[c + 1];
    double acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; i++) acc[i] = 0.0;
    bool any = false;
    bool tk[G], tk2[G];
    V v[G], v2[G];
#pragma unroll
    for (int i = 0; i < G; i++) load(b + i, e, tk[i], v[i]);
    for (int q0 = b; q0 < e; q0 += G) {
#pragma unroll
      for (int i = 0; i < G; i++) load(q0 + G + i, e, tk2[i], v2[i]);  // the next group, in flight
#pragma unroll
      for (int i = 0; i < G; i++) {
        if (!tk[i]) continue;
        any = true;
#pragma unroll
        for (int k = 0; k < VEC; k++) acc[k] += (double)v[i].f[k];
      }
#pragma unroll
      for (int i = 0; i < G; i++) {
        tk[i] = tk2[i];
        v[i] = v2[i];
      }
    }
    if (!any || !active) continue;
    const double rt = cell_x[c].w;
#pragma unroll
    for (int h = 0; h < VEC; h++) {
      const int d = VEC * lane + h;
      if (d >= ND) continue;
      int j, k, part;
      dof_decode(d, NT, j, k, part);
      const int o = tri(j) + k;
      const double val = acc[h] * sgn_pow(j) * t.anm[o] * pow(rt, -(double)(j + 1));
      double2 *dst = &L[c * NT + o];
      if (part == 0) dst->x += val;
      else dst->y += val;
    }
  }
}

int bits_for(long long v) {
  int b = 0;
  while ((1LL << b) <= v) b++;
  return b;
}

template <typename F>
void set_smem(F f, size_t bytes) {
  if (bytes > 48 * 1024) EXA_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// cuTensorMapEncodeTiled from the driver (no link-time dependency on libcuda).
EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// The bf16 source pieces Msb[cell][3 x NDP] as a 2-D tensor (3 NDP x ncells),
// read in boxes of one row x 64 elements (128 bytes) into the 128-byte-swizzled
// layout.
bool msb_tensor_map(CUtensorMap *map, const unsigned short *Msb, long long ncells, int NDP) {
  EncodeTiledFn fn = encode_tiled();
  if (!fn || ncells <= 0 || ncells > 0x7fffffffLL) return false;
  if ((reinterpret_cast<unsigned long long>(Msb) & 15ull) != 0) return false;
  const cuuint64_t dims[2] = {(cuuint64_t)(3 * NDP), (cuuint64_t)ncells};
  const cuuint64_t strides[1] = {(cuuint64_t)(3 * NDP * sizeof(unsigned short))};
  const cuuint32_t box[2] = {64, 1};
  const cuuint32_t estr[2] = {1, 1};
  return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void *)Msb, dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NDP>
void tma_launch(const CUtensorMap &map, M2LGemmBufs &g, const int *sv, long long chunks_max, int ncls, int *err,
                cudaStream_t st) {
  if constexpr (NDP == 64) {  // the two-K-block form (NDP = 112) measured slower than cp.async at P = 10
    constexpr size_t smem = tma_smem_bytes(NDP);
    set_smem(k_m2l_class_mma_tma<NDP>, smem);
    const int per_sm = (int)(233472 / (smem + 640 + 1024));
    const long long grid = std::min<long long>(chunks_max, (long long)kNumSMs * per_sm);
    k_m2l_class_mma_tma<NDP><<<(unsigned)grid, 128, smem, st>>>(map, g.chunks.p, g.cbase.p + ncls, sv, g.ssrc.p,
                                                                g.Kb.p, g.Y.p, err);
  }
}

template <int NDP>
void gemm64_launch(M2LGemmBufs &g, int cls0, int cls1, const int *sv, long long chunks_max, int ND, cudaStream_t st) {
  const size_t smem = gemm64_smem_bytes(NDP, ND);
  set_smem(k_m2l_class_gemm64<NDP>, smem);
  const int per_sm = std::max(1, std::min(2, (int)(233472 / (smem + 2048))));
  const long long grid = std::min<long long>(chunks_max, (long long)kNumSMs * per_sm);
  k_m2l_class_gemm64<NDP><<<(unsigned)grid, 256, smem, st>>>(g.chunks.p, g.cbase.p + cls0, g.cbase.p + cls1, cls0, sv,
                                                             g.ssrc.p, g.K64.p, g.Ms64r.p, g.Y64.p, ND);
  EXA_CHECK_LAUNCH();
}

template <typename T>
bool try_ensure(DBuf<T> &b, size_t n) {
  try {
    b.ensure(n);
    return true;
  } catch (const std::exception &) {
    cudaGetLastError();
    return false;
  }
}

}  // namespace

bool m2l_gemm_supported(int P) { return P == 4 || P == 6 || P == 8 || P == 10; }

// Where the class products beat the pair-by-pair kernel for one solve on a
// B200, measured on cube and Plummer systems of 20K-1M bodies (theta 0.4,
// ncrit 64): from about 0.15M pairs at P = 10, 1M at P = 8 and 8M at P = 6
// (at P = 4 the pair-by-pair code always wins), and only when the classes
// hold at least kMinPairsPerClass pairs on average, since every class costs
// an operator build: a 50K-body Plummer system at P = 10 (510K pairs, 73 per
// class) solved in 5.1 ms pair by pair and 6.6 ms with the products, a
// 100K-body cube (597K pairs, 89 per class) in 5.9 and 5.4 ms.
bool m2l_gemm_worthwhile(int P, long long n_m2l) {
  if (P == 6) return n_m2l >= 8000000;
  if (P == 8) return n_m2l >= 1000000;
  if (P == 10) return n_m2l >= 150000;
  return false;
}
constexpr long long kMinPairsPerClass = 80;

bool m2l_gemm(Context &C, const FmmArgs &a, M2LGemmBufs &g, long long n_m2l, int min_level, int max_dl) {
  const int P = a.P;
  if (!m2l_gemm_supported(P) || a.ncells <= 0 || n_m2l <= 0) return false;
  if (!g.force && !m2l_gemm_worthwhile(P, n_m2l)) return false;
  cudaStream_t st = a.stream;
  const DevTables &t = device_tables(P);
  const long long nc = a.ncells;
  const int NDP = ndp_of(P);
  // ---- classes
  // classes are far fewer than pairs (thousands to ~1e5): a table of about a
  // sixteenth of the pairs, within [2^14, 2^20] slots; a pair that finds no
  // slot stays with the pair-by-pair kernel
  long long hcap = 1 << 14;
  while (hcap < n_m2l / 16 && hcap < (1LL << 20)) hcap <<= 1;
  g.hk.ensure(hcap);
  g.hid.ensure(hcap);
  g.pair_slot.ensure(n_m2l);
  g.cnt.ensure(4);
  EXA_CUDA(cudaMemsetAsync(g.hk.p, 0xff, hcap * sizeof(unsigned long long), st));
  EXA_CUDA(cudaMemsetAsync(g.hid.p, 0xff, hcap * sizeof(int), st));
  EXA_CUDA(cudaMemsetAsync(g.cnt.p, 0, 4 * sizeof(int), st));
  k_pair_class<<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, a.cell_x, a.cell_pl, min_level,
                                            std::min(max_dl, 15), g.hk.p, hcap - 1, g.pair_slot.p);
  EXA_CHECK_LAUNCH();
  const int ccap = (int)std::min<long long>(hcap, (1LL << kClsBits) - 1);
  g.ck.ensure(ccap);
  g.ck_alt.ensure(ccap);
  g.cs.ensure(ccap);
  g.cs_alt.ensure(ccap);
  k_class_compact<<<kNumSMs * 4, 256, 0, st>>>(g.hk.p, hcap, g.ck.p, g.cs.p, g.cnt.p, ccap);
  EXA_CHECK_LAUNCH();
  int *ncls_h = reinterpret_cast<int *>(C.pin + kPinScratch);  // the context's pinned staging
  EXA_CUDA(cudaMemcpyAsync(ncls_h, g.cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st));
  EXA_CUDA(cudaStreamSynchronize(st));
  int ncls = *ncls_h;
  if (ncls <= 0) return false;
  if (!g.force && n_m2l < kMinPairsPerClass * (long long)ncls) return false;  // too many classes for their pairs
  if (ncls > ccap) ncls = ccap;  // the overflow classes' pairs stay per-pair
  bool alt = radix_sort_u64((uint64_t *)g.ck.p, g.cs.p, (uint64_t *)g.ck_alt.p, g.cs_alt.p, ncls, 0, 64, C.sort,
                            C.err.p, st);
  unsigned long long *ck = alt ? g.ck_alt.p : g.ck.p;
  int *cs = alt ? g.cs_alt.p : g.cs.p;
  k_class_ids<<<(ncls + 255) / 256, 256, 0, st>>>(cs, ncls, g.hid.p);
  EXA_CHECK_LAUNCH();
  const bool tc = g.tensor_cores;
  // P = 8 on the tensor cores: source pieces gathered by TMA (its tensor map made below).
  // At P = 10 (two 128-byte K-blocks, one CTA per SM either way) the cp.async
  // form is a little faster (M2L 16.4 vs 16.8 ms on a 1M-charge periodic box).
  CUtensorMap msb_map;
  bool use_tma = tc && NDP == 64 && g.tma && encode_tiled() != nullptr;
  if (tc) g.Kb.ensure((long long)ncls * 3 * (use_tma ? tma_kblocks(NDP) * NDP * 64 : NDP * NDP));
  else g.K.ensure((long long)ncls * NDP * NDP);
  {
    const size_t smem = tri(2 * P - 1) * sizeof(double2);
    float *Kt = tc ? nullptr : g.K.p;
    unsigned short *Kb = tc ? g.Kb.p : nullptr;
    auto build = [&](auto kernel) {
      kernel<<<ncls, 256, smem, st>>>(t, ck, P, Kt, Kb, nullptr, a.cell_x, a.cycle, nullptr);
      EXA_CHECK_LAUNCH();
    };
    switch (NDP) {
#define EXA_BUILD_K_CASE(N)                                      \
  case N:                                                        \
    if (!tc) build(k_build_K<N, kKFp32>);                   \
    else if (use_tma) build(k_build_K<N, kKSwizzled>);           \
    else build(k_build_K<N, kKCore>);                            \
    break;
      EXA_BUILD_K_CASE(16)
      EXA_BUILD_K_CASE(48)
      EXA_BUILD_K_CASE(64)
      EXA_BUILD_K_CASE(112)
#undef EXA_BUILD_K_CASE
      default: return false;
    }
  }
  if (tc) g.Msb.ensure(nc * 3 * NDP);
  else g.Msr.ensure(nc * NDP);
  if (use_tma && !msb_tensor_map(&msb_map, g.Msb.p, nc, NDP))
    throw std::runtime_error("TMA tensor map of the multipoles");
  k_scale_M_real<<<kNumSMs * 8, 256, 0, st>>>(t, a.M64, a.cell_x, nc, P, tc ? nullptr : g.Msr.p,
                                              tc ? g.Msb.p : nullptr, nullptr);
  EXA_CHECK_LAUNCH();
  // ---- pairs of classes with an operator, sorted by class
  g.taken.ensure(n_m2l);
  g.left_cnt.ensure(nc);
  g.left_off.ensure(nc + 1);
  g.left_src.ensure(n_m2l);
  g.skey.ensure(n_m2l);
  g.skey_alt.ensure(n_m2l);
  g.pval.ensure(n_m2l);
  g.pval_alt.ensure(n_m2l);
  k_gemm_flags<<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, g.pair_slot.p, g.hid.p, a.cell_pl, min_level,
                                            max_dl, g.taken.p, g.left_cnt.p, g.skey.p, g.pval.p);
  EXA_CHECK_LAUNCH();
  LeftScan ls{g.left_cnt.p, g.left_off.p, nc};
  launch_scan<1024, 8>(ls, nullptr, nc, nc, C.scan, C.err.p, st);
  k_left_fill<<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, g.taken.p, a.cell_pl, min_level, max_dl,
                                           g.left_off.p, g.left_src.p);
  EXA_CHECK_LAUNCH();
  const int end_bit = std::min(32, bits_for(ncls + 1));  // class ids; the untaken key 0xffffffff sorts last
  alt = radix_sort_u32(g.skey.p, g.pval.p, g.skey_alt.p, g.pval_alt.p, n_m2l, 0, end_bit, C.sort, C.err.p, st);
  const unsigned *sk = alt ? g.skey_alt.p : g.skey.p;
  const int *sv = alt ? g.pval_alt.p : g.pval.p;
  g.cstart.ensure(ncls + 1);
  g.cbase.ensure(ncls + 1);
  k_class_ranges<<<(ncls + 256) / 256, 256, 0, st>>>(sk, n_m2l, ncls, g.cstart.p);
  EXA_CHECK_LAUNCH();
  ChunkScan cs2{g.cstart.p, g.cbase.p, ncls};
  launch_scan<1024, 8>(cs2, nullptr, ncls, ncls, C.scan, C.err.p, st);
  const long long chunks_max = n_m2l / kChunk + ncls + 1;
  if (tc) {
    g.chunks.ensure(chunks_max);
    g.ssrc.ensure(n_m2l);
    k_chunk_table<<<(ncls + 255) / 256, 256, 0, st>>>(g.cstart.p, g.cbase.p, ncls, g.chunks.p);
    EXA_CHECK_LAUNCH();
    const int grid = (int)std::min<long long>(kNumSMs * 8, (n_m2l + 255) / 256);
    k_sorted_sources<<<grid, 256, 0, st>>>(sv, a.m2l_src, g.cstart.p + ncls, g.ssrc.p);
    EXA_CHECK_LAUNCH();
  }
  // ---- products per class chunk, then per-target sums
  g.Y.ensure(n_m2l * NDP);
  switch (NDP) {
#define EXA_GEMM_CASE(N)                                                                                      \
  case N: {                                                                                                   \
    if (use_tma) {                                                                                            \
      tma_launch<N>(msb_map, g, sv, chunks_max, ncls, C.err.p, st);                                           \
    } else if (tc) {                                                                                          \
      const size_t smem = mma_smem_bytes(N);                                                                  \
      set_smem(k_m2l_class_mma<N>, smem);                                                                     \
      const long long grid = std::min<long long>(chunks_max, (long long)kNumSMs * mma_ctas_per_sm(N));        \
      k_m2l_class_mma<N><<<(unsigned)grid, 128, smem, st>>>(g.chunks.p, g.cbase.p + ncls, sv, g.ssrc.p,       \
                                                            g.Kb.p, g.Msb.p, g.Y.p, C.err.p);                 \
    } else {                                                                                                  \
      const size_t smem = (size_t)(N * N + kChunk * (N + 4)) * sizeof(float);                                 \
      set_smem(k_m2l_class_gemm<N>, smem);                                                                    \
      k_m2l_class_gemm<N><<<(unsigned)chunks_max, 128, smem, st>>>(sk, sv, g.cstart.p, g.cbase.p, ncls,      \
                                                                   a.m2l_src, g.K.p, g.Msr.p, g.Y.p);         \
    }                                                                                                         \
    EXA_CHECK_LAUNCH();                                                                                       \
    k_m2l_class_reduce<N, float><<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, 0, nc, g.taken.p, g.Y.p, a.cell_x, t, P,  \
                                                              a.L64);                                         \
    EXA_CHECK_LAUNCH();                                                                                       \
    break;                                                                                                    \
  }
    EXA_GEMM_CASE(16)
    EXA_GEMM_CASE(48)
    EXA_GEMM_CASE(64)
    EXA_GEMM_CASE(112)
#undef EXA_GEMM_CASE
    default: return false;
  }
  return true;
}

// The plain method takes the products from this many pairs (0: never), by the
// pair count of a solve's or a forest's system alone, and every system goes by
// itself: a pair's contribution does not depend on the pairs beside it, nor on
// how the targets are cut into slabs, so a system's results are the same bits
// alone and in a forest.  M2L phase, pair by pair against products: 3.25 and
// 2.18 ms for 0.6M pairs at P = 10 (100K-body cube), 2.82 and 1.25 for 1.5M at
// P = 8 (200K-body cube), 2.16 and 1.87 for 3.3M at P = 6 (300K-body Plummer
// sphere); below the lines the products still won where classes were large (1.67
// and 0.80 ms for 0.3M at P = 10, 0.99 and 0.57 for 0.3M at P = 8, 0.97 and 0.86
// for 1.5M at P = 6), but the 0.5 ms of class work weighs more there.
long long m2l_gemm64_pairs(int P) { return P == 6 ? 3000000 : P == 8 ? 1000000 : P == 10 ? 400000 : 0; }

// And only where the classes, each of which costs an operator, save at least
// this many pairs' places in the pair-by-pair kernel's steps on average.
// Products against pair by pair over 62 systems of cubes, spheres, Plummer
// spheres and clumps of very different widths (30K to 1.5M bodies, theta 0.3 to
// 0.5): at P = 8 and 10 they lose at 33 (Plummer sphere, 31 pairs a class: 3.81
// against 2.97 and 10.3 against 7.13 ms), break even at 32 to 36 with half the
// pairs off the lattice and win from 41 on (clumps: 3.81 against 5.23 and 9.72
// against 13.0 ms); at P = 6 they lose at 175 (7.07 against 5.19) and win at 430
// (8.08 against 9.23).
int m2l_gemm64_places(int P) { return P == 6 ? 320 : 40; }

namespace {

// One system's pairs (targets [c0, c1), pairs [b, e)) through the class
// products.  Returns the pairs taken (0: none, and nothing was added).
long long m2l_gemm64_system(Context &C, const FmmArgs &a, M2LGemmBufs &g, int4 sys) {
  const int P = a.P, NDP = ndp_of(P), c0 = sys.x, c1 = sys.y, qb0 = sys.z;
  const long long np = (long long)sys.w - qb0;
  cudaStream_t st = a.stream;
  const DevTables &t = device_tables(P);
  // ---- classes
  const int limit = (int)(np / 16);  // no more classes than that pay in any case
  long long hcap = 1 << 14;
  while (hcap < 8LL * limit) hcap <<= 1;
  g.hk.ensure(hcap);
  g.hid.ensure(hcap);
  g.pair_slot.ensure(np);
  EXA_CUDA(cudaMemsetAsync(g.hk.p, 0xff, hcap * sizeof(unsigned long long), st));
  EXA_CUDA(cudaMemsetAsync(g.cnt.p, 0, 5 * sizeof(int), st));
  k_pair_class64<<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, a.m2l_src, c0, c1, qb0, a.cell_x, a.cell_pl, g.hk.p, hcap - 1,
                                              limit, g.pair_slot.p, g.cnt.p);
  EXA_CHECK_LAUNCH();
  // ---- slabs of whole targets, whose contributions fit the buffer
  long long rows = std::min(np, std::max<long long>(np / kMaxSlabs + 1, C.prm.m2l_work / 2 / (8LL * NDP)));
  int *cnt = reinterpret_cast<int *>(C.pin + kPinScratch);
  std::vector<int2> cut{make_int2(c0, qb0), make_int2(c1, sys.w)};
  auto read_counts = [&] {
    int2 *slab = reinterpret_cast<int2 *>(C.pin + kPinScratch) + 2;
    if (rows < np) {
      g.slabs.ensure(2 * kMaxSlabs + 2);
      k_slabs<<<1, 32, 0, st>>>(a.m2l_off, c0, c1, rows, g.slabs.p, g.cnt.p + 3);
      EXA_CHECK_LAUNCH();
      EXA_CUDA(cudaMemcpyAsync(slab, g.slabs.p, (2 * kMaxSlabs + 2) * sizeof(int2), cudaMemcpyDeviceToHost, st));
    }
    EXA_CUDA(cudaMemcpyAsync(cnt, g.cnt.p, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
    EXA_CUDA(cudaStreamSynchronize(st));
    if (rows < np) cut.assign(slab, slab + cnt[3] + 1);
  };
  read_counts();
  const int ncls = cnt[0];
  const long long taken = cnt[1];
  if (ncls <= 0 || ncls > limit || (long long)ncls * m2l_gemm64_places(P) > 32LL * cnt[2]) return 0;
  bool shorter = false;  // smaller slabs where memory is short
  while (!try_ensure(g.Y64, rows * NDP)) {
    if (rows <= np / kMaxSlabs + 1) throw std::runtime_error("no device memory for the M2L contributions");
    rows = std::max(rows / 2, np / kMaxSlabs + 1);
    shorter = true;
  }
  if (shorter) read_counts();
  const int nslab = (int)cut.size() - 1;
  long long most = 0;
  for (int i = 0; i < nslab; i++) most = std::max<long long>(most, cut[i + 1].y - cut[i].y);
  g.Y64.ensure(most * NDP);  // a target with more pairs than that is a slab of its own
  g.ck.ensure(ncls);
  k_class_ids64<<<kNumSMs * 4, 256, 0, st>>>(g.hk.p, hcap, g.ck.p, g.hid.p, g.cnt.p + 4);
  EXA_CHECK_LAUNCH();
  // ---- operators and multipoles
  const size_t smem_k = tri(2 * P - 1) * sizeof(double2);
  auto build = [&](int k0, int k1, const int *cstart) {
    auto launch = [&](auto kernel) {
      kernel<<<k1 - k0, 256, smem_k, st>>>(t, g.ck.p + k0, P, nullptr, nullptr, g.K64.p, a.cell_x, a.cycle, cstart);
      EXA_CHECK_LAUNCH();
    };
    if (NDP == 48) launch(k_build_K<48, kKFp64>);
    else if (NDP == 64) launch(k_build_K<64, kKFp64>);
    else launch(k_build_K<112, kKFp64>);
  };
  // all of them once where they fit their share of the workspace; else a batch
  // at a time, for each slab the ones it has pairs of
  const long long op = (long long)NDP * NDP;
  long long kcap = std::min<long long>(ncls, std::max<long long>(64, C.prm.m2l_work / 2 / (8 * op)));
  while (!try_ensure(g.K64, kcap * op)) {
    if (kcap <= 64) throw std::runtime_error("no device memory for the M2L operators");
    kcap = std::max<long long>(kcap / 2, 64);
  }
  if (kcap >= ncls) build(0, ncls, nullptr);
  g.Ms64r.ensure(a.ncells * NDP);
  k_scale_M_real<<<kNumSMs * 8, 256, 0, st>>>(t, a.M64 + (long long)c0 * t.nterm, a.cell_x + c0, c1 - c0, P, nullptr,
                                              nullptr, g.Ms64r.p + (long long)c0 * NDP);
  EXA_CHECK_LAUNCH();
  // ---- per slab: pairs sorted by class, products per class chunk, per-target sums
  const int end_bit = std::min(32, bits_for(ncls + 1));
  g.skey.ensure(most);
  g.skey_alt.ensure(most);
  g.pval.ensure(most);
  g.pval_alt.ensure(most);
  g.ssrc.ensure(most);
  g.cstart.ensure(ncls + 1);
  g.cbase.ensure(ncls + 1);
  g.chunks.ensure(most / kChunk + ncls + 1);
  for (int i = 0; i < nslab; i++) {
    const int qb = cut[i].y;
    const long long n = cut[i + 1].y - qb;
    if (n <= 0) continue;
    const int grid = (int)std::min<long long>(kNumSMs * 8, (n + 255) / 256);
    k_gemm_flags64<<<grid, 256, 0, st>>>(g.pair_slot.p + (qb - qb0), g.hid.p, n, g.taken.p + qb, g.skey.p, g.pval.p);
    EXA_CHECK_LAUNCH();
    const bool alt = radix_sort_u32(g.skey.p, g.pval.p, g.skey_alt.p, g.pval_alt.p, n, 0, end_bit, C.sort, C.err.p, st);
    const unsigned *sk = alt ? g.skey_alt.p : g.skey.p;
    const int *sv = alt ? g.pval_alt.p : g.pval.p;
    k_class_ranges<<<(ncls + 256) / 256, 256, 0, st>>>(sk, n, ncls, g.cstart.p);
    EXA_CHECK_LAUNCH();
    ChunkScan scan{g.cstart.p, g.cbase.p, ncls};
    launch_scan<1024, 8>(scan, nullptr, ncls, ncls, C.scan, C.err.p, st);
    k_chunk_table<<<(ncls + 255) / 256, 256, 0, st>>>(g.cstart.p, g.cbase.p, ncls, g.chunks.p);
    EXA_CHECK_LAUNCH();
    k_sorted_sources<<<grid, 256, 0, st>>>(sv, a.m2l_src + qb, g.cstart.p + ncls, g.ssrc.p);
    EXA_CHECK_LAUNCH();
    const long long chunks_max = n / kChunk + ncls + 1;
    auto products = [&](int k0, int k1) {
      if (NDP == 48) gemm64_launch<48>(g, k0, k1, sv, chunks_max, nd_of(P), st);
      else if (NDP == 64) gemm64_launch<64>(g, k0, k1, sv, chunks_max, nd_of(P), st);
      else gemm64_launch<112>(g, k0, k1, sv, chunks_max, nd_of(P), st);
    };
    if (kcap >= ncls) {
      products(0, ncls);
    } else {
      for (int k0 = 0; k0 < ncls; k0 += (int)kcap) {
        const int k1 = (int)std::min<long long>(ncls, k0 + kcap);
        build(k0, k1, g.cstart.p + k0);
        products(k0, k1);
      }
    }
    auto reduce = [&](auto kernel) {
      // Y64's first row is pair qb
      kernel<<<kNumSMs * 8, 256, 0, st>>>(a.m2l_off, cut[i].x, cut[i + 1].x, g.taken.p,
                                          g.Y64.p - (long long)qb * NDP, a.cell_x, t, P, a.L64);
      EXA_CHECK_LAUNCH();
    };
    if (NDP == 48) reduce(k_m2l_class_reduce<48, double>);
    else if (NDP == 64) reduce(k_m2l_class_reduce<64, double>);
    else reduce(k_m2l_class_reduce<112, double>);
  }
  return taken;
}

}  // namespace

long long m2l_gemm64_bytes(int P, long long pairs) {
  const long long least = m2l_gemm64_pairs(P), NDP = ndp_of(P);
  if (least <= 0 || pairs < least) return 0;
  const long long rows = std::min(pairs, kM2LWork / 2 / (8 * NDP));
  // a slab's contributions and sort; the operators; per pair the class table (at
  // most 12), its slot, the taken flag and the list of pairs left
  return rows * (8 * NDP + 24) + std::min(pairs / 16 * NDP * NDP * 8, kM2LWork / 2) + 21 * pairs;
}

long long m2l_gemm64(Context &C, const FmmArgs &a, M2LGemmBufs &g, long long n_m2l) {
  const long long least = m2l_gemm64_pairs(a.P), nc = a.ncells;
  if (least <= 0 || n_m2l < least || nc <= 0) return n_m2l;
  cudaStream_t st = a.stream;
  g.cnt.ensure(5);
  std::vector<int4> systems;
  if (!a.nsys) {
    systems.push_back(make_int4(0, (int)nc, 0, (int)n_m2l));
  } else {
    const int cap = (int)std::min<long long>(a.nsys, n_m2l / least);
    g.ranges.ensure(cap);
    EXA_CUDA(cudaMemsetAsync(g.cnt.p, 0, sizeof(int), st));
    k_sys_ranges<<<std::min(kNumSMs, div_up(a.nsys, 128)), 128, 0, st>>>(a.m2l_off, C.tree.sys_cell.p, a.nsys,
                                                                         (int)least, g.ranges.p, g.cnt.p);
    EXA_CHECK_LAUNCH();
    int *n = reinterpret_cast<int *>(C.pin + kPinScratch);
    EXA_CUDA(cudaMemcpyAsync(n, g.cnt.p, sizeof(int), cudaMemcpyDeviceToHost, st));
    EXA_CUDA(cudaStreamSynchronize(st));
    systems.resize(*n);
    if (*n > 0) {
      EXA_CUDA(cudaMemcpyAsync(systems.data(), g.ranges.p, *n * sizeof(int4), cudaMemcpyDeviceToHost, st));
      EXA_CUDA(cudaStreamSynchronize(st));
    }
  }
  if (systems.empty()) return n_m2l;
  g.taken.ensure(n_m2l);
  EXA_CUDA(cudaMemsetAsync(g.taken.p, 0, n_m2l, st));
  long long left = n_m2l;
  for (const int4 &sys : systems) left -= m2l_gemm64_system(C, a, g, sys);
  if (left == 0 || left == n_m2l) return left;
  g.left_cnt.ensure(nc);
  g.left_off.ensure(nc + 1);
  g.left_src.ensure(left);
  const int grid = (int)std::min<long long>(kNumSMs * 8, (nc + 7) / 8);
  k_left_count<<<grid, 256, 0, st>>>(a.m2l_off, nc, g.taken.p, g.left_cnt.p);
  EXA_CHECK_LAUNCH();
  LeftScan ls{g.left_cnt.p, g.left_off.p, nc};
  launch_scan<1024, 8>(ls, nullptr, nc, nc, C.scan, C.err.p, st);
  k_left_fill<<<grid, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, g.taken.p, a.cell_pl, 0, kMaxLevels, g.left_off.p,
                                    g.left_src.p);
  EXA_CHECK_LAUNCH();
  return left;
}
long long m2l_complement(Context &C, const FmmArgs &a, M2LGemmBufs &g, long long n_m2l, int min_level, int max_dl) {
  const long long nc = a.ncells;
  cudaStream_t st = a.stream;
  g.comp_cnt.ensure(nc);
  g.comp_off.ensure(nc + 1);
  g.comp_src.ensure(n_m2l > 0 ? n_m2l : 1);
  const int grid = (int)std::max<long long>(1, std::min<long long>(kNumSMs * 8, (nc + 7) / 8));
  k_complement_count<<<grid, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, a.cell_pl, min_level, max_dl, g.comp_cnt.p);
  EXA_CHECK_LAUNCH();
  LeftScan ls{g.comp_cnt.p, g.comp_off.p, nc};
  launch_scan<1024, 8>(ls, nullptr, nc, nc, C.scan, C.err.p, st);
  k_complement_fill<<<grid, 256, 0, st>>>(a.m2l_off, a.m2l_src, nc, a.cell_pl, min_level, max_dl, g.comp_off.p,
                                          g.comp_src.p);
  EXA_CHECK_LAUNCH();
  return nc;
}

}  // namespace exafmm_b200
