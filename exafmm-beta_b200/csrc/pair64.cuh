// FP64 pair arithmetic shared by the P2P kernel and the direct sum.
#pragma once
#include "common.cuh"

namespace exafmm_b200 {

// 1 / sqrt(r2); at r2 = 0 it is 0 and the charge q is dropped too, whatever it
// is (kernels/laplace.h:171 gives such a pair no weight).  The hardware's reciprocal square root of the high word (about 20
// bits) takes one third-order Householder step: with e = 1 - r2 y0^2,
//   1/sqrt(r2) = y0 (1 - e)^(-1/2) = y0 (1 + e/2 + 3/8 e^2 + O(5/16 e^3)),
// five FP64 operations, where rsqrt(double) costs about twice that and a
// branch.  Zero, subnormal, infinite and NaN arguments (one unsigned compare on
// the high word) take the library function, as every argument did before.
// The arguments of one step are tested together, so that the special case is
// one branch a step and the N chains interleave.
template <int N>
__device__ __forceinline__ void inv_dist(const double (&r2)[N], double (&q)[N], double (&inv)[N]) {
  bool special = false;
#pragma unroll
  for (int i = 0; i < N; i++) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(r2[i]));
    const double e = fma(-(r2[i] * y0), y0, 1.0);
    inv[i] = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    special |= (unsigned)__double2hiint(r2[i]) - 0x00100000u >= 0x7fe00000u;
  }
  if (special) {
#pragma unroll 1
    for (int i = 0; i < N; i++) {
      double v = r2[0];
#pragma unroll
      for (int k = 1; k < N; k++)
        if (k == i) v = r2[k];
      if ((unsigned)__double2hiint(v) - 0x00100000u < 0x7fe00000u) continue;
      const bool none = v == 0.0;
      v = none ? 0.0 : rsqrt(v);
#pragma unroll
      for (int k = 0; k < N; k++)
        if (k == i) {
          inv[k] = v;
          if (none) q[k] = 0.0;  // an infinite or NaN charge times 0 would be NaN
        }
    }
  }
}

// N pairs (separations d, charges q, which are used up), pair i into the sums
// acc[i / PER]: potential, and the three that are subtracted from the gradient.
template <int N, int PER>
__device__ __forceinline__ void pairs64(const double (&dx)[N], const double (&dy)[N], const double (&dz)[N],
                                        double (&q)[N], double (&acc)[N / PER][4]) {
  double r2[N], inv[N];
#pragma unroll
  for (int i = 0; i < N; i++) r2[i] = fma(dx[i], dx[i], fma(dy[i], dy[i], dz[i] * dz[i]));
  inv_dist(r2, q, inv);
#pragma unroll
  for (int i = 0; i < N; i++) {
    double(&a)[4] = acc[i / PER];
    const double qr = q[i] * inv[i];
    const double qr3 = qr * inv[i] * inv[i];  // in this order: a small charge very near does not overflow
    a[0] += qr;
    a[1] = fma(dx[i], qr3, a[1]);
    a[2] = fma(dy[i], qr3, a[2]);
    a[3] = fma(dz[i], qr3, a[3]);
  }
}

}  // namespace exafmm_b200
