// FP64 pair arithmetic shared by the P2P kernel and the direct sum.
#pragma once
#include "common.cuh"

namespace exafmm_b200 {

// N pairs (separations d and charges q, which are used up), pair i into the sums
// acc[i / PER]: the potential, and the three that are subtracted from the
// gradient.
//
// 1 / sqrt(r2): the hardware's reciprocal square root of the high word (about
// 20 bits) takes one third-order Householder step: with e = 1 - r2 y0^2,
//   1/sqrt(r2) = y0 (1 - e)^(-1/2) = y0 (1 + e/2 + 3/8 e^2 + O(5/16 e^3)),
// five FP64 operations.  Zero, subnormal, infinite and NaN arguments (one
// unsigned compare on the high word) are set apart; the arguments of one step
// are tested together, so that the special case is one branch a step and the N
// chains interleave.
//   * r2 = 0, every target's pair with itself: the charge is dropped, whatever
//     it is (kernels/laplace.h:171 gives such a pair no weight, and an infinite
//     or NaN charge times 0 would be NaN);
//   * the others, which hardly ever come, take the library function and put the
//     factors of 1/r into q and d: 1 / r^2 alone overflows for subnormal r2.
template <int N, int PER>
__device__ __forceinline__ void pairs64(double (&dx)[N], double (&dy)[N], double (&dz)[N], double (&q)[N],
                                        double (&acc)[N / PER][4]) {
  double r2[N], inv[N];
  bool special = false;
#pragma unroll
  for (int i = 0; i < N; i++) r2[i] = fma(dx[i], dx[i], fma(dy[i], dy[i], dz[i] * dz[i]));
  auto odd = [](double v) { return (unsigned)__double2hiint(v) - 0x00100000u >= 0x7fe00000u; };
#pragma unroll
  for (int i = 0; i < N; i++) {
    double y0;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(r2[i]));
    const double e = fma(-(r2[i] * y0), y0, 1.0);
    inv[i] = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    special |= odd(r2[i]);
  }
  if (special) {
    bool rare = false;
#pragma unroll
    for (int i = 0; i < N; i++) {
      if (!(__double2hiint(r2[i]) | __double2loint(r2[i]))) inv[i] = q[i] = 0.0;  // a sum of squares is never -0
      else rare |= odd(r2[i]);
    }
    if (rare) {
#pragma unroll 1
      for (int i = 0; i < N; i++) {
        double v = r2[0];
#pragma unroll
        for (int k = 1; k < N; k++)
          if (k == i) v = r2[k];
        if (!odd(v) || v == 0.0) continue;
        v = rsqrt(v);
#pragma unroll
        for (int k = 0; k < N; k++)
          if (k == i) {
            q[k] *= v;
            inv[k] = 1.0;
            dx[k] = dx[k] * v * v;
            dy[k] = dy[k] * v * v;
            dz[k] = dz[k] * v * v;
          }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < N; i++) {
    double(&a)[4] = acc[i / PER];
    const double qr = q[i] * inv[i];
    const double qr3 = qr * (inv[i] * inv[i]);
    a[0] += qr;
    a[1] = fma(dx[i], qr3, a[1]);
    a[2] = fma(dy[i], qr3, a[2]);
    a[3] = fma(dz[i], qr3, a[3]);
  }
}

}  // namespace exafmm_b200
