// Second and third derivatives of one AO, shared by the AO Hessian
// (ao_hessian.cu) and the adjoint (adjoint.cu).
#pragma once

#include <cuda_runtime.h>

namespace qb {

constexpr double kShiftD = 1.e-20;

// x^a and its first three derivatives (Leibniz, one factor x at a time)
template <typename F>
__device__ __forceinline__ void pow_derivs(F x, int a, F (&q)[4]) {
  if (a <= 3) {
    // without branches (lanes of a warp hold different exponents): with
    // f_i = x for i <= a, 1 otherwise, x^a = f1 f2 f3, and the derivatives
    // a x^(a-1), a (a-1) x^(a-2), a (a-1) (a-2) vanish where they must
    const F f1 = a >= 1 ? x : F(1), f2 = a >= 2 ? x : F(1), f3 = a >= 3 ? x : F(1);
    const F fa = F(a);
    q[2] = fa * (fa - F(1)) * f3;
    q[1] = fa * (f2 * f3);
    q[0] = f1 * (f2 * f3);
    q[3] = fa * (fa - F(1)) * (fa - F(2));
    return;
  }
  q[0] = F(1); q[1] = F(0); q[2] = F(0); q[3] = F(0);
  for (int i = 0; i < a; ++i) {
    q[3] = q[3] * x + F(3) * q[2];
    q[2] = q[2] * x + F(2) * q[1];
    q[1] = q[1] * x + q[0];
    q[0] = q[0] * x;
  }
}

// Hessian H[d][e] and gradient of the Laplacian T[d] of one AO (times its
// factor f), plus its gradient g[d], in arithmetic F.  The radial
// combinations that cancel near their zeros, lap R = 4 s R2 + 6 R1 and
// k3 = 20 R2 + 8 s R3, come in formed in FP64.
template <typename F>
__device__ __forceinline__ void ao_derivs(int code, F f, const F (&v)[3], const F (&R)[3], F lapR, F k3,
                                          F (&g)[3], F (&H)[3][3], F (&Tl)[3]) {
  const int ax = code & 15, by = (code >> 4) & 15, cz = (code >> 8) & 15, l = (code >> 12) & 15;
  F X[4], Y[4], Z[4];
  pow_derivs<F>(v[0], ax, X);
  pow_derivs<F>(v[1], by, Y);
  pow_derivs<F>(v[2], cz, Z);
  const F P = X[0] * Y[0] * Z[0] + (l >= 1 ? F(kShiftD) : F(0));
  const F Pd[3] = {X[1] * Y[0] * Z[0], X[0] * Y[1] * Z[0], X[0] * Y[0] * Z[1]};
  F Pdd[3][3];
  Pdd[0][0] = X[2] * Y[0] * Z[0];
  Pdd[1][1] = X[0] * Y[2] * Z[0];
  Pdd[2][2] = X[0] * Y[0] * Z[2];
  Pdd[0][1] = Pdd[1][0] = X[1] * Y[1] * Z[0];
  Pdd[0][2] = Pdd[2][0] = X[1] * Y[0] * Z[1];
  Pdd[1][2] = Pdd[2][1] = X[0] * Y[1] * Z[1];
  const F lapP = Pdd[0][0] + Pdd[1][1] + Pdd[2][2];
  const F dlapP[3] = {X[3] * Y[0] * Z[0] + X[1] * Y[2] * Z[0] + X[1] * Y[0] * Z[2],
                      X[2] * Y[1] * Z[0] + X[0] * Y[3] * Z[0] + X[0] * Y[1] * Z[2],
                      X[2] * Y[0] * Z[1] + X[0] * Y[2] * Z[1] + X[0] * Y[0] * Z[3]};
  const F Rd[3] = {F(2) * v[0] * R[1], F(2) * v[1] * R[1], F(2) * v[2] * R[1]};
  F Rdd[3][3];
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int e = 0; e < 3; ++e) Rdd[d][e] = F(4) * v[d] * v[e] * R[2] + (d == e ? F(2) * R[1] : F(0));
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    g[d] = f * (Pd[d] * R[0] + P * Rd[d]);
#pragma unroll
    for (int e = 0; e < 3; ++e) H[d][e] = f * (Pdd[d][e] * R[0] + Pd[d] * Rd[e] + Pd[e] * Rd[d] + P * Rdd[d][e]);
    F t = F(0);
#pragma unroll
    for (int e = 0; e < 3; ++e) t += Pdd[d][e] * Rd[e] + Pd[e] * Rdd[d][e];
    Tl[d] = f * (dlapP[d] * R[0] + lapP * Rd[d] + F(2) * t + Pd[d] * lapR + P * v[d] * k3);
  }
}

}  // namespace qb
