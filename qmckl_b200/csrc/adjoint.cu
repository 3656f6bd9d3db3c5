// Derivative kernels of the AO VGL: the AO Hessian getter and the adjoint of
// MO VGL with respect to the nuclear and point coordinates.
//
// Quantities (derivatives with respect to the point coordinates r; an AO
// centred on nucleus A depends on r - R_A, so d/dR_A = -d/dr):
//   radial part  R(s) = sum_j c_j exp(-a_j s), s = r^2, and its s-derivatives
//                R1 = -sum a c e, R2 = sum a^2 c e, R3 = -sum a^3 c e
//                d_d R = 2 x_d R1,  d_d d_e R = 4 x_d x_e R2 + 2 delta_de R1,
//                lap R = 4 s R2 + 6 R1,  d_d lap R = x_d (20 R2 + 8 s R3)
//   monomial     P = x^a y^b z^c with all derivatives up to third order
//   AO           chi = f P R;  H_de = d_d d_e chi;  T_d = d_d lap chi
// The reference forms the same quantities from the shell Hessian
// (qmckl_compute_ao_basis_shell_gaussian_hessian, org/qmckl_ao.org:5480-5580),
// the polynomial Hessian (qmckl_compute_ao_polynomial_hessian_doc, 7113-7236)
// and the AO Hessian (qmckl_compute_ao_hessian_doc, 9590-9720); its orbital
// forces (org/qmckl_forces.org:5688-6772) contract them with the MO
// coefficients.  Screening follows the forward kernels: nucleus skipped when
// r^2 > cutoff * range, primitives sorted by exponent with a break at
// a r^2 > cutoff, AO skipped when its contracted radial value is zero.
//
// Work decomposition: one warp per (point, nucleus block), as in the forward
// AO kernel: lanes stage the block's displacements and radial derivative sets
// in shared memory, then sweep the block's contiguous AO range.
//   MODE_HESSIAN  writes ao_hessian[3][point][4][ao] (coalesced rows).
//   MODE_ADJOINT  (mixed form) reads G[point][5][ao] = (W . C)[point][comp][ao], the loss
//                 weights pulled back through the MO coefficients, and forms
//                 q_d = G0 d_d chi + sum_e G_{1+e} H_ed + G4 T_d per AO.  A
//                 segmented warp reduction over the (contiguous) AOs of each
//                 nucleus feeds per-CTA shared accumulators of dL/dR (one
//                 device atomic per nucleus and CTA at the end); the sum over
//                 all AOs gives dL/dr of the point.
// The FP64 adjoint works on compact tiles instead (tile_deriv_kernel).
#include <algorithm>
#include <type_traits>

#include "kernels.cuh"

namespace qb {
namespace {

constexpr int kWarpsD = 8;
constexpr double kShiftD = 1.e-20;
constexpr int MODE_HESSIAN = 0, MODE_ADJOINT = 1;

struct DerivSmem {
  double rad[kBlockSlots][4];   // R, R1, R2, R3 of the block's shells
  double nuc[kBlockNuc][4];     // displacement, r^2 (negative when screened out)
  uint8_t act[kBlockSlots];     // the shells whose nucleus is in range
};

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

template <bool MIXED>
__device__ __forceinline__ void stage_deriv(const DevTables& T, DerivSmem& sm, const int4 blk, const int2 slots,
                                            double px, double py, double pz, double cutoff, int lane) {
  const int nn = blk.y - blk.x;
  if (lane < nn) {
    const int n = blk.x + lane;
    const int N = T.nucl_num;
    const double x = px - T.nucl_coord[n];
    const double y = py - T.nucl_coord[n + N];
    const double z = pz - T.nucl_coord[n + 2 * N];
    const double r2 = x * x + y * y + z * z;
    const bool in = !(r2 > cutoff * T.nucleus_range[n]);
    sm.nuc[lane][0] = x;
    sm.nuc[lane][1] = y;
    sm.nuc[lane][2] = z;
    sm.nuc[lane][3] = in ? r2 : -1.0;
  }
  __syncwarp();
  // shells of screened-out nuclei are not staged (the AO loop tests the nucleus first)
  const int nlive = pack_live_slots(T.slot_nuc, blk.x, slots, sm.nuc, sm.act, lane);
  for (int i = lane; i < nlive; i += 32) {
    const int ls = sm.act[i];
    const int s = slots.x + ls;
    const int nucl = T.slot_nuc[s];
    const double r2 = sm.nuc[nucl - blk.x][3];
    double acc[4] = {0., 0., 0., 0.};
    {
      const int2 cr = T.slot_coef[s];
      const int p0 = T.nuc_prim_start[nucl];
      for (int j = cr.x; j < cr.y; ++j) {
        const double a = T.expo[p0 + T.coef_prim[j]];
        const double ar2 = a * r2;
        if (ar2 > cutoff) break;   // primitives sorted by exponent
        const double e = (MIXED && ar2 <= 30.0) ? (double)expf(-(float)ar2) : exp(-ar2);
        const double ce = T.coef_val[j] * e;
        acc[0] += ce;
        acc[1] -= a * ce;
        acc[2] += a * a * ce;
        acc[3] -= a * a * a * ce;
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) sm.rad[ls][c] = acc[c];
  }
  __syncwarp();
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

// MODE_HESSIAN: out = ao_hessian[3][point_num][4][ao] (point_num points from
//   coord [3][cstride], cstride >= point_num).
// MODE_ADJOINT: G = [point_num][5][ao]; grad_nucl [nucl][3] -= sum q (per-CTA
//   shared accumulators when use_smem, else device atomics); grad_coord
//   ([3][gstride], may be null) += sum q.
// MIXED: FP32 exponentials where a r^2 <= 30; in MODE_ADJOINT also G in FP32
//   and the per-AO derivative arithmetic in FP32 (displacements, r^2, radial
//   sums and the cancelling radial combinations in FP64; q summed in FP64).
template <int MODE, bool MIXED>
__global__ void __launch_bounds__(kWarpsD * 32)
deriv_kernel(const DevTables T, const int64_t point_num, const double* __restrict__ coord, const int64_t cstride,
             const double cutoff, double* __restrict__ out, const void* __restrict__ Gv,
             double* __restrict__ grad_nucl, double* __restrict__ grad_coord, const int64_t gstride,
             const bool use_smem, const double* __restrict__ cusp_r) {
  using F = typename std::conditional<MIXED && MODE == MODE_ADJOINT, float, double>::type;
  const F* __restrict__ G = (const F*)Gv;
  __shared__ DerivSmem smem[kWarpsD];
  extern __shared__ double sacc[];   // [nucl][3] (MODE_ADJOINT with use_smem)
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  DerivSmem& sm = smem[warp];
  const int64_t A = T.ao_num;
  if (MODE == MODE_ADJOINT && use_smem) {
    for (int i = threadIdx.x; i < 3 * T.nucl_num; i += blockDim.x) sacc[i] = 0.0;
    __syncthreads();
  }
  const int64_t stride = (int64_t)gridDim.x * kWarpsD;
  // one warp per point, through its nucleus blocks (as the FP64 AO kernel)
  for (int64_t p = (int64_t)blockIdx.x * kWarpsD + warp; p < point_num; p += stride) {
   double pg[3] = {0., 0., 0.};
   for (int b = 0; b < T.nblock; ++b) {
    const int4 blk = T.block[b];
    const int2 slots = T.block_slots[b];
    stage_deriv<MIXED>(T, sm, blk, slots, coord[p], coord[p + cstride], coord[p + 2 * cstride], cutoff, lane);
    for (int k0 = blk.z; k0 < blk.w; k0 += 32) {
      const int k = k0 + lane;
      const bool valid = k < blk.w;
      int nl = kBlockNuc;   // past-the-end lanes form their own (last) segment
      F g[3] = {F(0), F(0), F(0)}, H[3][3] = {{F(0), F(0), F(0)}, {F(0), F(0), F(0)}, {F(0), F(0), F(0)}},
        Tl[3] = {F(0), F(0), F(0)};
      if (valid) {
        const int code = T.ao_code[k];
        const int slot = (code >> 16) & 255;
        nl = (code >> 24) & 31;
        const double r2 = sm.nuc[nl][3];
        const double* Rs = sm.rad[slot];
        if (r2 >= 0.0 && Rs[0] != 0.0 && !cusp_masked(cusp_r, (code >> 12) & 15, blk.x + nl, r2, false)) {
          const double lapR = 4.0 * r2 * Rs[2] + 6.0 * Rs[1];
          const double k3 = 20.0 * Rs[2] + 8.0 * r2 * Rs[3];
          const F v[3] = {(F)sm.nuc[nl][0], (F)sm.nuc[nl][1], (F)sm.nuc[nl][2]};
          const F R[3] = {(F)Rs[0], (F)Rs[1], (F)Rs[2]};
          ao_derivs<F>(code, (F)T.ao_factor[k], v, R, (F)lapR, (F)k3, g, H, Tl);
        }
      }
      if (MODE == MODE_HESSIAN) {
        if (valid) {
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            double* o = out + ((int64_t)i * point_num + p) * 4 * A;
            o[k] = H[i][0];
            o[A + k] = H[i][1];
            o[2 * A + k] = H[i][2];
            o[3 * A + k] = Tl[i];
          }
        }
      } else {
        double q[3] = {0., 0., 0.};
        if (valid) {
          const F* gr = G + p * 5 * A + k;
          const F G0 = gr[0], G1 = gr[A], G2 = gr[2 * A], G3 = gr[3 * A], G4 = gr[4 * A];
#pragma unroll
          for (int d = 0; d < 3; ++d)
            q[d] = (double)(G0 * g[d] + G1 * H[0][d] + G2 * H[1][d] + G3 * H[2][d] + G4 * Tl[d]);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) pg[d] += q[d];
        // segmented sum over lanes of the same nucleus (AOs of a nucleus are
        // contiguous, so segments are runs of lanes): the first lane of each
        // run ends up with the run's sum
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
          const int ko = __shfl_down_sync(0xffffffffu, nl, off);
          double o[3];
#pragma unroll
          for (int d = 0; d < 3; ++d) o[d] = __shfl_down_sync(0xffffffffu, q[d], off);
          if (lane + off < 32 && ko == nl) {
#pragma unroll
            for (int d = 0; d < 3; ++d) q[d] += o[d];
          }
        }
        const int kprev = __shfl_up_sync(0xffffffffu, nl, 1);
        if ((lane == 0 || kprev != nl) && nl < kBlockNuc) {
          const int n = blk.x + nl;
#pragma unroll
          for (int d = 0; d < 3; ++d) {
            if (use_smem) atomicAdd(&sacc[n * 3 + d], q[d]);
            else if (grad_nucl != nullptr) atomicAdd(&grad_nucl[n * 3 + d], -q[d]);
          }
        }
      }
    }
    __syncwarp();
   }
    if (MODE == MODE_ADJOINT && grad_coord != nullptr) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double s = pg[d];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
        pg[d] = s;
      }
      if (lane == 0) {
#pragma unroll
        for (int d = 0; d < 3; ++d) atomicAdd(&grad_coord[p + d * gstride], pg[d]);
      }
    }
    __syncwarp();
  }
  if (MODE == MODE_ADJOINT && use_smem && grad_nucl != nullptr) {
    __syncthreads();
    for (int i = threadIdx.x; i < 3 * T.nucl_num; i += blockDim.x)
      if (sacc[i] != 0.0) atomicAdd(&grad_nucl[i], -sacc[i]);
  }
}

template <int MODE>
cudaError_t launch_deriv(const DevTables& T, int64_t point_num, const double* coord, int64_t cstride, double cutoff,
                         bool mixed, double* out, const void* G, double* grad_nucl, double* grad_coord,
                         int64_t gstride, cudaStream_t s, const double* cusp_r = nullptr) {
  if (point_num <= 0) return cudaSuccess;
  const int grid = (int)std::min<int64_t>((point_num + kWarpsD - 1) / kWarpsD, 148 * 8);   // warps = points
  size_t dyn = 0;
  bool use_smem = false;
  if (MODE == MODE_ADJOINT) {
    dyn = sizeof(double) * 3 * (size_t)T.nucl_num;
    use_smem = dyn <= 64 * 1024;
    if (!use_smem) dyn = 0;
  }
  cudaError_t e = cudaSuccess;
  if (mixed || MODE == MODE_ADJOINT) {   // the FP64 adjoint: tile_deriv_kernel
    auto k = deriv_kernel<MODE, true>;
    if (dyn > 48 * 1024) e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn);
    if (e != cudaSuccess) return e;
    k<<<grid, kWarpsD * 32, dyn, s>>>(T, point_num, coord, cstride, cutoff, out, G, grad_nucl, grad_coord, gstride,
                                      use_smem, cusp_r);
  } else if constexpr (MODE == MODE_HESSIAN) {
    auto k = deriv_kernel<MODE, false>;
    k<<<grid, kWarpsD * 32, dyn, s>>>(T, point_num, coord, cstride, cutoff, out, G, grad_nucl, grad_coord, gstride,
                                      use_smem, cusp_r);
  }
  count_launch();
  return cudaGetLastError();
}

// One AO of the FP64 adjoint, exponents known at compile time: with the
// pulled-back weights (G0, g = G1..G3, G4) and P's derivatives,
//   q = R (G0 dP + HP g + G4 d lap P) + dP (g . dR + G4 lap R)
//       + dR (G0 P + g . dP + G4 lap P) + HR y + P v G4 k3
//       + 2 G4 HP dR,   y = P g + 2 G4 dP,  HR = 4 R2 v v^T + 2 R1 1,
// the terms of ao_derivs contracted before they are formed (70 instead of
// 200 operations per AO).
struct ShellRad {
  double v[3], R0, R1, R2, lapR, k3, Rd[3];
};
template <int a, int b, int c>
__device__ __forceinline__ void adj_ao(const ShellRad& S, const double (&xp)[4], const double (&yp)[4],
                                       const double (&zp)[4], double G0, double G1, double G2, double G3, double G4,
                                       double (&q)[3]) {
  // X[i] = i-th derivative of x^a, present when a >= i
  const double X0 = xp[a], Y0 = yp[b], Z0 = zp[c];
  const double X1 = a >= 1 ? (double)a * xp[a >= 1 ? a - 1 : 0] : 0.0, Y1 = b >= 1 ? (double)b * yp[b >= 1 ? b - 1 : 0] : 0.0,
               Z1 = c >= 1 ? (double)c * zp[c >= 1 ? c - 1 : 0] : 0.0;
  const double X2 = a >= 2 ? (double)(a * (a - 1)) * xp[a >= 2 ? a - 2 : 0] : 0.0,
               Y2 = b >= 2 ? (double)(b * (b - 1)) * yp[b >= 2 ? b - 2 : 0] : 0.0,
               Z2 = c >= 2 ? (double)(c * (c - 1)) * zp[c >= 2 ? c - 2 : 0] : 0.0;
  const double X3 = (double)(a * (a - 1) * (a - 2)), Y3 = (double)(b * (b - 1) * (b - 2)),
               Z3 = (double)(c * (c - 1) * (c - 2));
  const double yz = Y0 * Z0, xz = X0 * Z0, xy = X0 * Y0;
  const double P = X0 * yz + (a + b + c >= 1 ? kShiftD : 0.0);
  const double Px = a >= 1 ? X1 * yz : 0.0, Py = b >= 1 ? Y1 * xz : 0.0, Pz = c >= 1 ? Z1 * xy : 0.0;
  const double hx = S.R0 * G1 + 2.0 * G4 * S.Rd[0], hy = S.R0 * G2 + 2.0 * G4 * S.Rd[1],
               hz = S.R0 * G3 + 2.0 * G4 * S.Rd[2];
  double sx = G0 * Px, sy = G0 * Py, sz = G0 * Pz;          // times R0
  double tx = 0.0, ty = 0.0, tz = 0.0;                      // HP h
  double lapP = 0.0, lx = 0.0, ly = 0.0, lz = 0.0;          // lap P and its gradient
  if (a >= 2) { const double p = X2 * yz; tx += p * hx; lapP += p; }
  if (b >= 2) { const double p = Y2 * xz; ty += p * hy; lapP += p; }
  if (c >= 2) { const double p = Z2 * xy; tz += p * hz; lapP += p; }
  if (a >= 1 && b >= 1) { const double p = X1 * Y1 * Z0; tx += p * hy; ty += p * hx; }
  if (a >= 1 && c >= 1) { const double p = X1 * Y0 * Z1; tx += p * hz; tz += p * hx; }
  if (b >= 1 && c >= 1) { const double p = X0 * Y1 * Z1; ty += p * hz; tz += p * hy; }
  if (a >= 3) lx += X3 * yz;
  if (b >= 3) ly += Y3 * xz;
  if (c >= 3) lz += Z3 * xy;
  if (a >= 1 && b >= 2) lx += X1 * Y2 * Z0;
  if (a >= 1 && c >= 2) lx += X1 * Y0 * Z2;
  if (a >= 2 && b >= 1) ly += X2 * Y1 * Z0;
  if (b >= 1 && c >= 2) ly += X0 * Y1 * Z2;
  if (a >= 2 && c >= 1) lz += X2 * Y0 * Z1;
  if (b >= 2 && c >= 1) lz += X0 * Y2 * Z1;
  sx += G4 * lx;
  sy += G4 * ly;
  sz += G4 * lz;
  const double u = G1 * S.Rd[0] + G2 * S.Rd[1] + G3 * S.Rd[2] + G4 * S.lapR;
  const double w = G0 * P + (G1 * Px + G2 * Py + G3 * Pz) + G4 * lapP;
  const double y0 = P * G1 + 2.0 * G4 * Px, y1 = P * G2 + 2.0 * G4 * Py, y2 = P * G3 + 2.0 * G4 * Pz;
  const double vy = 4.0 * S.R2 * (S.v[0] * y0 + S.v[1] * y1 + S.v[2] * y2) + P * G4 * S.k3;
  const double r1 = 2.0 * S.R1;
  q[0] += S.R0 * sx + tx + Px * u + S.Rd[0] * w + S.v[0] * vy + r1 * y0;
  q[1] += S.R0 * sy + ty + Py * u + S.Rd[1] * w + S.v[1] * vy + r1 * y1;
  q[2] += S.R0 * sz + tz + Pz * u + S.Rd[2] * w + S.v[2] * vy + r1 * y2;
}

template <int L, int I>
__device__ __forceinline__ void adj_shell(const ShellRad& S, const double (&xp)[4], const double (&yp)[4],
                                          const double (&zp)[4], const double* __restrict__ gr, int64_t ld, int tp,
                                          const double* __restrict__ fac, double (&q)[3]) {
  constexpr int N = (L + 1) * (L + 2) / 2;
  if constexpr (I < N) {
    // the I-th monomial: row r of constant a = L - r holds r + 1 entries
    constexpr int r = I < 1 ? 0 : I < 3 ? 1 : I < 6 ? 2 : 3;
    constexpr int a = L - r, b = r - (I - r * (r + 1) / 2), c = L - a - b;
    const double f = fac[I];
    const double* p = gr + I * ld;
    adj_ao<a, b, c>(S, xp, yp, zp, f * p[0], f * p[tp], f * p[2 * tp], f * p[3 * tp], f * p[4 * tp], q);
    adj_shell<L, I + 1>(S, xp, yp, zp, gr, ld, tp, fac, q);
  }
}

// FP64 adjoint over compact tiles: a CTA per tile (gridDim.y of them when
// there are few tiles), lanes are points, the warps take contiguous runs of
// the tile's live shells.  The pulled-back weights G of the tile are read
// along the points; q of a point is kept in the lane over the warp's shells
// and summed over the warps in order (grad_coord is stored by a CTA that owns
// its points, added to by one that shares them), q of a nucleus is summed
// over the run of its shells and the lanes and added by one atomic.  0.14 ms on 20,352
// points of the 2000-AO molecule, bound by the latency of its FP64 chains (a
// warp per point over all AOs, with the AO derivatives formed first, 1.43 ms).
__global__ void __launch_bounds__(256)
tile_deriv_kernel(const DevTables T, const int64_t P, const double* __restrict__ coord, const int64_t cstride,
                  const int* __restrict__ perm, const int64_t tile0, const F64Shell* __restrict__ sh,
                  const double cutoff, const double* __restrict__ gc, const AdjTables adj, const int64_t kmax,
                  double* __restrict__ grad_nucl, double* __restrict__ grad_coord, const int64_t gstride) {
  constexpr int TP = 32, LD = 5 * TP + 4, NW = 8;
  __shared__ double sq[NW][3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile = blockIdx.x;
  const int64_t qi = (tile0 + tile) * TP + lane;
  const bool in = qi < P;
  const int64_t pi = in ? (perm ? (int64_t)perm[qi] : qi) : 0;
  const double px = in ? coord[pi] : 0.0, py = in ? coord[pi + cstride] : 0.0, pz = in ? coord[pi + 2 * cstride] : 0.0;
  const int n = adj.nlive[tile];
  const int part = (int)blockIdx.y * NW + warp, parts = (int)gridDim.y * NW;
  const int e0 = (int)((int64_t)n * part / parts), e1 = (int)((int64_t)n * (part + 1) / parts);
  const double* gt = gc + (size_t)tile * kmax * LD + lane;
  double pq[3] = {0., 0., 0.}, nq[3] = {0., 0., 0.};
  int nucl = -1;
  auto flush = [&]() {
    if (nucl >= 0 && grad_nucl != nullptr) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double s = nq[d];
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) atomicAdd(&grad_nucl[nucl * 3 + d], -s);
      }
    }
    nq[0] = nq[1] = nq[2] = 0.0;
  };
  for (int e = e0; e < e1; ++e) {
    const int2 le = adj.live[tile * T.shell_num + e];
    const F64Shell S = sh[le.x];
    if (S.nucl != nucl) {
      flush();
      nucl = S.nucl;
    }
    ShellRad R;
    R.v[0] = px - S.x;
    R.v[1] = py - S.y;
    R.v[2] = pz - S.z;
    const double r2 = R.v[0] * R.v[0] + R.v[1] * R.v[1] + R.v[2] * R.v[2];
    double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
    if (in && !(r2 > S.crange)) {
      for (int j = S.cb; j < S.ce; ++j) {
        const double2 ac = T.coef_ac[j];
        const double ar2 = ac.x * r2;
        if (ar2 > cutoff) break;   // primitives sorted by exponent
        const double ce = ac.y * exp(-ar2);
        a0 += ce;
        a1 -= ac.x * ce;
        a2 += ac.x * ac.x * ce;
        a3 -= ac.x * ac.x * ac.x * ce;
      }
    }
    if (a0 == 0.0) continue;   // the lane's point is beyond the shell
    R.R0 = a0;
    R.R1 = a1;
    R.R2 = a2;
    R.lapR = 4.0 * r2 * a2 + 6.0 * a1;
    R.k3 = 20.0 * a2 + 8.0 * r2 * a3;
#pragma unroll
    for (int d = 0; d < 3; ++d) R.Rd[d] = 2.0 * R.v[d] * a1;
    const double* gr = gt + (size_t)le.y * LD;
    const double* fac = T.ao_factor + S.a0;
    double q[3] = {0., 0., 0.};
    if (S.l <= 3) {
      const double x = R.v[0], y = R.v[1], z = R.v[2];
      const double xp[4] = {1.0, x, x * x, x * (x * x)}, yp[4] = {1.0, y, y * y, y * (y * y)},
                   zp[4] = {1.0, z, z * z, z * (z * z)};
      switch (S.l) {
        case 0: adj_shell<0, 0>(R, xp, yp, zp, gr, LD, TP, fac, q); break;
        case 1: adj_shell<1, 0>(R, xp, yp, zp, gr, LD, TP, fac, q); break;
        case 2: adj_shell<2, 0>(R, xp, yp, zp, gr, LD, TP, fac, q); break;
        default: adj_shell<3, 0>(R, xp, yp, zp, gr, LD, TP, fac, q);
      }
    } else {
      const double R3[3] = {a0, a1, a2};
      for (int i = 0; i < S.na; ++i) {
        double g[3], H[3][3], Tl[3];
        ao_derivs<double>(T.ao_code[S.a0 + i], fac[i], R.v, R3, R.lapR, R.k3, g, H, Tl);
        const double* p = gr + i * LD;
#pragma unroll
        for (int d = 0; d < 3; ++d)
          q[d] += p[0] * g[d] + p[TP] * H[0][d] + p[2 * TP] * H[1][d] + p[3 * TP] * H[2][d] + p[4 * TP] * Tl[d];
      }
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      pq[d] += q[d];
      nq[d] += q[d];
    }
  }
  __syncwarp();
  flush();
  if (grad_coord == nullptr) return;
#pragma unroll
  for (int d = 0; d < 3; ++d) sq[warp][d][lane] = pq[d];
  __syncthreads();
  if (warp < 3 && in) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) s += sq[w][warp][lane];
    if (gridDim.y == 1)
      grad_coord[pi + warp * gstride] = s;
    else
      atomicAdd(&grad_coord[pi + warp * gstride], s);
  }
}

// Orbital forces (derivatives with respect to the nuclear coordinates; the
// reference's qmckl_get_forces_* getters, org/qmckl_forces.org:5129-6880).
// Only the AOs of nucleus a depend on R_a, so each force is a contraction
// over that nucleus's AO range [nuc_ao[a].x, nuc_ao[a].y):
//   out[(a * R + r) * M + i] = -sum_k X_r[k] * Ct[k][i]
// with the row r and its source row X_r:
//   MODE 0 forces_mo_value [a][p][n][i]: R = 3P, r = 3p + n,         X_r = ao_vgl[p][1+n]
//   MODE 1 forces_mo_g [a][n][p][m][i]:  R = 9P, r = 3(nP + p) + m,  X_r = ao_hessian[n][p][m]
//   MODE 2 forces_mo_l [a][n][p][i]:     R = 3P, r = nP + p,         X_r = ao_hessian[n][p][3]
// One thread per output element, MOs fastest (coalesced Ct reads and stores).
template <int MODE>
__global__ void forces_mo_kernel(const int64_t P, const int64_t A, const int64_t M, const int N,
                                 const int2* __restrict__ nuc_ao, const double* __restrict__ X,
                                 const double* __restrict__ Ct, double* __restrict__ out) {
  const int64_t R = (MODE == 1 ? 9 : 3) * P;
  const int64_t total = (int64_t)N * R * M;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = u % M;
    const int64_t ar = u / M;
    const int a = (int)(ar / R);
    const int64_t r = ar - (int64_t)a * R;
    const double* xr;
    if (MODE == 0) {
      const int64_t p = r / 3, n = r - 3 * p;
      xr = X + (p * 5 + 1 + n) * A;
    } else if (MODE == 1) {
      const int64_t np = r / 3, m = r - 3 * np;
      xr = X + (np * 4 + m) * A;
    } else {
      xr = X + (r * 4 + 3) * A;
    }
    const int2 kr = nuc_ao[a];
    double acc = 0.0;
    for (int k = kr.x; k < kr.y; ++k) acc -= Ct[(int64_t)k * M + i] * xr[k];
    out[u] = acc;
  }
}

// forces_ao_value[a][p][n][k] = -ao_vgl[p][1+n][k] for the AOs of nucleus a, 0 elsewhere
__global__ void forces_ao_kernel(const int64_t P, const int64_t A, const int N, const int2* __restrict__ nuc_ao,
                                 const double* __restrict__ X, double* __restrict__ out) {
  const int64_t total = (int64_t)N * P * 3 * A;
  for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = u % A;
    const int64_t apn = u / A;
    const int64_t n = apn % 3, ap = apn / 3;
    const int64_t p = ap % P;
    const int a = (int)(ap / P);
    const int2 kr = nuc_ao[a];
    out[u] = (k >= kr.x && k < kr.y) ? -X[(p * 5 + 1 + n) * A + k] : 0.0;
  }
}

}  // namespace

cudaError_t launch_forces(int which, int64_t P, int64_t A, int64_t M, int N, const int2* nuc_ao, const double* X,
                          const double* Ct, double* out, cudaStream_t s) {
  if (P <= 0 || N <= 0) return cudaSuccess;
  const int64_t total = which == 3 ? (int64_t)N * P * 3 * A : (int64_t)N * (which == 1 ? 9 : 3) * P * M;
  const int grid = (int)std::min<int64_t>((total + 255) / 256, 148 * 16);
  switch (which) {
    case 0: forces_mo_kernel<0><<<grid, 256, 0, s>>>(P, A, M, N, nuc_ao, X, Ct, out); break;
    case 1: forces_mo_kernel<1><<<grid, 256, 0, s>>>(P, A, M, N, nuc_ao, X, Ct, out); break;
    case 2: forces_mo_kernel<2><<<grid, 256, 0, s>>>(P, A, M, N, nuc_ao, X, Ct, out); break;
    case 3: forces_ao_kernel<<<grid, 256, 0, s>>>(P, A, N, nuc_ao, X, out); break;
    default: return cudaErrorInvalidValue;
  }
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_ao_hessian(const DevTables& T, int64_t point_num, const double* coord, double cutoff, bool mixed,
                              double* ao_hessian, cudaStream_t s, const double* cusp_r) {
  return launch_deriv<MODE_HESSIAN>(T, point_num, coord, point_num, cutoff, mixed, ao_hessian, nullptr, nullptr,
                                    nullptr, 0, s, cusp_r);
}

cudaError_t launch_mo_adjoint_nuclear(const DevTables& T, int64_t point_num, const double* coord, int64_t cstride,
                                      double cutoff, const float* G, double* grad_nucl, double* grad_coord,
                                      int64_t gstride, cudaStream_t s) {
  return launch_deriv<MODE_ADJOINT>(T, point_num, coord, cstride, cutoff, true, nullptr, G, grad_nucl, grad_coord,
                                    gstride, s);
}

cudaError_t launch_tile_deriv(const DevTables& T, int64_t P, const double* coord, int64_t cstride, const int* perm,
                              int64_t tile0, int64_t ntiles, const F64Shell* sh, double cutoff, const F64Tiles& t,
                              double* grad_nucl, double* grad_coord, int64_t gstride, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  if (t.pts != 32) return cudaErrorInvalidValue;
  const int parts = (int)std::max<int64_t>(1, std::min<int64_t>(8, 2 * 148 / ntiles));
  tile_deriv_kernel<<<dim3((unsigned)ntiles, (unsigned)parts), 256, 0, s>>>(
      T, P, coord, cstride, perm, tile0, sh, cutoff, t.ac, t.adj, T.ao_num, grad_nucl, grad_coord, gstride);
  count_launch();
  return cudaGetLastError();
}

}  // namespace qb
