// The adjoint of MO VGL with respect to the nuclear and point coordinates, and
// the orbital forces.
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
// The adjoint works on compact tiles (tile_deriv_kernel): with the
// loss weights pulled back through the MO coefficients, G = W . C, it forms
// q_d = G0 d_d chi + sum_e G_{1+e} H_ed + G4 T_d per AO; -q summed over a
// nucleus's AOs and the points is dL/dR, q summed over all AOs dL/dr.
#include <algorithm>
#include <type_traits>

#include "ao_derivs.cuh"
#include "kernels.cuh"

namespace qb {
namespace {

// the derivative kernel shares tiles out below this many, among up to kDerivParts CTAs each
constexpr int64_t kDerivCtas = 6 * 148, kDerivParts = 24;

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

__device__ __forceinline__ double nan_d() { return __longlong_as_double(0x7ff8000000000000ll); }

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

// The adjoint over compact tiles: a CTA per tile (gridDim.y of them when
// there are few tiles), lanes are points, the warps take contiguous runs of
// the tile's live shells.  The pulled-back weights G of the tile are read
// along the points; q of a point is kept in the lane over the warp's shells
// and summed over the warps in order and, by sum_shares_kernel, over the
// tile's CTAs in order, so that grad_coord is the same in every run (on 313
// tiles in three parts a sum by the tile's last CTA, which waits for its
// atomics, took 96 us against 84); q of a nucleus is summed
// over the run of its shells and the lanes and added by one atomic.  0.13 ms on 20,352
// points of the 2000-AO molecule, bound by the latency of its FP64 chains (a
// warp per point over all AOs, with the AO derivatives formed first, 1.43 ms).
// gc: G[tile][m][LD], FP64 with LD = 164.  MIXED: G in FP32 with LD = 160, FP32
// exponentials where a r^2 <= 30 and FP32 per-AO derivative arithmetic
// (displacements, r^2, radial sums and the cancelling radial combinations in
// FP64; q summed in FP64); 0.18 ms, against 0.93 with a warp per point over all
// AOs.  Below 888 tiles (kDerivCtas) 2 to 24 CTAs share a tile: two at 636
// tiles, where it took 0.24 ms mixed and 0.14 FP64 with one.  adj.live null: all
// shells for every tile, G's rows the AOs.
template <bool MIXED>
__global__ void __launch_bounds__(256, MIXED ? 3 : 2)
tile_deriv_kernel(const DevTables T, const int64_t P, const double* __restrict__ coord, const int64_t cstride,
                  const int* __restrict__ perm, const int64_t tile0, const F64Shell* __restrict__ sh,
                  const double cutoff, const void* __restrict__ gcv, const AdjTables adj, const int64_t kmax,
                  double* __restrict__ grad_nucl, double* __restrict__ grad_coord, const int64_t gstride) {
  using F = typename std::conditional<MIXED, float, double>::type;
  constexpr int TP = 32, LD = 5 * TP + (MIXED ? 0 : 4), NW = 8;
  const F* __restrict__ gc = (const F*)gcv;
  __shared__ double sq[NW][3][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t tile = blockIdx.x;
  const int64_t qi = (tile0 + tile) * TP + lane;
  const bool in = qi < P;
  const int64_t pi = in ? (perm ? (int64_t)perm[qi] : qi) : 0;
  const double px = in ? coord[pi] : 0.0, py = in ? coord[pi + cstride] : 0.0, pz = in ? coord[pi + 2 * cstride] : 0.0;
  // with shells of l >= 4, T.shell_parts entries per shell share its AOs
  const int n = (adj.live != nullptr ? adj.nlive[tile] : T.shell_num) * T.shell_parts;
  const int part = (int)blockIdx.y * NW + warp, parts = (int)gridDim.y * NW;
  const int e0 = (int)((int64_t)n * part / parts), e1 = (int)((int64_t)n * (part + 1) / parts);
  const F* gt = gc + (size_t)tile * kmax * LD + lane;
  double pq[3] = {0., 0., 0.}, nq[3] = {0., 0., 0.};
  if (const unsigned int bad = adj.bad[tile]; bad != 0u && blockIdx.y == 0) {
    // weights that are not finite meet zero AOs (rare): NaN for their points
    // and for every nucleus
    const double nan = nan_d();
    if (warp == 0 && (bad >> lane & 1u)) pq[0] = pq[1] = pq[2] = nan;
    if (grad_nucl != nullptr)
      for (int i = threadIdx.x; i < 3 * T.nucl_num; i += 256) atomicAdd(&grad_nucl[i], nan);
  }
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
    int2 le = make_int2(e / T.shell_parts, 0);
    if (adj.live != nullptr) le = adj.live[tile * T.shell_num + le.x];
    const F64Shell S = sh[le.x];
    if (adj.live == nullptr) le.y = S.a0;
    const int sp = e % T.shell_parts;
    if (sp > 0 && S.l < 4) continue;
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
        const double e = MIXED && ar2 <= 30.0 ? (double)expf(-(float)ar2) : exp(-ar2);
        const double ce = ac.y * e;
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
    const F* gr = gt + (size_t)le.y * LD;
    const double* fac = T.ao_factor + S.a0;
    double q[3] = {0., 0., 0.};
    bool any_l = true;
    if constexpr (!MIXED) {
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
        any_l = false;
      }
    }
    if (any_l) {
      const F v[3] = {(F)R.v[0], (F)R.v[1], (F)R.v[2]}, R3[3] = {(F)a0, (F)a1, (F)a2};
      const int i0 = S.l < 4 ? 0 : S.na * sp / T.shell_parts, i1 = S.l < 4 ? S.na : S.na * (sp + 1) / T.shell_parts;
      for (int i = i0; i < i1; ++i) {
        F g[3], H[3][3], Tl[3];
        ao_derivs<F>(T.ao_code[S.a0 + i], (F)fac[i], v, R3, (F)R.lapR, (F)R.k3, g, H, Tl);
        const F* p = gr + i * LD;
        const F G0 = p[0], G1 = p[TP], G2 = p[2 * TP], G3 = p[3 * TP], G4 = p[4 * TP];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          q[d] += (double)(G0 * g[d] + G1 * H[0][d] + G2 * H[1][d] + G3 * H[2][d] + G4 * Tl[d]);
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
  if (warp < 3) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) s += sq[w][warp][lane];
    if (gridDim.y > 1)
      adj.share[((size_t)tile * gridDim.y + blockIdx.y) * 96 + warp * 32 + lane] = s;
    else if (in)
      grad_coord[pi + warp * gstride] = s;
  }
}

// grad_coord of tiles shared by `parts` CTAs: their shares summed in order.
__global__ void __launch_bounds__(192)
sum_shares_kernel(const int64_t P, const int* __restrict__ perm, const int64_t tile0, const int64_t ntiles,
                  const int parts, const double* __restrict__ share, double* __restrict__ grad_coord,
                  const int64_t gstride) {
  const int64_t i = (int64_t)blockIdx.x * 192 + threadIdx.x, tile = i / 96;
  const int at = (int)(i - tile * 96);
  const int64_t qi = (tile0 + tile) * 32 + (at & 31);
  if (tile >= ntiles || qi >= P) return;
  double s = 0.0;
  for (int r = 0; r < parts; ++r) s += share[((size_t)tile * parts + r) * 96 + at];
  grad_coord[(perm ? (int64_t)perm[qi] : qi) + (at >> 5) * gstride] = s;
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

// CTAs per tile: enough to fill the chip, up to 8, or up to 24 where there are
// shells (or parts of shells) for all their warps (60 points x 380 AOs, l up to
// 7: the mixed adjoint 93 us with 8, 79 with 24; x 1000 AOs 84 and 74).
static int deriv_parts(int64_t ntiles, int64_t entries) {
  const int64_t most = std::max<int64_t>(8, std::min<int64_t>(kDerivParts, entries / 8));
  return (int)std::max<int64_t>(1, std::min<int64_t>(most, (kDerivCtas + ntiles - 1) / ntiles));
}

size_t deriv_share_bytes(int64_t ntiles) {
  // CTAs that share tiles, for any count up to ntiles: kDerivParts per tile, and
  // below kDerivCtas + the tiles
  return sizeof(double) * 96 * (size_t)std::min<int64_t>(kDerivParts * ntiles, 2 * kDerivCtas);
}

cudaError_t launch_tile_deriv(const DevTables& T, int64_t P, const double* coord, int64_t cstride, const int* perm,
                              int64_t tile0, int64_t ntiles, const F64Shell* sh, double cutoff, const AdjTables& adj,
                              const void* g, bool mixed, double* grad_nucl, double* grad_coord, int64_t gstride,
                              cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  const int parts = deriv_parts(ntiles, (int64_t)T.shell_num * T.shell_parts);
  auto k = mixed ? tile_deriv_kernel<true> : tile_deriv_kernel<false>;
  k<<<dim3((unsigned)ntiles, (unsigned)parts), 256, 0, s>>>(T, P, coord, cstride, perm, tile0, sh, cutoff, g, adj, T.ao_num,
                                                            grad_nucl, grad_coord, gstride);
  count_launch();
  if (grad_coord != nullptr && parts > 1) {
    sum_shares_kernel<<<(unsigned)((ntiles + 1) / 2), 192, 0, s>>>(P, perm, tile0, ntiles, parts, adj.share, grad_coord,
                                                                   gstride);
    count_launch();
  }
  return cudaGetLastError();
}

}  // namespace qb
