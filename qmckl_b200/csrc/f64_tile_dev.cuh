// Device pieces of the FP64 kernels over tiles of spatially close points
// (f64_tiles.cu, ao_rows.cu): the tile's live shells, the radial part of a
// shell and its AOs, with a warp's lanes on points.
#pragma once

#include "kernels.cuh"

namespace qb {

constexpr double kShiftT = 1.e-20;

__device__ __forceinline__ double ipow_t(double x, int n) {
  double r = 1.0;
  for (int i = 0; i < n; ++i) r = r * x;
  return r;
}

// Radial VGL of one shell at one point (org/qmckl_ao.org:8798-8828); the
// arithmetic of ao_kernels.cu shell_radial.
template <int COMPS>
__device__ __forceinline__ void radial_t(const double2* __restrict__ prim, int cb, int ce, double x, double y, double z,
                                         double r2, double cutoff, bool dp_exp, double (&s)[5]) {
#pragma unroll
  for (int c = 0; c < 5; ++c) s[c] = 0.0;
  for (int j = cb; j < ce; ++j) {
    const double2 ac = prim[j];
    const double ar2 = ac.x * r2;
    if (ar2 > cutoff) break;   // primitives are sorted by exponent
    const double e = dp_exp ? exp(-ar2) : (double)expf(-(float)ar2);
    s[0] += ac.y * e;
    if (COMPS == 5) {
      double f = ac.x * e;
      f = -f - f;
      s[1] += ac.y * (f * x);
      s[2] += ac.y * (f * y);
      s[3] += ac.y * (f * z);
      s[4] += ac.y * (f * (3.0 - 2.0 * ar2));
    }
  }
}

// The product rule of one AO: v = P R (zero where !on) with P's derivatives.
template <int COMPS>
__device__ __forceinline__ void vgl_ao(bool on, double f, const double (&s)[5], double P0, double P1, double P2, double P3,
                                       double P4, double (&v)[COMPS]) {
  v[0] = on ? P0 * s[0] * f : 0.0;
  if constexpr (COMPS == 5) {
    v[1] = on ? (P1 * s[0] + P0 * s[1]) * f : 0.0;
    v[2] = on ? (P2 * s[0] + P0 * s[2]) * f : 0.0;
    v[3] = on ? (P3 * s[0] + P0 * s[3]) * f : 0.0;
    v[4] = on ? (P4 * s[0] + P0 * s[4] + 2.0 * (P1 * s[1] + P2 * s[2] + P3 * s[3])) * f : 0.0;
  }
}

// All AOs of a shell of angular momentum L <= 3 at the warp's 32 points, put(i,
// values) each: the cartesian exponents are compile-time constants.
template <int COMPS, int L, class Put>
__device__ __forceinline__ void emit_shell(Put put, bool on, const double* __restrict__ fac, const double (&s)[5],
                                           double x, double y, double z) {
  const double xp[4] = {1.0, x, x * x, x * (x * x)}, yp[4] = {1.0, y, y * y, y * (y * y)},
               zp[4] = {1.0, z, z * z, z * (z * z)};
  int i = 0;
#pragma unroll
  for (int a = L; a >= 0; --a)
#pragma unroll
    for (int b = L - a; b >= 0; --b) {
      const int c = L - a - b;
      const double yz = yp[b] * zp[c], xz = xp[a] * zp[c], xy = xp[a] * yp[b];
      const double P0 = xp[a] * yz + (L >= 1 ? kShiftT : 0.0);
      const double P1 = a ? (double)a * xp[a > 0 ? a - 1 : 0] * yz : 0.0;
      const double P2 = b ? (double)b * yp[b > 0 ? b - 1 : 0] * xz : 0.0;
      const double P3 = c ? (double)c * zp[c > 0 ? c - 1 : 0] * xy : 0.0;
      double P4 = 0.0;
      if (a >= 2) P4 += (double)(a * (a - 1)) * xp[a >= 2 ? a - 2 : 0] * yz;
      if (b >= 2) P4 += (double)(b * (b - 1)) * yp[b >= 2 ? b - 2 : 0] * xz;
      if (c >= 2) P4 += (double)(c * (c - 1)) * zp[c >= 2 ? c - 2 : 0] * xy;
      double v[COMPS];
      vgl_ao<COMPS>(on, fac[i], s, P0, P1, P2, P3, P4, v);
      put(i, v);
      ++i;
    }
}

// The same for L >= 4 (org/qmckl_ao.org:6624-6914).
template <int COMPS, class Put>
__device__ __forceinline__ void emit_shell_any(Put put, bool on, int L, int na, const double* __restrict__ fac,
                                               const double (&s)[5], double x, double y, double z) {
  int i = 0;
  for (int a = L; a >= 0; --a)
    for (int b = L - a; b >= 0 && i < na; --b, ++i) {
      const int c = L - a - b;
      const double pa = ipow_t(x, a), pb = ipow_t(y, b), pc = ipow_t(z, c);
      const double pa1 = a >= 1 ? ipow_t(x, a - 1) : 1.0, pb1 = b >= 1 ? ipow_t(y, b - 1) : 1.0,
                   pc1 = c >= 1 ? ipow_t(z, c - 1) : 1.0;
      const double pa2 = a >= 2 ? ipow_t(x, a - 2) : 1.0, pb2 = b >= 2 ? ipow_t(y, b - 2) : 1.0,
                   pc2 = c >= 2 ? ipow_t(z, c - 2) : 1.0;
      double xy = pa * pb, yz = pb * pc, xz = pa * pc;
      const double P0 = xy * pc + kShiftT;
      xy *= (double)c;
      xz *= (double)b;
      yz *= (double)a;
      double v[COMPS];
      vgl_ao<COMPS>(on, fac[i], s, P0, pa1 * yz, pb1 * xz, pc1 * xy,
                    (double)(a - 1) * pa2 * yz + (double)(b - 1) * pb2 * xz + (double)(c - 1) * pc2 * xy, v);
      put(i, v);
    }
}

// Live shells of a tile of TP points (np of them there; spts [3][TP] in
// shared memory) among sh[0, shell_num): live[.] = shell | mask of the 32-point
// groups it reaches << 24, in order, and lpos[.] = the AOs in front of it (both
// of shell_num entries of shared memory).  All NT threads of the CTA
// take part; returns the counts, after a barrier.
template <int TP>
struct TilePlan {
  unsigned long long wsum[32];
  double box[TP / 32][6];
  bool isnan_g[TP / 32];
  int nopen;
};
template <int TP, int NT>
__device__ __forceinline__ int2 tile_live_shells(TilePlan<TP>& pl, const double* spts, const int np,
                                                 const F64Shell* __restrict__ sh, const int shell_num, int* live,
                                                 int* lpos) {
  constexpr int G = TP / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) pl.nopen = 0;
  if (warp < G) {   // bounding box of each 32 points (NaN coordinates left out)
    const int i = max(0, min(32 * warp + lane, np - 1));
    bool bad = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double lo = spts[d * TP + i], hi = lo;
      bad = bad || isnan(lo);
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) {
        lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
      }
      if (lane == 0) {
        pl.box[warp][d] = lo;
        pl.box[warp][3 + d] = hi;
      }
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) pl.isnan_g[warp] = bad;
  }
  __syncthreads();
  // Live shells, one group of 32 points at a time: a shell beyond the group's
  // bounding box is dead, one that holds the group's first point is live, and
  // the rest (a fifth of them on the molecules of the tests), packed, are tested
  // point by point, a thread per shell.
  for (int s = tid; s < shell_num; s += NT) live[s] = 0;
#pragma unroll 1
  for (int g = 0; g < G; ++g) {
    if (32 * g >= np) break;
    for (int s = tid; s < shell_num; s += NT) {
      const F64Shell S = sh[s];
      if (S.r2max < 0.0) continue;   // no primitives
      // the margin covers the rounding of both distances
      const double bx = fmax(fmax(pl.box[g][0] - S.x, S.x - pl.box[g][3]), 0.0),
                   by = fmax(fmax(pl.box[g][1] - S.y, S.y - pl.box[g][4]), 0.0),
                   bz = fmax(fmax(pl.box[g][2] - S.z, S.z - pl.box[g][5]), 0.0);
      if (!pl.isnan_g[g] && (bx * bx + by * by + bz * bz) * (1.0 - 1e-9) > S.r2max) continue;
      const double x = spts[32 * g] - S.x, y = spts[TP + 32 * g] - S.y, z = spts[2 * TP + 32 * g] - S.z;
      if (x * x + y * y + z * z <= S.r2max)
        live[s] |= 1 << g;
      else
        lpos[atomicAdd(&pl.nopen, 1)] = s;
    }
    __syncthreads();
    const int n = pl.nopen, e = min(np, 32 * g + 32);
    for (int q = tid; q < n; q += NT) {
      const int s = lpos[q];
      const F64Shell S = sh[s];
      for (int i = 32 * g; i < e; i += 4) {
        bool in = false;
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          const int j = min(i + h, e - 1);
          const double x = spts[j] - S.x, y = spts[TP + j] - S.y, z = spts[2 * TP + j] - S.z;
          // a NaN distance counts as inside: the AO is then a NaN, not a zero
          in = in || !(x * x + y * y + z * z > S.r2max);
        }
        if (in) {
          live[s] |= 1 << g;
          break;
        }
      }
    }
    __syncthreads();
    if (tid == 0) pl.nopen = 0;
    __syncthreads();
  }
  // number them: thread tid owns shells [tid * per, (tid + 1) * per); the scan
  // counts AOs in the low and shells in the high half
  const int per = (shell_num + NT - 1) / NT;
  const int s0 = min(shell_num, tid * per), s1 = min(shell_num, s0 + per);
  unsigned long long local = 0ull;
  for (int s = s0; s < s1; ++s)
    if (live[s]) local += (1ull << 32) | (unsigned int)sh[s].na;
  unsigned long long incl = local;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += v;
  }
  if (lane == 31) pl.wsum[warp] = incl;
  __syncthreads();
  unsigned long long base = 0ull, total = 0ull;
  for (int w = 0; w < NT / 32; ++w) {
    if (w < warp) base += pl.wsum[w];
    total += pl.wsum[w];
  }
  const int nlive = (int)(total >> 32), nao = (int)(total & 0xffffffffull);
  base += incl - local;
  // compact in place: a thread's live shells move to smaller indices, so the
  // masks are read into registers before anyone writes
  int mk[4];
  const bool few = per <= 4;
  if (few) {
#pragma unroll
    for (int q = 0; q < 4; ++q) mk[q] = s0 + q < s1 ? live[s0 + q] : 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (mk[q]) {
        const int at = (int)(base >> 32), k = (int)(base & 0xffffffffull), s = s0 + q;
        live[at] = s | (mk[q] << 24);
        lpos[at] = k;
        base += (1ull << 32) | (unsigned int)sh[s].na;
      }
  } else {   // many shells: through the position array, then one more pass
    for (int s = s0; s < s1; ++s) lpos[s] = live[s];
    __syncthreads();
    const unsigned long long b0 = base;
    for (int s = s0; s < s1; ++s)
      if (lpos[s]) {
        live[(int)(base >> 32)] = s | (lpos[s] << 24);
        base += (1ull << 32);
      }
    __syncthreads();
    unsigned long long b = b0;
    int na_prev = 0;
    const int n_mine = (int)(base >> 32) - (int)(b0 >> 32);
    for (int q = 0; q < n_mine; ++q) {
      const int at = (int)(b0 >> 32) + q;
      b += (unsigned int)na_prev;
      na_prev = sh[live[at] & 0xffffff].na;
      lpos[at] = (int)(b & 0xffffffffull);
    }
  }
  __syncthreads();
  return make_int2(nlive, nao);
}

}  // namespace qb
