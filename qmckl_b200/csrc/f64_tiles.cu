// FP64 MO evaluation over spatial tiles: AO production into compact tiles,
// and the MO contraction of those tiles.
//
// The points are taken in a spatial order (perm) in tiles of TP.  A tile's
// live shells are those whose screening sphere (nucleus, squared radius
// beyond which all the shell's AOs are exact zeros, shell_r2max) holds one
// of its points; its K dimension is the list of their AOs, in the basis
// order.  On the 80-nucleus TZ molecule (2000 AOs) a tile of 32 points keeps
// 25% of the AOs, against 21% for a single point and 27% for 96.  An AO left
// out is an exact zero at every point of the tile, so a row's sum is the
// basis-order sum without zero terms (the order of the reference's own
// contraction, org/qmckl_mo.org:2015-2163, which skips the zero AOs of each
// point).
//
// Compact AO tile: ac[tile][k][LD], k along the tile's list, component c of
// point p at position c * TP + p, LD = COMPS * TP + 4 doubles (rows on
// distinct bank groups when they are copied to shared memory as they are).
#include <algorithm>

#include "kernels.cuh"

namespace qb {
namespace {

constexpr double kShiftT = 1.e-20;
constexpr int kAoThreads = 256;

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

// The product rule of one AO and its stores: v = P R with P's derivatives.
template <int COMPS, int TP>
__device__ __forceinline__ void put_ao(double* __restrict__ o, bool on, double f, const double (&s)[5], double P0,
                                       double P1, double P2, double P3, double P4) {
  o[0] = on ? P0 * s[0] * f : 0.0;
  if (COMPS == 5) {
    o[TP] = on ? (P1 * s[0] + P0 * s[1]) * f : 0.0;
    o[2 * TP] = on ? (P2 * s[0] + P0 * s[2]) * f : 0.0;
    o[3 * TP] = on ? (P3 * s[0] + P0 * s[3]) * f : 0.0;
    o[4 * TP] = on ? (P4 * s[0] + P0 * s[4] + 2.0 * (P1 * s[1] + P2 * s[2] + P3 * s[3])) * f : 0.0;
  }
}

// All AOs of a shell of angular momentum L <= 3 at the warp's 32 points: the
// cartesian exponents are compile-time constants.
template <int COMPS, int TP, int L>
__device__ __forceinline__ void emit_shell(double* __restrict__ o, int64_t ld, bool on, const double* __restrict__ fac,
                                           const double (&s)[5], double x, double y, double z) {
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
      put_ao<COMPS, TP>(o + i * ld, on, fac[i], s, P0, P1, P2, P3, P4);
      ++i;
    }
}

// The same for L >= 4 (org/qmckl_ao.org:6624-6914), its AOs [i0, i1).
template <int COMPS, int TP>
__device__ __forceinline__ void emit_shell_any(double* __restrict__ o, int64_t ld, bool on, int L, int i0, int i1,
                                               const double* __restrict__ fac, const double (&s)[5], double x, double y,
                                               double z) {
  int i = 0;
  for (int a = L; a >= 0; --a)
    for (int b = L - a; b >= 0 && i < i1; --b, ++i) {
      if (i < i0) continue;
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
      put_ao<COMPS, TP>(o + i * ld, on, fac[i], s, P0, pa1 * yz, pb1 * xz, pc1 * xy,
                        (double)(a - 1) * pa2 * yz + (double)(b - 1) * pb2 * xz + (double)(c - 1) * pc2 * xy);
    }
}

// AO production of a tile (blockIdx.x) by gridDim.y CTAs.  Each CTA finds the
// tile's live shells, numbers them by a scan, and its warps then claim (live
// shell, 32 points) units: the lanes are points, so the contraction loop, the
// angular momentum and every table read are uniform in the warp.  It is bound
// by the latency of the exponentials and table reads: 0.16 ms on 40,704
// points of the 2000-AO molecule, writing 0.85 GB (one warp per point with
// its lanes on the AOs, as the dense AO kernel works, visits every AO of
// every point and took 0.73 ms for the 3.3 GB array).  CTA 0 of the tile
// writes its AO list.
// Scratch: dynamic shared memory of 2 * shell_num ints; more shells than fit
// there come in windows [w0, w0 + shell_num) of all_shells, a launch each, that
// continue the tile's lists.
template <int COMPS, int TP, int PARTS>
__global__ void __launch_bounds__(kAoThreads, 4)
ao_tiles_kernel(const int64_t P, const double* __restrict__ coord, const int64_t cstride, const int* __restrict__ perm,
                const int64_t tile0, const int w0, const int shell_num, const int all_shells,
                const F64Shell* __restrict__ sh, const double2* __restrict__ prim, const double* __restrict__ factor, const double cutoff,
                const bool dp_exp, const double* __restrict__ cusp_r, const int64_t kmax, double* __restrict__ ac,
                int* __restrict__ klist, int* __restrict__ kcount, const AdjTables adj) {
  constexpr int G = TP / 32;
  constexpr int LD = COMPS * TP + 4;
  static_assert(TP % 32 == 0 && G <= 4, "a tile is 1 to 4 warps of points");
  __shared__ double spts[3 * TP];
  __shared__ unsigned long long wsum[kAoThreads / 32];
  __shared__ double box[G][6];
  __shared__ bool isnan_g[G];
  __shared__ int claim, nopen;
  extern __shared__ int sbuf[];
  int* live = sbuf;               // [shell_num] whether the shell is live, then [count] the live shells
  int* lpos = sbuf + shell_num;   // [count] first list position
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t tile = blockIdx.x;
  const int64_t p0 = (tile0 + tile) * TP;
  const int np = (int)(P - p0 < TP ? P - p0 : TP);
  for (int t = tid; t < 3 * TP; t += kAoThreads) {
    const int d = t / TP, i = t - d * TP;
    spts[t] = i < np ? coord[(perm ? (int64_t)perm[p0 + i] : p0 + i) + d * cstride] : 0.0;
  }
  if (tid == 0) claim = nopen = 0;
  sh += w0;
  const int k0 = w0 > 0 ? kcount[tile] : 0, q0 = w0 > 0 ? adj.nlive[tile] : 0;   // the lists of the windows before
  __syncthreads();
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
        box[warp][d] = lo;
        box[warp][3 + d] = hi;
      }
    }
    bad = __any_sync(0xffffffffu, bad);
    if (lane == 0) isnan_g[warp] = bad;
  }
  __syncthreads();
  // Live shells, one group of 32 points at a time: a shell beyond the group's
  // bounding box is dead, one that holds the group's first point is live, and
  // the rest (a fifth of them on the molecules of the tests), packed, are tested
  // point by point, a thread per shell.
  for (int s = tid; s < shell_num; s += kAoThreads) live[s] = 0;
#pragma unroll 1
  for (int g = 0; g < G; ++g) {
    if (32 * g >= np) break;
    for (int s = tid; s < shell_num; s += kAoThreads) {
      const F64Shell S = sh[s];
      if (S.r2max < 0.0) continue;   // no primitives
      // the margin covers the rounding of both distances
      const double bx = fmax(fmax(box[g][0] - S.x, S.x - box[g][3]), 0.0),
                   by = fmax(fmax(box[g][1] - S.y, S.y - box[g][4]), 0.0),
                   bz = fmax(fmax(box[g][2] - S.z, S.z - box[g][5]), 0.0);
      if (!isnan_g[g] && (bx * bx + by * by + bz * bz) * (1.0 - 1e-9) > S.r2max) continue;
      const double x = spts[32 * g] - S.x, y = spts[TP + 32 * g] - S.y, z = spts[2 * TP + 32 * g] - S.z;
      if (x * x + y * y + z * z <= S.r2max)
        live[s] = 1;
      else
        lpos[atomicAdd(&nopen, 1)] = s;
    }
    __syncthreads();
    const int n = nopen, e = min(np, 32 * g + 32);
    for (int q = tid; q < n; q += kAoThreads) {
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
          live[s] = 1;
          break;
        }
      }
    }
    __syncthreads();
    if (tid == 0) nopen = 0;
    __syncthreads();
  }
  // number them: thread tid owns shells [tid * per, (tid + 1) * per); the scan
  // counts AOs in the low and shells in the high half
  const int per = (shell_num + kAoThreads - 1) / kAoThreads;
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
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  unsigned long long base = 0ull, total = 0ull;
  for (int w = 0; w < kAoThreads / 32; ++w) {
    if (w < warp) base += wsum[w];
    total += wsum[w];
  }
  const int nlive = (int)(total >> 32), nao = (int)(total & 0xffffffffull);
  base += incl - local;
  // compact in place: a thread's live shells move to smaller indices, so the
  // flags are read into registers before anyone writes
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
        live[at] = s;
        lpos[at] = k;
        base += (1ull << 32) | (unsigned int)sh[s].na;
      }
  } else {   // many shells: through the position array, then one more pass
    for (int s = s0; s < s1; ++s) lpos[s] = live[s];
    __syncthreads();
    const unsigned long long b0 = base;
    for (int s = s0; s < s1; ++s)
      if (lpos[s]) {
        live[(int)(base >> 32)] = s;
        base += (1ull << 32);
      }
    __syncthreads();
    unsigned long long b = b0;
    int na_prev = 0;
    const int n_mine = (int)(base >> 32) - (int)(b0 >> 32);
    for (int q = 0; q < n_mine; ++q) {
      const int at = (int)(b0 >> 32) + q;
      b += (unsigned int)na_prev;
      na_prev = sh[live[at]].na;
      lpos[at] = (int)(b & 0xffffffffull);
    }
  }
  __syncthreads();
  if (blockIdx.y == 0) {
    int* kl = klist + tile * kmax;
    for (int q = tid; q < nlive; q += kAoThreads) {
      const F64Shell S = sh[live[q]];
      const int k = k0 + lpos[q];
      for (int i = 0; i < S.na; ++i) kl[k + i] = S.a0 + i;
      if (adj.live != nullptr) {
        adj.live[(int64_t)tile * all_shells + q0 + q] = make_int2(w0 + live[q], k);
        if (adj.inv != nullptr)
          for (int i = 0; i < S.na; ++i) adj.inv[tile * kmax + S.a0 + i] = k + i;
      }
    }
    if (tid == 0) {
      kcount[tile] = k0 + nao;
      if (adj.live != nullptr) {
        adj.nlive[tile] = q0 + nlive;
        adj.bad[tile] = 0u;
      }
    }
  }
  if (ac == nullptr) return;   // the lists only
  double* __restrict__ act = ac + (size_t)tile * kmax * LD;
  // Shells of l >= 4 are split over PARTS units, which form the radial part
  // again: with a unit each, their up to 36 AOs are the tile's critical path
  // (34 us, 18 split, on 100 points of a 5-atom molecule with l = 7).
  const int units = nlive * G * PARTS;
  for (;;) {
    int u = 0;
    if (lane == 0) u = atomicAdd(&claim, 1);
    u = __shfl_sync(0xffffffffu, u, 0) * (int)gridDim.y + (int)blockIdx.y;
    if (u >= units) break;
    const int part = u % PARTS;
    u /= PARTS;
    const int q = G == 1 ? u : u / G, g = G == 1 ? 0 : u % G;
    const F64Shell S = sh[live[q]];
    if (part > 0 && S.l < 4) continue;
    const int i = 32 * g + lane;
    double* o = act + (size_t)(k0 + lpos[q]) * LD + i;
    const double x = spts[i] - S.x, y = spts[TP + i] - S.y, z = spts[2 * TP + i] - S.z;
    const double r2 = x * x + y * y + z * z;
    double s[5] = {0., 0., 0., 0., 0.};
    bool on = i < np && !(r2 > S.crange);
    if (on) {
      radial_t<COMPS>(prim, S.cb, S.ce, x, y, z, r2, cutoff, dp_exp, s);
      on = s[0] != 0.0 && !cusp_masked(cusp_r, S.l, S.nucl, r2, COMPS == 1);
    }
    const double* fac = factor + S.a0;
    switch (S.l) {
      case 0: emit_shell<COMPS, TP, 0>(o, LD, on, fac, s, x, y, z); break;
      case 1: emit_shell<COMPS, TP, 1>(o, LD, on, fac, s, x, y, z); break;
      case 2: emit_shell<COMPS, TP, 2>(o, LD, on, fac, s, x, y, z); break;
      case 3: emit_shell<COMPS, TP, 3>(o, LD, on, fac, s, x, y, z); break;
      default:
        emit_shell_any<COMPS, TP>(o, LD, on, S.l, S.na * part / PARTS, S.na * (part + 1) / PARTS, fac, s, x, y,
                                  z);
    }
  }
}

__global__ void __launch_bounds__(256)
place_shells_kernel(const int n, const int nucl_num, const double* __restrict__ nucl_coord, F64Shell* __restrict__ sh) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const int m = sh[i].nucl;
  sh[i].x = nucl_coord[m];
  sh[i].y = nucl_coord[m + nucl_num];
  sh[i].z = nucl_coord[m + 2 * nucl_num];
}

// ------------------------------------------------------------ contraction

constexpr int BKT = 16;
constexpr int kListWin = 1024;   // list entries held in shared memory at a time

__device__ __forceinline__ void cp16(double* dst, const double* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes));
}
__device__ __forceinline__ void cp_commit_t() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_wait_t() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
__device__ __forceinline__ void dmma_t(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// out[point][c][n] = sum over the tile's list of ac[k][c][point] * Bt[list[k]][n]
// (Bt: coefficient_t, ldb even, 16-byte aligned rows) on the FP64 tensor pipe
// (mma.sync m8n8k4 f64, the only FP64 MMA of sm_100a), which bounds it: 37.0
// TFLOP/s measured with 4, 8, 16 or 20 warps per SM, but 30.7 with 10, since
// the pipe is per quarter of the SM and the warps are dealt to the quarters
// in turn.  So a CTA is a multiple of 4 warps, WM x WN of 8 MB rows x 8 NT
// columns each.  Large problems take all of a tile's rows (VGL: 160 = 4 x 40)
// by 80 columns, two CTAs per SM, so that one computes while the other waits
// for its step, loads or stores; few tiles are cut into row groups of one
// warp row (blockIdx.z) and narrower columns.  The column blocks are dealt to
// the warps in turn, from a warp that changes with the CTA, and blocks past N
// are skipped.  16-AO steps through STG stages of 16-byte cp.async; the AO
// rows are copied as they lie, the B rows are gathered by the list, which is
// staged in shared memory (read from global memory at each step it cost a
// load latency per step: 1.14 against 0.91 ms).  0.91 ms = 37 TFLOP/s of the
// executed products on 40,704 points, 2000 AOs, 160 MOs (1.10 ms = 30 TFLOP/s
// with 8-byte gathers of a dense AO array in 128-row tiles).  That form is at
// the 128 registers that two CTAs of 256 threads allow, and spills 28 bytes
// outside the k loop's products.
template <int COMPS, int TP, int MB, int WM, int WN, int NT, int STG>
__global__ void __launch_bounds__(32 * WM * WN, WM == 1 ? 5 : 2)
tile_gemm_kernel(const int64_t P, const int64_t tile0, const int64_t ntiles, const int64_t N,
                 const double* __restrict__ ac, const int* __restrict__ klist, const int* __restrict__ kcount,
                 const int64_t kmax, const int* __restrict__ perm, const double* __restrict__ Bt, const int64_t ldb,
                 double* __restrict__ C) {
  constexpr int ROWS = COMPS * TP, THREADS = 32 * WM * WN;
  constexpr int LD = ROWS + 4;                    // row stride of the AO tile
  constexpr int AR = 8 * MB * WM, LDA = AR + 4;   // rows of this CTA and their stride here
  static_assert(ROWS % AR == 0, "whole row groups");
  constexpr int BN = 8 * WN * NT, LDB = BN + 4;
  extern __shared__ __align__(16) double smem[];
  __shared__ int lwin[kListWin];
  double* As = smem;                       // [STG][BKT][LDA]
  double* Bs = smem + STG * BKT * LDA;     // [STG][BKT][LDB]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp / WN, wn = (warp + (int)(blockIdx.y + blockIdx.z)) % WN;
  const int g = lane >> 2, t = lane & 3;
  const int r0 = AR == ROWS ? 0 : (int)blockIdx.z * AR;
  const int64_t n0 = (int64_t)blockIdx.x * BN;
  const int nblk = (int)min((int64_t)(BN / 8), (N - n0 + 7) / 8);   // column blocks of this CTA
  const int nj = (nblk - wn + WN - 1) / WN;                         // of this warp: wn, wn + WN, ...
  for (int64_t tile = blockIdx.y; tile < ntiles; tile += gridDim.y) {
    const int nk = kcount[tile];
    const int* __restrict__ kl = klist + tile * kmax;
    const double* __restrict__ at = ac + (size_t)tile * kmax * LD + r0;
    const int ktiles = (nk + BKT - 1) / BKT;
    double acc[MB][NT][2];
#pragma unroll
    for (int i = 0; i < MB; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

    auto load = [&](int kt, int st) {
      const int k0 = kt * BKT;
      const int nv = min(BKT, nk - k0);   // rows past the list are zero-filled
      if (k0 % kListWin == 0) {           // the previous window's last use is a barrier ago
        for (int c = tid; c < min(kListWin, nk - k0); c += THREADS) lwin[c] = kl[k0 + c];
        __syncthreads();
      }
      double* as = As + st * BKT * LDA;
      if constexpr (AR == ROWS) {   // the step as it lies
        const double* src = at + (size_t)k0 * LD;
        const int cv = nv * (LD / 2);
#pragma unroll
        for (int i = 0; i < (BKT * LD / 2 + THREADS - 1) / THREADS; ++i) {
          const int c = tid + i * THREADS;
          if (c < BKT * LD / 2) cp16(as + 2 * c, c < cv ? src + 2 * c : at, c < cv ? 16 : 0);
        }
      } else {                      // its rows r0 .. r0 + AR, a warp per list entry
#pragma unroll
        for (int i = 0; i < BKT / (WM * WN); ++i) {
          const int row = warp + i * (WM * WN);
          const bool ok = row < nv;
          const double* src = ok ? at + (size_t)(k0 + row) * LD : at;
          for (int c = lane; c < AR / 2; c += 32) cp16(as + row * LDA + 2 * c, src + 2 * c, ok ? 16 : 0);
        }
      }
      double* bs = Bs + st * BKT * LDB;
#pragma unroll
      for (int i = 0; i < BKT / (WM * WN); ++i) {   // B rows, a warp per list entry
        const int row = warp + i * (WM * WN);
        const bool ok = row < nv;
        const double* src = Bt + n0 + (ok ? (int64_t)lwin[k0 % kListWin + row] * ldb : 0);
#pragma unroll
        for (int h = 0; h < (BN / 2 + 31) / 32; ++h) {
          const int c = lane + 32 * h;
          const bool in = ok && n0 + 2 * c < N;
          if (2 * c < BN) cp16(bs + row * LDB + 2 * c, in ? src + 2 * c : Bt, in ? 16 : 0);
        }
      }
    };
#pragma unroll
    for (int s = 0; s < STG - 1; ++s) {
      if (s < ktiles) load(s, s);
      cp_commit_t();
    }
    int st = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      cp_wait_t<STG - 2>();
      __syncthreads();
      if (kt + STG - 1 < ktiles) load(kt + STG - 1, st == 0 ? STG - 1 : st - 1);
      cp_commit_t();
      const double* as = As + st * BKT * LDA + wm * (8 * MB) + g;
      const double* bs = Bs + st * BKT * LDB + wn * 8 + g;
      st = st + 1 == STG ? 0 : st + 1;
#pragma unroll
      for (int kk = 0; kk < BKT; kk += 4) {
        double af[MB], bf[NT];
#pragma unroll
        for (int i = 0; i < MB; ++i) af[i] = as[(kk + t) * LDA + i * 8];
#pragma unroll
        for (int j = 0; j < NT; ++j) bf[j] = bs[(kk + t) * LDB + j * (8 * WN)];
#pragma unroll
        for (int j = 0; j < NT; ++j)
          if (j < nj) {   // uniform in the warp
#pragma unroll
            for (int i = 0; i < MB; ++i) dmma_t(acc[i][j][0], acc[i][j][1], af[i], bf[j]);
          }
      }
    }
    cp_wait_t<0>();
    __syncthreads();   // the stages are refilled for the next tile
    const bool pairs = (N & 1) == 0 && (reinterpret_cast<uintptr_t>(C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < MB; ++i) {
      const int r = r0 + wm * (8 * MB) + i * 8 + g;
      const int c = r / TP, p = r % TP;
      const int64_t q = (tile0 + tile) * TP + p;
      if (q >= P) continue;
      double* crow = C + ((perm ? (int64_t)perm[q] : q) * COMPS + c) * N;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int64_t n = n0 + (wn + j * WN) * 8 + 2 * t;
        if (n + 1 < N && pairs) {
          *reinterpret_cast<double2*>(crow + n) = make_double2(acc[i][j][0], acc[i][j][1]);
        } else {
          if (n < N) crow[n] = acc[i][j][0];
          if (n + 1 < N) crow[n + 1] = acc[i][j][1];
        }
      }
    }
  }
}

template <int COMPS, int TP, int MB, int WM, int WN, int NT, int STG>
cudaError_t run_tile_gemm(int64_t P, int64_t tile0, int64_t ntiles, int64_t N, const F64Tiles& t, int64_t kmax,
                          const int* perm, const double* Bt, int64_t ldb, double* C, cudaStream_t s) {
  constexpr int AR = 8 * MB * WM, BN = 8 * WN * NT;
  const size_t smem = sizeof(double) * STG * BKT * (AR + 4 + BN + 4);
  auto kern = tile_gemm_kernel<COMPS, TP, MB, WM, WN, NT, STG>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((N + BN - 1) / BN), (unsigned)std::min<int64_t>(ntiles, 65535), COMPS * TP / AR);
  kern<<<grid, 32 * WM * WN, smem, s>>>(P, tile0, ntiles, N, t.ac, t.klist, t.kcount, kmax, perm, Bt, ldb, C);
  count_launch();
  return cudaGetLastError();
}

// ---------------------------------------------------------------- adjoint

constexpr int kAdjPts = 32, kAdjRows = 5 * kAdjPts, kAdjLd = kAdjRows + 4;   // tiles of 32 points

// Loss weights in tile order: ws[tile][c * 32 + p][ldw] = w[perm point][c][.]
// (zero past the MOs and past the points), and the tile's points with weights
// that are not finite; a warp per row.
__global__ void __launch_bounds__(256)
weight_tiles_kernel(const int64_t P, const int64_t tile0, const int64_t rows, const double* __restrict__ w,
                    const int64_t M, const int* __restrict__ perm, double* __restrict__ ws, const int64_t ldw,
                    unsigned int* __restrict__ bad) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 8) {
    const int64_t tile = r / kAdjRows;
    const int pos = (int)(r - tile * kAdjRows), c = pos / kAdjPts;
    const int64_t q = (tile0 + tile) * kAdjPts + pos % kAdjPts;
    double* o = ws + r * ldw;
    if (q < P) {
      const double* src = w + ((perm ? (int64_t)perm[q] : q) * 5 + c) * M;
      bool off = false;
      for (int64_t n = lane; n < ldw; n += 32) {
        const double x = n < M ? src[n] : 0.0;
        off = off || !isfinite(x);
        o[n] = x;
      }
      if (__any_sync(0xffffffffu, off) && lane == 0) atomicOr(&bad[tile], 1u << (pos % kAdjPts));
    } else {
      for (int64_t n = lane; n < ldw; n += 32) o[n] = 0.0;
    }
  }
}

// The two contractions of the adjoint over a tile's AO list, 32 MF list rows by
// 80 columns per CTA (8 warps as 4 x 2), 16-step k in STG stages of 16-byte
// cp.async, two CTAs per SM; bound by the FP64 tensor pipe as the forward.
//   COEF: part[tile][m][n] = sum over the tile's positions of ac[m][pos] *
//         ws[pos][n], the tile's share of dL/dC (columns: MOs)
//   else: ac[m][pos] = sum over MOs of Ct[list[m]][mo] * ws[pos][mo], the
//         weights pulled back to the AOs (columns: positions; overwrites ac)
// The 8-row and 8-column blocks are dealt to the warps in turn and blocks past
// the list or the columns are skipped.  Tiles of 32 points, although their
// products are short (160 rows): tiles of 128 points keep 31% of the AOs of
// the 2000-AO molecule against 25%, and with their dead 32-point groups
// skipped the warps wait for one another (0.68 and 0.64 ms against 0.56 and
// 0.57 = 30 TFLOP/s on 20,352 points; as dense products over all AOs they
// took 3.3 and 2.2 ms).
template <bool COEF, int MF, int STG>
__global__ void __launch_bounds__(256, 2)
adj_gemm_kernel(double* __restrict__ ac, const int* __restrict__ klist, const int* __restrict__ kcount,
                const int64_t kmax, const int64_t M, const double* __restrict__ ws, const int64_t ldw,
                const double* __restrict__ Ct, const int64_t ldc, double* __restrict__ part) {
  constexpr int BM = 32 * MF, NT = 5, BN = 80, LDR = BKT + 4, LDB = BN + 4;
  constexpr int B_STAGE = COEF ? BKT * LDB : BN * LDR;
  extern __shared__ __align__(16) double smem[];
  double* As = smem;                          // [STG][BM][LDR]
  double* Bs = smem + STG * BM * LDR;        // COEF: [STG][BKT][LDB], else [STG][BN][LDR]
  const int64_t tile = blockIdx.z;
  const int nk = kcount[tile];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int turn = (int)(blockIdx.y + blockIdx.z);
  const int wm = ((warp >> 1) + turn) & 3, wn = (warp + turn) & 1;
  const int g = lane >> 2, t = lane & 3;
  const int n0 = (int)blockIdx.x * BN;
  const int K = COEF ? kAdjRows : (int)M;
  const int ncol = COEF ? (int)M : kAdjRows;
  const int ktiles = (K + BKT - 1) / BKT;
  const int nj = (min(BN / 8, (ncol - n0 + 7) / 8) - wn + 1) / 2;     // column blocks wn, wn + 2, ...
  const double* wt = ws + (size_t)tile * kAdjRows * ldw;
  for (int m0 = (int)blockIdx.y * BM; m0 < nk; m0 += (int)gridDim.y * BM) {
    const int ni = (min(4 * MF, (nk - m0 + 7) / 8) - wm + 3) / 4;           // row blocks wm, wm + 4, ...
    // the MF A rows this thread copies a 16-byte piece of
    const int a_r = tid >> 3, a_c = (tid & 7) * 2;
    const double* arow[MF];
#pragma unroll
    for (int i = 0; i < MF; ++i) {
      const int m = m0 + a_r + 32 * i;
      arow[i] = m >= nk ? nullptr
                : COEF  ? ac + ((size_t)tile * kmax + m) * kAdjLd + a_c
                        : Ct + (int64_t)klist[tile * kmax + m] * ldc + a_c;
    }
    double acc[MF][NT][2];
#pragma unroll
    for (int i = 0; i < MF; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
    auto load = [&](int kt, int st) {
      const int k0 = kt * BKT;
      double* as = As + st * BM * LDR + a_r * LDR + a_c;
      const bool ka = k0 + a_c < K;   // pairs: the pad of an odd row length is zero
#pragma unroll
      for (int i = 0; i < MF; ++i) {
        const bool ok = ka && arow[i] != nullptr;
        cp16(as + 32 * i * LDR, ok ? arow[i] + k0 : ws, ok ? 16 : 0);
      }
      double* bs = Bs + st * B_STAGE;
      if constexpr (COEF) {
#pragma unroll
        for (int i = 0; i < BKT / 8; ++i) {
          const int row = warp + 8 * i;
          const double* src = wt + (int64_t)(k0 + row) * ldw + n0;
#pragma unroll
          for (int h = 0; h < (BN / 2 + 31) / 32; ++h) {
            const int c = lane + 32 * h;
            const bool ok = n0 + 2 * c < (int)ldw;
            if (2 * c < BN) cp16(bs + row * LDB + 2 * c, ok ? src + 2 * c : ws, ok ? 16 : 0);
          }
        }
      } else {
        for (int r = a_r; r < BN; r += 32) {
          const bool ok = ka && n0 + r < ncol;
          cp16(bs + r * LDR + a_c, ok ? wt + (int64_t)(n0 + r) * ldw + k0 + a_c : ws, ok ? 16 : 0);
        }
      }
    };
#pragma unroll
    for (int s = 0; s < STG - 1; ++s) {
      if (s < ktiles) load(s, s);
      cp_commit_t();
    }
    int st = 0;
    for (int kt = 0; kt < ktiles; ++kt) {
      cp_wait_t<STG - 2>();
      __syncthreads();
      if (kt + STG - 1 < ktiles) load(kt + STG - 1, st == 0 ? STG - 1 : st - 1);
      cp_commit_t();
      const double* as = As + st * BM * LDR + (wm * 8 + g) * LDR + t;
      const double* bs = COEF ? Bs + st * B_STAGE + t * LDB + wn * 8 + g : Bs + st * B_STAGE + (wn * 8 + g) * LDR + t;
      st = st + 1 == STG ? 0 : st + 1;
#pragma unroll
      for (int kk = 0; kk < BKT; kk += 4) {
        double bf[NT];
#pragma unroll
        for (int j = 0; j < NT; ++j) bf[j] = COEF ? bs[kk * LDB + j * 16] : bs[j * 16 * LDR + kk];
#pragma unroll
        for (int i = 0; i < MF; ++i)
          if (i < ni) {   // uniform in the warp
            const double af = as[i * 32 * LDR + kk];
#pragma unroll
            for (int j = 0; j < NT; ++j)
              if (j < nj) dmma_t(acc[i][j][0], acc[i][j][1], af, bf[j]);
          }
      }
    }
    cp_wait_t<0>();
    __syncthreads();   // the stages are refilled for the next rows
#pragma unroll
    for (int i = 0; i < MF; ++i) {
      const int m = m0 + (4 * i + wm) * 8 + g;
      if (m >= nk) continue;
      double* o = COEF ? part + ((size_t)tile * kmax + m) * ldw : ac + ((size_t)tile * kmax + m) * kAdjLd;
#pragma unroll
      for (int j = 0; j < NT; ++j) {
        const int n = n0 + (wn + 2 * j) * 8 + 2 * t;
        if (n < (COEF ? (int)ldw : ncol)) *reinterpret_cast<double2*>(o + n) = make_double2(acc[i][j][0], acc[i][j][1]);
      }
    }
  }
}

// grad[n][k] (+)= sum over the tiles, in order, of part[tile][inv[tile][k]][n]
// (inv < 0: AO k is not in the tile's list, and only a weight that is not
// finite, times that zero, adds to the sum).  A warp per AO and 64 MOs, with
// the list positions of the next 32 tiles in flight beside eight rows; 16 AOs
// x 64 MOs per CTA, transposed through shared memory.
__global__ void __launch_bounds__(512)
sum_tiles_kernel(const double* __restrict__ part, const int* __restrict__ inv, const unsigned int* __restrict__ bad,
                 const double* __restrict__ ws, const int64_t ntiles, const int64_t kmax, const int64_t A,
                 const int64_t M, const int64_t ldw, double* __restrict__ grad, const bool accumulate) {
  __shared__ double tr[64][17];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t k = (int64_t)blockIdx.x * 16 + warp, n = (int64_t)blockIdx.y * 64 + 2 * lane;
  double2 v = make_double2(0.0, 0.0);
  if (k < A) {
    int next = lane < ntiles ? inv[lane * kmax + k] : -1;
    for (int64_t t0 = 0; t0 < ntiles; t0 += 32) {
      const int at = next;
      next = t0 + 32 + lane < ntiles ? inv[(t0 + 32 + lane) * kmax + k] : -1;
      const unsigned int pts = at < 0 && t0 + lane < ntiles ? bad[t0 + lane] : 0u;
      for (unsigned int q = __ballot_sync(0xffffffffu, pts != 0u); q; q &= q - 1) {   // rare
        const int b = __ffs(q) - 1;
        for (unsigned int p = __shfl_sync(0xffffffffu, pts, b); p; p &= p - 1)
          for (int c = 0; c < 5; ++c) {
            const double* row = ws + ((size_t)(t0 + b) * kAdjRows + c * kAdjPts + __ffs(p) - 1) * ldw;
            if (n < ldw) {
              v.x += 0.0 * row[n];
              v.y += 0.0 * row[n + 1];
            }
          }
      }
      unsigned int m = __ballot_sync(0xffffffffu, at >= 0);
      while (m) {
        double2 x[8];
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          x[h] = make_double2(0.0, 0.0);
          if (m) {
            const int b = __ffs(m) - 1;
            m &= m - 1;
            const int row = __shfl_sync(0xffffffffu, at, b);
            if (n < ldw) x[h] = *reinterpret_cast<const double2*>(part + ((size_t)(t0 + b) * kmax + row) * ldw + n);
          }
        }
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          v.x += x[h].x;
          v.y += x[h].y;
        }
      }
    }
  }
  tr[2 * lane][warp] = v.x;
  tr[2 * lane + 1][warp] = v.y;
  __syncthreads();
  for (int i = threadIdx.x; i < 64 * 16; i += 512) {
    const int64_t n2 = (int64_t)blockIdx.y * 64 + i / 16, k2 = (int64_t)blockIdx.x * 16 + i % 16;
    if (n2 < M && k2 < A) {
      double* o = grad + n2 * A + k2;
      *o = accumulate ? *o + tr[i / 16][i % 16] : tr[i / 16][i % 16];
    }
  }
}

template <bool COEF, int MF, int STG>
cudaError_t run_adj_gemm(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws, int64_t ldw,
                         const double* Ct, int64_t ldc, double* part, cudaStream_t s) {
  constexpr int BM = 32 * MF, BN = 80;
  const size_t smem = sizeof(double) * STG * (BM * (BKT + 4) + (COEF ? BKT * (BN + 4) : BN * (BKT + 4)));
  auto kern = adj_gemm_kernel<COEF, MF, STG>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t ncol = COEF ? M : kAdjRows;
  // a tile's list holds a quarter to a half of the AOs: a CTA takes row block
  // after row block beyond half of them
  const int64_t gy = (ao_num + 2 * BM - 1) / (2 * BM);
  for (int64_t z0 = 0; z0 < ntiles; z0 += 65535) {   // grid.z limit
    const int64_t nz = std::min<int64_t>(65535, ntiles - z0);
    dim3 grid((unsigned)((ncol + BN - 1) / BN), (unsigned)std::min<int64_t>(65535, gy), (unsigned)nz);
    kern<<<grid, 256, smem, s>>>(t.ac + (size_t)z0 * ao_num * kAdjLd, t.klist + z0 * ao_num, t.kcount + z0, ao_num, M,
                                 ws + (size_t)z0 * kAdjRows * ldw, ldw, Ct, ldc,
                                 COEF ? part + (size_t)z0 * ao_num * ldw : nullptr);
    count_launch();
  }
  return cudaGetLastError();
}

// Blocks of 128 list rows when they give about a CTA per SM (lists of a
// quarter of the AOs), else of 32: 10 tiles of a 500-AO molecule 17 and 12
// us against 56 and 30; 32 tiles of a 3750-AO one 157 and 156 us with 128,
// 189 and 169 with 32.
template <bool COEF>
cudaError_t pick_adj_gemm(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws, int64_t ldw,
                          const double* Ct, int64_t ldc, double* part, cudaStream_t s) {
  const int64_t ctas = ntiles * (((COEF ? M : kAdjRows) + 79) / 80) * std::max<int64_t>(1, ao_num / 512);
  return ctas < 148 ? run_adj_gemm<COEF, 1, 5>(ntiles, ao_num, M, t, ws, ldw, Ct, ldc, part, s)
                    : run_adj_gemm<COEF, 4, 3>(ntiles, ao_num, M, t, ws, ldw, Ct, ldc, part, s);
}

}  // namespace

// VGL tiles of 32 points (one warp of points, 160 contraction rows).  Value
// tiles of 128 points where that gives four CTAs per SM, else of 32.
int f64_tile_points(int comps, int64_t P) { return comps == 5 || P < 4 * 148 * 128 ? 32 : 128; }

size_t f64_tile_bytes(int comps, int pts, int64_t ao_num) {
  const size_t ld = (size_t)comps * pts + 4;
  return sizeof(double) * ld * (size_t)ao_num + sizeof(int) * ((size_t)ao_num + 1);
}

F64Tiles f64_tiles_at(void* scratch, int64_t ntiles, int comps, int pts, int64_t ao_num) {
  const size_t ld = (size_t)comps * pts + 4;
  F64Tiles t{};
  t.pts = pts;
  t.ac = (double*)scratch;
  t.klist = (int*)(t.ac + ld * (size_t)ao_num * (size_t)ntiles);
  t.kcount = t.klist + ao_num * ntiles;
  return t;
}

cudaError_t launch_place_shells(const DevTables& T, F64Shell* sh, cudaStream_t s) {
  if (T.shell_num <= 0) return cudaSuccess;
  place_shells_kernel<<<(unsigned)((T.shell_num + 255) / 256), 256, 0, s>>>(T.shell_num, T.nucl_num, T.nucl_coord, sh);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_ao_tiles(const DevTables& T, int64_t P, int comps, const double* coord, int64_t cstride,
                            const int* perm, int64_t tile0, int64_t ntiles, const F64Shell* sh, double cutoff,
                            bool dp_exp, const double* cusp_r, const F64Tiles& t, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  if (!(comps == 5 && t.pts == 32) && !(comps == 1 && (t.pts == 32 || t.pts == 128))) return cudaErrorInvalidValue;
  // in windows for the adjoint only: the forward refuses so many shells
  constexpr int kWindow = 200 * 1024 / (2 * (int)sizeof(int));
  if (T.shell_num > kWindow && t.adj.live == nullptr) return cudaErrorInvalidValue;
  const size_t sm = sizeof(int) * 2 * (size_t)std::min(T.shell_num, kWindow);
  auto kern = T.shell_parts > 1
                  ? (comps == 5 ? ao_tiles_kernel<5, 32, 4>
                                : (t.pts == 32 ? ao_tiles_kernel<1, 32, 4> : ao_tiles_kernel<1, 128, 4>))
                  : (comps == 5 ? ao_tiles_kernel<5, 32, 1>
                                : (t.pts == 32 ? ao_tiles_kernel<1, 32, 1> : ao_tiles_kernel<1, 128, 1>));
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kWindow * 2 * (int)sizeof(int));
  if (e != cudaSuccess) return e;
  // few tiles: several CTAs share one, so that its shells are spread over SMs
  // (not over windows: a window reads the counts that the one before wrote)
  const int parts = t.ac == nullptr || T.shell_num > kWindow
                        ? 1
                        : (int)std::max<int64_t>(1, std::min<int64_t>(8, (8 * 148 + ntiles - 1) / ntiles));
  for (int w0 = 0; w0 < T.shell_num; w0 += kWindow) {
    kern<<<dim3((unsigned)ntiles, (unsigned)parts), kAoThreads, sm, s>>>(
        P, coord, cstride, perm, tile0, w0, std::min(kWindow, T.shell_num - w0), T.shell_num, sh, T.coef_ac, T.ao_factor,
        cutoff, dp_exp, cusp_r, T.ao_num, t.ac, t.klist, t.kcount, t.adj);
    count_launch();
  }
  return cudaGetLastError();
}

cudaError_t launch_tile_gemm(int64_t P, int comps, int64_t tile0, int64_t ntiles, int64_t N, int64_t ao_num,
                             const F64Tiles& t, const int* perm, const double* Bt, int64_t ldb, double* C,
                             cudaStream_t s) {
  if (ntiles <= 0 || N <= 0) return cudaSuccess;
  if ((ldb & 1) != 0 || (reinterpret_cast<uintptr_t>(Bt) & 15) != 0) return cudaErrorInvalidValue;
  auto go = [&](auto launch) { return launch(P, tile0, ntiles, N, t, ao_num, perm, Bt, ldb, C, s); };
  if (comps == 5 && t.pts == 32) {
    // 160 x 80 tiles from four CTAs per SM on; below, row groups: on 136
    // points of a 263-AO, 224-MO molecule 15 us against 57 with whole tiles
    if (ntiles * ((N + 79) / 80) >= 4 * 148) return go(run_tile_gemm<5, 32, 5, 4, 2, 5, 3>);
    if (ntiles * 4 * ((N + 63) / 64) >= 2 * 148) return go(run_tile_gemm<5, 32, 5, 1, 4, 2, 3>);
    return go(run_tile_gemm<5, 32, 5, 1, 4, 1, 6>);
  }
  if (comps == 1 && t.pts == 128) return go(run_tile_gemm<1, 128, 4, 4, 2, 5, 3>);
  if (comps == 1 && t.pts == 32) {
    if (ntiles * ((N + 63) / 64) >= 2 * 148) return go(run_tile_gemm<1, 32, 4, 1, 4, 2, 3>);
    return go(run_tile_gemm<1, 32, 4, 1, 4, 1, 6>);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_weight_tiles(int64_t P, int64_t tile0, int64_t ntiles, const double* w, int64_t M, const int* perm,
                                double* ws, int64_t ldw, unsigned int* bad, cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  const int64_t rows = ntiles * kAdjRows;
  const unsigned grid = (unsigned)std::min<int64_t>((rows + 7) / 8, 148 * 32);
  weight_tiles_kernel<<<grid, 256, 0, s>>>(P, tile0, rows, w, M, perm, ws, ldw, bad);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_adj_coef(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws, int64_t ldw,
                            double* part, double* grad, bool accumulate, cudaStream_t s) {
  if (ntiles <= 0 || M <= 0) return cudaSuccess;
  if (t.pts != kAdjPts) return cudaErrorInvalidValue;
  cudaError_t e = pick_adj_gemm<true>(ntiles, ao_num, M, t, ws, ldw, nullptr, 0, part, s);
  if (e != cudaSuccess) return e;
  dim3 grid((unsigned)((ao_num + 15) / 16), (unsigned)((M + 63) / 64));
  sum_tiles_kernel<<<grid, 512, 0, s>>>(part, t.adj.inv, t.adj.bad, ws, ntiles, ao_num, ao_num, M, ldw, grad,
                                         accumulate);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_adj_pullback(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws,
                                int64_t ldw, const double* Ct, int64_t ldc, cudaStream_t s) {
  if (ntiles <= 0 || M <= 0) return cudaSuccess;
  if (t.pts != kAdjPts) return cudaErrorInvalidValue;
  return pick_adj_gemm<false>(ntiles, ao_num, M, t, ws, ldw, Ct, ldc, nullptr, s);
}

}  // namespace qb
