// AO arrays through row images in shared memory: the AO Hessian
// ao_hessian[3][point][4][ao] (FP64, qmckl_compute_ao_hessian_doc,
// org/qmckl_ao.org:9590-9720) and the AO VGL as 3 bfloat16 pieces (split.cuh)
// for the mixed-form adjoint (the arithmetic of ao_kernels.cu).
//
// The arrays are mostly exact zeros (79% on the 2000-AO molecule) and, without
// the work that visiting the zeros takes, bound by the HBM writes.  Both
// kernels evaluate the AOs of live shells only, into an image of the rows in
// shared memory that is otherwise zero, write the image out and put the zeros
// back.
#include <algorithm>

#include "ao_derivs.cuh"
#include "f64_tile_dev.cuh"
#include "split.cuh"
#include "tc_ptx.cuh"

namespace qb {
namespace {

// ---------------------------------------------------------------- Hessian

// A CTA of 128 threads takes (point, segment of AOs) items: it packs the
// segment's live shells, forms their radial parts and then their AOs, a
// thread per AO, into the image of the 12 rows; each row leaves in one bulk
// copy and the entries written are zeroed again once the copies have read
// them.  Six CTAs per SM overlap the arithmetic of some with the copies of the
// others.  Segments are multiples of 32 AOs, so that the copies write whole
// 128-byte lines where the row length allows.  0.123 ms on 5,087 points x 1000
// AOs (0.49 GB: 4.0 TB/s); a warp per point over all its AOs with stores from
// registers, 0.20 ms; tiles of points as in ao_pieces_kernel, 0.18 ms (the few
// live shells of a segment keep too few warps busy with 12 rows per AO).
constexpr int kHessRows = 12, kThreadsH = 128;
constexpr int kHessRad = 7;   // R, R1, R2, R3, displacement

__global__ void __launch_bounds__(kThreadsH)
ao_hessian_kernel(const int64_t P, const double* __restrict__ coord, const F64Shell* __restrict__ sh,
                  const double2* __restrict__ prim, const int32_t* __restrict__ ao_code,
                  const double* __restrict__ factor, const int2* __restrict__ segs, const int nseg, const int width,
                  const int max_shells, const int A, const double cutoff, const bool fp32_exp,
                  const double* __restrict__ cusp_r, double* __restrict__ out) {
  extern __shared__ __align__(16) uint8_t smem_r[];
  const int rs = width + 2;                                     // row stride of the image
  double* img = (double*)smem_r;                                // [12][rs]
  double* rad = img + kHessRows * rs;                           // [max_shells][kHessRad]
  uint32_t* lists = (uint32_t*)(rad + (size_t)max_shells * kHessRad);   // [2][width] live slot << 16 | AO
  int* live = (int*)(lists + 2 * width);                        // [max_shells]
  __shared__ unsigned int count[2];                             // live shells << 16 | live AOs
  __shared__ int shifts[2][kHessRows];                          // 16-byte phase of the rows, this and the previous item
  const int tid = threadIdx.x;
  for (int i = tid; i < kHessRows * rs / 2; i += kThreadsH) reinterpret_cast<uint4*>(img)[i] = make_uint4(0u, 0u, 0u, 0u);
  if (tid < 2) count[tid] = 0u;
  __syncthreads();
  const int64_t items = P * nseg;
  int pn = 0, buf = 0;   // live AOs of the previous item
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x, buf ^= 1) {
    const int64_t p = it / nseg;
    const int sg = (int)(it - p * nseg);
    const int a0 = sg * width, a1 = min(A, a0 + width);
    const int2 sr = segs[sg];
    const double px = coord[p], py = coord[p + P], pz = coord[p + 2 * P];
    uint32_t* list = lists + buf * width;
    auto row_addr = [&](int r) { return out + (((r >> 2) * P + p) * 4 + (r & 3)) * A + a0; };
    // a row's first element sits at the 16-byte phase that it has in the output
    if (tid < kHessRows) shifts[buf][tid] = (int)((reinterpret_cast<uintptr_t>(row_addr(tid)) >> 3) & 1);
    // the live shells and the list of their AOs in the segment
    for (int s = sr.x + tid; s < sr.y; s += kThreadsH) {
      const F64Shell S = sh[s];
      const double x = px - S.x, y = py - S.y, z = pz - S.z;
      const double r2 = x * x + y * y + z * z;
      if (!(r2 > S.r2max) && S.cb < S.ce) {
        const int k0 = max(S.a0, a0), k1 = min(S.a0 + S.na, a1);
        const unsigned int at = atomicAdd(&count[buf], (1u << 16) | (unsigned int)(k1 - k0));
        const int slot = (int)(at >> 16), q = (int)(at & 0xffffu);
        live[slot] = s;
        for (int k = k0; k < k1; ++k) list[q + k - k0] = ((uint32_t)slot << 16) | (uint32_t)(k - a0);
      }
    }
    __syncthreads();
    const int nlive = (int)(count[buf] >> 16), nao = (int)(count[buf] & 0xffffu);
    if (tid == 0) count[buf ^ 1] = 0u;
    // radial parts
    for (int q = tid; q < nlive; q += kThreadsH) {
      const F64Shell S = sh[live[q]];
      const double x = px - S.x, y = py - S.y, z = pz - S.z;
      const double r2 = x * x + y * y + z * z;
      double a[4] = {0., 0., 0., 0.};
      if (!(r2 > S.crange)) {
        for (int j = S.cb; j < S.ce; ++j) {
          const double2 ac = prim[j];
          const double ar2 = ac.x * r2;
          if (ar2 > cutoff) break;   // primitives are sorted by exponent
          const double e = (fp32_exp && ar2 <= 30.0) ? (double)expf(-(float)ar2) : exp(-ar2);
          const double ce = ac.y * e;
          a[0] += ce;
          a[1] -= ac.x * ce;
          a[2] += ac.x * ac.x * ce;
          a[3] -= ac.x * ac.x * ac.x * ce;
        }
        if (cusp_r != nullptr && cusp_masked(cusp_r, S.l, S.nucl, r2, false)) a[0] = 0.0;
      }
      double* o = rad + q * kHessRad;
#pragma unroll
      for (int c = 0; c < 4; ++c) o[c] = a[c];
      o[4] = x;
      o[5] = y;
      o[6] = z;
    }
    // the copies of the previous item have read the image: zero its entries
    if (tid < kHessRows) tcx::bulk_wait_read();
    __syncthreads();
    {
      const uint32_t* old = lists + (buf ^ 1) * width;
      for (int i = tid; i < pn; i += kThreadsH) {
        const int k = (int)(old[i] & 0xffffu);
#pragma unroll
        for (int r = 0; r < kHessRows; ++r) img[r * rs + shifts[buf ^ 1][r] + k] = 0.0;
      }
    }
    __syncthreads();
    // the live AOs
    for (int i = tid; i < nao; i += kThreadsH) {
      const int k = (int)(list[i] & 0xffffu);
      const double* s = rad + (list[i] >> 16) * kHessRad;
      if (s[0] == 0.0) continue;
      const double v[3] = {s[4], s[5], s[6]}, R[3] = {s[0], s[1], s[2]};
      const double r2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
      double g[3], H[3][3], Tl[3];
      ao_derivs<double>(ao_code[a0 + k], factor[a0 + k], v, R, 4.0 * r2 * s[2] + 6.0 * s[1],
                        20.0 * s[2] + 8.0 * r2 * s[3], g, H, Tl);
#pragma unroll
      for (int d = 0; d < 3; ++d) {
#pragma unroll
        for (int m = 0; m < 4; ++m) img[(4 * d + m) * rs + shifts[buf][4 * d + m] + k] = m < 3 ? H[d][m] : Tl[d];
      }
    }
    tcx::fence_async_smem();
    __syncthreads();
    if (tid < kHessRows) {
      double* g = row_addr(tid);
      const int sf = shifts[buf][tid], n = a1 - a0;
      const double* s = img + tid * rs + sf;
      const int head = sf, body = (n - head) / 2 * 2;
      if (head) g[0] = s[0];
      if (head + body < n) g[n - 1] = s[n - 1];
      if (body > 0) tcx::bulk_store(g + head, s + head, (uint32_t)body * 8u);
      tcx::bulk_commit();
    }
    pn = nao;
  }
  if (tid < kHessRows) tcx::bulk_wait_read();
}

// ----------------------------------------------------------------- pieces

// A CTA of four warps takes a tile of 32 spatially close points: it lists the
// shells that reach the tile, then goes through segments of 32 AOs: its warps,
// lanes on the points, form the segment's live shells into the image of the
// tile's 15 x 32 rows; then all threads write the image out row by row, each
// putting the zeros back where it read.  With lanes on the points every branch,
// table read and contraction loop is uniform in a warp and dead AOs cost only
// their zeros.  0.41 ms on 20,352 points x 2000 AOs (1.22 GB: 3.0 TB/s),
// bound by the waits between the two phases; a warp per point over all its
// AOs, with 2-byte stores from registers, took 0.56 ms.
constexpr int TPR = 32;      // points of a tile
constexpr int kThreadsR = 128;
constexpr int kPieceW = 32, kPieceRows = 15;
constexpr int kPiecePs = kPieceRows * kPieceW + 8;   // point stride: the lanes' stores spread over the banks
constexpr size_t kPieceImage = sizeof(uint16_t) * TPR * kPiecePs;

__global__ void __launch_bounds__(kThreadsR, 4)
ao_pieces_kernel(const int64_t P, const double* __restrict__ coord, const int* __restrict__ perm,
                 const F64Shell* __restrict__ sh, const double2* __restrict__ prim,
                 const double* __restrict__ factor, const int2* __restrict__ segs, const int nseg, const int part_shells,
                 const double cutoff, const bool dp_exp, uint16_t* __restrict__ out, const int64_t lda,
                 const int64_t pstride) {
  using E = uint16_t;
  constexpr int W = kPieceW, ROWS = kPieceRows, PS = kPiecePs, V = 8, NW = kThreadsR / 32;
  extern __shared__ __align__(16) uint8_t smem_r[];
  E* img = (E*)smem_r;
  int* live = (int*)(smem_r + kPieceImage);
  int* lao = live + part_shells;   // the live shells' first AO | AO count << 24
  __shared__ double spts[3 * TPR];
  __shared__ E* rowp[TPR * ROWS];  // the tile's rows in the output
  __shared__ TilePlan<TPR> pl;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t p0 = (int64_t)blockIdx.x * TPR;
  const int np = (int)(P - p0 < TPR ? P - p0 : TPR);
  const int g0 = (int)((int64_t)nseg * blockIdx.y / gridDim.y), g1 = (int)((int64_t)nseg * (blockIdx.y + 1) / gridDim.y);
  const int sbase = segs[g0].x, scount = segs[g1 - 1].y - sbase;
  for (int t = tid; t < 3 * TPR; t += kThreadsR) {
    const int d = t / TPR, i = t - d * TPR;
    spts[t] = i < np ? coord[(perm ? (int64_t)perm[p0 + i] : p0 + i) + d * P] : 0.0;
  }
  for (int rr = tid; rr < np * ROWS; rr += kThreadsR) {
    const int i = rr / ROWS, r = rr - i * ROWS;
    const int64_t p = perm ? (int64_t)perm[p0 + i] : p0 + i;
    rowp[rr] = out + (r / 5) * pstride + (p * 5 + r % 5) * lda;
  }
  for (int i = tid; i < (int)(kPieceImage / 16); i += kThreadsR)
    reinterpret_cast<uint4*>(img)[i] = make_uint4(0u, 0u, 0u, 0u);
  __syncthreads();
  const int nlive = tile_live_shells<TPR, kThreadsR>(pl, spts, np, sh + sbase, scount, live, lao).x;
  for (int q = tid; q < nlive; q += kThreadsR) {
    const int s = sbase + (live[q] & 0xffffff);
    live[q] = s;
    lao[q] = sh[s].a0 | (sh[s].na << 24);
  }
  __syncthreads();
  const double px = spts[lane], py = spts[TPR + lane], pz = spts[2 * TPR + lane];
  E* mine = img + lane * PS;
  int q0 = 0;   // first live shell with AOs in the segment
  for (int sg = g0; sg < g1; ++sg) {
    const int a0 = sg * W, a1 = a0 + W;
    while (q0 < nlive && (lao[q0] & 0xffffff) + (int)((unsigned int)lao[q0] >> 24) <= a0) ++q0;
    for (int q = q0 + warp; q < nlive && (lao[q] & 0xffffff) < a1; q += NW) {
      const F64Shell S = sh[live[q]];
      const double x = px - S.x, y = py - S.y, z = pz - S.z;
      const double r2 = x * x + y * y + z * z;
      bool on = lane < np && !(r2 > S.crange);
      const double* fac = factor + S.a0;
      const int k0 = S.a0 - a0;   // the shell's first AO in the segment's numbering
      double s[5] = {0., 0., 0., 0., 0.};
      if (on) {
        radial_t<5>(prim, S.cb, S.ce, x, y, z, r2, cutoff, dp_exp, s);
        on = s[0] != 0.0;
      }
      auto put = [&](int i, const double (&v)[5]) {
        const int k = k0 + i;
        if (k < 0 || k >= W || !on) return;   // zeros are there
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          uint16_t pc[3];
          split3_bf16(v[c], pc);
#pragma unroll
          for (int h = 0; h < 3; ++h) mine[(h * 5 + c) * W + k] = pc[h];
        }
      };
      switch (S.l) {
        case 0: emit_shell<5, 0>(put, on, fac, s, x, y, z); break;
        case 1: emit_shell<5, 1>(put, on, fac, s, x, y, z); break;
        case 2: emit_shell<5, 2>(put, on, fac, s, x, y, z); break;
        case 3: emit_shell<5, 3>(put, on, fac, s, x, y, z); break;
        default: emit_shell_any<5>(put, on, S.l, S.na, fac, s, x, y, z);
      }
    }
    __syncthreads();
    // the rows, 16 bytes per thread and step, and the zeros back in place: the
    // thread keeps its piece k of a row and steps over the rows
    constexpr int CW = W / V, RSTEP = kThreadsR / CW;
    const int end = min((int)lda - a0, W);   // to the row's padded end, a multiple of 8
    const int k = (tid % CW) * V;
#pragma unroll 4
    for (int rr = tid / CW; rr < np * ROWS; rr += RSTEP) {
      uint4* src = reinterpret_cast<uint4*>(img + rr * W + rr / ROWS * V + k);
      const uint4 v = *src;
      *src = make_uint4(0u, 0u, 0u, 0u);
      if (k < end) __stcs(reinterpret_cast<uint4*>(rowp[rr] + a0 + k), v);   // written once, not read here
    }
    __syncthreads();
  }
}

}  // namespace

int ao_segment_width(int array, int64_t ao_num) {
  if (array == 1) return kPieceW;
  const int64_t n = std::max<int64_t>(1, (ao_num + 255) / 256);   // at most 256 AOs: 12-row images of 25 KB
  return (int)std::max<int64_t>(32, ((ao_num + n - 1) / n + 31) / 32 * 32);
}

cudaError_t launch_ao_hessian(const DevTables& T, const AoRowTables& R, int64_t point_num, const double* coord,
                              double cutoff, bool mixed, double* ao_hessian, cudaStream_t s, const double* cusp_r) {
  if (point_num <= 0 || T.ao_num <= 0) return cudaSuccess;
  const AoSegments& g = R.seg[0];
  const int max_shells = std::max(1, g.run_shells[1]);
  const size_t smem = sizeof(double) * kHessRows * (size_t)(g.width + 2) + sizeof(double) * kHessRad * (size_t)max_shells +
                      sizeof(uint32_t) * 2 * (size_t)g.width + sizeof(int) * (size_t)max_shells;
  cudaError_t e = cudaFuncSetAttribute(ao_hessian_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t per_sm = std::min<int64_t>(12, std::max<int64_t>(1, (int64_t)(227 * 1024) / (int64_t)(smem + 2048)));
  const int64_t grid = std::min<int64_t>(point_num * g.nseg, 148 * per_sm);
  ao_hessian_kernel<<<(unsigned)grid, kThreadsH, smem, s>>>(point_num, coord, R.sh, T.coef_ac, T.ao_code, T.ao_factor,
                                                            g.seg, g.nseg, g.width, max_shells, T.ao_num, cutoff, mixed,
                                                            cusp_r, ao_hessian);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_ao_vgl_pieces(const DevTables& T, const AoRowTables& R, int64_t point_num, const double* coord,
                                 const int* perm, double cutoff, bool dp_exp, void* pieces, int64_t lda, int64_t pstride,
                                 cudaStream_t s) {
  if (point_num <= 0 || T.ao_num <= 0) return cudaSuccess;
  if (lda < T.ao_num || lda - T.ao_num >= 8 || lda % 8 != 0 || pstride % 8 != 0) return cudaErrorInvalidValue;
  const AoSegments& g = R.seg[1];
  const int64_t tiles = (point_num + TPR - 1) / TPR;
  if (tiles > 0x7fffffff) return cudaErrorInvalidValue;
  // a tile's segments over several CTAs: enough of them to fill the SMs evenly
  // (each lists the shells of its own segments only), and as many as keep a
  // part's shells within 32 KB
  int64_t parts = std::min<int64_t>(g.nseg, std::max<int64_t>(1, (32 * 148 + tiles - 1) / tiles));
  while (parts < g.nseg && g.run_shells[(size_t)((g.nseg + parts - 1) / parts)] > 4096) ++parts;
  const int part_shells = g.run_shells[(size_t)((g.nseg + parts - 1) / parts)];
  const size_t smem = kPieceImage + sizeof(int) * 2 * (size_t)part_shells;
  cudaError_t e = cudaFuncSetAttribute(ao_pieces_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  ao_pieces_kernel<<<dim3((unsigned)tiles, (unsigned)parts), kThreadsR, smem, s>>>(
      point_num, coord, perm, R.sh, T.coef_ac, T.ao_factor, g.seg, g.nseg, part_shells, cutoff, dp_exp, (uint16_t*)pieces,
      lda, pstride);
  count_launch();
  return cudaGetLastError();
}

}  // namespace qb
