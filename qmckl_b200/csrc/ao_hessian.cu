// AO Hessian ao_hessian[3][point][4][ao]: second derivatives and Laplacian
// gradients of the AOs with respect to the nuclear coordinates
// (qmckl_compute_ao_hessian_doc, org/qmckl_ao.org:9590-9720).
//
// Most of the array is exact zeros (79% on a 2000-AO molecule) and, without
// the work that visiting them takes, bound by the HBM writes.  A CTA of 128
// threads takes (point, segment of AOs) items: it packs the segment's live
// shells, forms their radial parts and then their AOs, a thread per AO, into
// an image of the 12 rows that is otherwise zero; each row leaves in one bulk
// copy and the entries written are zeroed again once the copies have read
// them.  Several CTAs per SM overlap the arithmetic of some with the copies of
// the others.  Segments are multiples of 32 AOs, so that the copies write
// whole 128-byte lines where the row length allows.
//
// 5,087 points x 1000 AOs (0.49 GB): 0.124 ms, 3.9 TB/s.  A warp per point
// over all its AOs with stores from registers took 0.198 ms, tiles of 32
// points with lanes on the points 0.18 ms (the few live shells of a segment
// keep too few warps busy with 12 rows per AO).
#include <algorithm>

#include "ao_derivs.cuh"
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace qb {
namespace {

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

}  // namespace

int hessian_segment_width(int64_t ao_num) {
  const int64_t n = std::max<int64_t>(1, (ao_num + 255) / 256);   // at most 256 AOs: 12-row images of 25 KB
  return (int)std::max<int64_t>(32, ((ao_num + n - 1) / n + 31) / 32 * 32);
}

cudaError_t launch_ao_hessian(const DevTables& T, const AoSegments& g, int64_t point_num, const double* coord,
                              double cutoff, bool mixed, double* ao_hessian, cudaStream_t s, const double* cusp_r) {
  if (point_num <= 0 || T.ao_num <= 0) return cudaSuccess;
  const int max_shells = std::max(1, g.max_shells);
  const size_t smem = sizeof(double) * kHessRows * (size_t)(g.width + 2) + sizeof(double) * kHessRad * (size_t)max_shells +
                      sizeof(uint32_t) * 2 * (size_t)g.width + sizeof(int) * (size_t)max_shells;
  cudaError_t e = cudaFuncSetAttribute(ao_hessian_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - 1024);
  if (e != cudaSuccess) return e;
  const int64_t per_sm = std::min<int64_t>(12, std::max<int64_t>(1, (int64_t)(227 * 1024) / (int64_t)(smem + 2048)));
  const int64_t grid = std::min<int64_t>(point_num * g.nseg, 148 * per_sm);
  ao_hessian_kernel<<<(unsigned)grid, kThreadsH, smem, s>>>(point_num, coord, g.sh, T.coef_ac, T.ao_code, T.ao_factor,
                                                            g.seg, g.nseg, g.width, max_shells, T.ao_num, cutoff, mixed,
                                                            cusp_r, ao_hessian);
  count_launch();
  return cudaGetLastError();
}

}  // namespace qb
