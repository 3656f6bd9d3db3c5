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
// keep too few warps busy with 12 rows per AO).  Small molecules at many points
// take the warp per point (hessian_by_warps).
#include <algorithm>

#include "ao_derivs.cuh"
#include "kernels.cuh"
#include "tc_ptx.cuh"

namespace qb {
namespace {

constexpr int kHessRows = 12, kThreadsH = 128;
constexpr int kHessRad = 7;   // R, R1, R2, R3, displacement

// CTAs per SM: as many as the registers allow (80 a thread).  More, where small
// images left room for them, ran as a second, nearly empty wave of CTAs that
// each had as many items as the first (20,000 points x 400 AOs 0.30 ms with 7,
// 0.22 with 6).
constexpr int kHessCtas = 6;

__global__ void __launch_bounds__(kThreadsH, kHessCtas)
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

// The same with a warp per point over all its AOs, lanes on the AOs, and stores
// from registers: through the point's nucleus blocks, the lanes stage a block's
// displacements and radial parts in shared memory, then sweep its AOs.
constexpr int kWarpsH = 8;
struct HessSmem {
  double rad[kBlockSlots][4];   // R, R1, R2, R3 of the block's shells
  double nuc[kBlockNuc][4];     // displacement, r^2 (negative when screened out)
  uint8_t act[kBlockSlots];     // the shells whose nucleus is in range
};

__global__ void __launch_bounds__(kWarpsH * 32)
ao_hessian_warp_kernel(const DevTables T, const int64_t P, const double* __restrict__ coord, const double cutoff,
                       const bool fp32_exp, const double* __restrict__ cusp_r, double* __restrict__ out) {
  __shared__ HessSmem smem[kWarpsH];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  HessSmem& sm = smem[warp];
  const int64_t A = T.ao_num;
  for (int64_t p = (int64_t)blockIdx.x * kWarpsH + warp; p < P; p += (int64_t)gridDim.x * kWarpsH) {
    for (int b = 0; b < T.nblock; ++b) {
      const int4 blk = T.block[b];
      const int2 slots = T.block_slots[b];
      if (lane < blk.y - blk.x) {
        const int n = blk.x + lane, N = T.nucl_num;
        const double x = coord[p] - T.nucl_coord[n], y = coord[p + P] - T.nucl_coord[n + N],
                     z = coord[p + 2 * P] - T.nucl_coord[n + 2 * N];
        const double r2 = x * x + y * y + z * z;
        sm.nuc[lane][0] = x;
        sm.nuc[lane][1] = y;
        sm.nuc[lane][2] = z;
        sm.nuc[lane][3] = !(r2 > cutoff * T.nucleus_range[n]) ? r2 : -1.0;
      }
      __syncwarp();
      const int nlive = pack_live_slots(T.slot_nuc, blk.x, slots, sm.nuc, sm.act, lane);
      for (int i = lane; i < nlive; i += 32) {
        const int ls = sm.act[i], s = slots.x + ls;
        const double r2 = sm.nuc[T.slot_nuc[s] - blk.x][3];
        const int2 cr = T.slot_coef[s];
        double a[4] = {0., 0., 0., 0.};
        for (int j = cr.x; j < cr.y; ++j) {
          const double2 ac = T.coef_ac[j];
          const double ar2 = ac.x * r2;
          if (ar2 > cutoff) break;   // primitives are sorted by exponent
          const double e = (fp32_exp && ar2 <= 30.0) ? (double)expf(-(float)ar2) : exp(-ar2);
          const double ce = ac.y * e;
          a[0] += ce;
          a[1] -= ac.x * ce;
          a[2] += ac.x * ac.x * ce;
          a[3] -= ac.x * ac.x * ac.x * ce;
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) sm.rad[ls][c] = a[c];
      }
      __syncwarp();
      for (int k = blk.z + lane; k < blk.w; k += 32) {
        const int code = T.ao_code[k];
        const double* nc = sm.nuc[(code >> 24) & 31];
        const double* R = sm.rad[(code >> 16) & 255];
        const double r2 = nc[3];
        double g[3], H[3][3] = {{0., 0., 0.}, {0., 0., 0.}, {0., 0., 0.}}, Tl[3] = {0., 0., 0.};
        if (!(r2 < 0.0) && R[0] != 0.0 &&   // a NaN distance gives NaNs
            !cusp_masked(cusp_r, (code >> 12) & 15, blk.x + ((code >> 24) & 31), r2, false)) {
          const double v[3] = {nc[0], nc[1], nc[2]}, R3[3] = {R[0], R[1], R[2]};
          ao_derivs<double>(code, T.ao_factor[k], v, R3, 4.0 * r2 * R[2] + 6.0 * R[1], 20.0 * R[2] + 8.0 * r2 * R[3], g,
                            H, Tl);
        }
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          double* o = out + (((int64_t)d * P + p) * 4) * A + k;
          o[0] = H[d][0];
          o[A] = H[d][1];
          o[2 * A] = H[d][2];
          o[3 * A] = Tl[d];
        }
      }
      __syncwarp();
    }
  }
}

}  // namespace

// Segments of at most 256 AOs (images of 25 KB, six CTAs per SM; 320 on 600 or
// 800 AOs of s, p and d shells is the same or slower).  With shells of high
// angular momentum an item's radial parts are few, and its fixed cost counts:
// 320 (10,000 points x 914 AOs 0.30 -> 0.25 ms).  Molecules of up to 448 AOs with
// no more shells than threads in one (10,000 points x 380 AOs 0.115 -> 0.098 ms;
// 400 AOs of 180 shells are slower in one).
int hessian_segment_width(int64_t ao_num, int64_t shell_num) {
  if (ao_num <= 448 && shell_num <= kThreadsH) return (int)std::max<int64_t>(32, (ao_num + 31) / 32 * 32);
  const int64_t limit = ao_num >= 5 * shell_num ? 320 : 256;
  const int64_t n = std::max<int64_t>(1, (ao_num + limit - 1) / limit);
  return (int)std::max<int64_t>(32, ((ao_num + n - 1) / n + 31) / 32 * 32);
}

// Where a warp per point is the faster one: an image costs 4 to 7 ns per segment
// and point however few AOs it holds, a warp about 0.03 ns per AO once there are
// points for all warps.  Up to 208 AOs from 10 points per AO on (40,000 points x
// 55 AOs 84 against 171 us, x 200 AOs 199 against 213 to 271; 1,000 points x 200
// AOs 15 against 13).  With shells of high angular momentum, most of whose work
// is the AOs', up to 640 AOs from 5,000 points on (10,000 x 519 AOs 158 against
// 176 us) and any from 20,000 on (40,000 x 638 AOs 0.61 against 0.67 ms, x 914
// AOs 0.88 to 1.11 against 0.74 to 0.98).
static bool hessian_by_warps(const DevTables& T, int64_t points) {
  if (T.ao_num <= 208) return points >= std::max<int64_t>(1000, 10 * (int64_t)T.ao_num);
  if (T.ao_num < 5 * T.shell_num) return false;
  return points >= (T.ao_num <= 272 ? 10 * (int64_t)T.ao_num : T.ao_num <= 640 ? 5000 : 20000);
}

cudaError_t launch_ao_hessian(const DevTables& T, const AoSegments& g, int64_t point_num, const double* coord,
                              double cutoff, bool mixed, double* ao_hessian, cudaStream_t s, const double* cusp_r) {
  if (point_num <= 0 || T.ao_num <= 0) return cudaSuccess;
  if (hessian_by_warps(T, point_num)) {
    const int64_t grid = std::min<int64_t>((point_num + kWarpsH - 1) / kWarpsH, 148 * 8);
    ao_hessian_warp_kernel<<<(unsigned)grid, kWarpsH * 32, 0, s>>>(T, point_num, coord, cutoff, mixed, cusp_r,
                                                                   ao_hessian);
    count_launch();
    return cudaGetLastError();
  }
  const int max_shells = std::max(1, g.max_shells);
  const size_t smem = sizeof(double) * kHessRows * (size_t)(g.width + 2) + sizeof(double) * kHessRad * (size_t)max_shells +
                      sizeof(uint32_t) * 2 * (size_t)g.width + sizeof(int) * (size_t)max_shells;
  cudaError_t e = cudaFuncSetAttribute(ao_hessian_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem - 1024);
  if (e != cudaSuccess) return e;
  const int64_t per_sm = std::min<int64_t>(kHessCtas, std::max<int64_t>(1, (int64_t)(227 * 1024) / (int64_t)(smem + 2048)));
  const int64_t grid = std::min<int64_t>(point_num * g.nseg, 148 * per_sm);
  ao_hessian_kernel<<<(unsigned)grid, kThreadsH, smem, s>>>(point_num, coord, g.sh, T.coef_ac, T.ao_code, T.ao_factor,
                                                            g.seg, g.nseg, g.width, max_shells, T.ao_num, cutoff, mixed,
                                                            cusp_r, ao_hessian);
  count_launch();
  return cudaGetLastError();
}

}  // namespace qb
