// Spatial order of the points.
//
// Tiles of spatially close points share their zero AOs, which the tile
// kernels skip.  Points are put in the Morton order of the cells of a 32^3
// grid over the box of the nuclei (coordinates clamped), points of one cell in
// their own order: a stable least-significant-digit radix sort of the 15-bit
// cell codes in two passes (8 and 7 bits), so that the order, and with it
// the tiles and their sums taken in tile order (dL/dC), are the same in every
// run.
//
// The sort is bound by launches and load latencies, not by its bytes.  Up to
// kOneCta points one CTA does all of it in one launch; above it takes three: the
// digit counts of the first pass, its scatter, which also counts the second
// pass's digits, and the second scatter; every scatter CTA sums the counts of
// all for itself, so that their number is bounded (with 4096 points each, 8
// million points cost 0.65 ms more).  Kernel times: 1,920 points 8 us in one
// launch, 40,704 points 22 us in three (27 us with a count launch per pass).
// As cell counting, a one-CTA scan of the 32 K cells and an unordered scatter
// (four launches with the memset) the mixed evaluation of 1,920 points took
// 44.8 us against 31.8, the mixed value of 10,000 points of a 90-AO molecule
// 53.5 against 54.4 (57.8 with a count launch per pass), that of 40,704 points
// 91.3 against 90.4 (94.5).
#include <algorithm>

#include "kernels.cuh"
#include "mo_tc.cuh"

namespace qb {
namespace {

constexpr int kDigits = 256;
constexpr int kOneCta = 4096;
constexpr int kCtas = 64;         // CTAs of a pass, when that gives runs of kMinRun to kMaxRun points
constexpr int kMinRun = 1024, kMaxRun = 4096;
constexpr int64_t kMaxCtas = 592;   // 4 per SM

__device__ __forceinline__ unsigned int spread5(unsigned int x) {   // 5 bits -> every third bit
  x &= 31u;
  x = (x | (x << 8)) & 0x0300F00Fu;
  x = (x | (x << 4)) & 0x030C30C3u;
  x = (x | (x << 2)) & 0x09249249u;
  return x;
}

__device__ __forceinline__ unsigned int cell_code(const double* __restrict__ coord, int64_t cstride, int64_t p,
                                                  double3 origin, double inv_cell) {
  unsigned int c[3];
  const double o[3] = {origin.x, origin.y, origin.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const double v = floor((coord[p + d * cstride] - o[d]) * inv_cell);
    c[d] = (unsigned int)(int)fmin(31.0, fmax(0.0, v));
  }
  return spread5(c[0]) | (spread5(c[1]) << 1) | (spread5(c[2]) << 2);
}

// Lanes of the warp that hold the same 8-bit digit (among those that are on):
// eight ballots (match.any took several times as long on random digits).
__device__ __forceinline__ unsigned int same_digit(unsigned int d, bool on) {
  unsigned int m = __ballot_sync(0xffffffffu, on);
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const unsigned int v = __ballot_sync(0xffffffffu, (d >> b) & 1u);
    m &= ((d >> b) & 1u) ? v : ~v;
  }
  return m;
}

// A warp's items [b, e), a contiguous run of at most 32 R: the digit of item
// b + 32 r + lane in dig[r], its rank among the warp's items of that digit in
// rank[r], the digits' counts in wh.
template <int R, class Count, class Digit>
__device__ __forceinline__ void warp_ranks(int b, int e, Count* wh, int lane, Digit digit, unsigned char (&dig)[R],
                                           unsigned short (&rank)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) dig[r] = b + 32 * r + lane < e ? (unsigned char)digit(b + 32 * r + lane) : 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (b + 32 * r >= e) break;   // uniform in the warp
    const bool on = b + 32 * r + lane < e;
    const unsigned int d = dig[r], same = same_digit(d, on), before = __popc(same & ((1u << lane) - 1u));
    const unsigned int at = wh[d];
    __syncwarp();
    rank[r] = (unsigned short)(at + before);
    if (on && before == 0u) wh[d] = (Count)(at + __popc(same));
    __syncwarp();
  }
}

// wh[w][d] <- the position of the first item of digit d in warp w: the items
// of smaller digits, those of digit d in front of this CTA and those of the
// CTA's warps before w.  256 Q threads: thread (q, d) takes NW / Q warps.
// With several CTAs, thread d < 256 brings its digit's total over all of them
// and its count before these items; with one (ONE) both follow from wh.
// Returns the items of digit d in the thread's warps.
template <int NW, int Q, bool ONE, class Count>
__device__ __forceinline__ unsigned int warp_offsets(Count (*wh)[kDigits], unsigned int (*part)[kDigits], unsigned int* dsum,
                                             unsigned int all, unsigned int in_front, int tid) {
  constexpr int W = NW / Q;
  const int lane = tid & 31, warp = tid >> 5, d = tid & (kDigits - 1), q = tid / kDigits;
  unsigned int c[W], mine = 0u;
#pragma unroll
  for (int w = 0; w < W; ++w) mine += c[w] = wh[q * W + w][d];
  part[q][d] = mine;
  __syncthreads();
  if (tid < kDigits) {
    if (ONE) {
      all = 0u;
#pragma unroll
      for (int i = 0; i < Q; ++i) all += part[i][d];
      in_front = 0u;
    }
    unsigned int incl = all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) dsum[warp] = incl;
    all = incl - all + in_front;   // within the thread's 32 digits
  }
  __syncthreads();
  if (tid < kDigits) {
#pragma unroll
    for (int w = 0; w < 8; ++w)
      if (w < warp) all += dsum[w];
    // first position of each quarter's warps
#pragma unroll
    for (int i = 0; i < Q; ++i) {
      const unsigned int n = part[i][d];
      part[i][d] = all;
      all += n;
    }
  }
  __syncthreads();
  unsigned int run = part[q][d];
#pragma unroll
  for (int w = 0; w < W; ++w) {
    wh[q * W + w][d] = (Count)run;
    run += c[w];
  }
  __syncthreads();
  return mine;
}

__global__ void __launch_bounds__(1024)
order_one_kernel(const double* __restrict__ coord, const int P, const int64_t cstride, const double3 origin,
                 const double inv_cell, int* __restrict__ perm) {
  constexpr int NW = 32, R = kOneCta / (32 * NW);
  __shared__ __align__(4) unsigned short wh[NW][kDigits];   // positions below kOneCta
  __shared__ unsigned int part[4][kDigits], dsum[8];
  __shared__ unsigned short code[kOneCta], idx[kOneCta];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int seg = ((P + NW - 1) / NW + 31) / 32 * 32;
  const int b = min(P, warp * seg), e = min(P, b + seg);
  unsigned char dig[R];
  unsigned short rank[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = tid + 1024 * r;
    if (i < P) code[i] = (unsigned short)cell_code(coord, cstride, i, origin, inv_cell);
  }
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
    for (int i = 0; i < NW * kDigits / 2048; ++i) reinterpret_cast<unsigned int*>(&wh[0][0])[tid + 1024 * i] = 0u;
    __syncthreads();
    warp_ranks<R>(b, e, wh[warp], lane,
                  [&](int i) { return pass == 0 ? code[i] & 255 : code[idx[i]] >> 8; }, dig, rank);
    __syncthreads();
    warp_offsets<NW, 4, true>(wh, part, dsum, 0u, 0u, tid);
    unsigned short item[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = b + 32 * r + lane;
      if (i < e) item[r] = pass == 0 ? (unsigned short)i : idx[i];
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = b + 32 * r + lane;
      if (i >= e) continue;
      const int at = wh[warp][dig[r]] + rank[r];
      if (pass == 0) idx[at] = item[r];
      else perm[at] = item[r];
    }
    __syncthreads();
  }
}

// Cell codes, and the counts of their low digits in each CTA's run of points,
// hist[cta][256]; the counts of the second pass, taken while the first one
// scatters, are cleared.
__global__ void __launch_bounds__(256)
order_hist_kernel(const double* __restrict__ coord, const int64_t P, const int64_t cstride, const double3 origin,
                  const double inv_cell, const int64_t run, unsigned short* __restrict__ code,
                  unsigned int* __restrict__ hist, unsigned int* __restrict__ hist2) {
  __shared__ unsigned int h[kDigits];
  const int tid = threadIdx.x;
  h[tid] = 0u;
  hist2[(size_t)blockIdx.x * kDigits + tid] = 0u;
  __syncthreads();
  const int64_t b = blockIdx.x * run, e = min(P, b + run);
  for (int64_t i = b + tid; i < e; i += 256) {
    const unsigned int c = cell_code(coord, cstride, i, origin, inv_cell);
    code[i] = (unsigned short)c;
    atomicAdd(&h[c & 255u], 1u);
  }
  __syncthreads();
  hist[(size_t)blockIdx.x * kDigits + tid] = h[tid];
}

// One pass over the CTA's run, kMaxRun points at a time: their places by the
// pass's digit.  The first pass also counts the high digits of the runs that
// its points go to.
template <int PASS>
__global__ void __launch_bounds__(256)
order_scatter_kernel(const int64_t P, const int64_t run, const unsigned short* __restrict__ code,
                     const int* __restrict__ src, const unsigned int* __restrict__ hist, int* __restrict__ dst,
                     unsigned int* __restrict__ hist2) {
  constexpr int NW = 8, R = kMaxRun / (32 * NW);
  __shared__ unsigned int wh[NW][kDigits];
  __shared__ unsigned int part[1][kDigits], dsum[8];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t end = min(P, (blockIdx.x + 1) * run);
  unsigned int all = 0u, in_front = 0u;
  for (int64_t b0 = blockIdx.x * run; b0 < end; b0 += kMaxRun) {
    const int step = (int)min((int64_t)kMaxRun, run), n = (int)min((int64_t)step, end - b0), seg = step / NW;
    const int b = min(n, warp * seg), e = min(n, b + seg);
    unsigned char dig[R];
    unsigned short rank[R];
#pragma unroll
    for (int w = 0; w < NW; ++w) wh[w][tid] = 0u;
    __syncthreads();
    warp_ranks<R>(b, e, wh[warp], lane,
                  [&](int i) { return PASS == 0 ? code[b0 + i] & 255 : code[src[b0 + i]] >> 8; }, dig, rank);
    if (b0 == blockIdx.x * run) {
      for (int c0 = 0; c0 < (int)gridDim.x; c0 += 32) {
        unsigned int v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = c0 + j < (int)gridDim.x ? hist[(size_t)(c0 + j) * kDigits + tid] : 0u;
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          all += v[j];
          if (c0 + j < (int)blockIdx.x) in_front += v[j];
        }
      }
    }
    __syncthreads();
    in_front += warp_offsets<NW, 1, false>(wh, part, dsum, all, in_front, tid);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = b + 32 * r + lane;
      if (i >= e) continue;
      const unsigned int at = wh[warp][dig[r]] + rank[r];
      dst[at] = PASS == 0 ? (int)(b0 + i) : src[b0 + i];
      if (PASS == 0) atomicAdd(&hist2[(size_t)(at / (unsigned int)run) * kDigits + (code[b0 + i] >> 8)], 1u);
    }
    __syncthreads();   // wh is cleared for the next points
  }
}

size_t code_bytes(int64_t P) { return (sizeof(unsigned short) * (size_t)P + 255) / 256 * 256; }

// points per CTA of the multi-CTA passes: whole warp rounds (8 warps x 32
// points) of up to kMaxRun, then whole kMaxRuns that leave at most kMaxCtas
// CTAs, each of which reads the counts of all
int64_t order_run(int64_t P) {
  const int64_t want = (P + kCtas - 1) / kCtas;
  if (P > kMaxCtas * kMaxRun) return ((P + kMaxCtas - 1) / kMaxCtas + kMaxRun - 1) / kMaxRun * kMaxRun;
  return (std::min<int64_t>(kMaxRun, std::max<int64_t>(kMinRun, want)) + 255) / 256 * 256;
}
int64_t order_ctas(int64_t P) { return (P + order_run(P) - 1) / order_run(P); }

}  // namespace

// The count of CTAs falls where a run grows (64 at 65,536 points, 52 at
// 65,537); the two histograms get room for the most that any count up to
// point_num takes, so that scratch made for a count serves every smaller one.
size_t point_order_bytes(int64_t point_num) {
  if (point_num <= kOneCta) return 0;
  const int64_t most = std::min(kMaxCtas, std::max<int64_t>(kCtas, (point_num + kMaxRun - 1) / kMaxRun));
  return code_bytes(point_num) + 2 * sizeof(unsigned int) * kDigits * (size_t)most + sizeof(int) * (size_t)point_num;
}

cudaError_t point_order(const double* coord, int64_t point_num, const double* box_lo, const double* box_hi,
                        void* scratch, int* perm, cudaStream_t s, int64_t cstride) {
  if (cstride < point_num) cstride = point_num;
  if (point_num <= 0) return cudaSuccess;
  // 32 cells per axis over the box of the nuclei (cells at least 1 bohr wide)
  double ext = 0.0;
  for (int d = 0; d < 3; ++d) ext = std::max(ext, box_hi[d] - box_lo[d]);
  const double inv = 1.0 / std::max(1.0, ext / 32.0);
  const double3 origin = make_double3(box_lo[0], box_lo[1], box_lo[2]);
  if (point_num <= kOneCta) {
    order_one_kernel<<<1, 1024, 0, s>>>(coord, (int)point_num, cstride, origin, inv, perm);
    count_launch();
    return cudaGetLastError();
  }
  unsigned short* code = (unsigned short*)scratch;
  unsigned int* hist = (unsigned int*)((uint8_t*)scratch + code_bytes(point_num));
  const int64_t run = order_run(point_num);
  const unsigned ctas = (unsigned)order_ctas(point_num);
  unsigned int* hist2 = hist + (size_t)ctas * kDigits;
  int* mid = (int*)(hist2 + (size_t)ctas * kDigits);
  order_hist_kernel<<<ctas, 256, 0, s>>>(coord, point_num, cstride, origin, inv, run, code, hist, hist2);
  order_scatter_kernel<0><<<ctas, 256, 0, s>>>(point_num, run, code, nullptr, hist, mid, hist2);
  order_scatter_kernel<1><<<ctas, 256, 0, s>>>(point_num, run, code, mid, hist2, perm, nullptr);
  count_launch(3);
  return cudaGetLastError();
}

}  // namespace qb
