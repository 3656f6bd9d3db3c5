// Device-side tables and kernel launchers of the orbital-evaluation path.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace qb {

// Limits of the per-warp shared-memory staging in the AO kernels.  A nucleus
// block holds at most kBlockNuc nuclei and kBlockSlots shells; finalization
// rejects a basis with more than kBlockSlots shells on one nucleus.
constexpr int kBlockNuc = 32;
constexpr int kBlockSlots = 64;

// Basis tables in device memory (one allocation; see device.cu).
//
// Nuclei are grouped into blocks of consecutive nuclei.  A block's AOs are
// contiguous ([ao_begin, ao_end)) because AOs are numbered nucleus by nucleus.
// The block's shells are its "slots" (block-local shell numbering) and each AO
// carries its slot, its block-local nucleus and its cartesian powers.
struct DevTables {
  int32_t nucl_num, shell_num, prim_num, ao_num, nblock, nslot;
  int32_t shell_parts;            // parts of a shell that separate warps take: 4 with shells of l >= 4, else 1
  const double* nucl_coord;       // [3][nucl]
  const double* nucleus_range;    // [nucl]
  const int32_t* nuc_prim_start;  // [nucl+1] into expo (sorted, de-duplicated per nucleus)
  const double* expo;             // [sum of unique primitives]
  const int4* block;              // [nblock] (nuc_begin, nuc_end, ao_begin, ao_end)
  const int2* block_slots;        // [nblock] (slot_begin, slot_end)
  const int32_t* slot_nuc;        // [nslot] global nucleus of a slot
  const int2* slot_coef;          // [nslot] (begin, end) into coef_prim / coef_val
  const int32_t* coef_prim;       // nucleus-local index of the sorted primitive
  const double* coef_val;         // normalized, merged coefficient
  const int32_t* ao_code;         // [ao] a | b<<4 | c<<8 | l<<12 | slot<<16 | nuc_local<<24
  const double* ao_factor;        // [ao]
  // tables of the primitive / shell getters (unsorted, as set by the user)
  const int32_t* prim_nuc;        // [prim]
  const double* prim_expo;        // [prim]
  const double* prim_coef;        // [prim] normalized coefficient
  const int32_t* shell_nuc;       // [shell]
  const int2* shell_prims;        // [shell] (prim_begin, prim_end)
  // tables of the fused AO -> MO kernel (global shell numbering)
  const int32_t* ao_shell;        // [ao] shell of each AO
  const int2* shell_coef;         // [shell] (begin, end) into coef_prim / coef_val
  const double2* coef_ac;         // [coefficient entry] (exponent, coefficient): coef_val with its exponent
};

// Global count of kernels launched by this library.
void count_launch(int n = 1);

// Cusp adjustment of the MOs (org/qmckl_mo.org:2839, 3133, 2659): the s AOs
// of a nucleus are left out of the MO sums at points closer to it than its
// radius cusp_r[nucl] (strictly for MO values, r <= r_cusp for the VGL and the
// Hessian).  r2 < 0 marks a nucleus screened out (its AOs vanish anyway).
__device__ __forceinline__ bool cusp_masked(const double* cusp_r, int l, int nucl, double r2, bool strict) {
  if (cusp_r == nullptr || l != 0 || r2 < 0.0) return false;
  const double r = sqrt(r2), R = cusp_r[nucl];
  return strict ? (r < R) : (r <= R);
}

// Whole warp: the positions (relative to slots.x) of a nucleus block's shells
// whose nucleus is in range of the point (nuc[.][3] not negative), packed in slot
// order into act; returns their count.  The radial staging then runs over
// the live shells only, in as few 32-lane passes as they need.
__device__ __forceinline__ int pack_live_slots(const int32_t* __restrict__ slot_nuc, int blk_first, int2 slots,
                                               const double (*nuc)[4], uint8_t* act, int lane) {
  int n = 0;
  for (int s0 = slots.x; s0 < slots.y; s0 += 32) {
    const int s = s0 + lane;
    const bool live = s < slots.y && !(nuc[slot_nuc[s] - blk_first][3] < 0.0);
    const unsigned int m = __ballot_sync(0xffffffffu, live);
    if (live) act[n + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(s - slots.x);
    n += __popc(m);
  }
  __syncwarp();
  return n;
}

// A block's most shared memory.  A kernel whose dynamic shared memory differs
// from call to call is opted in to all of it (less its static part), never to a
// call's size: the attribute belongs to the kernel, and another thread's
// smaller call could lower it between a call's opt-in and its launch.
constexpr int kMaxSmem = 232448;

// AO kernels (ao_kernels.cu).  coord is [3][point_num].  All return
// cudaGetLastError() after the launch.
// cusp_r (optional, [nucl]): the AOs that the cusp adjustment leaves out of
// the MO sums are written as zero (the arrays then only feed the MO step).
cudaError_t launch_ao_vgl_f64(const DevTables& T, int64_t point_num, const double* coord,
                              double cutoff, bool dp_exp, double* ao_vgl, cudaStream_t s,
                              const double* cusp_r = nullptr);
cudaError_t launch_ao_value_f64(const DevTables& T, int64_t point_num, const double* coord,
                                double cutoff, bool dp_exp, double* ao_value, cudaStream_t s,
                                const double* cusp_r = nullptr);
// The same FP64 AO VGL stored as 3 bfloat16 pieces (split.cuh) of rows
// p*5 + c: pieces[q * pstride + row * lda + ao] (lda, pstride multiples of 8).
cudaError_t launch_ao_vgl_pieces(const DevTables& T, int64_t point_num, const double* coord, double cutoff,
                                 bool dp_exp, void* pieces, int64_t lda, int64_t pstride, cudaStream_t s);
// AO Hessian (ao_hessian.cu): the shell records and segments of `width` =
// hessian_segment_width AOs, the shells [seg.x, seg.y) with AOs in
// each; at most max_shells of them.
struct F64Shell;
struct AoSegments {
  const F64Shell* sh;
  const int2* seg;
  int nseg, width, max_shells;
};
int hessian_segment_width(int64_t ao_num, int64_t shell_num);
// ao_hessian [3][point_num][4][ao]; `mixed`: FP32 exponentials where a r^2 <= 30.
cudaError_t launch_ao_hessian(const DevTables& T, const AoSegments& g, int64_t point_num, const double* coord,
                              double cutoff, bool mixed, double* ao_hessian, cudaStream_t s,
                              const double* cusp_r = nullptr);
// Cusp adjustment (cusp.cu, org/qmckl_mo.org:2807-2860, 3099-3185,
// 2629-2697): adds, for every nucleus closer to a point than its radius, the
// cubic c0 + c1 r + c2 r^2 + c3 r^3 (prm [nucl][4][mo]) to the point's MO
// values (comps 1, r <= r_cusp) or its value, gradient and Laplacian
// (comps 5, r < r_cusp) in out[point][comps][mo]; its Hessian to
// out[3][point][3][mo].  coord [3][cstride].
cudaError_t launch_cusp_mo(int64_t P, int comps, const double* coord, int64_t cstride, int N, const double* nucl,
                           const double* r_cusp, const double* prm, int M, double* out, cudaStream_t s);
cudaError_t launch_cusp_hessian(int64_t P, const double* coord, int N, const double* nucl, const double* r_cusp,
                                const double* prm, int M, double* out, cudaStream_t s);
// en_distance[point][nucl] (org/qmckl_electron.org:1357-1393)
cudaError_t launch_en_distance(int64_t P, const double* coord, int N, const double* nucl, double* out,
                               cudaStream_t s);
cudaError_t launch_primitive_vgl(const DevTables& T, int64_t point_num, const double* coord,
                                 double cutoff, double* prim_vgl, cudaStream_t s);
cudaError_t launch_shell_vgl(const DevTables& T, int64_t point_num, const double* coord,
                             double cutoff, double* shell_vgl, cudaStream_t s);

// Mixed-form AO kernel: writes the AO matrix A[(point,comp)][k] as `pieces`
// bfloat16 matrices (A = sum of pieces), each [5*point_num][lda], lda >= ao_num,
// pieces at stride piece_stride elements.
cudaError_t launch_ao_vgl_split(const DevTables& T, int64_t point_num, const double* coord,
                                double cutoff, int pieces, void* a_pieces, int64_t lda,
                                int64_t piece_stride, cudaStream_t s);

// FP64 GEMM C[M][N] = A[M][K] * B[K][N], row-major with leading dimensions (gemm_f64.cu).
cudaError_t launch_gemm_f64(int64_t M, int64_t N, int64_t K, const double* A, int64_t lda,
                            const double* B, int64_t ldb, double* C, int64_t ldc, cudaStream_t s);

// Tile-sparse FP64 MO evaluation (f64_tiles.cu).  One record per shell: its
// nucleus and the squared radius beyond which its AOs are exact zeros
// (r2max, negative: no primitives), the nucleus screening bound
// cutoff * range, its AOs [a0, a0 + na), its (exponent, coefficient) entries
// [cb, ce) of DevTables::coef_ac, its angular momentum and nucleus.
struct F64Shell {
  double x, y, z, r2max, crange;
  int32_t a0, na, cb, ce, l, nucl;
};
// The nuclei's positions (T.nucl_coord) into the records of T.shell_num shells.
cudaError_t launch_place_shells(const DevTables& T, F64Shell* sh, cudaStream_t s);
// Compact tiles of pts = f64_tile_points points each, f64_tile_bytes per
// tile: ac[tile][ao_num][comps * pts + 4] (the first kcount[tile] rows hold
// the tile's live AOs klist[tile][.]).
// For the adjoint also: inv[tile][ao_num], the list position of each AO
// (preset to -1; may be null); live[tile][shell_num], the live shells (shell,
// first list position), nlive[tile] of them; bad[tile], the points of the tile
// (bits) with a loss weight that is not finite, set by the kernels that lay
// out the weights after launch_ao_tiles has cleared it.  Such a weight times
// an AO that is exactly zero is a NaN of dL/dC, dL/dR and dL/dr, also where the
// AO is in no list.  share: deriv_share_bytes, the shares of dL/dr of the CTAs
// that share a tile.
struct AdjTables {
  int* inv;
  int2* live;
  int* nlive;
  unsigned int* bad;
  double* share;
};
size_t deriv_share_bytes(int64_t ntiles);
struct F64Tiles {
  int pts;
  double* ac;
  int* klist;
  int* kcount;
  AdjTables adj;
};
int f64_tile_points(int comps, int64_t P);
size_t f64_tile_bytes(int comps, int pts, int64_t ao_num);
F64Tiles f64_tiles_at(void* scratch, int64_t ntiles, int comps, int pts, int64_t ao_num);
// The AO tiles (or, with t.ac null, only their lists) [tile0, tile0 + ntiles) of
// the points in the order perm
// (null: as they are), coord [3][cstride]; cusp_r as in launch_ao_vgl_f64.
cudaError_t launch_ao_tiles(const DevTables& T, int64_t P, int comps, const double* coord, int64_t cstride,
                            const int* perm, int64_t tile0, int64_t ntiles, const F64Shell* sh, double cutoff,
                            bool dp_exp, const double* cusp_r, const F64Tiles& t, cudaStream_t s);
// C[point][comps][N] of those tiles' points = AO tile * Bt (coefficient_t
// with ldb even and 16-byte aligned rows).
cudaError_t launch_tile_gemm(int64_t P, int comps, int64_t tile0, int64_t ntiles, int64_t N, int64_t ao_num,
                             const F64Tiles& t, const int* perm, const double* Bt, int64_t ldb, double* C,
                             cudaStream_t s);

// FP64 adjoint of the MO VGL over compact VGL tiles (f64_tiles.cu,
// adjoint.cu) with their AdjTables.
// Weights in tile order: ws[tile][c * 32 + p][ldw], ldw even; bad as AdjTables.
cudaError_t launch_weight_tiles(int64_t P, int64_t tile0, int64_t ntiles, const double* w, int64_t M, const int* perm,
                                double* ws, int64_t ldw, unsigned int* bad, cudaStream_t s);
// grad[mo][ao] (+)= AO^T W of the tiles; part [ntiles][ao_num][ldw].
cudaError_t launch_adj_coef(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws, int64_t ldw,
                            double* part, double* grad, bool accumulate, cudaStream_t s);
// t.ac <- W C, the weights pulled back to the tiles' AOs (Ct: coefficient_t
// with ldc even, zero past the MOs).
cudaError_t launch_adj_pullback(int64_t ntiles, int64_t ao_num, int64_t M, const F64Tiles& t, const double* ws,
                                int64_t ldw, const double* Ct, int64_t ldc, cudaStream_t s);
// grad_nucl [nucl][3] -= and grad_coord [3][gstride] =, either
// may be null, from the pulled-back weights g of the tiles' listed AOs (all AOs
// where adj.live is null): FP64
// [tile][ao_num][164], or (mixed) FP32 [tile][ao_num][160] with FP32
// exponentials where a r^2 <= 30 and FP32 per-AO derivative arithmetic.
cudaError_t launch_tile_deriv(const DevTables& T, int64_t P, const double* coord, int64_t cstride, const int* perm,
                              int64_t tile0, int64_t ntiles, const F64Shell* sh, double cutoff, const AdjTables& adj,
                              const void* g, bool mixed, double* grad_nucl, double* grad_coord, int64_t gstride,
                              cudaStream_t s);

// out[n][m] = (out[n][m] +) sum_z part[z][m][n]  (fixed summation order)
cudaError_t launch_add_transposed(const double* part, int splits, int64_t M, int64_t N, double* out, bool accumulate,
                                  cudaStream_t s);

// Orbital forces (adjoint.cu): which = 0 forces_mo_value, 1 forces_mo_g,
// 2 forces_mo_l (from X = ao_vgl for 0, ao_hessian for 1 and 2, and
// Ct = coefficient_t [ao][mo]), 3 forces_ao_value (from X = ao_vgl).
// nuc_ao[a] = AO range of nucleus a.
cudaError_t launch_forces(int which, int64_t P, int64_t A, int64_t M, int N, const int2* nuc_ao, const double* X,
                          const double* Ct, double* out, cudaStream_t s);

}  // namespace qb
