// Large-front kernels (fronts with more than 96 rows), 64-column blocks.
//
// Factorization, per block J = [j0, j0+w) of a front (right-looking):
//   k_gather8   extend-add of the children's updates (once per level);
//   k_panel64   every CTA factors the w x w diagonal block with the blocked
//               dense routine (cta_ldlt, which also forms L_JJ^-1); CTA 0
//               stores the factored block (dcache) and L_JJ^-1 (the inverse-
//               block cache, reused by the selected inverse); each CTA forms
//               its 64 rows L_i = F_i L_JJ^-T D_J^-1 as one tensor-core GEMM
//               (or one CTA per front factors the block and k_rows64 forms the
//               rows; or k_diag_next factors it while step J - 1 is in work);
//   update      F[i,j] -= sum_{t in J} L_it d_t L_jt on 64x64 tiles of the lower
//               trailing matrix (tensor-core tiles, operands staged with cp.async;
//               update64w8_body in snode_persist.cuh, launched as k_update64w8).
// Selected inverse: matrix products over the whole front (k_si_gemm).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "dense_ldlt.cuh"
#include "devsym.hpp"

namespace inla {
namespace {

constexpr int kB64 = 64;         // block-column width
constexpr int kPanelRows = 64;   // rows per panel GEMM sub-block
constexpr int kLd64 = dense_ld(kB64);
constexpr int kULd64 = dense_uld(kB64);
constexpr int kPanelSmem = (2 * kB64 * kLd64 + 8 * kULd64 + kDenseScratch) * 8;
constexpr int kSiStages = 2, kSiCtas = 3;
constexpr int kSiGemmSmem = kSiStages * 64 * kLd64 * 8;  // stage buffers

__device__ __forceinline__ int lg_k(const DevSym& S, int s) { return S.first[s + 1] - S.first[s]; }
__device__ __forceinline__ int lg_m(const DevSym& S, int s) { return S.rowptr[s + 1] - S.rowptr[s]; }

__device__ __forceinline__ void mma884(double& c0, double& c1, double a, double b) { dmma884(c0, c1, a, b); }

__device__ __forceinline__ const double* linv_block(const DevSym& S, const double* linv, int b, int s, int blk) {
  return linv + (int64_t)b * S.lstride + ((int64_t)S.lbo[s] + blk) * (kB64 * kB64);
}

// Extend-add of the children's updates into parent columns [c0, c1) (gcols columns per CTA, at most
// kGatherCols, fewer when the slice would not fit): every warp assembles columns of its own in shared
// memory (panel columns start from the filled values, update columns from zero), adds the children's
// columns that fall on it in child order (targets are distinct within one child, so an entry's sum has a
// fixed order) and writes the column's lower part back once. No warp waits for another. A host table
// lists these columns (DevSym::gcol), 32 read at a time, one per lane, so a child without the column
// costs nothing and there is one dependent load between the list and the values. What bounds it is the
// latency of the loads: eight per lane are in flight, of one long column or of up to eight short ones.
// Measured (one child after the other for the whole CTA, two barriers each -> a warp per column searching
// every child's range -> lists and eight pieces): level launches of SPDE 200^2 at B = 10 1.20 -> 1.12 ->
// 0.70 ms, at B = 30 3.40 -> 2.58 -> 2.00 ms. Fronts of the grouped model 24x24x14 have 20 to 324 iid
// children (B = 2): persistent factorization 2.72 -> 1.69 ms before the lists.
constexpr int kGatherCols = 8;

__device__ __forceinline__ GatherCol gather_shfl(const GatherCol& d, int lane) {
  GatherCol r;
  r.src = __shfl_sync(0xffffffffu, d.src, lane);
  r.len = __shfl_sync(0xffffffffu, d.len, lane);
  r.rel = __shfl_sync(0xffffffffu, d.rel, lane);
  return r;
}

// One warp: column `col` of front s (ld m) of problem b in g[0 .. m).
__device__ __forceinline__ void gather_column(const DevSym& S, int s, double* Fb, double* Fs, int k, int m, int col,
                                              double* g) {
  const int lane = threadIdx.x & 31;
  for (int row = col + lane; row < m; row += 32) {
    if (col < k) cp_async8(&g[row], Fs + row + (int64_t)col * m);
    else g[row] = 0.0;
  }
  cp_async_commit();
  const int row0 = S.rowptr[s] + col, e0 = S.rsp[row0], n = S.rsp[row0 + 1] - e0;
  const GatherCol* list = S.gcol + S.gptr[s] + e0;
  bool ready = false;  // the panel values have landed
  auto settle = [&] {
    if (!ready) cp_async_wait<0>();
    ready = true;
    __syncwarp();
  };
  for (int qb = 0; qb < n; qb += 32) {
    const GatherCol mine = qb + lane < n ? list[qb + lane] : GatherCol{0, 0, 0};
    const int cnt = min(32, n - qb);
    GatherCol d = gather_shfl(mine, 0);
    for (int at = 0, off = lane; at < cnt;) {  // 32 rows of a column at a time, eight such pieces in flight
      double v[8];
      int dst[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        dst[u] = -1;
        if (at >= cnt) continue;
        if (off < d.len) {
          v[u] = Fb[d.src + off];
          dst[u] = S.relx[d.rel + off];
        }
        off += 32;
        if (off - lane >= d.len) {
          off = lane;
          if (++at < cnt) d = gather_shfl(mine, at);
        }
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        settle();
        if (dst[u] >= 0) g[dst[u]] += v[u];
      }
    }
  }
  settle();
  for (int row = col + lane; row < m; row += 32) Fs[row + (int64_t)col * m] = g[row];
}

// Chunk z of front s, problem b (any block size; gsl: [gcols][m] doubles of shared memory).
__device__ __forceinline__ void gather8_body(const DevSym& S, int s, int b, int z, double* __restrict__ F,
                                             int64_t fstride, int gcols, double* gsl) {
  if (front_skipped(S, s, b)) return;
  const int k = lg_k(S, s), m = lg_m(S, s);
  const int c0 = z * gcols;
  if (c0 >= m) return;
  const int c1 = min(c0 + gcols, m);
  double* Fb = F + (int64_t)b * fstride;
  for (int cc = threadIdx.x >> 5; cc < c1 - c0; cc += blockDim.x >> 5)
    gather_column(S, s, Fb, Fb + S.fptr[s], k, m, c0 + cc, gsl + (int64_t)cc * m);
}

// 48 registers, five CTAs per SM: SPDE 200^2 at B = 10 / 30 0.70 / 2.00 ms per factorization (four CTAs
// 0.76 / 2.16, six with spills 0.79 / 2.22).
__global__ void __launch_bounds__(256, 5) k_gather8(DevSym S, const int* __restrict__ list, double* __restrict__ F,
                                                 int64_t fstride, int gcols) {
  extern __shared__ double gsl[];  // [gcols][m] column slice
  gather8_body(S, list[blockIdx.x], blockIdx.y, blockIdx.z, F, fstride, gcols, gsl);
}

// Sigma restricted to the below-rows of s, gathered from the parent's Sigma
// front into the trailing block (lower triangle), columns [c0, c1) of it.
__device__ __forceinline__ void si_gather8_body(const DevSym& S, int s, int b, int z, double* __restrict__ Sg,
                                                int64_t fstride) {
  const int k = lg_k(S, s), m = lg_m(S, s), r = m - k;
  if (r == 0) return;
  const int c0 = z * kGatherCols;
  if (c0 >= r) return;
  const int c1 = min(c0 + kGatherCols, r);
  const int p = S.parent[s];
  const int mp = lg_m(S, p);
  const double* __restrict__ Sp = Sg + (int64_t)b * fstride + S.fptr[p];
  double* Ss = Sg + (int64_t)b * fstride + S.fptr[s];
  const int* __restrict__ rel = S.relx + S.rowptr[s] + k;
  const int total = (c1 - c0) * r;
  int e = threadIdx.x;
  for (; e + 3 * (int)blockDim.x < total; e += 4 * blockDim.x) {
    double v[4];
    int64_t dst[4];
    bool ok[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int ee = e + u * blockDim.x;
      const int jj = c0 + ee / r, ii = ee - (ee / r) * r;
      ok[u] = ii >= jj;
      const int pi = ok[u] ? rel[ii] : 0, pj = ok[u] ? rel[jj] : 0;
      v[u] = ok[u] ? (pi >= pj ? Sp[pi + (int64_t)pj * mp] : Sp[pj + (int64_t)pi * mp]) : 0.0;
      dst[u] = (k + ii) + (int64_t)(k + jj) * m;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (ok[u]) Ss[dst[u]] = v[u];
  }
  for (; e < total; e += blockDim.x) {
    const int jj = c0 + e / r, ii = e - (e / r) * r;
    if (ii < jj) continue;
    const int pi = rel[ii], pj = rel[jj];
    Ss[(k + ii) + (int64_t)(k + jj) * m] = pi >= pj ? Sp[pi + (int64_t)pj * mp] : Sp[pj + (int64_t)pi * mp];
  }
}

__global__ void __launch_bounds__(256) k_si_gather8(DevSym S, const int* __restrict__ list, double* __restrict__ Sg,
                                                    int64_t fstride) {
  si_gather8_body(S, list[blockIdx.x], blockIdx.y, blockIdx.z, Sg, fstride);
}

// The factored diagonal block goes to dcache[(list index, problem)] (written by
// CTA 0): the other CTAs of this launch still read the unfactored block from
// the front, so it is copied into the front by the trailing update (tile 0) of the same step.
// Each CTA: blocked LDL^T + inverse of the diagonal block, then the rows
// [r0, r0 + rpc) (rpc a multiple of 64) in 64-row sub-blocks, each
// X = F_rows (L_JJ^-T D^-1) as one tensor-core GEMM. The row sub-blocks are
// staged in the diagonal block's buffer once it is no longer needed, which
// keeps the CTA at 84 KB of shared memory (two CTAs per SM).
// Block J = [j0, j0 + 64) of front s, problem b, row CTA z (256 threads). dc: this front's and
// problem's slot of the factored-diagonal-block cache (written when z == 0), or nullptr in the chain
// form (one CTA per front and problem, rpc = 0), which writes the factored block into the front.
__device__ __forceinline__ void panel64_body(const DevSym& S, int s, int b, int z, int j0, int rpc,
                                             double* __restrict__ F, int64_t fstride, double* __restrict__ dc,
                                             double* __restrict__ linv, double* smem64) {
  constexpr int ld = kLd64;  if (front_skipped(S, s, b)) return;

  double* Ds = smem64;         // [64 cols][ld]: diagonal block, factored in place; then row sub-blocks
  double* Li = Ds + kB64 * ld; // L_JJ^-1, then Bm[u + t*ld] = Li[t][u] / d_t
  double* U = Li + kB64 * ld;  // [8][kULd64] scratch of cta_ldlt, then 1 / d_t
  double* ws = U + 8 * kULd64;
  const int k = lg_k(S, s), m = lg_m(S, s);
  if (j0 >= k) return;
  const int w = min(kB64, k - j0);
  const int r0 = j0 + w + z * rpc;
  if (z > 0 && r0 >= m) return;
  const int r1 = min(m, r0 + rpc);
  double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  const double* D0 = Fs + j0 + (int64_t)j0 * m;
  for (int e = threadIdx.x; e < kB64 * kB64; e += blockDim.x) {
    const int c = e >> 6, r = e & 63;
    if (r < w && c < w && r >= c) cp_async8(&Ds[r + c * ld], D0 + r + (int64_t)c * m);
    else Ds[r + c * ld] = 0.0;
    Li[r + c * ld] = 0.0;
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  cta_ldlt<true>(Ds, ld, w, w, Li, ld, U, kULd64, ws);
  if (z == 0) {
    double* lc = const_cast<double*>(linv_block(S, linv, b, s, j0 / kB64));
    for (int e = threadIdx.x; e < kB64 * kB64; e += blockDim.x) {
      const int c = e >> 6, r = e & 63;
      lc[e] = Li[r + c * ld];  // zero outside the w x w lower triangle
      if (dc) dc[e] = (r < w && c < w) ? Ds[r + c * ld] : 0.0;
      else if (r < w && c < w && r >= c) Fs[(j0 + r) + (int64_t)(j0 + c) * m] = Ds[r + c * ld];
    }
    // chain form: the next diagonal block's task reads the unscaled rows from their mirror position
    // while the row tasks scale them in place
    if (!dc && j0 + kB64 < k)
      for (int e = threadIdx.x; e < kB64 * kB64; e += blockDim.x) {
        const int c = e & 63, r = e >> 6, i = j0 + kB64 + r;
        if (i < m) Fs[(j0 + c) + (int64_t)i * m] = Fs[i + (int64_t)(j0 + c) * m];
      }
  }
  if (r0 >= r1) return;
  double* dinv = U;
  if (threadIdx.x < kB64) dinv[threadIdx.x] = threadIdx.x < w ? 1.0 / Ds[threadIdx.x * (ld + 1)] : 0.0;
  __syncthreads();
  double bv[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int e = threadIdx.x + 256 * q, u = e & 63, t = e >> 6;
    bv[q] = Li[t + u * ld] * dinv[t];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int e = threadIdx.x + 256 * q, u = e & 63, t = e >> 6;
    Li[u + t * ld] = bv[q];
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wr = (warp & 1) * 32, wc = (warp >> 1) * 16;
  const int g = lane >> 2, tg = lane & 3;
  const int wk = (w + 3) & ~3;
  double* Fa = Ds;  // row sub-block: Fa[t*ld + r] = F[rb + r, j0 + t]
  for (int rb = r0; rb < r1; rb += kPanelRows) {
    const int rows = min(kPanelRows, r1 - rb);
    __syncthreads();  // previous sub-block (or the diagonal block) fully consumed
    for (int e = threadIdx.x; e < kB64 * kPanelRows; e += blockDim.x) {
      const int c = e >> 6, r = e & 63;
      if (r < rows && c < w) cp_async8(&Fa[c * ld + r], Fs + (rb + r) + (int64_t)(j0 + c) * m);
      else Fa[c * ld + r] = 0.0;
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    // X (64 x 64) = Fa (64 x w) * Bm (w x 64); warp tile 32 x 16
    double acc[4][2][2];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q) acc[a][q][0] = acc[a][q][1] = 0.0;
#pragma unroll 4
    for (int kk = 0; kk < wk; kk += 4) {
      double af[4], bf[2];
#pragma unroll
      for (int a = 0; a < 4; ++a) af[a] = Fa[(kk + tg) * ld + wr + a * 8 + g];
#pragma unroll
      for (int q = 0; q < 2; ++q) bf[q] = Li[(kk + tg) + (wc + q * 8 + g) * ld];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int q = 0; q < 2; ++q) mma884(acc[a][q][0], acc[a][q][1], af[a], bf[q]);
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int r = wr + a * 8 + g, t = wc + q * 8 + tg * 2 + h;
          if (r < rows && t < w) Fs[(rb + r) + (int64_t)(j0 + t) * m] = acc[a][q][h];
        }
  }
}

__global__ void __launch_bounds__(256, 2) k_panel64(DevSym S, const int* __restrict__ list, int j0, int rpc,
                                                 double* __restrict__ F, int64_t fstride,
                                                 double* __restrict__ dcache, double* __restrict__ linv) {
  extern __shared__ double smem64[];
  double* dc = dcache ? dcache + ((int64_t)blockIdx.x * gridDim.y + blockIdx.y) * (kB64 * kB64) : nullptr;
  panel64_body(S, list[blockIdx.x], blockIdx.y, blockIdx.z, j0, rpc, F, fstride, dc, linv, smem64);
}

// Rows of a 64-column block from this step's factored diagonal block (dcache:
// L_JJ with D on the diagonal, written by k_panel64 launched with rpc = 0;
// linv: L_JJ^-1): X = F_rows L_JJ^-T D^-1 for the 64 rows of CTA z, one
// tensor-core GEMM. Used when many fronts x problems share a step, where a
// factorization per row CTA would be redundant work.
constexpr int kRowsSmem = (2 * kB64 * kLd64 + kB64) * 8;
// Row block z of block J of front s, problem b (256 threads); dc as in panel64_body (nullptr: D is
// read from the front).
__device__ __forceinline__ void rows64_body(const DevSym& S, int s, int b, int z, int j0, double* __restrict__ F,
                                            int64_t fstride, const double* __restrict__ dc,
                                            const double* __restrict__ linv, double* smr) {
  if (front_skipped(S, s, b)) return;
  constexpr int ld = kLd64;
  double* Bm = smr;               // Bm[u + t*ld] = L_JJ^-1[t][u] / d_t
  double* Fa = Bm + kB64 * ld;    // Fa[t*ld + r] = F[r0 + r, j0 + t]
  double* dinv = Fa + kB64 * ld;  // [kB64]
  const int k = lg_k(S, s), m = lg_m(S, s);
  if (j0 >= k) return;
  const int w = min(kB64, k - j0);
  const int r0 = j0 + w + z * kPanelRows;
  if (r0 >= m) return;
  const int rows = min(kPanelRows, m - r0);
  double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  for (int e = threadIdx.x; e < kB64 * kPanelRows; e += blockDim.x) {
    const int c = e >> 6, r = e & 63;
    if (r < rows && c < w) cp_async8(&Fa[c * ld + r], Fs + (r0 + r) + (int64_t)(j0 + c) * m);
    else Fa[c * ld + r] = 0.0;
  }
  cp_async_commit();
  const double* lc = linv_block(S, linv, b, s, j0 / kB64);
  const double* dg = dc ? dc : Fs + j0 + (int64_t)j0 * m;  // d_t at dg[t * ds]
  const int64_t ds = dc ? kB64 + 1 : m + 1;
  if (threadIdx.x < kB64) dinv[threadIdx.x] = threadIdx.x < w ? 1.0 / dg[threadIdx.x * ds] : 0.0;
  __syncthreads();
  double lv[16];
#pragma unroll
  for (int q = 0; q < 16; ++q) lv[q] = lc[threadIdx.x + 256 * q];  // L_JJ^-1 column-major: (t, u) at t + 64 u
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int e = threadIdx.x + 256 * q, t = e & 63, u = e >> 6;
    Bm[u + t * ld] = lv[q] * dinv[t];
  }
  cp_async_wait<0>();
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wr = (warp & 1) * 32, wc = (warp >> 1) * 16;
  const int g = lane >> 2, tg = lane & 3;
  const int wk = (wr >= rows || wc >= w) ? 0 : (w + 3) & ~3;
  double acc[4][2][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[a][q][0] = acc[a][q][1] = 0.0;
#pragma unroll 4
  for (int kk = 0; kk < wk; kk += 4) {
    double af[4], bf[2];
#pragma unroll
    for (int a = 0; a < 4; ++a) af[a] = Fa[(kk + tg) * ld + wr + a * 8 + g];
#pragma unroll
    for (int q = 0; q < 2; ++q) bf[q] = Bm[(kk + tg) + (wc + q * 8 + g) * ld];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q) mma884(acc[a][q][0], acc[a][q][1], af[a], bf[q]);
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = wr + a * 8 + g, t = wc + q * 8 + tg * 2 + h;
        if (r < rows && t < w) Fs[(r0 + r) + (int64_t)(j0 + t) * m] = acc[a][q][h];
      }
}

__global__ void __launch_bounds__(256) k_rows64(DevSym S, const int* __restrict__ list, int j0,
                                                double* __restrict__ F, int64_t fstride,
                                                const double* __restrict__ dcache, const double* __restrict__ linv) {
  extern __shared__ double smr[];
  const double* dc = dcache ? dcache + ((int64_t)blockIdx.x * gridDim.y + blockIdx.y) * (kB64 * kB64) : nullptr;
  rows64_body(S, list[blockIdx.x], blockIdx.y, blockIdx.z, j0, F, fstride, dc, linv, smr);
}

constexpr int kUT64 = 64;

// ---------------------------------------------------------------------------
// triangular sweeps in 32-column blocks: the diagonal block is solved by one
// warp with shuffles, the rows below it are updated by the whole CTA
// (two barriers per block instead of one per column)
// ---------------------------------------------------------------------------

// v plus the children's update entries of front row `row` (of the concatenated structures), in child
// order, eight loads in flight. One child after the other for the whole CTA, a barrier each, cost a
// memory latency per child: fronts of grouped models have 20 to 324 of them (persistent solve of the
// group model 24x24x14, B = 2: 1.30 -> 0.51 ms).
__device__ __forceinline__ double fwd_row_start(const DevSym& S, int row, const double* __restrict__ ub, double v) {
  int q = S.rsp[row];
  const int e = S.rsp[row + 1];
  for (; q + 8 <= e; q += 8) {
    double u[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) u[i] = ub[S.rss[q + i]];
#pragma unroll
    for (int i = 0; i < 8; ++i) v += u[i];
  }
  for (; q < e; ++q) v += ub[S.rss[q]];
  return v;
}

// Forward sweep of front s, problem b (NT threads; y: m + 2 + 32 * 33 doubles of shared memory).
template <int NT>
__device__ __forceinline__ void fwd32_body(const DevSym& S, int s, int b, const double* __restrict__ F,
                                           int64_t fstride, double* __restrict__ xp, double* __restrict__ ub,
                                           int64_t ustride, double* y) {
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  double* ubb = ub + (int64_t)b * ustride;
  for (int t = threadIdx.x; t < m; t += NT)
    y[t] = fwd_row_start(S, S.rowptr[s] + t, ubb, t < k ? xb[f + t] : 0.0);
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Ls = y + ((m + 1) & ~1);  // [32][33] strictly lower part of the block's diagonal tile
  for (int jb = 0; jb < k; jb += 32) {
    const int wb = min(32, k - jb);
    for (int e = threadIdx.x; e < 32 * 32; e += NT) {
      const int r = e & 31, c = e >> 5;
      Ls[r * 33 + c] = (c < r && r < wb) ? Fs[(jb + r) + (int64_t)(jb + c) * m] : 0.0;
    }
    __syncthreads();
    if (warp == 0) {
      double yi = lane < wb ? y[jb + lane] : 0.0;
#pragma unroll 8
      for (int j = 0; j < 32; ++j) {
        const double yj = __shfl_sync(0xffffffffu, yi, j);
        yi -= Ls[lane * 33 + j] * yj;
      }
      if (lane < wb) y[jb + lane] = yi;
    }
    __syncthreads();
    for (int r = jb + wb + threadIdx.x; r < m; r += NT) {
      // all (up to 32) loads of the row issued together, four partial sums
      double a[4] = {0.0, 0.0, 0.0, 0.0};
      const double* Lr = Fs + r + (int64_t)jb * m;
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (j < wb) a[j & 3] += Lr[(int64_t)j * m] * y[jb + j];
      y[r] -= (a[0] + a[1]) + (a[2] + a[3]);
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < m; t += NT) {
    if (t < k) xb[f + t] = y[t] / Fs[t + (int64_t)t * m];
    else ubb[S.uoff[s] + t - k] = y[t];
  }
}

template <int NT>
__global__ void __launch_bounds__(NT, 8) k_fwd32(DevSym S, const int* __restrict__ list, const double* __restrict__ F,
                                              int64_t fstride, double* __restrict__ xp, double* __restrict__ ub,
                                              int64_t ustride) {
  extern __shared__ double y[];
  fwd32_body<NT>(S, list[blockIdx.x], blockIdx.y, F, fstride, xp, ub, ustride, y);
}

// Backward sweep of front s, problem b (NT threads; x: m + 2 + 32 * 33 doubles of shared memory).
template <int NT>
__device__ __forceinline__ void bwd32_body(const DevSym& S, int s, int b, const double* __restrict__ F,
                                           int64_t fstride, double* __restrict__ xp, double* x) {
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  const int* R = S.rows + S.rowptr[s];
  for (int t = threadIdx.x; t < m; t += NT) x[t] = xb[R[t]];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* Ls = x + ((m + 1) & ~1);  // [32][33] strictly lower part of the block's diagonal tile
  const int nblk = (k + 31) / 32;
  for (int bi = nblk - 1; bi >= 0; --bi) {
    const int jb = bi * 32, wb = min(32, k - jb), i0 = jb + wb;
    // x_j -= sum_{i >= i0} L_ij x_i for the block's columns (warp per column)
    for (int j = jb + warp; j < jb + wb; j += NT / 32) {
      const double* Lj = Fs + (int64_t)j * m;
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
      int i = i0 + lane;
      for (; i + 96 < m; i += 128) {
        a0 += Lj[i] * x[i];
        a1 += Lj[i + 32] * x[i + 32];
        a2 += Lj[i + 64] * x[i + 64];
        a3 += Lj[i + 96] * x[i + 96];
      }
      for (; i < m; i += 32) a0 += Lj[i] * x[i];
      double acc = (a0 + a1) + (a2 + a3);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      if (lane == 0) x[j] -= acc;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * 32; e += NT) {
      const int r = e & 31, c = e >> 5;
      Ls[r * 33 + c] = (c < r && r < wb) ? Fs[(jb + r) + (int64_t)(jb + c) * m] : 0.0;
    }
    __syncthreads();
    if (warp == 0) {
      // lane j holds x_{jb+j}; unit upper L_JJ^T solved from the last row up
      double xj = lane < wb ? x[jb + lane] : 0.0;
#pragma unroll 8
      for (int i = 31; i >= 0; --i) {
        const double xi = __shfl_sync(0xffffffffu, xj, i);
        xj -= Ls[i * 33 + lane] * xi;
      }
      if (lane < wb) x[jb + lane] = xj;
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < k; t += NT) xb[f + t] = x[t];
}

template <int NT>
__global__ void __launch_bounds__(NT, 8) k_bwd32(DevSym S, const int* __restrict__ list, const double* __restrict__ F,
                                              int64_t fstride, double* __restrict__ xp) {
  extern __shared__ double x[];
  bwd32_body<NT>(S, list[blockIdx.x], blockIdx.y, F, fstride, xp, x);
}

// Sweeps of the large fronts (those with cached 64 x 64 inverse blocks), 64-column blocks:
// the diagonal block is applied as a product with its cached inverse L_JJ^-1 (no sequential
// substitution chain), and the rows below (forward) or the column sums (backward) are spread
// over the CTA. NT threads; NT / 64 threads share one row of the inverse-block product (their
// partial sums are combined by shuffles in a fixed order). Shared memory: m + 2 doubles.
template <int NT>
__device__ __forceinline__ double inv_block_dot(const double* __restrict__ lc, const double* v, int wb, bool trans) {
  constexpr int kP = NT / 64;
  const int r = threadIdx.x / kP, q = threadIdx.x % kP;
  double acc = 0.0;
  if (r < wb) {
    if (!trans) {  // (L^-1 v)_r = sum_{c <= r} L^-1[r][c] v_c
      for (int c = q; c <= r; c += kP) acc += lc[r + 64 * c] * v[c];
    } else {  // (L^-T v)_r = sum_{c >= r} L^-1[c][r] v_c
      for (int c = r + q; c < wb; c += kP) acc += lc[c + 64 * r] * v[c];
    }
  }
#pragma unroll
  for (int o = 1; o < kP; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  return acc;
}

// Forward sweep of large front s, problem b (NT = 256 threads). kDeep: two rows per pass and
// 32 loads per row instead of one row and 16 (more loads in flight, more registers); the
// result is the same either way.
template <int NT, bool kDeep = true>
__device__ __forceinline__ void fwd64_body(const DevSym& S, int s, int b, const double* __restrict__ F,
                                           int64_t fstride, const double* __restrict__ linv,
                                           double* __restrict__ xp, double* __restrict__ ub, int64_t ustride,
                                           double* y) {
  static_assert(NT % 64 == 0 && NT / 64 <= 32, "whole rows of the inverse-block product per warp");
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  double* ubb = ub + (int64_t)b * ustride;
  for (int t = threadIdx.x; t < m; t += NT)
    y[t] = fwd_row_start(S, S.rowptr[s] + t, ubb, t < k ? xb[f + t] : 0.0);
  __syncthreads();
  const int nblk = (k + kB64 - 1) / kB64;
  for (int bi = 0; bi < nblk; ++bi) {
    const int jb = bi * kB64, wb = min(kB64, k - jb);
    const double v = inv_block_dot<NT>(linv_block(S, linv, b, s, bi), y + jb, wb, false);
    __syncthreads();  // every read of y_J is done
    if (threadIdx.x % (NT / 64) == 0 && threadIdx.x / (NT / 64) < wb) y[jb + threadIdx.x / (NT / 64)] = v;
    __syncthreads();
    // rows below: one thread per row (kDeep: two rows per pass, 32 loads of each in flight;
    // otherwise one row, 16 loads: the panel streams from DRAM, so the loads in flight set the
    // rate), eight partial sums per row in column order
    for (int r = jb + wb + threadIdx.x; r < m; r += (kDeep ? 2 : 1) * NT) {
      const int r2 = r + NT;
      const bool two = kDeep && r2 < m;
      double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      double c[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
      const double* Lr = Fs + r + (int64_t)jb * m;
      constexpr int kJ = kDeep ? 32 : 16;  // loads of a row per pass
      for (int j0 = 0; j0 < wb; j0 += kJ) {
        double la[kJ], lb[kDeep ? kJ : 1];
#pragma unroll
        for (int u = 0; u < kJ; ++u) {
          const bool ok = j0 + u < wb;
          la[u] = ok ? Lr[(int64_t)(j0 + u) * m] : 0.0;
          if (kDeep) lb[kDeep ? u : 0] = ok && two ? Lr[(int64_t)(j0 + u) * m + NT] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kJ; ++u) {
          const double yj = j0 + u < wb ? y[jb + j0 + u] : 0.0;
          a[u & 7] += la[u] * yj;
          if (kDeep) c[u & 7] += lb[kDeep ? u : 0] * yj;
        }
      }
      y[r] -= ((a[0] + a[1]) + (a[2] + a[3])) + ((a[4] + a[5]) + (a[6] + a[7]));
      if (two) y[r2] -= ((c[0] + c[1]) + (c[2] + c[3])) + ((c[4] + c[5]) + (c[6] + c[7]));
    }
    __syncthreads();
  }
  for (int t = threadIdx.x; t < m; t += NT) {
    if (t < k) xb[f + t] = y[t] / Fs[t + (int64_t)t * m];
    else ubb[S.uoff[s] + t - k] = y[t];
  }
}

// kDeep: the register-hungry form (one CTA per SM) for launches with few CTAs; the other
// (two CTAs per SM) for wide levels. Both give the same result.
template <int NT, bool kDeep>
__global__ void __launch_bounds__(NT, kDeep ? 1 : 2) k_fwd64(DevSym S, const int* __restrict__ list,
                                                             const double* __restrict__ F, int64_t fstride,
                                                             const double* __restrict__ linv,
                                                             double* __restrict__ xp, double* __restrict__ ub,
                                                             int64_t ustride) {
  extern __shared__ double y[];
  fwd64_body<NT, kDeep>(S, list[blockIdx.x], blockIdx.y, F, fstride, linv, xp, ub, ustride, y);
}

// Backward sweep of large front s, problem b (NT = 256 threads). kDeep: four rows per pass
// instead of two (more loads in flight); every lane still visits its rows in increasing
// order, so the result is the same either way.
template <int NT, bool kDeep = true>
__device__ __forceinline__ void bwd64_body(const DevSym& S, int s, int b, const double* __restrict__ F,
                                           int64_t fstride, const double* __restrict__ linv,
                                           double* __restrict__ xp, double* x) {
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  const int* R = S.rows + S.rowptr[s];
  for (int t = threadIdx.x; t < m; t += NT) x[t] = xb[R[t]];
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nblk = (k + kB64 - 1) / kB64;
  for (int bi = nblk - 1; bi >= 0; --bi) {
    const int jb = bi * kB64, wb = min(kB64, k - jb), i0 = jb + wb;
    // x_j -= sum_{i >= i0} L_ij x_i for the block's columns: warp w takes the columns
    // j = jb + w + (NT / 32) c, all of them at once (lane l: rows i0 + l + 32 t, four rows per
    // pass), so that every lane keeps kR * kC loads in flight; a butterfly per column at the end
    {
      constexpr int kW = NT / 32, kC = 64 / kW;  // columns per warp
      double acc[kC];
#pragma unroll
      for (int c = 0; c < kC; ++c) acc[c] = 0.0;
      constexpr int kR = kDeep ? 4 : 2;  // rows per lane and pass
      for (int i = i0 + lane; i < m; i += 32 * kR) {
        double lv[kR][kC], xv[kR];
#pragma unroll
        for (int t = 0; t < kR; ++t) {
          const int it = i + 32 * t;
          xv[t] = it < m ? x[it] : 0.0;
#pragma unroll
          for (int c = 0; c < kC; ++c) {
            const int j = warp + kW * c;
            lv[t][c] = (it < m && j < wb) ? Fs[it + (int64_t)(jb + j) * m] : 0.0;
          }
        }
#pragma unroll
        for (int t = 0; t < kR; ++t)
#pragma unroll
          for (int c = 0; c < kC; ++c) acc[c] += lv[t][c] * xv[t];
      }
#pragma unroll
      for (int c = 0; c < kC; ++c) {
        double v = acc[c];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        const int j = warp + kW * c;
        if (lane == 0 && j < wb) x[jb + j] -= v;
      }
    }
    __syncthreads();
    const double v = inv_block_dot<NT>(linv_block(S, linv, b, s, bi), x + jb, wb, true);
    __syncthreads();
    if (threadIdx.x % (NT / 64) == 0 && threadIdx.x / (NT / 64) < wb) x[jb + threadIdx.x / (NT / 64)] = v;
    __syncthreads();
  }
  for (int t = threadIdx.x; t < k; t += NT) xb[f + t] = x[t];
}

template <int NT, bool kDeep>
__global__ void __launch_bounds__(NT, kDeep ? 1 : 2) k_bwd64(DevSym S, const int* __restrict__ list,
                                                             const double* __restrict__ F, int64_t fstride,
                                                             const double* __restrict__ linv,
                                                             double* __restrict__ xp) {
  extern __shared__ double x[];
  bwd64_body<NT, kDeep>(S, list[blockIdx.x], blockIdx.y, F, fstride, linv, xp, x);
}

// Sweeps of fronts with m <= 32 rows (one 32-column block): one warp per (front,
// problem), kTinySweepWarps per CTA. Lane t holds entry t of the front's vector; the
// arithmetic follows k_fwd32 / k_bwd32 step for step (sequential shuffle chain on the
// diagonal block, the same four partial sums for the rows below, the same xor tree
// for the column sums), so the results equal theirs.
constexpr int kTinySweepWarps = 8;

// One warp: forward sweep of tiny front s, problem b (y: 32 doubles of shared memory).
__device__ __forceinline__ void fwd_tiny_warp(const DevSym& S, int s, int b, const double* __restrict__ F,
                                              int64_t fstride, double* __restrict__ xp, double* __restrict__ ub,
                                              int64_t ustride, double* y) {
  const int lane = threadIdx.x & 31;
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  double* ubb = ub + (int64_t)b * ustride;
  double yi = lane < m ? fwd_row_start(S, S.rowptr[s] + lane, ubb, lane < k ? xb[f + lane] : 0.0) : 0.0;
  {  // diagonal block: unit lower L_JJ
    double yd = lane < k ? yi : 0.0;
    for (int j = 0; j < k; ++j) {
      const double yj = __shfl_sync(0xffffffffu, yd, j);
      if (lane > j && lane < k) yd -= Fs[lane + (int64_t)j * m] * yj;
    }
    if (lane < k) yi = yd;
    y[lane] = yi;
  }
  __syncwarp();
  if (lane >= k && lane < m) {  // rows below the block
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    const double* Lr = Fs + lane;
    for (int j = 0; j < k; ++j) a[j & 3] += Lr[(int64_t)j * m] * y[j];
    yi -= (a[0] + a[1]) + (a[2] + a[3]);
  }
  if (lane < k) xb[f + lane] = yi / Fs[lane + (int64_t)lane * m];
  else if (lane < m) ubb[S.uoff[s] + lane - k] = yi;
}

__global__ void __launch_bounds__(32 * kTinySweepWarps) k_fwd_tiny(DevSym S, const int* __restrict__ list, int nlist,
                                                                   const double* __restrict__ F, int64_t fstride,
                                                                   double* __restrict__ xp, double* __restrict__ ub,
                                                                   int64_t ustride) {
  __shared__ double sy[kTinySweepWarps][32];
  const int warp = threadIdx.x >> 5;
  const int idx = blockIdx.x * kTinySweepWarps + warp;
  if (idx >= nlist) return;  // the whole warp leaves; only warp-level synchronization follows
  fwd_tiny_warp(S, list[idx], blockIdx.y, F, fstride, xp, ub, ustride, sy[warp]);
}

// One warp: backward sweep of tiny front s, problem b (registers and shuffles only).
__device__ __forceinline__ void bwd_tiny_warp(const DevSym& S, int s, int b, const double* __restrict__ F,
                                              int64_t fstride, double* __restrict__ xp) {
  const int lane = threadIdx.x & 31;
  const int k = lg_k(S, s), m = lg_m(S, s), f = S.first[s];
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* xb = xp + (int64_t)b * S.n;
  double xl = lane < m ? xb[S.rows[S.rowptr[s] + lane]] : 0.0;
  // x_j -= sum_{i >= k} L_ij x_i for the block's columns: as in k_bwd32, lane l holds the
  // term of row k + l and the butterfly total of lane 0 is used
  const int ri = k + lane;
  const double xs = __shfl_sync(0xffffffffu, xl, ri & 31);
  for (int j = 0; j < k; ++j) {
    double acc = ri < m ? Fs[ri + (int64_t)j * m] * xs : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    acc = __shfl_sync(0xffffffffu, acc, 0);
    if (lane == j) xl -= acc;
  }
  // unit upper L_JJ^T from the last row up
  for (int i = k - 1; i >= 0; --i) {
    const double xi = __shfl_sync(0xffffffffu, xl, i);
    if (lane < i) xl -= Fs[i + (int64_t)lane * m] * xi;
  }
  if (lane < k) xb[f + lane] = xl;
}

__global__ void __launch_bounds__(32 * kTinySweepWarps) k_bwd_tiny(DevSym S, const int* __restrict__ list, int nlist,
                                                                   const double* __restrict__ F, int64_t fstride,
                                                                   double* __restrict__ xp) {
  const int warp = threadIdx.x >> 5;
  const int idx = blockIdx.x * kTinySweepWarps + warp;
  if (idx >= nlist) return;  // the whole warp leaves; only warp-level synchronization follows
  bwd_tiny_warp(S, list[idx], blockIdx.y, F, fstride, xp);
}

// ---------------------------------------------------------------------------
// selected inverse
// ---------------------------------------------------------------------------

constexpr int kSiT = 64;  // rows of B per tile

// ---------------------------------------------------------------------------
// Selected inverse of the large fronts as matrix products over the whole front. With K the k pivot
// rows, B the r rows below, X = L_KK^-1 and W = L_BK X:
//   Sigma_BK = -Sigma_BB W,   Sigma_KK = X^T D^-1 X - W^T Sigma_BK,
// the closed form of the Takahashi recurrence S_ij = -sum_{l>j} L_lj S_li, S_jj = 1/d_j - sum_{l>j}
// L_lj S_lj over the block K (Sigma_BB comes from the parent). X is built from the cached 64 x 64
// inverses by doubling: for neighbouring block ranges 1 and 2, X_21 = -X_22 (L_21 X_11).
//
// The blockwise recurrence takes two dependent launches per 64 pivot columns (22 for the 644-column
// root front of the SPDE 200^2 model); this takes 2 log2(k / 64) + 3 with the same number of products,
// every launch over all tiles of the level. Measured, SPDE 200^2 posterior, all products of the large
// fronts: 1.71 -> 1.02 ms at B = 1 (1.27 with 64-row tiles only), 3.69 -> 2.95 ms at B = 10, 4.66 ->
// 3.98 ms at B = 15. Chains of launches bound the small batches, padding of 100- to 200-row fronts to
// 64 x 64 tiles the large ones.
//
// X and W live transposed in the strictly upper triangle of the front's Sigma buffer (block (I, J) of X
// at (J, I), W at (K, B)), which nothing else uses; the products L_21 X_11 in the lower block that
// Sigma_KK takes at the end. One CTA per 64 x 64 tile, K in chunks of 32 through two cp.async stages (three
// CTAs per SM; a third stage would leave two).
// ---------------------------------------------------------------------------
enum SiMode : int {
  SI_T = 0,      // T = L_21 X_11                      (lower block (I, J))
  SI_X = 1,      // X_21 = -X_22 T                     (transposed, upper block)
  SI_W = 2,      // W = L_BK X                         (transposed, upper block)
  SI_BK = 3,     // Sigma_BK = -Sigma_BB W
  SI_KK = 4,     // Sigma_KK = X^T D^-1 X - W^T Sigma_BK
};

// A launch of k_si_gemm over the large fronts of a level: tiles z0 .. z0 + tiles of every front, in 32-row
// halves or whole (SI_T, SI_X: z0 = 0).
struct SiLaunch {
  int mode, hb, z0, tiles;
  bool half;
};

// Tiles of the joins of ranges of hb blocks (SI_T, SI_X) of a front of nblk blocks: hb x hb per pair of whole
// ranges, and the rows that exist of a last, partial pair.
__host__ __device__ inline int si_join_tiles(int nblk, int hb) {
  const int pairs = nblk / (2 * hb), rest = nblk - 2 * hb * pairs - hb;
  return pairs * hb * hb + (rest > 0 ? rest * hb : 0);
}

// Rows i0 .. i1, columns from j0 and K range t0 .. t1 of tile z (all in rows of a front of k pivots and m
// rows); TM = 32: z counts halves. False: the front has no such tile. Within a join the tiles with the longest
// K range come first: in an order that mixes them the launch waits for SMs that got several long ones (SI_T
// of the last join, 900 pivots at B = 7 72 -> 56 us; all joins of 6000 pivots, SI_T 2.20 -> 1.93 ms, SI_X 1.62 ->
// 1.42 ms).
struct SiTile {
  int i0, i1, j0, t0, t1;
};
template <int MODE, int TM>
__host__ __device__ __forceinline__ bool si_tile(int z, int hb, int k, int m, SiTile& o) {
  const int nblk = (k + kB64 - 1) / kB64, rt = (m - k + kSiT - 1) / kSiT;
  const int half = TM == 32 ? (z & 1) : 0;
  if (TM == 32) z >>= 1;
  auto lower = [](int a, int b) { return a < b ? a : b; };
  if (MODE == SI_T || MODE == SI_X) {
    const int pr = z / (hb * hb), q = z - pr * hb * hb, first = 2 * pr * hb;
    const int rows = lower(hb, nblk - first - hb);
    if (q >= rows * hb) return false;
    const int I = first + hb + (MODE == SI_T ? q % rows : rows - 1 - q / hb);
    const int J = first + (MODE == SI_T ? q / rows : q % hb);
    o.i0 = I * kB64;
    o.i1 = lower(k, o.i0 + kB64);
    o.j0 = J * kB64;
    o.t0 = MODE == SI_T ? o.j0 : (first + hb) * kB64;
    o.t1 = MODE == SI_T ? (first + hb) * kB64 : o.i1;
  } else if (MODE == SI_W || MODE == SI_BK) {
    const int I = z / nblk, J = z - I * nblk;
    if (I >= rt) return false;
    o.i0 = k + I * kSiT;
    o.i1 = lower(m, o.i0 + kSiT);
    o.j0 = J * kB64;
    o.t0 = MODE == SI_W ? o.j0 : k;
    o.t1 = MODE == SI_W ? k : m;
  } else {
    if (z >= nblk * (nblk + 1) / 2) return false;
    int I = 0, rem = z;
    while (rem > I) rem -= ++I;
    o.i0 = I * kB64;
    o.i1 = lower(k, o.i0 + kB64);
    o.j0 = rem * kB64;
    o.t0 = o.i0 + 32 * half;  // X is lower triangular
    o.t1 = m;
  }
  if (TM == 32) {
    o.i0 += 32 * half;
    o.i1 = lower(o.i1, o.i0 + 32);
  }
  return o.i0 < o.i1;
}

// Tile z of front s, problem b. hb: block count of the ranges joined (SI_T, SI_X). TM = 32 cuts every
// tile into two CTAs of 32 rows, for launches whose 64-row tiles would leave SMs idle (the K loop of
// one 64 x 64 tile is 1.1 us per chunk at the tensor-core rate of one SM); an entry's sum is the same.
template <int MODE, int TM>
__device__ __forceinline__ void si_gemm_body(const DevSym& S, int s, int b, int z, int hb,
                                             const double* __restrict__ F, double* __restrict__ Sg, int64_t fstride,
                                             const double* __restrict__ linv, double* smem64) {
  constexpr int ld = kLd64, kBuf = 64 * kLd64;  // one stage: As[32][ld], Bs[32][ld]
  __shared__ double scale[kSiStages][32];
  const int k = lg_k(S, s), m = lg_m(S, s);
  SiTile tile;
  if (!si_tile<MODE, TM>(z, hb, k, m, tile)) return;
  const int i0 = tile.i0, i1 = tile.i1, j0 = tile.j0, t0 = tile.t0, t1 = tile.t1;
  const int j1 = min(k, j0 + kB64);
  const double* Fs = F + (int64_t)b * fstride + S.fptr[s];
  double* Ss = Sg + (int64_t)b * fstride + S.fptr[s];
  const double* lb = linv + (int64_t)b * S.lstride + (int64_t)S.lbo[s] * (kB64 * kB64);
  // address of X (t < k) or W (t >= k) at (t, c), c < k, in a block on or below the diagonal
  auto xw = [&](int t, int c) -> const double* {
    const int cb = c >> 6;
    if ((t >> 6) == cb && t < k) return lb + (int64_t)cb * (kB64 * kB64) + (t & 63) + (c & 63) * kB64;
    return Ss + c + (int64_t)t * m;
  };
  auto load_chunk = [&](int c0, int buf) {
    double* As = smem64 + buf * kBuf;
    double* Bs = As + 32 * ld;
    constexpr bool a_along_t = MODE == SI_X;
#pragma unroll
    for (int u = 0; u < TM / 8; ++u) {
      const int e = threadIdx.x + 256 * u;
      bool along_t = a_along_t;
      if (MODE == SI_BK) along_t = i0 + TM - 1 < c0;  // above the diagonal: stored at (t, i)
      const int l = along_t ? (e & 31) : (e / TM), ii = along_t ? (e >> 5) : (e % TM);
      const int t = c0 + l, i = i0 + ii;
      double* dst = As + l * ld + ii;
      if (t < t1 && i < i1) {
        const double* src;
        if (MODE == SI_T || MODE == SI_W) src = Fs + i + (int64_t)t * m;
        else if (MODE == SI_X) src = xw(i, t);
        else if (MODE == SI_BK) src = i >= t ? Ss + i + (int64_t)t * m : Ss + t + (int64_t)i * m;
        else src = xw(t, i);
        cp_async8(dst, src);
      } else {
        *dst = 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int e = threadIdx.x + 256 * u;
      const bool along_t = MODE == SI_X || (MODE == SI_KK && c0 >= k);
      const int l = along_t ? (e & 31) : (e >> 6), jj = along_t ? (e >> 5) : (e & 63);
      const int t = c0 + l, j = j0 + jj;
      double* dst = Bs + l * ld + jj;
      if (t < t1 && j < j1) {
        const double* src;
        if (MODE == SI_X) src = Ss + t + (int64_t)j * m;
        else if (MODE == SI_BK) src = Ss + j + (int64_t)t * m;
        else if (MODE == SI_KK && t >= k) src = Ss + t + (int64_t)j * m;
        else src = xw(t, j);
        cp_async8(dst, src);
      } else {
        *dst = 0.0;
      }
    }
    if (MODE == SI_KK && threadIdx.x < 32) {
      const int t = c0 + threadIdx.x;
      scale[buf][threadIdx.x] = t < k ? 1.0 / Fs[t + (int64_t)t * m] : -1.0;
    }
    cp_async_commit();
  };
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int NA = TM / 16;  // 8-row sub-tiles of a warp
  const int wi = (warp & 1) * (TM / 2), wj = (warp >> 1) * 16;
  const int g = lane >> 2, tg = lane & 3;
  const bool wact = i0 + wi < i1 && j0 + wj < j1;
  double acc[NA][2][2];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q) acc[a][q][0] = acc[a][q][1] = 0.0;
  const int nc = (t1 - t0 + 31) / 32;
  load_chunk(t0, 0);
  for (int c = 0; c < nc; ++c) {
    cp_async_wait<0>();
    __syncthreads();  // chunk c has landed, and every warp is done with chunk c - 1
    if (c + 1 < nc) load_chunk(t0 + 32 * (c + 1), (c + 1) % kSiStages);
    const double* As = smem64 + (c % kSiStages) * kBuf;
    const double* Bs = As + 32 * ld;
    if (wact) {
#pragma unroll
      for (int kk = 0; kk < 32; kk += 4) {
        double af[NA], bf[2];
#pragma unroll
        for (int a = 0; a < NA; ++a) af[a] = As[(kk + tg) * ld + wi + a * 8 + g];
#pragma unroll
        for (int q = 0; q < 2; ++q) bf[q] = Bs[(kk + tg) * ld + wj + q * 8 + g];
        if (MODE == SI_KK) {
          const double sc = scale[c % kSiStages][kk + tg];
          bf[0] *= sc;
          bf[1] *= sc;
        }
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
          for (int q = 0; q < 2; ++q) mma884(acc[a][q][0], acc[a][q][1], af[a], bf[q]);
      }
    }
  }
  constexpr double sign = (MODE == SI_X || MODE == SI_BK) ? -1.0 : 1.0;
  if (MODE == SI_X || MODE == SI_W) {  // transposed output: through shared memory, contiguous over j
    __syncthreads();
    double* Gs = smem64;  // [64][ld]
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h) Gs[(wi + a * 8 + g) * ld + wj + q * 8 + tg * 2 + h] = sign * acc[a][q][h];
    __syncthreads();
    for (int e = threadIdx.x; e < TM * kB64; e += 256) {
      const int ii = e >> 6, jj = e & 63;
      if (i0 + ii < i1 && j0 + jj < j1) Ss[(j0 + jj) + (int64_t)(i0 + ii) * m] = Gs[ii * ld + jj];
    }
    return;
  }
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int i = i0 + wi + a * 8 + g, j = j0 + wj + q * 8 + tg * 2 + h;
        if (i < i1 && j < j1 && (MODE != SI_KK || i >= j)) Ss[i + (int64_t)j * m] = sign * acc[a][q][h];
      }
}

// arg: hb (SI_T, SI_X: always one launch), else the launch's first tile (a parameter of its own for all modes
// spills in SI_T and SI_X; without the assumption SI_KK is 3 % slower).
template <int MODE, int TM>
__global__ void __launch_bounds__(256, kSiCtas) k_si_gemm(DevSym S, const int* __restrict__ list, int arg,
                                                    const double* __restrict__ F, double* __restrict__ Sg,
                                                    int64_t fstride, const double* __restrict__ linv) {
  extern __shared__ double smem64[];
  constexpr bool join = MODE == SI_T || MODE == SI_X;
  const int z = join ? blockIdx.z : arg + blockIdx.z;
  __builtin_assume(z >= 0);
  si_gemm_body<MODE, TM>(S, list[blockIdx.x], blockIdx.y, z, join ? arg : 0, F, Sg,
                         fstride, linv, smem64);
}

}  // namespace
}  // namespace inla
