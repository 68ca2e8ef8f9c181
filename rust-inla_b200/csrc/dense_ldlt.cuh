// Blocked dense LDL^T of a symmetric block held in shared memory.
//
// The pivots are taken 8 at a time. One warp factors the 8 x 8 diagonal block with every lane
// holding the whole block in registers (warp_ldlt8: no exchange on the pivot chain) and forms its
// inverse Lam = L_kk^-1. The rows below and the trailing matrix are updated by all warps with FP64
// tensor-core tiles (mma.sync m8n8k4):
//   U_bk = A_bk Lam^T            (= L_bk D_k),  L_bk = U_bk D_k^-1
//   A_bb -= L_bk U_bk^T          (lower triangle)
// which is the right-looking blocked LDL^T (Golub & Van Loan, Matrix
// Computations, 4th ed., Sec. 4.2) with the diagonal-block solve done through
// the explicit inverse of the unit triangle. The pivot warp looks ahead: it updates the next
// diagonal block itself and factors it while the other warps update the rest. Optionally the
// inverse of the whole unit lower factor of the leading kp x kp block is accumulated as well
// (block forward elimination: Li_k <- Lam Li_k, Li_b <- Li_b - L_bk Li_k).
#pragma once
#include <cstdint>
#include <type_traits>

#include <cuda_runtime.h>

namespace inla {
namespace {

__device__ __forceinline__ void dmma884(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}

// 8-byte asynchronous global -> shared copies (many in flight per thread).
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N));
}

constexpr int kLamLd = 20;  // leading dimension of a 16 x 16 Lam block (== 4 mod 16: conflict-free tiles)
// Shared scratch of the blocked routine (doubles): two buffers of Lam (8 x 8) and 1 / d.
constexpr int kLam8Ld = 12;
constexpr int kLam8Buf = 8 * kLam8Ld + 8;
constexpr int kDenseScratch = 2 * kLam8Buf;

// Leading dimension for an m-row block in shared memory: >= m and == 4 (mod 16),
// so the 16 lanes of a half-warp reading an 8 x 4 fragment hit 16 distinct banks.
__host__ __device__ constexpr int dense_ld(int m) { return ((m + 11) / 16) * 16 + 4; }
// Leading dimension of the 8-column U buffer of cta_ldlt (rows rounded up to 8).
__host__ __device__ constexpr int dense_uld(int m) { return dense_ld(m + 8); }

// Barrier id: `arrive` counts the caller's warp in without waiting.
__device__ __forceinline__ void bar_sync_id(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive_id(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// 1 / d for 2^-1000 <= |d| < 2^1000 (rcp_in_range) without a branch: the hardware approximation y and one step
// of the third-order Householder iteration y (1 + e + e^2). PTX has y look at the 20 leading mantissa bits of d
// and set as many, so |e| < 2^-18, and the neglected e^3 y is below half a unit in the last place: the result
// lies within one unit of the correctly rounded 1 / d (measured over two million mantissas: 0.03 % differ, the
// worst is 0.506 units off). Outside the range y may be flushed; warp_ldlt8 then
// repeats the block with 1.0 / d. With 1.0 / d throughout the 64 x 64 block of cta_ldlt takes 14.9 k cycles with
// the inverse and 13.3 k without, with this 13.6 k and 11.4 k.
__device__ __forceinline__ double rcp_straight(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ bool rcp_in_range(double d) {  // by the high word of |d|
  return (unsigned)(__double2hiint(d) & 0x7fffffff) - 0x01700000u < 0x7d000000u;
}

// One warp: what warp_ldlt8 leaves in A, Lam and di, with 1.0 / d for every pivot, from the copy of the block
// that Lam holds. Rarely taken, so it works in shared memory, lane i on row i (then on column i of L^-1),
// and is a call: unrolled beside the fast pass it spills in k_panel64 and k_diag_next (5 to 7 % slower).
__device__ __noinline__ void warp_ldlt8_div(double* A, int lda, int w, double* Lam, double* di) {
  const int lane = threadIdx.x & 31;
  if (lane < 8)
    for (int j = 0; j <= lane; ++j)
      if (lane >= w) Lam[lane + j * kLam8Ld] = lane == j ? 1.0 : 0.0;
  __syncwarp();
#pragma unroll 1
  for (int p = 0; p < 8; ++p) {
    const double r = 1.0 / Lam[p + p * kLam8Ld];
    const bool below = lane > p && lane < 8;
    const double l = below ? Lam[lane + p * kLam8Ld] * r : 0.0;
    if (below)
#pragma unroll 1
      for (int j = p + 1; j <= lane; ++j) Lam[lane + j * kLam8Ld] -= l * Lam[j + p * kLam8Ld];
    __syncwarp();
    if (below) Lam[lane + p * kLam8Ld] = l;
    if (lane == 0) di[p] = r;
    if (lane >= p && lane < w) A[lane + p * lda] = lane == p ? Lam[p + p * kLam8Ld] : l;
    __syncwarp();
  }
  double x[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    x[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int p = 0; p < i; ++p) x[i] -= Lam[i + p * kLam8Ld] * x[p];
  }
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (lane < 8) Lam[i + lane * kLam8Ld] = x[i];
  __syncwarp();
}

// One warp: LDL^T and inverse of the w x w (w <= 8) leading block of A (shared memory, column-major,
// even leading dimension lda, 16-byte aligned; lower triangle read). On exit A holds L strictly below
// the diagonal and D on it (inside w x w only); Lam (ld kLam8Ld) holds L^-1 as an 8 x 8 unit lower
// triangle (identity beyond w), di[t] = 1 / d_t (1 beyond w), and lam0 / lam1 the lane's entries
// (g, tg) and (g, tg + 4) of Lam (g = lane / 4, tg = lane % 4: its tensor-core fragments).
// The chain per pivot is a reciprocal and two dependent FMAs. Exchanging the
// pivot column between lanes put a store -> __syncwarp -> load (40 cycles) and the issue of the
// exchanged row's loads on it as well: 360 cycles per pivot for 16 x 16 blocks. So every lane repeats
// the block's 112 products instead, which fit in the shadow of the reciprocals.
__device__ __forceinline__ void warp_ldlt8(double* A, int lda, int w, double* Lam, double* di, double& lam0,
                                           double& lam1) {
  const int lane = threadIdx.x & 31, g = lane >> 2, tg = lane & 3;
  double a[8][8];  // a[i][j], i >= j
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = j & ~1; i < 8; i += 2) {
      const double2 v = *reinterpret_cast<const double2*>(A + i + j * lda);
      if (i >= j) a[i][j] = v.x;
      a[i + 1][j] = v.y;
    }
  if (w < 8) {
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int i = j; i < 8; ++i)
        if (i >= w) a[i][j] = (i == j) ? 1.0 : 0.0;
  }
  // the block as it came, for a second pass (A is overwritten as the columns are finished)
  Lam[g + tg * kLam8Ld] = A[g + tg * lda];
  Lam[g + (tg + 4) * kLam8Ld] = A[g + (tg + 4) * lda];
  __syncwarp();  // every lane has read the block that lane 0 overwrites
  // Right-looking elimination of the block and of the columns tg and tg + 4 of L^-1 (x0, x1: rows 4 to 7
  // of the latter). A finished column leaves for shared memory at once (lane 0), which frees its registers.
  double x0[8], x1[4];
  const int lim = lane == 0 ? w : 0;
  bool in_range = true;
#pragma unroll
  for (int i = 0; i < 8; ++i) x0[i] = (i == tg) ? 1.0 : 0.0;
#pragma unroll
  for (int i = 0; i < 4; ++i) x1[i] = (i == tg) ? 1.0 : 0.0;
#pragma unroll
  for (int p = 0; p < 8; ++p) {
    in_range = in_range && rcp_in_range(a[p][p]);
    const double r = rcp_straight(a[p][p]);
    if (lane == 0) di[p] = r;
    if (p < lim) A[p + p * lda] = a[p][p];
    double l[8];
#pragma unroll
    for (int i = p + 1; i < 8; ++i) l[i] = a[i][p] * r;
#pragma unroll
    for (int j = p + 1; j < 8; ++j)
#pragma unroll
      for (int i = j; i < 8; ++i) a[i][j] -= l[i] * a[j][p];
#pragma unroll
    for (int i = p + 1; i < 8; ++i) {
      if (i < lim) A[i + p * lda] = l[i];
      x0[i] -= l[i] * x0[p];
      if (p >= 4) x1[i - 4] -= l[i] * x1[p - 4];
    }
  }
  if (!in_range) {  // every lane alike
    __syncwarp();
    warp_ldlt8_div(A, lda, w, Lam, di);
    lam0 = Lam[g + tg * kLam8Ld];
    lam1 = Lam[g + (tg + 4) * kLam8Ld];
    return;
  }
  lam0 = x0[0];
  lam1 = 0.0;
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    if (g == i) lam0 = x0[i];
    if (i >= 4 && g == i) lam1 = x1[i - 4];
  }
  Lam[g + tg * kLam8Ld] = lam0;
  Lam[g + (tg + 4) * kLam8Ld] = lam1;
}

// One warp: Lam = L^-1 of the unit lower w x w (w <= 16) block of L (shared
// memory, column-major, leading dimension ldl; the diagonal is not read),
// identity-padded to 16 x 16 (ld kLamLd). Forward elimination
// Lam[i,:] -= L[i,p] Lam[p,:] for i > p, one __syncwarp per step; xbuf: 32 doubles.
__device__ __forceinline__ void warp_trinv16(const double* L, int ldl, int w, double* Lam, double* xbuf) {
  const int lane = threadIdx.x & 31, r = lane >> 1, h = lane & 1;
  double li[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) li[q] = (r == h + 2 * q) ? 1.0 : 0.0;
#pragma unroll 16
  for (int p = 0; p < 16; ++p) {
    double* row = xbuf + (p & 1) * 16;
    const double lrp = (r > p && r < w && p < w) ? L[r + p * ldl] : 0.0;
    if (r == p) {
#pragma unroll
      for (int q = 0; q < 8; ++q) row[h + 2 * q] = li[q];
    }
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 8; ++q) li[q] -= lrp * row[h + 2 * q];
  }
#pragma unroll
  for (int q = 0; q < 8; ++q) Lam[r + (h + 2 * q) * kLamLd] = li[q];
  __syncwarp();
}

// Partial LDL^T of the m x m symmetric matrix A (shared memory, column-major, 16-byte aligned, even
// leading dimension lda, lower triangle), eliminating the first kp columns.
// On exit A[:, :kp] holds L (unit, strictly lower) with D on the diagonal and
// the lower triangle of A[kp:, kp:] holds the Schur complement. With kInv, Li
// (shared, leading dimension ldi, kp x kp) receives the inverse of the unit
// lower factor of the leading kp x kp block (Li must be zero on entry). Called
// by all threads of the CTA (at least two warps); U: 8 x ldu doubles with ldu = dense_uld(m);
// ws: kDenseScratch doubles (16-byte aligned). Ends with a barrier. Uses barrier 1.
//
// Per block of 8 pivots the pivot warp (warp 0) runs factor -> its own 8 rows below -> the next
// diagonal tile without waiting for the others; they wait for Lam (barrier 0), form their rows, wait
// for the pivot warp's rows (barrier 1, which the pivot warp only counts into), and update the
// trailing tiles while the pivot warp is already in the next block. What bounds it is the pivot
// warp's chain. Lam and 1 / d are double-buffered: they are overwritten two blocks later, after a
// barrier that every reader has passed.
// Measured for a 64 x 64 block with its inverse, one CTA of 256 threads: 13.6 k cycles (11.4 k without the
// inverse); the 16-wide form it replaces (one warp factoring 16 x 16 with the others waiting, three barriers
// per block): 32.7 k (25.5 k).
template <bool kInv>
__device__ __forceinline__ void cta_ldlt(double* A, int lda, int m, int kp, double* Li, int ldi, double* U, int ldu, double* ws) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int g = lane >> 2, tg = lane & 3;
  int buf = 0;
  // callers with kp <= 64 would get eight copies of the body: 18 k cycles instead of 14 k, and 21 k the
  // first time through (instruction fetch)
#pragma unroll 1
  for (int o = 0; o < kp; o += 8, buf ^= 1) {
    const int w = min(8, kp - o);
    double* lam = ws + buf * kLam8Buf;
    double* di = lam + 8 * kLam8Ld;
    const int base = o + w, nb = m - base, T = (nb + 7) >> 3;
    const bool w0 = tg < w, w1 = tg + 4 < w;
    double lam0, lam1;
    if (warp == 0) {
      warp_ldlt8(A + o + o * lda, lda, w, lam, di, lam0, lam1);
      if (kInv) {
        if (g < w && w0) Li[(o + g) + (o + tg) * ldi] = lam0;
        if (g < w && w1) Li[(o + g) + (o + tg + 4) * ldi] = lam1;
      }
    }
    __syncthreads();
    const double* Ar = A + base + g + (o + tg) * lda;  // the lane's operand entry of row task 0
    // rows of 8-row task t: U = A Lam^T and L = U D^-1
    auto form_rows = [&](int t) {
      const int i = base + 8 * t + g;
      const double a0 = (w0 && i < m) ? Ar[8 * t] : 0.0;
      const double a1 = (w1 && i < m) ? Ar[8 * t + 4 * lda] : 0.0;
      const double d0 = di[2 * tg], d1 = di[2 * tg + 1];
      double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0;
      dmma884(c0, c1, a0, lam0);
      dmma884(e0, e1, a1, lam1);
      c0 += e0;
      c1 += e1;
      __syncwarp();
      const bool k0 = i < m && 2 * tg < w, k1 = i < m && 2 * tg + 1 < w;
      double* Ut = U + 2 * tg * ldu + 8 * t + g;
      double* At = A + i + (o + 2 * tg) * lda;
      Ut[0] = k0 ? c0 : 0.0;
      Ut[ldu] = k1 ? c1 : 0.0;
      if (k0) At[0] = c0 * d0;
      if (k1) At[lda] = c1 * d1;
    };
    // C[8 I + g, 2 tg + h] -= L_I B for N row tiles I = I0, I0 + 1, ... of one column of tiles (the
    // lane's operand entries b0, b1), all loads before the first store. Rows r with max(lo, diag + h)
    // <= r < rows (r counted from `base`) are updated.
    auto column = [&](auto ntiles, int I0, double b0, double b1, double* C, int ldc, int diag, int lo, int rows) {
      constexpr int N = decltype(ntiles)::value;
      double a0[N], a1[N], v[N][2], c[N][2];
      bool ok[N][2];
#pragma unroll
      for (int q = 0; q < N; ++q) {
        const int r = 8 * (I0 + q) + g;
        a0[q] = (w0 && r < rows) ? Ar[8 * (I0 + q)] : 0.0;
        a1[q] = (w1 && r < rows) ? Ar[8 * (I0 + q) + 4 * lda] : 0.0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          ok[q][h] = r < rows && r >= diag + h && r >= lo;
          v[q][h] = ok[q][h] ? C[8 * (I0 + q) + h * ldc] : 0.0;
          c[q][h] = 0.0;
        }
      }
#pragma unroll
      for (int q = 0; q < N; ++q) dmma884(c[q][0], c[q][1], a0[q], b0);
#pragma unroll
      for (int q = 0; q < N; ++q) dmma884(c[q][0], c[q][1], a1[q], b1);
#pragma unroll
      for (int q = 0; q < N; ++q)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (ok[q][h]) C[8 * (I0 + q) + h * ldc] = v[q][h] - c[q][h];
    };
    const std::integral_constant<int, 1> one{};
    const std::integral_constant<int, 4> four{};
    if (warp == 0) {
      if (T > 0) {
        form_rows(0);
        __syncwarp();
        bar_arrive_id(1, blockDim.x);
        const double* Ub = U + tg * ldu + g;
        column(one, 0, Ub[0], Ub[4 * ldu], A + base + g + (base + 2 * tg) * lda, lda, 2 * tg, 0, nb);
        __syncwarp();
      }
      continue;
    }
    lam0 = lam[g + tg * kLam8Ld];
    lam1 = lam[g + (tg + 4) * kLam8Ld];
#pragma unroll 1
    for (int t = warp; t < T; t += nw - 1) form_rows(t);
    if (kInv) {
      // Li_k[:, :o] <- Lam Li_k[:, :o]  (8 columns per task)
#pragma unroll 1
      for (int t = warp - 1; t < (o >> 3); t += nw - 1) {
        const double* Lb = Li + (o + tg) + (8 * t + g) * ldi;
        const double b0 = w0 ? Lb[0] : 0.0, b1 = w1 ? Lb[4] : 0.0;
        double c0 = 0.0, c1 = 0.0, e0 = 0.0, e1 = 0.0;
        dmma884(c0, c1, lam0, b0);
        dmma884(e0, e1, lam1, b1);
        __syncwarp();
        if (g < w) {
          Li[(o + g) + (8 * t + 2 * tg) * ldi] = c0 + e0;
          Li[(o + g) + (8 * t + 2 * tg + 1) * ldi] = c1 + e1;
        }
      }
    }
    if (T == 0) continue;
    bar_sync_id(1, blockDim.x);
    // Trailing tiles A_IJ -= L_I U_J^T (I >= J) and, with kInv, Li_IJ -= L_I Li_kJ for the rows of
    // later blocks inside kp: one task is up to four row tiles of a tile column.
    const int Tc = kInv ? base >> 3 : 0;
    const int nbi = kp - base;
    int left = warp - 1;  // tasks to skip before this warp's next one
#pragma unroll 1
    for (int I0 = 0; I0 < T; I0 += 4) {
      const int nj = min(T, I0 + 4), ni = 8 * I0 < nbi ? Tc : 0;
#pragma unroll 1
      for (; left < nj + ni; left += nw - 1) {
        if (left < nj) {
          const int J = left, c = 8 * J + 2 * tg;
          const double* Ub = U + tg * ldu + 8 * J + g;
          // the first eight rows of column 0 are the pivot warp's
          column(four, I0, Ub[0], Ub[4 * ldu], A + base + g + (base + c) * lda, lda, c, J == 0 ? 8 : 0, nb);
        } else if (kInv) {
          const int J = left - nj, c = 8 * J + 2 * tg;
          const double* Lb = Li + (o + tg) + (8 * J + g) * ldi;
          column(four, I0, Lb[0], Lb[4], Li + base + g + c * ldi, ldi, -8, 0, nbi);  // w = 8: rows follow
        }
      }
      left -= nj + ni;
    }
  }
  __syncthreads();
}

}  // namespace
}  // namespace inla
