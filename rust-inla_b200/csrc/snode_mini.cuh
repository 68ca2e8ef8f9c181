// Trees of fronts with at most eight rows (independent AR1-type models: half a million fronts of at
// most seven rows on 30 to 40 levels, most of them links of a chain). A launch per level and a warp
// per front spends the time on launches with few fronts and on warps with 25 idle lanes. Here
// consecutive levels whose fronts all have at most kMiniM rows form a band; the fronts of a band that
// hang together through parent links are one task, handled front by front by eight lanes (lane i owns
// row i), and one launch does all tasks of a band. Everything a front needs from another front of its
// band was written by the same eight lanes, so warp synchronization orders it.
//
// Bounded by the latency of a front's dependent loads (descriptor, structure, values) times the length
// of a task; 4 fronts per warp and 32 per CTA in 18 KB keep up to 256 fronts per SM in flight instead
// of 24. A front of a task costs 5 to 6 us however many run beside it, so bands are short: 4 levels
// take 0.23 ms per factorization of the models below, 8 levels 0.37 (tasks of up to 20 fronts), 16
// levels 0.58.
// 96 uneven AR1 + iid models (134 k fronts, 39 levels, B = 2), per call: factorization 465 -> 229 us,
// forward sweep 349 -> 158, backward sweep 215 -> 99, selected inverse 700 -> 270.
//
// Per front the arithmetic and its order are those of the one-warp kernels (factor_tiny_warp,
// fwd_tiny_warp, bwd_tiny_warp, k_selinv_tiny): same bits.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "devsym.hpp"
#include "snode_kernels.cuh"
#include "snode_large.cuh"

namespace inla {
namespace {

constexpr int kMiniM = 8;          // rows of a front
constexpr int kMiniLd = kMiniM + 1;
constexpr int kMiniLevels = 4;     // levels of a band
constexpr int kMiniGroups = 32;    // tasks per CTA (8 lanes each)
constexpr int kMiniThreads = kMiniGroups * 8;

// The caller's task: fronts list[f0 .. f0 + len), and the longest task of the warp.
struct MiniTask {
  int f0, len, longest;
};
__device__ __forceinline__ MiniTask mini_task(const DevSym& S, const int* __restrict__ ptr,
                                              const int* __restrict__ list, int ntask, int b, bool skip) {
  MiniTask t{0, 0, 0};
  const int c = blockIdx.x * kMiniGroups + (threadIdx.x >> 3);
  if (c < ntask) {
    t.f0 = ptr[c];
    t.len = ptr[c + 1] - t.f0;
    if (skip && front_skipped(S, list[t.f0], b)) t.len = 0;  // a task lies within one model
  }
  t.longest = __reduce_max_sync(0xffffffffu, t.len);
  return t;
}

__global__ void __launch_bounds__(kMiniThreads) k_factor_mini(DevSym S, const int* __restrict__ ptr,
                                                              const int* __restrict__ list, int ntask,
                                                              double* __restrict__ F, int64_t fstride) {
  __shared__ double sA[kMiniGroups][kMiniM * kMiniLd];
  const int l = threadIdx.x & 7, b = blockIdx.y;
  double* A = sA[threadIdx.x >> 3];
  double* Fb = F + (int64_t)b * fstride;
  const MiniTask T = mini_task(S, ptr, list, ntask, b, true);
  for (int it = 0; it < T.longest; ++it) {
    const bool on = it < T.len;
    const int s = on ? list[T.f0 + it] : 0;
    const int k = on ? sn_k(S, s) : 0, m = on ? sn_m(S, s) : 0;
    double* Fs = Fb + S.fptr[s];
    const int q0 = S.child_ptr[s], nch = on ? S.child_ptr[s + 1] - q0 : 0;
    const int kmax = __reduce_max_sync(0xffffffffu, k), cmax = __reduce_max_sync(0xffffffffu, nch);
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) A[l + j * kMiniLd] = (l < m && j < k) ? Fs[l + j * m] : 0.0;
    __syncwarp();
    for (int q = 0; q < cmax; ++q) {
      int rel = 0, rc = 0;
      double v[kMiniM];
      if (q < nch) {
        const int c = S.child_list[q0 + q], kc = sn_k(S, c), mc = sn_m(S, c);
        rc = mc - kc;
        const double* Uc = Fb + S.fptr[c] + (int64_t)kc * mc + kc;
        if (l < rc) {
          rel = S.relx[S.rowptr[c] + kc + l];
#pragma unroll
          for (int j = 0; j < kMiniM; ++j) v[j] = j <= l ? Uc[l + j * mc] : 0.0;
        }
      }
#pragma unroll
      for (int j = 0; j < kMiniM; ++j) {
        const int pc = __shfl_sync(0xffffffffu, rel, j, 8);
        if (l < rc && j <= l) A[rel + pc * kMiniLd] += v[j];
      }
      __syncwarp();
    }
    double a[kMiniM];
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) a[j] = A[l + j * kMiniLd];
#pragma unroll
    for (int p = 0; p < kMiniM; ++p) {
      if (p >= kmax) break;
      const double d = __shfl_sync(0xffffffffu, a[p], p, 8);
      const bool below = p < k && l > p && l < m;
      const double lip = below ? a[p] / d : 0.0;
#pragma unroll
      for (int j = p + 1; j < kMiniM; ++j) {
        const double u = __shfl_sync(0xffffffffu, a[p], j, 8);
        if (below && j <= l) a[j] -= lip * u;
      }
      if (below) a[p] = lip;
    }
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (l < m && j <= l) Fs[l + j * m] = a[j];
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kMiniThreads) k_fwd_mini(DevSym S, const int* __restrict__ ptr,
                                                           const int* __restrict__ list, int ntask,
                                                           const double* __restrict__ F, int64_t fstride, double* xp,
                                                           double* ub, int64_t ustride) {
  const int l = threadIdx.x & 7, b = blockIdx.y;
  const double* Fb = F + (int64_t)b * fstride;
  double* xb = xp + (int64_t)b * S.n;
  double* ubb = ub + (int64_t)b * ustride;
  const MiniTask T = mini_task(S, ptr, list, ntask, b, false);
  for (int it = 0; it < T.longest; ++it) {
    const bool on = it < T.len;
    const int s = on ? list[T.f0 + it] : 0;
    const int k = on ? lg_k(S, s) : 0, m = on ? lg_m(S, s) : 0, f = S.first[s];
    const double* Fs = Fb + S.fptr[s];
    const int kmax = __reduce_max_sync(0xffffffffu, k);
    double L[kMiniM];  // row l of the panel, D at l < k
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) L[j] = (l < m && j < k && j <= l) ? Fs[l + j * m] : 0.0;
    double yi = 0.0;
    if (l < m) {
      yi = l < k ? xb[f + l] : 0.0;
      const int row = S.rowptr[s] + l;
      for (int q = S.rsp[row], e = S.rsp[row + 1]; q < e; ++q) yi += ubb[S.rss[q]];
    }
    double yd = l < k ? yi : 0.0;
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (j >= kmax) break;
      const double yj = __shfl_sync(0xffffffffu, yd, j, 8);
      if (j < k && l > j && l < k) yd -= L[j] * yj;
    }
    double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (j >= kmax) break;
      const double yj = __shfl_sync(0xffffffffu, yd, j, 8);
      if (j < k) a[j & 3] += L[j] * yj;
    }
    double d = 1.0;
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (j == l) d = L[j];
    if (l < k) xb[f + l] = yd / d;
    else if (l < m) ubb[S.uoff[s] + l - k] = yi - ((a[0] + a[1]) + (a[2] + a[3]));
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kMiniThreads) k_bwd_mini(DevSym S, const int* __restrict__ ptr,
                                                           const int* __restrict__ list, int ntask,
                                                           const double* __restrict__ F, int64_t fstride, double* xp) {
  const int l = threadIdx.x & 7, b = blockIdx.y;
  const double* Fb = F + (int64_t)b * fstride;
  double* xb = xp + (int64_t)b * S.n;
  const MiniTask T = mini_task(S, ptr, list, ntask, b, false);
  for (int it = 0; it < T.longest; ++it) {  // parents first
    const bool on = it < T.len;
    const int s = on ? list[T.f0 + T.len - 1 - it] : 0;
    const int k = on ? lg_k(S, s) : 0, m = on ? lg_m(S, s) : 0, f = S.first[s];
    const double* Fs = Fb + S.fptr[s];
    const int kmax = __reduce_max_sync(0xffffffffu, k);
    const int ri = k + l;
    double Lb[kMiniM], Lc[kMiniM];  // L[ri][j] and L[i][l]
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      Lb[j] = (ri < m && j < k) ? Fs[ri + j * m] : 0.0;
      Lc[j] = (j < k && l < j) ? Fs[j + l * m] : 0.0;
    }
    double xl = l < m ? xb[S.rows[S.rowptr[s] + l]] : 0.0;
    const double xs = __shfl_sync(0xffffffffu, xl, ri & 7, 8);
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (j >= kmax) break;
      double acc = ri < m ? Lb[j] * xs : 0.0;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, 8);
      acc = __shfl_sync(0xffffffffu, acc, 0, 8);
      if (l == j && j < k) xl -= acc;
    }
#pragma unroll
    for (int i = kMiniM - 1; i >= 0; --i) {
      if (i >= kmax) continue;
      const double xi = __shfl_sync(0xffffffffu, xl, i, 8);
      if (i < k && l < i) xl -= Lc[i] * xi;
    }
    if (l < k) xb[f + l] = xl;
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kMiniThreads) k_selinv_mini(DevSym S, const int* __restrict__ ptr,
                                                              const int* __restrict__ list, int ntask,
                                                              const double* __restrict__ F, double* Sg,
                                                              int64_t fstride) {
  __shared__ double sS[kMiniGroups][kMiniM * kMiniLd];
  __shared__ double sL[kMiniGroups][kMiniM * kMiniLd];
  const int l = threadIdx.x & 7, b = blockIdx.y;
  double* Sm = sS[threadIdx.x >> 3];
  double* L = sL[threadIdx.x >> 3];
  const double* Fb = F + (int64_t)b * fstride;
  double* Sb = Sg + (int64_t)b * fstride;
  const MiniTask T = mini_task(S, ptr, list, ntask, b, false);
  for (int it = 0; it < T.longest; ++it) {  // parents first
    const bool on = it < T.len;
    const int s = on ? list[T.f0 + T.len - 1 - it] : 0;
    const int k = on ? sn_k(S, s) : 0, m = on ? sn_m(S, s) : 0, r = m - k;
    const double* Fs = Fb + S.fptr[s];
    double* Ss = Sb + S.fptr[s];
    const int kmax = __reduce_max_sync(0xffffffffu, k);
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (l < m && j < k) L[l + j * kMiniLd] = Fs[l + j * m];
    if (r > 0) {
      const int p = S.parent[s], mp = sn_m(S, p);
      const double* Sp = Sb + S.fptr[p];
      const int* rel = S.relx + S.rowptr[s] + k;
      if (l < r) {
        const int ri = rel[l];
        double v[kMiniM];
#pragma unroll
        for (int j = 0; j < kMiniM; ++j) v[j] = j <= l ? parent_sigma(Sp, mp, ri, rel[j]) : 0.0;
#pragma unroll
        for (int j = 0; j < kMiniM; ++j)
          if (j <= l) {
            Sm[(k + l) + (k + j) * kMiniLd] = v[j];
            Sm[(k + j) + (k + l) * kMiniLd] = v[j];
          }
      }
    }
    __syncwarp();
    for (int jj = kmax - 1; jj >= 0; --jj) {
      const bool col = jj < k, mine = col && l > jj && l < m;
      double acc = 0.0;
      if (mine)
        for (int i = jj + 1; i < m; ++i) acc += L[i + jj * kMiniLd] * Sm[i + l * kMiniLd];
      __syncwarp();
      if (mine) {
        Sm[l + jj * kMiniLd] = -acc;
        Sm[jj + l * kMiniLd] = -acc;
      }
      __syncwarp();
      double t = mine ? L[l + jj * kMiniLd] * Sm[l + jj * kMiniLd] : 0.0;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o, 8);
      if (col && l == 0) Sm[jj + jj * kMiniLd] = 1.0 / L[jj + jj * kMiniLd] - t;
      __syncwarp();
    }
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (l < m && j <= l) Ss[l + j * m] = Sm[l + j * kMiniLd];
    __syncwarp();
  }
}

}  // namespace
}  // namespace inla
