// Trees of fronts with at most eight rows (independent AR1-type models: half a million fronts of at
// most seven rows on 30 to 40 levels, most of them links of a chain). A launch per level and a warp
// per front spends the time on launches with few fronts and on warps with 25 idle lanes. Here
// consecutive levels whose fronts all have at most kMiniM rows form a band; the fronts of a band that
// hang together through parent links are one task, handled front by front by eight lanes (lane i owns
// row i), and one launch does all tasks of a band. Everything a front needs from another front of its
// band was written by the same eight lanes, so warp synchronization orders it.
//
// Bounded by the instructions and the load latency of one front after the other in a task (2.7 us per
// front of the factorization with few tasks on the chip; with many, half of the issue slots are taken).
// So what a front needs besides its children's results is loaded before the front below it is finished:
// its line of the front table (two ahead), the panel (copied to shared memory without going through
// registers), its children's lines and its rows' places. Reading these through list, first, rowptr, fptr
// and child_list when the front's turn came cost 5 to 6 us per front. Bands are short because a task is as
// long as the fronts that hang together: 4 levels give tasks of up to 9 fronts and 0.17 ms per
// factorization of the models below, 6 levels 0.25, 8 levels 0.34.
// Those are chains. Where fronts branch, a band stops before the level that would make a task longer than
// kMiniTask fronts: a star or a nested grouping is one component, and without the limit one task. Star of
// 24 000 leaves, factorization / solve / selected inverse without the limit 25.6 / 24.9 / 23.5 ms, with it
// 12.6 / 0.98 / 0.04 ms (12.6 for 4 to 40 fronts). 1000 stars of 12 leaves, one task each: selected inverse
// 23 us, in level launches 28; 200 of 60: 101 / 88 / 71 us as tasks, 79 / 30 / 30 in level launches; one of
// 40: 65 / 51 / 50 and 47 / 20 / 14. Adding a child from outside the band takes a quarter of a front's time:
// chain of 100 hubs with 400 leaves each 2.49 / 0.35 / 0.09 ms with fronts counted alone, 1.83 / 0.23 / 0.10
// with the children counted; 2000 hubs of 10 leaves 241 / 127 / 82 and 154 / 96 / 60 us (weights 1 / 2 and
// 1 / 8: 166 and 187 us). 96 uneven AR1 + iid models: the same within 2 % for every limit and weight.
// Registers: a spill costs more than a resident CTA gains (factorization, 4 / 5 / 6 / 8 CTAs of 128
// threads: 172 / 179 / 200 / 251 us); leaving the unrolled loops at the warp's largest front costs more
// than the skipped steps (224 us).
// 96 uneven AR1 + iid models (134 k fronts, 39 levels, B = 2), per call, level launches -> bands -> with
// the loads ahead: factorization 465 -> 229 -> 172 us, forward sweep 349 -> 164 -> 106, backward sweep
// 215 -> 100 -> 82, selected inverse 700 -> 275 -> 158.
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
constexpr int kMiniTask = 16;      // fronts of a task
constexpr int kMiniChildren = 4;   // children from outside the band that count as a front
constexpr int kMiniGroups = 16;    // tasks per CTA (8 lanes each)
constexpr int kMiniThreads = kMiniGroups * 8;

// The caller's task: fronts f0 .. f0 + len of the table, and the longest task of the warp.
struct MiniTask {
  int f0, len, longest;
};
__device__ __forceinline__ MiniTask mini_task(const DevSym& S, const MiniTables& M, int ntask, int b, bool skip) {
  MiniTask t{0, 0, 0};
  const int c = blockIdx.x * kMiniGroups + (threadIdx.x >> 3);
  if (c < ntask) {
    t.f0 = M.ptr[c];
    t.len = M.ptr[c + 1] - t.f0;
    if (skip && front_skipped(S, M.list[t.f0], b)) t.len = 0;  // a task lies within one model
  }
  t.longest = __reduce_max_sync(0xffffffffu, t.len);
  return t;
}
// Front `it` of the task, parents first for `Up` = false; a front without rows past the end.
template <bool Up>
__device__ __forceinline__ MiniFront mini_front(const MiniTables& M, const MiniTask& T, int it) {
  if (it >= T.len) return MiniFront{};
  return M.front[T.f0 + (Up ? it : T.len - 1 - it)];
}

__global__ void __launch_bounds__(kMiniThreads, 4) k_factor_mini(DevSym S, MiniTables M, int ntask,
                                                              double* __restrict__ F, int64_t fstride) {
  __shared__ double sA[2][kMiniGroups][kMiniM * kMiniLd];
  const int l = threadIdx.x & 7, b = blockIdx.y;
  double* Fb = F + (int64_t)b * fstride;
  const MiniTask T = mini_task(S, M, ntask, b, true);
  MiniFront cur = mini_front<true>(M, T, 0), nxt = mini_front<true>(M, T, 1);
  MiniChild ch{0, 0, 0};  // child l of the front that comes next
  auto prefetch = [&](const MiniFront& f, double* A) {
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (l < f.m && j < f.k) cp_async8(&A[l + j * kMiniLd], Fb + f.fptr + l + j * f.m);
      else A[l + j * kMiniLd] = 0.0;
    }
    cp_async_commit();
    if (l < f.nch) ch = M.child[f.child0 + l];
  };
  prefetch(cur, sA[0][threadIdx.x >> 3]);
  for (int it = 0; it < T.longest; ++it) {
    const int k = cur.k, m = cur.m, nch = cur.nch, child0 = cur.child0;
    double* Fs = Fb + cur.fptr;
    double* A = sA[it & 1][threadIdx.x >> 3];
    const int kmax = __reduce_max_sync(0xffffffffu, k), cmax = __reduce_max_sync(0xffffffffu, nch);
    MiniChild mine = ch;
    double v[kMiniM];  // row l of the update of child q, and its place in the parent
    int rel, rc;
    auto fetch = [&](int q) {
      const int64_t src = __shfl_sync(0xffffffffu, mine.src, q & 7, 8);
      const int dim = __shfl_sync(0xffffffffu, mine.dim, q & 7, 8);
      const int r0 = __shfl_sync(0xffffffffu, mine.rel, q & 7, 8);
      rc = q < nch ? dim & 15 : 0;
      rel = 0;
      if (l < rc) {
        rel = S.relx[r0 + l];
#pragma unroll
        for (int j = 0; j < kMiniM; ++j) v[j] = j <= l ? Fb[src + l + (int64_t)j * (dim >> 4)] : 0.0;
      }
    };
    fetch(0);
    cur = nxt;
    nxt = mini_front<true>(M, T, it + 2);
    prefetch(cur, sA[(it + 1) & 1][threadIdx.x >> 3]);
    cp_async_wait<1>();
    __syncwarp();
    for (int q = 0; q < cmax; ++q) {
      if (q) {
        if ((q & 7) == 0 && q + l < nch) mine = M.child[child0 + q + l];
        fetch(q);
      }
      double t[kMiniM];  // the targets of one child are distinct: all loads before the stores
      int at[kMiniM];
#pragma unroll
      for (int j = 0; j < kMiniM; ++j) {
        at[j] = rel + __shfl_sync(0xffffffffu, rel, j, 8) * kMiniLd;
        if (l < rc && j <= l) t[j] = A[at[j]];
      }
#pragma unroll
      for (int j = 0; j < kMiniM; ++j)
        if (l < rc && j <= l) A[at[j]] = t[j] + v[j];
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

__global__ void __launch_bounds__(kMiniThreads, 6) k_fwd_mini(DevSym S, MiniTables M, int ntask,
                                                           const double* __restrict__ F, int64_t fstride, double* xp,
                                                           double* ub, int64_t ustride) {
  __shared__ double sL[2][kMiniM][kMiniThreads];  // row l of the panels (D at l < k), per thread
  const int l = threadIdx.x & 7, b = blockIdx.y;
  const double* Fb = F + (int64_t)b * fstride;
  double* xb = xp + (int64_t)b * S.n;
  double* ubb = ub + (int64_t)b * ustride;
  const MiniTask T = mini_task(S, M, ntask, b, false);
  // fronts it, it + 1, it + 2; of front it: the right-hand side and the first two of the row's children
  // entries; of front it + 1: the row's range of entries
  MiniFront cur = mini_front<true>(M, T, 0), nxt = mini_front<true>(M, T, 1), nx2 = mini_front<true>(M, T, 2);
  double x = 0.0;
  int e0 = 0, e1 = 0, n0 = 0, n1 = 0, s0 = 0, s1 = 0;
  auto range = [&](const MiniFront& f) {
    n0 = n1 = 0;
    if (l < f.m) {
      n0 = S.rsp[f.rowptr + l];
      n1 = S.rsp[f.rowptr + l + 1];
    }
  };
  auto prefetch = [&](const MiniFront& f, int it) {
    e0 = n0;
    e1 = n1;
    if (e0 < e1) s0 = S.rss[e0];
    if (e0 + 1 < e1) s1 = S.rss[e0 + 1];
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (l < f.m && j < f.k && j <= l) cp_async8(&sL[it & 1][j][threadIdx.x], Fb + f.fptr + l + j * f.m);
    cp_async_commit();
    x = l < f.k ? xb[f.first + l] : 0.0;
  };
  range(cur);
  prefetch(cur, 0);
  range(nxt);
  for (int it = 0; it < T.longest; ++it) {
    const int k = cur.k, m = cur.m, f = cur.first, uo = cur.uoff;
    const int kmax = __reduce_max_sync(0xffffffffu, k);
    const double u0 = e0 < e1 ? ubb[s0] : 0.0, u1 = e0 + 1 < e1 ? ubb[s1] : 0.0;
    double yi = x;
    const int q0 = e0, q1 = e1;
    cur = nxt;
    nxt = nx2;
    nx2 = mini_front<true>(M, T, it + 3);
    prefetch(cur, it + 1);
    range(nxt);
    if (q0 < q1) yi += u0;
    if (q0 + 1 < q1) yi += u1;
    for (int q = q0 + 2; q < q1; ++q) yi += ubb[S.rss[q]];
    cp_async_wait<1>();
    double L[kMiniM];
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) L[j] = (l < m && j < k && j <= l) ? sL[it & 1][j][threadIdx.x] : 0.0;
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
    if (l < k) xb[f + l] = yd / sL[it & 1][l][threadIdx.x];
    else if (l < m) ubb[uo + l - k] = yi - ((a[0] + a[1]) + (a[2] + a[3]));
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kMiniThreads, 6) k_bwd_mini(DevSym S, MiniTables M, int ntask,
                                                           const double* __restrict__ F, int64_t fstride, double* xp) {
  __shared__ double sB[2][kMiniM][kMiniThreads], sC[2][kMiniM][kMiniThreads];  // L[k + l][j], L[j][l]
  const int l = threadIdx.x & 7, b = blockIdx.y;
  const double* Fb = F + (int64_t)b * fstride;
  double* xb = xp + (int64_t)b * S.n;
  const MiniTask T = mini_task(S, M, ntask, b, false);
  MiniFront cur = mini_front<false>(M, T, 0), nxt = mini_front<false>(M, T, 1);
  int row = 0;
  auto prefetch = [&](const MiniFront& f, int it) {
    const double* Fs = Fb + f.fptr;
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (f.k + l < f.m && j < f.k) cp_async8(&sB[it & 1][j][threadIdx.x], Fs + f.k + l + j * f.m);
      if (j < f.k && l < j) cp_async8(&sC[it & 1][j][threadIdx.x], Fs + j + l * f.m);
    }
    cp_async_commit();
    if (l < f.m) row = S.rows[f.rowptr + l];
  };
  prefetch(cur, 0);
  for (int it = 0; it < T.longest; ++it) {
    const int k = cur.k, m = cur.m, f = cur.first, ri = k + l;
    const int kmax = __reduce_max_sync(0xffffffffu, k);
    double xl = l < m ? xb[row] : 0.0;
    cur = nxt;
    nxt = mini_front<false>(M, T, it + 2);
    prefetch(cur, it + 1);
    cp_async_wait<1>();
    const double xs = __shfl_sync(0xffffffffu, xl, ri & 7, 8);
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      if (j >= kmax) break;
      double acc = ri < m && j < k ? sB[it & 1][j][threadIdx.x] * xs : 0.0;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, 8);
      acc = __shfl_sync(0xffffffffu, acc, 0, 8);
      if (l == j && j < k) xl -= acc;
    }
#pragma unroll
    for (int i = kMiniM - 1; i >= 0; --i) {
      if (i >= kmax) continue;
      const double xi = __shfl_sync(0xffffffffu, xl, i, 8);
      if (i < k && l < i) xl -= sC[it & 1][i][threadIdx.x] * xi;
    }
    if (l < k) xb[f + l] = xl;
    __syncwarp();
  }
}

__global__ void __launch_bounds__(kMiniThreads, 6) k_selinv_mini(DevSym S, MiniTables M, int ntask,
                                                              const double* __restrict__ F, double* Sg,
                                                              int64_t fstride) {
  __shared__ double sS[kMiniGroups][kMiniM * kMiniLd];
  __shared__ double sL[kMiniGroups][kMiniM * kMiniLd];
  const int l = threadIdx.x & 7, b = blockIdx.y;
  double* Sm = sS[threadIdx.x >> 3];
  double* L = sL[threadIdx.x >> 3];
  const double* Fb = F + (int64_t)b * fstride;
  double* Sb = Sg + (int64_t)b * fstride;
  const MiniTask T = mini_task(S, M, ntask, b, false);
  MiniFront cur = mini_front<false>(M, T, 0), nxt = mini_front<false>(M, T, 1);
  double pv[kMiniM];  // row l of the panel, and the place of below-row l, of the front that comes next
  int rel = 0;
  auto prefetch = [&](const MiniFront& f) {
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) pv[j] = (l < f.m && j < f.k) ? Fb[f.fptr + l + j * f.m] : 0.0;
    if (l < f.m - f.k) rel = S.relx[f.rowptr + f.k + l];
  };
  prefetch(cur);
  for (int it = 0; it < T.longest; ++it) {
    const int k = cur.k, m = cur.m, r = m - k;
    double* Ss = Sb + cur.fptr;
    const int kmax = __reduce_max_sync(0xffffffffu, k);
    double v[kMiniM];
#pragma unroll
    for (int j = 0; j < kMiniM; ++j) {
      const int rj = __shfl_sync(0xffffffffu, rel, j, 8);
      v[j] = j <= l && l < r ? parent_sigma(Sb + cur.pptr, cur.pm, rel, rj) : 0.0;
      if (l < m && j < k) L[l + j * kMiniLd] = pv[j];
    }
    cur = nxt;
    nxt = mini_front<false>(M, T, it + 2);
    prefetch(cur);
#pragma unroll
    for (int j = 0; j < kMiniM; ++j)
      if (j <= l && l < r) {
        Sm[(k + l) + (k + j) * kMiniLd] = v[j];
        Sm[(k + j) + (k + l) * kMiniLd] = v[j];
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
