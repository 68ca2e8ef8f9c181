// Host orchestration of the batched supernodal kernels.
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <atomic>
#include <list>
#include <mutex>

#include "gpu_factor.hpp"
#include "host_par.hpp"
#include "snode_kernels.cuh"
#include "snode_large.cuh"
#include "snode_mini.cuh"
#include "snode_persist.cuh"

namespace inla {

namespace {
inline int cdiv(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// Panel forms of a level's large fronts (entries of the per-level schedule).
constexpr char kFormSplit = 0, kFormFused = 1, kFormLookahead = 2, kNumForms = 3;
// Process-wide panel form for engines built from now on: -1 the autotuner's choice per level
// (default), otherwise that form at every level.
std::atomic<int> g_panel_form{-1};

// Trailing-update tile on eight warps (32 x 16 warp tiles; the body the persistent schedule
// runs too), two CTAs per SM: 16 warps per SM where the four-warp form with 32 x 32 warp tiles
// fitted 12 (168 registers, 70 KB of staging). Measured on the SPDE 200^2 factorization: 7 %
// faster at B = 1, 3 % at B = 7, 2 % at B = 21.
__global__ void __launch_bounds__(256, 2) k_update64w8(DevSym S, const int* __restrict__ list, int j0,
                                                         double* __restrict__ F, int64_t fstride,
                                                         const double* __restrict__ dcache) {
  extern __shared__ double smu[];
  const double* dc = dcache ? dcache + ((int64_t)blockIdx.x * gridDim.y + blockIdx.y) * (kB64 * kB64) : nullptr;
  update64w8_body(S, list[blockIdx.x], blockIdx.y, blockIdx.z, j0, F, fstride, dc, smu);
}

// Diagonal blocks of step j0 >= 64 in the look-ahead form, one CTA per (front, problem).
__global__ void __launch_bounds__(256, 2) k_diag_next(DevSym S, const int* __restrict__ list, int j0,
                                                      double* __restrict__ F, int64_t fstride,
                                                      double* __restrict__ linv) {
  extern __shared__ double smu[];
  diag_next_body(S, list[blockIdx.x], blockIdx.y, j0, F, fstride, linv, smu);
}

// Parent columns per extend-add CTA: the m-row slice must fit in shared memory.
inline int gather_cols(int m) { return std::max(1, std::min(kGatherCols, (200 * 1024) / (8 * std::max(m, 1)))); }

// The dynamic shared-memory limit is an attribute of the kernel on the current
// device, shared by every engine in the process. Engines of different sizes
// need different limits, so the attribute only ever rises: a smaller engine
// built later must not lower it below what a larger one still launches with.
std::mutex g_smem_mu;
std::map<std::pair<const void*, int>, int> g_smem_set;  // (kernel, device) -> limit set

template <class K>
void set_smem(K kernel, int bytes) {
  int dev = 0;
  INLA_CUDA(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(g_smem_mu);
  int& cur = g_smem_set[{(const void*)kernel, dev}];
  if (bytes <= cur) return;
  INLA_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
  cur = bytes;
}
}  // namespace

// Host tables of a symbolic analysis that the engine uploads (32-bit supernode arrays, front
// offsets, the panel map and the front positions of the input entries). They depend on the
// analysis only, so they are built once per analysis id and shared by every engine created on
// it (a model rebuilt on the same mesh skips the ~10-20 ms of building them); at most
// kMapsCacheBytes are kept, most recently used first.
namespace {
constexpr size_t kMapsCacheBytes = size_t(1) << 30;
std::mutex g_maps_mu;
std::list<std::pair<uint64_t, std::shared_ptr<const HostMaps>>> g_maps;
size_t g_maps_bytes = 0;

size_t host_maps_bytes(const HostMaps& M) {
  return sizeof(int) * (M.first.size() + M.rowptr.size() + M.rows.size() + M.relx.size() + M.child_ptr.size() +
                        M.child_list.size() + M.parent.size() + M.uoff.size() + M.perm.size() + M.pmap.size() + M.rsp.size() + M.rss.size()) +
         sizeof(int64_t) * (M.fptr.size() + M.lptr.size() + M.dpos.size() + M.spos.size() + M.spos_full.size());
}

std::shared_ptr<const HostMaps> build_host_maps(const Symbolic& S) {
  auto out = std::make_shared<HostMaps>();
  HostMaps& M = *out;
  const int64_t ns = S.nsuper, n = S.n;
  const int64_t nnz_ = (int64_t)S.rowidx.size();
  std::vector<int>&first = M.first, &rowptr = M.rowptr, &rows = M.rows, &relx = M.relx, &child_ptr = M.child_ptr,
                   &child_list = M.child_list, &parent = M.parent, &uoff = M.uoff, &perm = M.perm;
  std::vector<int64_t>&fptr = M.fptr, &lptr = M.lptr, &dpos = M.dpos;
  first.resize(ns + 1);
  rowptr.resize(ns + 1);
  rows.resize(S.sn_rows.size());
  relx.assign(S.sn_rows.size(), -1);
  child_ptr.resize(ns + 1);
  child_list.resize(S.child_list.size());
  parent.resize(ns);
  uoff.assign(ns + 1, 0);
  perm.resize(n);
  fptr.assign(ns + 1, 0);
  lptr.resize(ns + 1);
  dpos.resize(n);
  for (int64_t s = 0; s <= ns; ++s) {
    first[s] = (int)S.sn_first[s];
    rowptr[s] = (int)S.sn_rowptr[s];
    child_ptr[s] = (int)S.child_ptr[s];
    lptr[s] = S.sn_lptr[s];
  }
  for (size_t i = 0; i < S.sn_rows.size(); ++i) rows[i] = (int)S.sn_rows[i];
  for (size_t i = 0; i < S.child_list.size(); ++i) child_list[i] = (int)S.child_list[i];
  for (int64_t s = 0; s < ns; ++s) {
    int64_t k = S.sn_first[s + 1] - S.sn_first[s], m = S.sn_rowptr[s + 1] - S.sn_rowptr[s];
    parent[s] = (int)S.sn_parent[s];
    fptr[s + 1] = fptr[s] + m * m;
    uoff[s + 1] = uoff[s] + (int)(m - k);
    for (int64_t t = 0; t < m - k; ++t) relx[S.sn_rowptr[s] + k + t] = S.rel[S.rel_ptr[s] + t];
    for (int64_t j = S.sn_first[s]; j < S.sn_first[s + 1]; ++j) {
      int64_t c = j - S.sn_first[s];
      dpos[j] = fptr[s] + c * (m + 1);
    }
  }
  for (int64_t j = 0; j < n; ++j) perm[j] = (int)S.perm[j];

  // children's update entries per front row, in child order
  {
    const size_t nrows = S.sn_rows.size();
    std::vector<int>&rsp = M.rsp, &rss = M.rss;
    rsp.assign(nrows + 1, 0);
    rss.resize(std::max(uoff[ns], 1));
    auto each = [&](auto&& use) {  // (row of the parent, update entry), children in their list's order
      for (int64_t s = 0; s < ns; ++s)
        for (int q = child_ptr[s]; q < child_ptr[s + 1]; ++q) {
          const int c = child_list[q], kc = first[c + 1] - first[c], rc = uoff[c + 1] - uoff[c];
          for (int t = 0; t < rc; ++t) use(rowptr[s] + relx[rowptr[c] + kc + t], uoff[c] + t);
        }
    };
    each([&](int row, int) { ++rsp[row + 1]; });
    for (size_t i = 0; i < nrows; ++i) rsp[i + 1] += rsp[i];
    std::vector<int> fill(rsp.begin(), rsp.end() - 1);
    each([&](int row, int src) { rss[fill[row]++] = src; });
  }

  // panel map (compact panel index -> input entry) and front positions of input entries
  std::vector<int>& pmap = M.pmap;
  std::vector<int64_t>&spos = M.spos, &spos_full = M.spos_full;
  pmap.assign(S.nnz_l_stored, -1);
  spos.assign(nnz_, -1);
  spos_full.assign(nnz_, -1);
  parallel_for(n, [&](int64_t c0, int64_t c1) {  // disjoint writes: entry p, panel slot qmap[p]
    for (int64_t c = c0; c < c1; ++c)
      for (int64_t p = S.colptr[c]; p < S.colptr[c + 1]; ++p) {
        int64_t i = S.iperm[S.rowidx[p]], j = S.iperm[c];
        int64_t lo = std::min(i, j), hi = std::max(i, j);
        int64_t s = S.col_to_sn[lo];
        const int64_t* R = S.sn_rows.data() + S.sn_rowptr[s];
        int64_t m = S.sn_rowptr[s + 1] - S.sn_rowptr[s];
        const int64_t* it = std::lower_bound(R, R + m, hi);
        if (it == R + m || *it != hi) throw std::runtime_error("entry outside the filled pattern");
        spos_full[p] = fptr[s] + (lo - S.sn_first[s]) * m + (it - R);
        int64_t q = S.qmap[p];
        if (q < 0) continue;
        pmap[q] = (int)p;
        spos[p] = spos_full[p];
      }
  });
  return out;
}
}  // namespace

void release_host_maps() {
  std::lock_guard<std::mutex> lk(g_maps_mu);
  g_maps.clear();
  g_maps_bytes = 0;
}

std::shared_ptr<const HostMaps> host_maps(const Symbolic& S) {
  // without the symbolic cache every engine has an analysis of its own: nothing to share
  static const bool on = std::getenv("INLA_NO_SYMBOLIC_CACHE") == nullptr;
  if (!on) return build_host_maps(S);
  if (S.id != 0) {
    std::lock_guard<std::mutex> lk(g_maps_mu);
    for (auto it = g_maps.begin(); it != g_maps.end(); ++it)
      if (it->first == S.id) {
        g_maps.splice(g_maps.begin(), g_maps, it);
        return g_maps.front().second;
      }
  }
  std::shared_ptr<const HostMaps> m = build_host_maps(S);
  if (S.id != 0) {
    const size_t bytes = host_maps_bytes(*m);
    std::lock_guard<std::mutex> lk(g_maps_mu);
    if (bytes <= kMapsCacheBytes / 2) {
      g_maps.emplace_front(S.id, m);
      g_maps_bytes += bytes;
      while (g_maps_bytes > kMapsCacheBytes && g_maps.size() > 1) {
        g_maps_bytes -= host_maps_bytes(*g_maps.back().second);
        g_maps.pop_back();
      }
    }
  }
  return m;
}

GpuFactor::GpuFactor(const Symbolic& sym, int max_batch, cudaStream_t stream)
    : sym_(sym), max_batch_(max_batch), stream_(stream) {
  const auto tstart = std::chrono::steady_clock::now();
  if (max_batch < 1) throw std::runtime_error("max_batch must be >= 1");
  const Symbolic& S = sym_;
  const int64_t ns = S.nsuper, n = S.n;
  nnz_ = (int64_t)S.rowidx.size();
  if (n >= (1LL << 31) || (int64_t)S.sn_rows.size() >= (1LL << 31) || nnz_ >= (1LL << 31))
    throw std::runtime_error("problem too large for 32-bit indices");
  if (S.max_m > 25600) throw std::runtime_error("front with more than 25600 rows (extend-add slice exceeds shared memory)");

  const std::shared_ptr<const HostMaps> maps = host_maps(S);
  const HostMaps& M = *maps;
  const std::vector<int>&first = M.first, &rowptr = M.rowptr, &rows = M.rows, &relx = M.relx,
                  &child_ptr = M.child_ptr, &child_list = M.child_list, &parent = M.parent, &uoff = M.uoff,
                  &perm = M.perm, &pmap = M.pmap;
  const std::vector<int64_t>&fptr = M.fptr, &lptr = M.lptr, &dpos = M.dpos, &spos = M.spos,
                      &spos_full = M.spos_full;
  ftotal_ = fptr[ns];
  usum_ = uoff[ns];

  const auto tm1 = std::chrono::steady_clock::now();
  d_first_.upload(first, stream_);
  d_rowptr_.upload(rowptr, stream_);
  d_rows_.upload(rows, stream_);
  d_relx_.upload(relx, stream_);
  d_child_ptr_.upload(child_ptr, stream_);
  d_child_list_.upload(child_list, stream_);
  d_parent_.upload(parent, stream_);
  d_uoff_.upload(uoff, stream_);
  d_perm_.upload(perm, stream_);
  d_rsp_.upload(M.rsp, stream_);
  d_rss_.upload(M.rss, stream_);
  d_fptr_.upload(fptr, stream_);
  d_lptr_.upload(lptr, stream_);
  d_dpos_.upload(dpos, stream_);
  d_pmap_.upload(pmap, stream_);
  spos_.upload(spos, stream_);
  spos_full_.upload(spos_full, stream_);

  ds_.n = (int)n;
  ds_.ns = (int)ns;
  ds_.first = d_first_.p;
  ds_.rowptr = d_rowptr_.p;
  ds_.rows = d_rows_.p;
  ds_.relx = d_relx_.p;
  ds_.fptr = d_fptr_.p;
  ds_.lptr = d_lptr_.p;
  ds_.child_ptr = d_child_ptr_.p;
  ds_.child_list = d_child_list_.p;
  ds_.parent = d_parent_.p;
  ds_.uoff = d_uoff_.p;
  ds_.dpos = d_dpos_.p;
  ds_.perm = d_perm_.p;
  ds_.rsp = d_rsp_.p;
  ds_.rss = d_rss_.p;

  const auto tm2 = std::chrono::steady_clock::now();
  // inverse-block cache: one 64 x 64 block per 64 pivot columns of every large front
  {
    std::vector<int> lbo(ns, -1);
    int64_t nblk = 0;
    for (int64_t s = 0; s < ns; ++s) {
      const int64_t k = S.sn_first[s + 1] - S.sn_first[s], m = S.sn_rowptr[s + 1] - S.sn_rowptr[s];
      if (m > kSmallB) {
        lbo[s] = (int)nblk;
        nblk += cdiv(k, kB64);
      }
    }
    d_lbo_.upload(lbo, stream_);
    ds_.lbo = d_lbo_.p;
    ds_.lstride = nblk * kB64 * kB64;
    linv_.alloc((size_t)max_batch_ * std::max<int64_t>(ds_.lstride, 1));
  }
  // value-fill chunks over the compact panel numbering (kFillChunk entries for
  // the input-values fill, kFillModelChunk for the component-model fill)
  {
    ntot_ = S.sn_lptr[ns];
    auto chunk_table = [&](int chunk, int& count, DBuf<int>& dst) {
      count = std::max(1, cdiv(ntot_, chunk));
      std::vector<int> csn(count + 1);
      int64_t s = 0;
      for (int c = 0; c < count; ++c) {
        const int64_t e = (int64_t)c * chunk;
        while (s + 1 < ns && S.sn_lptr[s + 1] <= e) ++s;
        csn[c] = (int)s;
      }
      csn[count] = (int)(ns - 1);
      dst.upload(csn, stream_);
    };
    chunk_table(kFillChunk, nfill_, d_csn_);
    chunk_table(kFillModelChunk, nfillm_, d_csnm_);
  }
  nldchunk_ = std::max(1, cdiv(n, kLogdetChunk));
  ldpart_.alloc((size_t)max_batch_ * nldchunk_);
  ldflag_.alloc((size_t)max_batch_ * nldchunk_);
  ldticket_.alloc((size_t)max_batch_);
  INLA_CUDA(cudaMemsetAsync(ldticket_.p, 0, sizeof(unsigned) * max_batch_, stream_));

  const auto tm3 = std::chrono::steady_clock::now();
  plan_levels(M);
  // children's columns of the large fronts (DevSym::gcol)
  {
    std::vector<int64_t> gptr(ns, 0);
    std::vector<GatherCol> gcol;
    std::vector<int> cursor;
    bool large = false;
    for (const LevelPlan& P : levels_)
      for (int s : P.large) {
        large = true;
        const int* rsp = M.rsp.data() + rowptr[s];
        const int m = rowptr[s + 1] - rowptr[s];
        gptr[s] = (int64_t)gcol.size() - rsp[0];
        gcol.resize(gcol.size() + (rsp[m] - rsp[0]));
        cursor.assign(rsp, rsp + m);
        for (int64_t q = S.child_ptr[s]; q < S.child_ptr[s + 1]; ++q) {
          const int c = (int)S.child_list[q];
          const int kc = first[c + 1] - first[c], mc = rowptr[c + 1] - rowptr[c];
          for (int i = kc; i < mc; ++i)
            gcol[gptr[s] + cursor[relx[rowptr[c] + i]]++] = {fptr[c] + (int64_t)i * mc + i, mc - i, rowptr[c] + i};
        }
      }
    if (large) {  // also where no large front has children: the kernel reads gptr
      d_gptr_.upload(gptr, stream_);
      d_gcol_.upload(gcol, stream_);
      ds_.gptr = d_gptr_.p;
      ds_.gcol = d_gcol_.p;
    }
  }

  // the look-ahead form needs its stream where a large front has more than one block of pivots
  if (std::any_of(levels_.begin(), levels_.end(), [](const LevelPlan& P) { return P.kmax_large > kB64; }))
    chain_.create();
  panel_form_ = g_panel_form.load();
  plan_persist();
  const auto ta = std::chrono::steady_clock::now();
  F_.alloc((size_t)max_batch_ * ftotal_);
  xp_.alloc((size_t)max_batch_ * n);
  ub_.alloc((size_t)max_batch_ * std::max<int64_t>(usum_, 1));
  logdet_.alloc(max_batch_);
  status_.alloc(max_batch_);

  {
    int64_t nlmax = 1;
    for (const LevelPlan& P : levels_) nlmax = std::max<int64_t>(nlmax, (int64_t)P.large.size());
    dcache_.alloc((size_t)nlmax * max_batch_ * kB64 * kB64);
  }
  set_smem(k_factor_small<128>, small_factor_smem(kSmallA));
  set_smem(k_factor_small<256>, small_factor_smem(kSmallB));
  set_smem(k_selinv_small<256>, small_selinv_smem(kSiSmall, kSiSmall));
  set_smem(k_panel64, kPanelSmem);
  {
    int dev = 0;
    INLA_CUDA(cudaGetDevice(&dev));
    INLA_CUDA(cudaDeviceGetAttribute(&num_sms_, cudaDevAttrMultiProcessorCount, dev));
  }
  {  // key of the tuning table: FNV-1a over the supernode partition and row counts
    uint64_t h = 1469598103934665603ull;
    auto mix = [&](int64_t v) {
      for (int b = 0; b < 8; ++b) h = (h ^ (uint64_t)((v >> (8 * b)) & 0xff)) * 1099511628211ull;
    };
    mix(n);
    mix(ns);
    mix(num_sms_);
    for (int64_t s = 0; s <= ns; ++s) mix(S.sn_first[s]), mix(S.sn_rowptr[s]);
    struct_hash_ = h;
  }
  set_smem(k_update64w8, kPersistUpdSmem);
  set_smem(k_diag_next, kPanelSmem);
  set_smem(k_rows64, kRowsSmem);
  set_smem(k_fwd32<128>, (int)((S.max_m + 2 + 32 * 33) * 8));
  set_smem(k_bwd32<128>, (int)((S.max_m + 2 + 32 * 33) * 8));
  set_smem(k_fwd64<256, true>, (int)((S.max_m + 2) * 8));
  set_smem(k_fwd64<256, false>, (int)((S.max_m + 2) * 8));
  set_smem(k_bwd64<256, true>, (int)((S.max_m + 2) * 8));
  set_smem(k_bwd64<256, false>, (int)((S.max_m + 2) * 8));
  set_smem(k_gather8, 200 * 1024 + 8 * kGatherCols * 8);
  auto si_smem = [](auto... kern) { (set_smem(kern, kSiGemmSmem), ...); };
  si_smem(k_si_gemm<SI_T, 64>, k_si_gemm<SI_X, 64>, k_si_gemm<SI_W, 64>, k_si_gemm<SI_BK, 64>, k_si_gemm<SI_KK, 64>,
          k_si_gemm<SI_T, 32>, k_si_gemm<SI_X, 32>, k_si_gemm<SI_W, 32>, k_si_gemm<SI_BK, 32>, k_si_gemm<SI_KK, 32>);
  if (persist_) {
    set_smem(k_factor_persist, persist_smem_);
    int per_sm = 0;
    INLA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_factor_persist, kPersistThreads,
                                                            persist_smem_));
    persist_grid_ = std::max(1, per_sm) * num_sms_;
    if (per_sm < 1) persist_ = false;
  }
  if (solve_persist_) {
    set_smem(k_solve_persist, solve_smem_);
    int per_sm = 0;
    INLA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve_persist, kPersistThreads, solve_smem_));
    solve_grid_ = std::max(1, per_sm) * num_sms_;
    if (per_sm < 1) solve_persist_ = false;
  }
  INLA_CUDA(cudaStreamSynchronize(stream_));
  if (std::getenv("INLA_DEBUG"))
    std::fprintf(stderr, "device factor: maps %.1f ms, symbolic uploads %.1f ms, caches %.1f ms, levels %.1f ms, buffers %.1f ms (%d slots)\n",
                 std::chrono::duration<double, std::milli>(tm1 - tstart).count(),
                 std::chrono::duration<double, std::milli>(tm2 - tm1).count(),
                 std::chrono::duration<double, std::milli>(tm3 - tm2).count(),
                 std::chrono::duration<double, std::milli>(ta - tm3).count(),
                 std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - ta).count(),
                 max_batch_);
}

GpuFactor::~GpuFactor() {
  for (auto& kv : graphs_) cudaGraphExecDestroy(kv.second.exec);
}

// Level plans of a symbolic analysis (host lists; offsets into the flattened device list).
std::vector<LevelPlan> make_level_plans(const Symbolic& S, std::vector<int>& flat) {
  std::vector<LevelPlan> levels(S.nlevels);
  flat.clear();
  // fronts of at most kTinyM rows: one warp each (INLA_NO_TINY_FRONTS keeps them on k_factor_small)
  static const bool tiny_on = std::getenv("INLA_NO_TINY_FRONTS") == nullptr;
  constexpr int kSmallA = GpuFactor::kSmallA, kSmallB = GpuFactor::kSmallB, kSiSmall = GpuFactor::kSiSmall;
  for (int32_t l = 0; l < S.nlevels; ++l) {
    LevelPlan& P = levels[l];
    for (int64_t t = S.level_ptr[l]; t < S.level_ptr[l + 1]; ++t) {
      int s = (int)S.level_list[t];
      int k = (int)(S.sn_first[s + 1] - S.sn_first[s]);
      int m = (int)(S.sn_rowptr[s + 1] - S.sn_rowptr[s]);
      P.all.push_back(s);
      P.mmax_all = std::max(P.mmax_all, m);
      if (!(tiny_on && m <= kTinyM)) {
        P.nontiny.push_back(s);
        P.mmax_nontiny = std::max(P.mmax_nontiny, m);
      }
      if (tiny_on && m <= kTinyM) {
        P.tiny.push_back(s);
      } else if (m <= kSmallA) {
        P.small_a.push_back(s);
        P.mmax_a = std::max(P.mmax_a, m);
      } else if (m <= kSmallB) {
        P.small_b.push_back(s);
        P.mmax_b = std::max(P.mmax_b, m);
      } else {
        P.large.push_back(s);
        P.kmax_large = std::max(P.kmax_large, k);
        P.mmax_large = std::max(P.mmax_large, m);
      }
      if (tiny_on && m <= kTinyM) {
        P.si_tiny.push_back(s);
      } else if (m <= kSiSmall) {
        P.si_small.push_back(s);
        P.mmax_si_small = std::max(P.mmax_si_small, m);
        P.kmax_si_small = std::max(P.kmax_si_small, k);
      } else {
        P.si_large.push_back(s);
        P.kmax_si_large = std::max(P.kmax_si_large, k);
        P.mmax_si_large = std::max(P.mmax_si_large, m);
        P.rmax_si_large = std::max(P.rmax_si_large, m - k);
      }
    }
    auto put = [&](const std::vector<int>& v) {
      int off = (int)flat.size();
      flat.insert(flat.end(), v.begin(), v.end());
      return off;
    };
    P.off_tiny = put(P.tiny);
    P.off_small_a = put(P.small_a);
    P.off_small_b = put(P.small_b);
    P.off_large = put(P.large);
    P.off_all = put(P.all);
    P.off_nontiny = put(P.nontiny);
    P.off_si_tiny = put(P.si_tiny);
    P.off_si_small = put(P.si_small);
    P.off_si_large = put(P.si_large);
  }
  return levels;
}

void GpuFactor::plan_levels(const HostMaps& maps) {
  std::vector<int> flat;
  levels_ = make_level_plans(sym_, flat);
  d_lists_.upload(flat, stream_);
  plan_minis(maps);
}

// Bands of up to kMiniLevels consecutive levels whose fronts all have at most kMiniM rows, cut into the
// tasks of snode_mini.cuh: the fronts of a band that are connected through parent links, children
// first. A level joins the band below it only while no task's cost exceeds kMiniTask fronts, a child from
// outside the band counting 1 / kMiniChildren of a front.
// (INLA_NO_TINY_FRONTS switches these off with the other small-front kernels.)
void make_mini_plan(const Symbolic& S, const std::vector<LevelPlan>& levels, MiniPlan& pl) {
  const int L = (int)levels.size();
  pl = MiniPlan();
  pl.at.assign(L, -1);
  static const bool on = std::getenv("INLA_NO_TINY_FRONTS") == nullptr;
  if (!on) return;
  std::vector<int64_t> cost(S.nsuper, 0);  // of the band's fronts in the subtree of a front of the band
  std::vector<int> task(S.nsuper, -1);     // task of a front within the band being built
  for (int l = 0; l < L;) {
    int e = l;
    for (; e < L && e - l < kMiniLevels && levels[e].mmax_all <= kMiniM; ++e) {
      int64_t most = 0;
      for (int s : levels[e].all) {
        cost[s] = kMiniChildren;
        for (int64_t q = S.child_ptr[s]; q < S.child_ptr[s + 1]; ++q)
          cost[s] += std::max<int64_t>(cost[S.child_list[q]], 1);
        most = std::max(most, cost[s]);
      }
      if (most > kMiniTask * kMiniChildren) break;
    }
    for (int q = l; q < std::min(L, e + 1); ++q)
      for (int s : levels[q].all) cost[s] = 0;
    if (e - l < 2) {  // a single level gains nothing over the level kernels
      l = std::max(e, l + 1);
      continue;
    }
    // from the top level down: a front joins its parent's task if the parent lies in the band
    const int off = (int)pl.ptr.size() - 1;
    std::vector<std::vector<int>> tasks;
    for (int q = e - 1; q >= l; --q)
      for (int s : levels[q].all) {
        const int64_t p = S.sn_parent[s];
        task[s] = p >= 0 && task[p] >= 0 ? task[p] : (int)tasks.size();
        if (task[s] == (int)tasks.size()) tasks.emplace_back();
        tasks[task[s]].push_back(s);
      }
    // similar lengths side by side: the four tasks of a warp run for the longest of them
    std::stable_sort(tasks.begin(), tasks.end(),
                     [](const std::vector<int>& a, const std::vector<int>& b) { return a.size() > b.size(); });
    pl.longest = std::max(pl.longest, (int)tasks[0].size());
    for (const std::vector<int>& t : tasks) {
      pl.list.insert(pl.list.end(), t.rbegin(), t.rend());
      pl.ptr.push_back((int)pl.list.size());
    }
    for (int q = l; q < e; ++q) {
      pl.at[q] = (int)pl.bands.size();
      for (int s : levels[q].all) task[s] = -1;
    }
    pl.bands.push_back({l, e, off, (int)tasks.size()});
    l = e;
  }
}

// Host check of the bands: every front of a band's levels in exactly one of its tasks, after its
// children of the band, which lie in the same task; no task longer than kMiniTask. Returns an empty
// string or the first violation.
std::string check_mini_plan(const Symbolic& S, const std::vector<LevelPlan>& levels, const MiniPlan& pl) {
  std::vector<int> band(S.nsuper, -1), task(S.nsuper, -1);
  for (size_t i = 0; i < pl.bands.size(); ++i)
    for (int q = pl.bands[i].l0; q < pl.bands[i].l1; ++q)
      for (int s : levels[q].all) band[s] = (int)i;
  for (size_t i = 0; i < pl.bands.size(); ++i) {
    const MiniBand& M = pl.bands[i];
    const std::string at = "band " + std::to_string(i) + ": ";
    for (int t = M.off; t < M.off + M.ntask; ++t) {
      const int len = pl.ptr[t + 1] - pl.ptr[t];
      if (len < 1 || len > kMiniTask || len > pl.longest) return at + "task of " + std::to_string(len) + " fronts";
      for (int f = pl.ptr[t]; f < pl.ptr[t + 1]; ++f) {
        const int s = pl.list[f];
        if (band[s] != (int)i || task[s] >= 0) return at + "front of another band or twice";
        if (S.sn_rowptr[s + 1] - S.sn_rowptr[s] > kMiniM) return at + "front too large";
        for (int64_t q = S.child_ptr[s]; q < S.child_ptr[s + 1]; ++q) {
          const int c = (int)S.child_list[q];
          if (band[c] == (int)i && task[c] != t) return at + "front before its children";
        }
        task[s] = t;
      }
    }
  }
  for (int64_t s = 0; s < S.nsuper; ++s)
    if (band[s] >= 0 && task[s] < 0) return "front " + std::to_string(s) + " in no task";
  return std::string();
}

void GpuFactor::plan_minis(const HostMaps& maps) {
  MiniPlan pl;
  make_mini_plan(sym_, levels_, pl);
  bands_ = pl.bands;
  band_at_ = pl.at;
  const std::vector<int>& list = pl.list;
  if (bands_.empty()) return;
  std::vector<MiniFront> front;
  std::vector<MiniChild> child;
  front.reserve(list.size());
  auto rows = [&](int s) { return maps.rowptr[s + 1] - maps.rowptr[s]; };
  auto pivots = [&](int s) { return maps.first[s + 1] - maps.first[s]; };
  for (int s : list) {
    const int p = maps.parent[s], c0 = maps.child_ptr[s], c1 = maps.child_ptr[s + 1];
    front.push_back({maps.fptr[s], maps.rowptr[s], maps.first[s], pivots(s), rows(s), (int)child.size(), c1 - c0,
                     p < 0 ? 0 : maps.fptr[p], p < 0 ? 0 : rows(p), maps.uoff[s]});
    for (int q = c0; q < c1; ++q) {
      const int c = maps.child_list[q], kc = pivots(c), mc = rows(c);
      child.push_back({maps.fptr[c] + (int64_t)kc * mc + kc, maps.rowptr[c] + kc, mc * 16 + (mc - kc)});
    }
  }
  d_mptr_.upload(pl.ptr, stream_);
  d_mlist_.upload(list, stream_);
  d_mfront_.upload(front, stream_);
  d_mchild_.upload(child, stream_);
}

// ---------------------------------------------------------------------------
// Persistent schedule: the task queue of k_factor_persist (see snode_persist.cuh).
// Per level: tiny fronts in groups of eight, small fronts, then the large fronts phase by
// phase (extend-add chunks; per 64-column block the diagonal block, the row blocks and the
// trailing-update tiles). Each phase of a level is one group; within a group the tasks of
// problem 0 come first, then problem 1, and so on.
// ---------------------------------------------------------------------------
namespace {
// Process-wide schedule mode for engines built from now on: 0 level launches only, 1 measured
// per batch size (default), 2 persistent wherever it fits. INLA_NO_PERSIST in the environment
// starts it at 0; inla_set_persistent_schedule changes it.
std::atomic<int> g_persist_default{-1};
// measured choices per (supernodal structure, batch size): true = persistent
struct SchedChoice {
  bool factor, solve;
};
std::mutex g_sched_mu;
std::map<std::pair<uint64_t, int>, SchedChoice> g_sched;
}  // namespace

void set_persistent_default(int mode) { g_persist_default.store(mode < 0 ? 0 : (mode > 2 ? 2 : mode)); }

void set_panel_form(int form) { g_panel_form.store(form < 0 || form >= kNumForms ? -1 : form); }

// The task queue of the persistent schedule for one problem (host arrays).
bool make_persist_plan(const Symbolic& S, const std::vector<LevelPlan>& levels, PersistPlan& out) {
  const int ns = (int)S.nsuper;
  constexpr int kGatherBudget = 110 * 1024;  // bytes of one extend-add column slice
  int smem = std::max({kPersistTinySmem, small_factor_smem(GpuFactor::kSmallB), kPanelSmem, kRowsSmem,
                       kPersistUpdSmem});
  PersistPlan& pl = out;
  pl = PersistPlan();
  pl.gstart = {0};
  pl.total.assign(ns, 0);
  auto push = [&](int type, int sn, int sub, int need, int j0, int arg) {
    pl.task.insert(pl.task.end(), {type, sn, sub, need, j0, arg});
  };
  auto close_group = [&] {
    const int cnt = (int)(pl.task.size() / 6);
    if (cnt > pl.gstart.back()) pl.gstart.push_back(cnt);
  };
  struct Phase {
    int type, count, j0, sub0, need, arg;  // tasks sub0 .. sub0 + count - 1
  };
  for (const LevelPlan& P : levels) {
    for (size_t i = 0; i < P.tiny.size(); i += kPersistTinyWarps) {
      const int cnt = (int)std::min<size_t>(kPersistTinyWarps, P.tiny.size() - i);
      push(PT_TINY, (int)pl.tiny.size(), cnt, 0, 0, 0);
      for (int u = 0; u < cnt; ++u) {
        pl.tiny.push_back(P.tiny[i + u]);
        pl.total[P.tiny[i + u]] = 1;
      }
    }
    close_group();
    for (const std::vector<int>* v : {&P.small_a, &P.small_b})
      for (int sn : *v) {
        push(PT_SMALL, sn, 0, 0, 0, 0);
        pl.total[sn] = 1;
      }
    close_group();
    if (P.large.empty()) continue;
    // phases of every large front: extend-add, first diagonal block, then per block J the next diagonal
    // block, the rows and the update
    std::vector<std::vector<Phase>> ph(P.large.size());
    size_t maxp = 0;
    for (size_t f = 0; f < P.large.size(); ++f) {
      const int sn = P.large[f];
      const int k = (int)(S.sn_first[sn + 1] - S.sn_first[sn]), m = (int)(S.sn_rowptr[sn + 1] - S.sn_rowptr[sn]);
      const int gcols = std::max(1, std::min(kGatherCols, kGatherBudget / (8 * m)));
      smem = std::max(smem, gcols * m * 8);
      ++pl.nlarge;
      const int nz = cdiv(m, gcols);
      ph[f].push_back({PT_GATHER, nz, 0, 0, 0, gcols});
      ph[f].push_back({PT_DIAG, 1, 0, 0, nz, 0});
      int done = nz;  // extend-add, row and update tasks so far
      for (int j0 = 0; j0 < k; j0 += kB64) {
        const int w = std::min(kB64, k - j0), below = std::max(m - j0 - w, 0);
        const int nt = cdiv(below, kUT64), nrow = cdiv(below, kPanelRows);
        const bool next = j0 + kB64 < k;  // then tile 0 of the update is the next diagonal block's
        const int diags = j0 / kB64 + 1;
        ph[f].push_back({PT_NEXT, next ? 1 : 0, j0 + kB64, 0, done, diags});
        ph[f].push_back({PT_ROWS, nrow, j0, 0, done, diags});
        done += nrow;
        const int ntile = nt * (nt + 1) / 2 - (next ? 1 : 0);
        ph[f].push_back({PT_UPDATE, ntile, j0, next ? 1 : 0, done, 0});
        done += ntile;
      }
      maxp = std::max(maxp, ph[f].size());
      pl.total[sn] = done;
    }
    for (size_t p = 0; p < maxp; ++p) {
      for (size_t f = 0; f < P.large.size(); ++f) {
        if (p >= ph[f].size()) continue;
        const Phase& x = ph[f][p];
        for (int u = 0; u < x.count; ++u) push(x.type, P.large[f], x.sub0 + u, x.need, x.j0, x.arg);
      }
      close_group();
    }
  }
  pl.smem = smem;
  if (pl.tiny.empty()) pl.tiny.push_back(0);
  return smem <= 227 * 1024 && pl.gstart.size() > 1;
}

// Host check of the schedule's invariants: processed one task at a time in queue order (one
// problem), every task's dependencies are complete when it is reached (so the smallest
// unfinished task of the GPU queue can always run), the counts that a task of a large front waits for
// cover everything it reads (derived here from the front's shape, not from the queue), every part of a
// step is there once, every front ends with its completion count, and every table index is in range.
// Returns an empty string or the first violation.
std::string check_persist_plan(const Symbolic& S, const PersistPlan& pl) {
  const int ns = (int)S.nsuper;
  const int ntask = (int)(pl.task.size() / 6);
  if (pl.gstart.back() != ntask) return "group table does not cover the tasks";
  for (size_t g = 0; g + 1 < pl.gstart.size(); ++g)
    if (pl.gstart[g + 1] <= pl.gstart[g]) return "empty or decreasing group " + std::to_string(g);
  std::vector<int> prog(ns, 0), diag(ns, 0);
  auto children_done = [&](int sn) {
    for (int64_t q = S.child_ptr[sn]; q < S.child_ptr[sn + 1]; ++q) {
      const int c = (int)S.child_list[q];
      if (prog[c] != pl.total[c]) return false;
    }
    return true;
  };
  auto pivots = [&](int sn) { return (int)(S.sn_first[sn + 1] - S.sn_first[sn]); };
  auto height = [&](int sn) { return (int)(S.sn_rowptr[sn + 1] - S.sn_rowptr[sn]); };
  auto blocks = [&](int sn) { return cdiv(pivots(sn), kB64); };
  // large fronts: columns per extend-add task, and tasks of every (step, type) reached so far
  std::vector<int> gcols_of(ns, 0);
  std::map<std::pair<int, int>, std::pair<int, int>> parts;  // (front, step) -> rows, tiles
  auto below = [&](int sn, int J) { return std::max(height(sn) - std::min((J + 1) * kB64, pivots(sn)), 0); };
  auto row_tasks = [&](int sn, int J) { return cdiv(below(sn, J), kPanelRows); };
  // the first 64 x 64 tile below step J is the next diagonal block's while there is one
  auto first_tile = [&](int sn, int J) { return J + 1 < blocks(sn) ? 1 : 0; };
  auto end_tile = [&](int sn, int J) { return cdiv(below(sn, J), kUT64) * (cdiv(below(sn, J), kUT64) + 1) / 2; };
  auto before = [&](int sn, int J) {  // extend-add tasks, and rows and tiles of the steps before J
    int c = cdiv(height(sn), std::max(gcols_of[sn], 1));
    for (int q = 0; q < J; ++q) c += row_tasks(sn, q) + end_tile(sn, q) - first_tile(sn, q);
    return c;
  };
  for (int t = 0; t < ntask; ++t) {
    const int* T = pl.task.data() + 6 * t;
    const int type = T[0], sn = T[1], sub = T[2], need = T[3];
    const std::string at = "task " + std::to_string(t) + ": ";
    if (type == PT_TINY) {
      if (sub < 1 || sub > kPersistTinyWarps || sn < 0 || sn + sub > (int)pl.tiny.size()) return at + "tiny range";
      for (int u = 0; u < sub; ++u) {
        const int f = pl.tiny[sn + u];
        if (f < 0 || f >= ns || !children_done(f)) return at + "tiny front before its children";
        if (height(f) > kTinyM) return at + "front too large for a warp";
      }
      for (int u = 0; u < sub; ++u) ++prog[pl.tiny[sn + u]];
      continue;
    }
    if (sn < 0 || sn >= ns) return at + "front out of range";
    const int k = pivots(sn), m = height(sn);
    if (type == PT_SMALL) {
      if (m > GpuFactor::kSmallB) return at + "front too large for the small body";
      if (!children_done(sn)) return at + "small front before its children";
    } else if (type == PT_GATHER) {
      if (m <= GpuFactor::kSmallB || !children_done(sn)) return at + "extend-add before the children";
      const int gcols = T[5];
      if (gcols < 1 || (int64_t)gcols * m * 8 > pl.smem) return at + "extend-add slice exceeds shared memory";
      if (gcols_of[sn] == 0) gcols_of[sn] = gcols;
      if (gcols != gcols_of[sn]) return at + "extend-add slices of different widths";
      if (sub >= cdiv(m, gcols)) return at + "extend-add chunk out of range";
      if (need != 0 || prog[sn] != sub) return at + "extend-add count";
    } else if (type == PT_DIAG || type == PT_NEXT || type == PT_ROWS || type == PT_UPDATE) {
      if (m <= GpuFactor::kSmallB) return at + "step of a front that is not large";
      if (T[4] < 0 || T[4] >= k || T[4] % kB64) return at + "block column out of range";
      if (prog[sn] < need || diag[sn] < T[5]) return at + "phase before its predecessors";
      const int J = T[4] / kB64;
      if (type == PT_DIAG || type == PT_NEXT) {
        // the first block after the extend-add; block J after block J - 1 and, for its tile and its mirror
        // rows, after the updates of step J - 2
        if (J != diag[sn] || (type == PT_DIAG) != (J == 0) || T[5] < J) return at + "diagonal block order";
        if (need < before(sn, std::max(J - 1, 0))) return at + "diagonal block does not wait for its updates";
        ++diag[sn];
        continue;
      }
      std::pair<int, int>& part = parts[{sn, J}];
      if (type == PT_ROWS) {
        if (T[5] < J + 1 || need < before(sn, J)) return at + "rows do not wait for their diagonal block or updates";
        if (sub != part.first++ || sub >= row_tasks(sn, J)) return at + "row block out of order or range";
      } else {
        if (need < before(sn, J) + row_tasks(sn, J)) return at + "update does not wait for its rows";
        if (sub != first_tile(sn, J) + part.second++ || sub >= end_tile(sn, J)) return at + "tile out of order or range";
      }
    } else {
      return at + "unknown task type";
    }
    ++prog[sn];
  }
  for (int sn = 0; sn < ns; ++sn)
    if (pl.total[sn] < 1 || prog[sn] != pl.total[sn] ||
        (height(sn) > GpuFactor::kSmallB && (diag[sn] != blocks(sn) || prog[sn] != before(sn, blocks(sn)))))
      return "front " + std::to_string(sn) + " incomplete";
  return std::string();
}

void make_solve_plan(const Symbolic& S, const std::vector<LevelPlan>& levels, PersistPlan& pl) {
  pl = PersistPlan();
  pl.gstart = {0};
  auto push = [&](int type, int sn, int sub) { pl.task.insert(pl.task.end(), {type, sn, sub, 0, 0, 0}); };
  auto close_group = [&] {
    const int cnt = (int)(pl.task.size() / 6);
    if (cnt > pl.gstart.back()) pl.gstart.push_back(cnt);
  };
  auto tiny_tasks = [&](const std::vector<int>& v, int type) {
    for (size_t i = 0; i < v.size(); i += kPersistTinyWarps) {
      const int cnt = (int)std::min<size_t>(kPersistTinyWarps, v.size() - i);
      push(type, (int)pl.tiny.size(), cnt);
      for (int u = 0; u < cnt; ++u) pl.tiny.push_back(v[i + u]);
    }
    close_group();
  };
  int mmax = 0;
  for (const LevelPlan& P : levels) {
    tiny_tasks(P.tiny, ST_FWD_TINY);
    for (int sn : P.nontiny) push(ST_FWD, sn, 0);
    close_group();
    mmax = std::max(mmax, P.mmax_nontiny);
  }
  for (size_t l = levels.size(); l-- > 0;) {
    for (int sn : levels[l].nontiny) push(ST_BWD, sn, 0);
    close_group();
    tiny_tasks(levels[l].tiny, ST_BWD_TINY);
  }
  pl.smem = std::max(kPersistTinyWarps * 32, mmax + 2 + 32 * 33) * 8;
  if (pl.tiny.empty()) pl.tiny.push_back(0);
}

// As check_persist_plan, for the solve queue: forward tasks after their children's forward
// tasks, backward tasks after their parent's backward task (roots: after their own forward).
std::string check_solve_plan(const Symbolic& S, const PersistPlan& pl) {
  const int ns = (int)S.nsuper;
  const int ntask = (int)(pl.task.size() / 6);
  if (pl.gstart.back() != ntask) return "group table does not cover the tasks";
  std::vector<int> pf(ns, 0), pb(ns, 0);
  auto ready = [&](int type, int sn) {
    if (type == ST_FWD_TINY || type == ST_FWD) {
      for (int64_t q = S.child_ptr[sn]; q < S.child_ptr[sn + 1]; ++q)
        if (pf[S.child_list[q]] != 1) return false;
      return pf[sn] == 0;
    }
    const int64_t p = S.sn_parent[sn];
    return pb[sn] == 0 && (p < 0 ? pf[sn] == 1 : pb[p] == 1);
  };
  for (int t = 0; t < ntask; ++t) {
    const int* T = pl.task.data() + 6 * t;
    const bool tiny = T[0] == ST_FWD_TINY || T[0] == ST_BWD_TINY;
    const bool fwd = T[0] == ST_FWD_TINY || T[0] == ST_FWD;
    const int cnt = tiny ? T[2] : 1;
    for (int u = 0; u < cnt; ++u) {
      const int sn = tiny ? pl.tiny[T[1] + u] : T[1];
      if (sn < 0 || sn >= ns || !ready(T[0], sn)) return "task " + std::to_string(t) + " before its dependencies";
      if (tiny && S.sn_rowptr[sn + 1] - S.sn_rowptr[sn] > kTinyM) return "tiny task with a wide front";
      (fwd ? pf : pb)[sn] = 1;
    }
  }
  for (int sn = 0; sn < ns; ++sn)
    if (pf[sn] != 1 || pb[sn] != 1) return "front " + std::to_string(sn) + " not swept";
  return std::string();
}

void GpuFactor::plan_solve_persist() {
  PersistPlan pl;
  make_solve_plan(sym_, levels_, pl);
  if (pl.smem > 227 * 1024 || pl.gstart.size() < 2) return;
  const int ns = (int)sym_.nsuper;
  solve_groups_ = (int)pl.gstart.size() - 1;
  d_sgstart_.upload(pl.gstart, stream_);
  d_stask_.upload(pl.task, stream_);
  d_stiny_.upload(pl.tiny, stream_);
  d_sstate_.alloc(2 + 2 * (size_t)max_batch_ * ns);
  INLA_CUDA(cudaMemsetAsync(d_sstate_.p, 0, sizeof(int) * (2 + 2 * (size_t)max_batch_ * ns), stream_));
  solve_smem_ = pl.smem;
  solve_persist_ = true;
}

constexpr int64_t kPersistPairs = 1 << 17;  // (large front, problem) pairs

void GpuFactor::plan_persist() {
  int def = g_persist_default.load();
  if (def < 0) {
    def = std::getenv("INLA_NO_PERSIST") ? 0 : 1;
    int expect = -1;
    g_persist_default.compare_exchange_strong(expect, def);
    def = g_persist_default.load();
  }
  if (def == 0) return;
  persist_mode_ = def;
  if (const char* w = std::getenv("INLA_PERSIST_WAIT_MS")) persist_limit_ns_ = (long long)(std::atof(w) * 1e6);
  PersistPlan pl;
  if (!make_persist_plan(sym_, levels_, pl)) return;  // a front too wide for the schedule's shared memory
  const int ns = (int)sym_.nsuper;
  // With this many large fronts every step of a level fills the GPU, and the queue only adds its waits: 4400
  // fronts of 100 rows at B = 30 35.1 ms by level launches, 54.2 ms persistent; 600 trees of seven fronts of 150
  // and 300 rows at B = 32 170 and 266 ms. Not worth timing both.
  if ((int64_t)pl.nlarge * max_batch_ > kPersistPairs) return;
  persist_groups_ = (int)pl.gstart.size() - 1;
  d_pgstart_.upload(pl.gstart, stream_);
  d_ptask_.upload(pl.task, stream_);
  d_ptiny_.upload(pl.tiny, stream_);
  d_ptotal_.upload(pl.total, stream_);
  d_pstate_.alloc(2 + 2 * (size_t)max_batch_ * ns);
  INLA_CUDA(cudaMemsetAsync(d_pstate_.p, 0, sizeof(int) * (2 + 2 * (size_t)max_batch_ * ns), stream_));
  persist_smem_ = pl.smem;
  persist_ = true;
  plan_solve_persist();
}

void GpuFactor::set_front_groups(const std::vector<int>& fseg) {
  if ((int64_t)fseg.size() != sym_.nsuper) throw std::runtime_error("one group per front expected");
  d_fseg_.upload(fseg, stream_);
}

void GpuFactor::run_factor_persist(int B, const int* total_override, long long limit_ns,
                                   const unsigned char* active, int nseg) {
  const int ns = (int)sym_.nsuper;
  // head and the completion counts start at zero; the error record (word 0) stays until read
  INLA_CUDA(cudaMemsetAsync(d_pstate_.p + 1, 0, sizeof(int) * (1 + 2 * (size_t)B * ns), stream_));
  PersistArgs a;
  a.S = ds_;
  a.F = F_.p;
  a.fstride = ftotal_;
  a.B = B;
  a.ngroups = persist_groups_;
  a.gstart = d_pgstart_.p;
  a.task = reinterpret_cast<const PersistTask*>(d_ptask_.p);
  a.tiny_list = d_ptiny_.p;
  a.total = total_override ? total_override : d_ptotal_.p;
  a.prog = d_pstate_.p + 2;
  a.dprog = d_pstate_.p + 2 + (size_t)B * ns;
  a.head = reinterpret_cast<unsigned*>(d_pstate_.p + 1);
  a.err = d_pstate_.p;
  a.linv = linv_.p;
  a.limit_ns = limit_ns > 0 ? limit_ns : persist_limit_ns_;
  if (active) {
    a.S.active = active;
    a.S.fseg = d_fseg_.p;
    a.S.nseg = nseg;
  }
  k_factor_persist<<<persist_grid_, kPersistThreads, persist_smem_, stream_>>>(a);
  k_logdet_chunks<<<dim3(nldchunk_, B), 256, 0, stream_>>>(ds_, F_.p, ftotal_, ldpart_.p, ldflag_.p, ldticket_.p,
                                                           logdet_.p, status_.p, d_pstate_.p);
  launches_ += 2;
}

// Persistent or level launches for batch size B: fixed by the mode, or measured on the
// first factorization at B (the level sequence in its tuned form and the persistent launch, with their
// value fills, each after a warm-up as the graph it runs as, with CUDA events on the engine's stream) and
// kept for the structure and B. Launched directly, a level sequence takes longer than its graph: the grouped
// model 24x24x14 at B = 2 1.69 ms against 1.67 persistent, and the evaluation 22.0 ms persistent, 21.2 by
// level launches; binary trees of dense blocks lost up to 13 % by that.
// Where the factorization is persistent, the triangular solve's two schedules are timed in
// the same way: which is faster depends on the tree, not on its depth alone.
// Level launches / persistent: 13 levels (n = 900, AMD) 187 / 169 us, 28 levels (n = 10 000, AMD) 519 / 450, 3-D
// grid of 22^3 350 / 336, but 2-D grids of 60^2 and 300^2 under nested dissection 193 / 224 and 488 / 607, binary
// trees of dense 60-column blocks, 3 / 5 / 7 / 8 levels, 41 / 52, 69 / 83, 223 / 302, 513 / 776.
bool GpuFactor::use_persist(int B, const std::function<void()>& fill) {
  if (!persist_) return false;
  if (persist_mode_ == 2) return true;
  auto it = persist_at_.find(B);
  if (it != persist_at_.end()) return it->second;
  {
    std::lock_guard<std::mutex> lk(g_sched_mu);
    auto g = g_sched.find({struct_hash_, B});
    if (g != g_sched.end()) {
      solve_persist_at_[B] = g->second.solve;
      return persist_at_[B] = g->second.factor;
    }
  }
  const std::vector<char>* pol = schedule(B, fill);
  const float tl = time_graph([&] {
    fill();
    run_factor_levels(B, pol);
  });
  const float tp = time_graph([&] {
    fill();
    run_factor_persist(B);
  });
  const bool pick = tp < tl;
  bool pick_solve = false;
  if (pick && solve_persist_) {
    INLA_CUDA(cudaMemsetAsync(xp_.p, 0, sizeof(double) * B * sym_.n, stream_));
    const float sl = time_graph([&] { solve_levels(B, 0); });
    const float sp = time_graph([&] { solve_queue(B, 0); });
    pick_solve = sp < sl;
    if (std::getenv("INLA_DEBUG"))
      std::fprintf(stderr, "solve B=%d: level launches %.3f ms, persistent %.3f ms -> %s\n", B, sl, sp,
                   pick_solve ? "persistent" : "levels");
  }
  check_schedule();
  if (std::getenv("INLA_DEBUG"))
    std::fprintf(stderr, "schedule B=%d: level launches %.3f ms, persistent %.3f ms -> %s\n", B, tl, tp,
                 pick ? "persistent" : "levels");
  {
    std::lock_guard<std::mutex> lk(g_sched_mu);
    g_sched[{struct_hash_, B}] = {pick, pick_solve};
  }
  solve_persist_at_[B] = pick_solve;
  return persist_at_[B] = pick;
}

// Milliseconds of a launch sequence run as a graph (after a warm-up), or launched directly where it cannot be
// captured.
float GpuFactor::time_graph(const std::function<void()>& body) {
  const int64_t before = launches_;
  cudaGraph_t g = nullptr;
  cudaGraphExec_t ex = nullptr;
  if (use_graphs_) {
    INLA_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    bool ok = true;
    try {
      body();
    } catch (...) {
      ok = false;  // the direct run below throws it again
    }
    ok = cudaGetLastError() == cudaSuccess && ok;
    if (cudaStreamEndCapture(stream_, &g) != cudaSuccess || !ok || cudaGraphInstantiate(&ex, g, 0) != cudaSuccess) {
      ex = nullptr;
      cudaGetLastError();  // the capture's errors are not sticky
    }
    if (g) cudaGraphDestroy(g);
  }
  auto run = [&] {
    if (ex) INLA_CUDA(cudaGraphLaunch(ex, stream_));
    else body();
  };
  cudaEvent_t e[2];
  for (auto& x : e) INLA_CUDA(cudaEventCreate(&x));
  run();
  INLA_CUDA(cudaEventRecord(e[0], stream_));
  run();
  INLA_CUDA(cudaEventRecord(e[1], stream_));
  INLA_CUDA(cudaStreamSynchronize(stream_));
  float ms = 0.f;
  INLA_CUDA(cudaEventElapsedTime(&ms, e[0], e[1]));
  for (auto& x : e) cudaEventDestroy(x);
  if (ex) cudaGraphExecDestroy(ex);
  launches_ = before;
  return ms;
}

void GpuFactor::check_schedule() {
  if (!persist_) return;
  int err = 0, serr = 0;
  INLA_CUDA(cudaMemcpyAsync(&err, d_pstate_.p, sizeof(int), cudaMemcpyDeviceToHost, stream_));
  if (solve_persist_) INLA_CUDA(cudaMemcpyAsync(&serr, d_sstate_.p, sizeof(int), cudaMemcpyDeviceToHost, stream_));
  INLA_CUDA(cudaStreamSynchronize(stream_));
  if (err == 0 && serr == 0) return;
  INLA_CUDA(cudaMemsetAsync(d_pstate_.p, 0, sizeof(int), stream_));
  if (solve_persist_) INLA_CUDA(cudaMemsetAsync(d_sstate_.p, 0, sizeof(int), stream_));
  INLA_CUDA(cudaStreamSynchronize(stream_));
  if (err == 0) err = serr;
  throw CudaError("persistent factorization stopped: a dependency wait ran out (code " + std::to_string(err) + ")",
                  (int)cudaErrorLaunchTimeout);
}

namespace {
__global__ void k_reciprocal(int64_t n, const double* __restrict__ x, double* __restrict__ y) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) y[i] = rcp_in_range(x[i]) ? rcp_straight(x[i]) : 1.0 / x[i];
}
}  // namespace

void reciprocal_selftest(int64_t n, const double* x, double* y) {
  if (n == 0) return;
  DBuf<double> dx, dy;
  dx.alloc(n);
  dy.alloc(n);
  INLA_CUDA(cudaMemcpy(dx.p, x, sizeof(double) * n, cudaMemcpyHostToDevice));
  k_reciprocal<<<(unsigned)cdiv(n, 256), 256>>>(n, dx.p, dy.p);
  INLA_CUDA(cudaGetLastError());
  INLA_CUDA(cudaMemcpy(y, dy.p, sizeof(double) * n, cudaMemcpyDeviceToHost));
}

int GpuFactor::persist_wait_limit_selftest(double limit_ms) {
  if (!persist_) return -1;
  const int ns = (int)sym_.nsuper;
  // completion counts no front can reach: every front with children waits until the limit
  std::vector<int> never(ns, 1 << 30);
  DBuf<int> d_never;
  d_never.upload(never, stream_);
  INLA_CUDA(cudaMemsetAsync(F_.p, 0, sizeof(double) * ftotal_, stream_));  // a defined input for the fronts that run
  run_factor_persist(1, d_never.p, (long long)(limit_ms * 1e6));
  INLA_CUDA(cudaGetLastError());
  int err = 0;
  INLA_CUDA(cudaMemcpyAsync(&err, d_pstate_.p, sizeof(int), cudaMemcpyDeviceToHost, stream_));
  INLA_CUDA(cudaStreamSynchronize(stream_));
  INLA_CUDA(cudaMemsetAsync(d_pstate_.p, 0, sizeof(int), stream_));
  INLA_CUDA(cudaStreamSynchronize(stream_));
  return err;
}

void GpuFactor::run_factor_levels(int B, const std::vector<char>* fuse, cudaEvent_t* ev) {
  const int64_t fs = ftotal_;
  for (size_t li = 0; li < levels_.size(); ++li) {
    const LevelPlan& P = levels_[li];
    if (band_at_[li] >= 0) {
      const MiniBand& M = bands_[band_at_[li]];
      if ((int)li == M.l0) {
        k_factor_mini<<<dim3(cdiv(M.ntask, kMiniGroups), B), kMiniThreads, 0, stream_>>>(
            ds_, mini_tables(M.off), M.ntask, F_.p, fs);
        ++launches_;
      }
      if (ev) {
        INLA_CUDA(cudaEventRecord(ev[2 * li], stream_));
        INLA_CUDA(cudaEventRecord(ev[2 * li + 1], stream_));
      }
      continue;
    }
    if (!P.tiny.empty()) {
      const int nt = (int)P.tiny.size();
      k_factor_tiny<<<dim3(cdiv(nt, kTinyWarps), B), 32 * kTinyWarps, 0, stream_>>>(ds_, d_lists_.p + P.off_tiny, nt,
                                                                                 F_.p, fs);
      ++launches_;
    }
    if (!P.small_a.empty()) {
      dim3 g((unsigned)P.small_a.size(), B);
      k_factor_small<128><<<g, 128, small_factor_smem(P.mmax_a), stream_>>>(ds_, d_lists_.p + P.off_small_a, F_.p,
                                                                             fs);
      ++launches_;
    }
    if (!P.small_b.empty()) {
      dim3 g((unsigned)P.small_b.size(), B);
      k_factor_small<256><<<g, 256, small_factor_smem(P.mmax_b), stream_>>>(ds_, d_lists_.p + P.off_small_b, F_.p,
                                                                             fs);
      ++launches_;
    }
    if (ev) INLA_CUDA(cudaEventRecord(ev[2 * li], stream_));
    if (!P.large.empty()) {
      const int nl = (int)P.large.size();
      const int* lst = d_lists_.p + P.off_large;
      const int gcols = gather_cols(P.mmax_large);
      k_gather8<<<dim3(nl, B, cdiv(P.mmax_large, gcols)), 256, gcols * P.mmax_large * 8, stream_>>>(
          ds_, lst, F_.p, fs, gcols);
      ++launches_;
      const int form = fuse ? (*fuse)[li] : -1;
      for (int j0 = 0; j0 < P.kmax_large; j0 += kB64) {
        int rows = P.mmax_large - j0;
        const int nrb = std::max(1, cdiv(rows, kPanelRows));
        int nt = cdiv(rows, kUT64);
        const dim3 ug(nl, B, std::max(1, nt * (nt + 1) / 2));
        if (form == kFormLookahead) {
          // The pivot chain runs on a stream of its own: the diagonal block of step J + 1 depends on
          // the one of step J and on the updates of step J - 1, and runs beside the rows and updates
          // of step J.
          if (j0 == 0) {
            k_panel64<<<dim3(nl, B, 1), 256, kPanelSmem, stream_>>>(ds_, lst, j0, 0, F_.p, fs, nullptr, linv_.p);
            ++launches_;
          }
          const bool next = j0 + kB64 < P.kmax_large;
          if (next) {
            INLA_CUDA(cudaEventRecord(chain_.fork, stream_));
            INLA_CUDA(cudaStreamWaitEvent(chain_.stream, chain_.fork, 0));
            k_diag_next<<<dim3(nl, B), 256, kPanelSmem, chain_.stream>>>(ds_, lst, j0 + kB64, F_.p, fs, linv_.p);
            INLA_CUDA(cudaEventRecord(chain_.join, chain_.stream));
            ++launches_;
          }
          k_rows64<<<dim3(nl, B, nrb), 256, kRowsSmem, stream_>>>(ds_, lst, j0, F_.p, fs, nullptr, linv_.p);
          k_update64w8<<<ug, 256, kPersistUpdSmem, stream_>>>(ds_, lst, j0, F_.p, fs, nullptr);
          if (next) INLA_CUDA(cudaStreamWaitEvent(stream_, chain_.join, 0));
          launches_ += 2;
          continue;
        }
        // While every (front, problem, 64-row block) gets its own CTA within about
        // one wave (two CTAs per SM), each row CTA factors the diagonal block
        // itself (one launch). Beyond that, one CTA per (front, problem) factors
        // it and k_rows64 forms the rows from the cached factor (no redundant
        // factorizations).
        const int per = std::max(1, (2 * num_sms_) / std::max(1, nl * B));
        const bool fused = form >= 0 ? form == kFormFused : per >= nrb;
        if (fused) {
          k_panel64<<<dim3(nl, B, nrb), 256, kPanelSmem, stream_>>>(ds_, lst, j0, kPanelRows, F_.p, fs, dcache_.p,
                                                                     linv_.p);
        } else {
          k_panel64<<<dim3(nl, B, 1), 256, kPanelSmem, stream_>>>(ds_, lst, j0, 0, F_.p, fs, dcache_.p, linv_.p);
          k_rows64<<<dim3(nl, B, nrb), 256, kRowsSmem, stream_>>>(ds_, lst, j0, F_.p, fs, dcache_.p, linv_.p);
          ++launches_;
        }
        k_update64w8<<<ug, 256, kPersistUpdSmem, stream_>>>(ds_, lst, j0, F_.p, fs, dcache_.p);
        launches_ += 2;
      }
    }
    if (ev) INLA_CUDA(cudaEventRecord(ev[2 * li + 1], stream_));
  }
  k_logdet_chunks<<<dim3(nldchunk_, B), 256, 0, stream_>>>(ds_, F_.p, fs, ldpart_.p, ldflag_.p, ldticket_.p,
                                                           logdet_.p, status_.p);
  ++launches_;
}

// ---------------------------------------------------------------------------
// Panel-schedule autotuner. For every level with large fronts the panel step has
// three forms with bit-identical results: "split" (one CTA per front factors the
// 64 x 64 diagonal block, k_rows64 forms the rows from the cached factor, then the
// trailing update: three launches per step), "fused" (each of the nrb row CTAs
// factors the diagonal block itself, then the update: two launches) and
// "look-ahead" (rows and update, and beside them on a stream of its own k_diag_next, which
// needs only the previous diagonal block: three launches per step). Which is faster
// depends on the level's fronts, the batch size and the GPU, so on the first
// factorization at a batch size B the level sequence runs once in each form
// (after a fill, untimed warm-up first) with CUDA events around every level's
// large-front work, and each level keeps the fastest form. Decisions are kept in a
// process-wide table keyed by the supernodal structure and B, so later handles on
// the same pattern reuse them. INLA_NO_AUTOTUNE in the environment keeps the
// occupancy rule (fused while every row CTA fits in about one wave, else split).
// ---------------------------------------------------------------------------
namespace {
std::mutex g_tune_mu;
std::map<std::pair<uint64_t, int>, std::vector<char>> g_tune;  // (structure hash, B) -> schedule
}  // namespace

const std::vector<char>* GpuFactor::schedule(int B, const std::function<void()>& fill) {
  static const bool off = std::getenv("INLA_NO_AUTOTUNE") != nullptr;
  if (off) return nullptr;
  bool any_large = false;
  for (const LevelPlan& P : levels_) any_large = any_large || !P.large.empty();
  if (!any_large) return nullptr;
  auto it = fuse_.find(B);
  if (it != fuse_.end()) return &it->second;
  if (panel_form_ >= 0) return &(fuse_[B] = std::vector<char>(levels_.size(), (char)panel_form_));
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    auto g = g_tune.find({struct_hash_, B});
    if (g != g_tune.end()) return &(fuse_[B] = g->second);
  }
  const size_t L = levels_.size();
  std::vector<cudaEvent_t> ev(2 * L);
  for (auto& e : ev) INLA_CUDA(cudaEventCreate(&e));
  std::vector<double> t[kNumForms];
  for (int form = 0; form < kNumForms; ++form) {
    const std::vector<char> pol(L, (char)form);
    fill();
    run_factor_levels(B, &pol, nullptr);  // warm-up (module load, caches)
    fill();
    run_factor_levels(B, &pol, ev.data());
    INLA_CUDA(cudaStreamSynchronize(stream_));
    t[form].assign(L, 0.0);
    for (size_t l = 0; l < L; ++l) {
      float ms = 0.f;
      INLA_CUDA(cudaEventElapsedTime(&ms, ev[2 * l], ev[2 * l + 1]));
      t[form][l] = ms;
    }
  }
  for (auto& e : ev) cudaEventDestroy(e);
  std::vector<char> best(L, kFormSplit);
  double tot[kNumForms] = {0.0, 0.0, 0.0}, tbest = 0.0;
  for (size_t l = 0; l < L; ++l) {
    for (int f = 0; f < kNumForms; ++f) {
      tot[f] += t[f][l];
      if (t[f][l] < t[(int)best[l]][l]) best[l] = (char)f;
    }
    tbest += t[(int)best[l]][l];
  }
  if (std::getenv("INLA_DEBUG"))
    std::fprintf(stderr, "autotune B=%d: split %.3f ms, fused %.3f ms, look-ahead %.3f ms, per-level best %.3f ms\n",
                 B, tot[kFormSplit], tot[kFormFused], tot[kFormLookahead], tbest);
  {
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tune[{struct_hash_, B}] = best;
  }
  return &(fuse_[B] = best);
}

template <class Body>
void GpuFactor::launch_cached(const std::vector<int64_t>& key, Body&& body) {
  if (!use_graphs_ || uncaptured_.count(key)) {
    body();
    INLA_CUDA(cudaGetLastError());
    return;
  }
  auto it = graphs_.find(key);
  if (it == graphs_.end()) {
    const int64_t before = launches_;
    INLA_CUDA(cudaStreamBeginCapture(stream_, cudaStreamCaptureModeThreadLocal));
    bool host_error = false;
    try {
      body();
    } catch (...) {
      host_error = true;
    }
    // A launch rejected during capture (configuration, resources, a call that
    // capture does not allow) returns its error here and invalidates the capture.
    const cudaError_t launch_err = cudaGetLastError();
    cudaGraph_t g = nullptr;
    const cudaError_t end_err = cudaStreamEndCapture(stream_, &g);
    const int64_t captured = launches_ - before;
    launches_ = before;
    if (host_error || launch_err != cudaSuccess || end_err != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      cudaGetLastError();  // the capture's errors are not sticky: clear them
      // Keep the handle usable: this key runs without a graph from now on. A
      // host-side exception of the body surfaces again, with its message, from
      // the direct run.
      const cudaError_t why = launch_err != cudaSuccess ? launch_err : end_err;
      std::fprintf(stderr, "inla_b200: CUDA graph capture of launch sequence %lld failed (%s); running it uncaptured\n",
                   (long long)key[0], host_error ? "host exception" : cudaGetErrorString(why));
      uncaptured_.insert(key);
      ++capture_failures_;
      body();
      const cudaError_t run_err = cudaGetLastError();
      if (run_err != cudaSuccess)
        throw CudaError(std::string("launch sequence failed (capture: ") + cudaGetErrorString(why) +
                            "; direct run: " + cudaGetErrorString(run_err) + ")",
                        (int)run_err);
      return;
    }
    cudaGraphExec_t ex = nullptr;
    cudaError_t e = cudaGraphInstantiate(&ex, g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) throw CudaError(std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e), (int)e);
    it = graphs_.emplace(key, GraphEntry{ex, captured}).first;
  }
  INLA_CUDA(cudaGraphLaunch(it->second.exec, stream_));
  launches_ += it->second.nkernels;
}

void GpuFactor::factor_values(const double* d_vals, int B) {
  if (B < 1 || B > max_batch_) throw std::runtime_error("batch size out of range");
  auto fill = [&] {
    k_fill_panels<<<dim3(nfill_, B), 256, 0, stream_>>>(ds_, d_csn_.p, ntot_, d_pmap_.p, d_vals, nnz_, F_.p,
                                                        ftotal_);
    ++launches_;
  };
  const bool per = use_persist(B, fill);  // settled before any capture
  const std::vector<char>* pol = per ? nullptr : schedule(B, fill);
  launch_cached({1, B, (int64_t)(uintptr_t)d_vals, per}, [&] {
    fill();
    if (per) run_factor_persist(B);
    else run_factor_levels(B, pol);
  });
}

void GpuFactor::factor_model(int ncomp, const double* d_comp, const double* d_coef, double diag_add,
                             const unsigned char* d_pdiag, const int* d_cptr, const int* d_cobs,
                             const double* d_cprod, const double* d_w, int64_t wstride, int B, int nprior,
                             double diag_add_post, const int* d_pseg, int nseg, const unsigned char* d_active) {
  if (B < 1 || B > max_batch_) throw std::runtime_error("batch size out of range");
  if (nprior < 0 || nprior > B) throw std::runtime_error("prior count out of range");
  if (ncomp < 1 || ncomp > 8) throw std::runtime_error("1..8 precision components supported");
  int64_t dbits, dpbits;
  std::memcpy(&dbits, &diag_add, sizeof(dbits));
  std::memcpy(&dpbits, &diag_add_post, sizeof(dpbits));

  const unsigned char* fill_mask = nullptr;  // the measurements below fill and factorize every pair
  auto fill = [&] {
    k_fill_panels_model<<<dim3(nfillm_), 256, 0, stream_>>>(ds_, d_csnm_.p, ntot_, d_pmap_.p, ncomp, d_comp, nnz_,
                                                            d_coef, diag_add, d_pdiag, d_cptr, d_cobs, d_cprod, d_w,
                                                            wstride, B, nprior, diag_add_post, d_pseg, nseg, F_.p,
                                                            ftotal_, d_fseg_.p, fill_mask);
    ++launches_;
  };
  const bool per = use_persist(B, fill);  // settled before any capture
  if (!d_fseg_.p) d_active = nullptr;
  fill_mask = d_active;
  const std::vector<char>* pol = per ? nullptr : schedule(B, fill);
  launch_cached({2, B, ncomp, (int64_t)(uintptr_t)d_comp, (int64_t)(uintptr_t)d_coef, dbits,
                 (int64_t)(uintptr_t)d_pdiag, (int64_t)(uintptr_t)d_cptr, (int64_t)(uintptr_t)d_cobs,
                 (int64_t)(uintptr_t)d_cprod, (int64_t)(uintptr_t)d_w, wstride, nprior, dpbits,
                 (int64_t)(uintptr_t)d_pseg, nseg, (int64_t)(uintptr_t)d_active, per},
                [&] {
                  fill();
                  if (per) {
                    run_factor_persist(B, nullptr, 0, d_active, nseg);
                  } else {
                    const DevSym plain = ds_;
                    if (d_active) {  // the level kernels read the mask through the device view
                      ds_.active = d_active;
                      ds_.fseg = d_fseg_.p;
                      ds_.nseg = nseg;
                    }
                    run_factor_levels(B, pol);
                    ds_ = plain;
                  }
                });
}

void GpuFactor::solve(double* d_x, int64_t xstride, int B, int slot0) {
  if (B < 1 || slot0 < 0 || slot0 + B > max_batch_) throw std::runtime_error("batch size out of range");
  const int n = (int)sym_.n;
  dim3 gp(cdiv(n, 256) > 1024 ? 1024 : cdiv(n, 256), B);
  auto pa = solve_persist_at_.find(B);
  const bool per = solve_persist_ && (persist_mode_ == 2 || (pa != solve_persist_at_.end() && pa->second));
  launch_cached({3, B, (int64_t)(uintptr_t)d_x, xstride, slot0, per}, [&] {
    k_permute_in<<<gp, 256, 0, stream_>>>(n, d_perm_.p, d_x, xstride, xp_.p);
    if (per) solve_queue(B, slot0);
    else solve_levels(B, slot0);
    k_permute_out<<<gp, 256, 0, stream_>>>(n, d_perm_.p, xp_.p, d_x, xstride);
    launches_ += 2;
  });
}

void GpuFactor::solve_queue(int B, int slot0) {
  const int ns = (int)sym_.nsuper;
  INLA_CUDA(cudaMemsetAsync(d_sstate_.p + 1, 0, sizeof(int) * (1 + 2 * (size_t)B * ns), stream_));
  SolveArgs a;
  a.S = ds_;
  a.F = F_.p + (int64_t)slot0 * ftotal_;
  a.fstride = ftotal_;
  a.B = B;
  a.ngroups = solve_groups_;
  a.gstart = d_sgstart_.p;
  a.task = reinterpret_cast<const PersistTask*>(d_stask_.p);
  a.tiny_list = d_stiny_.p;
  a.linv = linv_.p + (int64_t)slot0 * ds_.lstride;
  a.xp = xp_.p;
  a.ub = ub_.p;
  a.ustride = std::max<int64_t>(usum_, 1);
  a.progf = d_sstate_.p + 2;
  a.progb = d_sstate_.p + 2 + (size_t)B * ns;
  a.head = reinterpret_cast<unsigned*>(d_sstate_.p + 1);
  a.err = d_sstate_.p;
  a.limit_ns = persist_limit_ns_;
  k_solve_persist<<<solve_grid_, kPersistThreads, solve_smem_, stream_>>>(a);
  ++launches_;
}

// Fronts of up to kSmallB rows (contiguous lists small_a, small_b) in 32-column blocks by one CTA each;
// larger fronts in 64-column blocks with their cached inverse blocks.
void GpuFactor::solve_levels(int B, int slot0) {
  const int64_t fs = ftotal_, us = std::max<int64_t>(usum_, 1);
  const double* Fp = F_.p + (int64_t)slot0 * fs;
  const double* Lp = linv_.p + (int64_t)slot0 * ds_.lstride;
  for (size_t li = 0; li < levels_.size(); ++li) {
    const LevelPlan& P = levels_[li];
    if (band_at_[li] >= 0) {
      const MiniBand& M = bands_[band_at_[li]];
      if ((int)li != M.l0) continue;
      k_fwd_mini<<<dim3(cdiv(M.ntask, kMiniGroups), B), kMiniThreads, 0, stream_>>>(
          ds_, mini_tables(M.off), M.ntask, Fp, fs, xp_.p, ub_.p, us);
      ++launches_;
      continue;
    }
    if (!P.tiny.empty()) {
      const int nt = (int)P.tiny.size();
      k_fwd_tiny<<<dim3(cdiv(nt, kTinySweepWarps), B), 32 * kTinySweepWarps, 0, stream_>>>(
          ds_, d_lists_.p + P.off_tiny, nt, Fp, fs, xp_.p, ub_.p, us);
      ++launches_;
    }
    const int nsm = (int)(P.small_a.size() + P.small_b.size());
    if (nsm > 0) {
      k_fwd32<128><<<dim3((unsigned)nsm, B), 128, (std::max(P.mmax_a, P.mmax_b) + 2 + 32 * 33) * 8, stream_>>>(
          ds_, d_lists_.p + P.off_small_a, Fp, fs, xp_.p, ub_.p, us);
      ++launches_;
    }
    if (!P.large.empty()) {
      const dim3 g((unsigned)P.large.size(), B);
      const int sm = (P.mmax_large + 2) * 8;
      if ((int64_t)P.large.size() * B <= num_sms_)
        k_fwd64<256, true><<<g, 256, sm, stream_>>>(ds_, d_lists_.p + P.off_large, Fp, fs, Lp, xp_.p, ub_.p, us);
      else
        k_fwd64<256, false><<<g, 256, sm, stream_>>>(ds_, d_lists_.p + P.off_large, Fp, fs, Lp, xp_.p, ub_.p, us);
      ++launches_;
    }
  }
  for (int l = (int)levels_.size() - 1; l >= 0; --l) {
    const LevelPlan& P = levels_[l];
    if (band_at_[l] >= 0) {
      const MiniBand& M = bands_[band_at_[l]];
      if (l != M.l0) continue;
      k_bwd_mini<<<dim3(cdiv(M.ntask, kMiniGroups), B), kMiniThreads, 0, stream_>>>(
          ds_, mini_tables(M.off), M.ntask, Fp, fs, xp_.p);
      ++launches_;
      continue;
    }
    if (!P.tiny.empty()) {
      const int nt = (int)P.tiny.size();
      k_bwd_tiny<<<dim3(cdiv(nt, kTinySweepWarps), B), 32 * kTinySweepWarps, 0, stream_>>>(
          ds_, d_lists_.p + P.off_tiny, nt, Fp, fs, xp_.p);
      ++launches_;
    }
    const int nsm = (int)(P.small_a.size() + P.small_b.size());
    if (nsm > 0) {
      k_bwd32<128><<<dim3((unsigned)nsm, B), 128, (std::max(P.mmax_a, P.mmax_b) + 2 + 32 * 33) * 8, stream_>>>(
          ds_, d_lists_.p + P.off_small_a, Fp, fs, xp_.p);
      ++launches_;
    }
    if (!P.large.empty()) {
      const dim3 g((unsigned)P.large.size(), B);
      const int sm = (P.mmax_large + 2) * 8;
      if ((int64_t)P.large.size() * B <= num_sms_)
        k_bwd64<256, true><<<g, 256, sm, stream_>>>(ds_, d_lists_.p + P.off_large, Fp, fs, Lp, xp_.p);
      else
        k_bwd64<256, false><<<g, 256, sm, stream_>>>(ds_, d_lists_.p + P.off_large, Fp, fs, Lp, xp_.p);
      ++launches_;
    }
  }
}

// Launches of the products of a level whose large fronts have at most kmax pivots and rmax rows below them,
// for `pairs` (front, problem) pairs. Only tiles that exist are counted: the count decides between whole
// tiles and 32-row halves, and a launch takes at most kMaxGridZ of them.
constexpr int kMaxGridZ = 65535;
std::vector<SiLaunch> si_launches(int kmax, int rmax, int64_t pairs, int sms) {
  std::vector<SiLaunch> out;
  auto add = [&](int mode, int hb, int64_t tiles) {
    const bool half = pairs * tiles <= sms;
    for (int64_t z0 = 0; z0 < tiles; z0 += kMaxGridZ)
      out.push_back({mode, hb, (int)z0, (int)std::min<int64_t>(kMaxGridZ, tiles - z0), half});
  };
  const int nblk = cdiv(kmax, kB64);
  for (int hb = 1; hb < nblk; hb *= 2) {
    add(SI_T, hb, si_join_tiles(nblk, hb));
    add(SI_X, hb, si_join_tiles(nblk, hb));
  }
  const int64_t below = (int64_t)cdiv(rmax, kSiT) * nblk;
  add(SI_W, 0, below);
  add(SI_BK, 0, below);
  add(SI_KK, 0, (int64_t)nblk * (nblk + 1) / 2);
  return out;
}

// Host check of those launches for every front of an analysis at batch size B: grids within the limits, and
// every tile of every product computed exactly once.
std::string check_selinv_launches(const Symbolic& S, const std::vector<LevelPlan>& levels, int B, int sms,
                                  int64_t* info3) {
  int64_t nlaunch = 0, zmax = 0, ctas = 0;
  for (const LevelPlan& P : levels) {
    if (P.si_large.empty()) continue;
    const std::vector<SiLaunch> launches =
        si_launches(P.kmax_si_large, P.rmax_si_large, (int64_t)P.si_large.size() * B, sms);
    for (const SiLaunch& x : launches) {
      const int64_t z = x.half ? 2 * (int64_t)x.tiles : x.tiles;
      if (z < 1 || z > kMaxGridZ || (x.hb > 0 && x.z0 > 0)) return "grid of " + std::to_string(z) + " tiles";
      ++nlaunch;
      zmax = std::max(zmax, z);
      ctas += z;
    }
    for (int s : P.si_large) {
      const int k = (int)(S.sn_first[s + 1] - S.sn_first[s]), m = (int)(S.sn_rowptr[s + 1] - S.sn_rowptr[s]);
      const int nblk = cdiv(k, kB64), rt = cdiv(m - k, kSiT);
      std::map<std::pair<int, int>, std::vector<int64_t>> rows;  // (mode, hb): rows done of every 64-column block
      for (const SiLaunch& x : launches) {
        std::vector<int64_t>& seen = rows[{x.mode, x.hb}];
        seen.resize((size_t)nblk * (nblk + rt), 0);
        for (int z = 0; z < (x.half ? 2 : 1) * x.tiles; ++z) {
          auto tile = [&](auto mode) {
            constexpr int M = decltype(mode)::value;
            SiTile t;
            const bool ok = x.half ? si_tile<M, 32>(x.z0 + z, x.hb, k, m, t) : si_tile<M, 64>(x.z0 + z, x.hb, k, m, t);
            if (!ok) return true;
            const bool below = M == SI_W || M == SI_BK;
            if (t.i0 < 0 || t.i1 > (below ? m : k) || t.j0 < 0 || t.j0 >= k || t.t0 > t.t1 || t.t1 > m) return false;
            const int I = below ? nblk + (t.i0 - k) / kSiT : t.i0 / kB64;
            seen[(size_t)I * nblk + t.j0 / kB64] += t.i1 - t.i0;
            return true;
          };
          bool ok = true;
          if (x.mode == SI_T) ok = tile(std::integral_constant<int, SI_T>());
          else if (x.mode == SI_X) ok = tile(std::integral_constant<int, SI_X>());
          else if (x.mode == SI_W) ok = tile(std::integral_constant<int, SI_W>());
          else if (x.mode == SI_BK) ok = tile(std::integral_constant<int, SI_BK>());
          else ok = tile(std::integral_constant<int, SI_KK>());
          if (!ok) return "tile out of range";
        }
      }
      for (int hb = 1; hb < nblk; hb *= 2)
        if (!rows.count({SI_T, hb}) || !rows.count({SI_X, hb})) return "a join is missing";
      if (!rows.count({SI_KK, 0}) || (rt > 0 && (!rows.count({SI_W, 0}) || !rows.count({SI_BK, 0}))))
        return "a product is missing";
      for (const auto& r : rows) {
        const int mode = r.first.first, hb = r.first.second;
        for (int I = 0; I < nblk + rt; ++I)
          for (int J = 0; J < nblk; ++J) {
            bool want = I < nblk && I >= J;  // SI_KK
            if (mode == SI_T || mode == SI_X) want = I < nblk && I / (2 * hb) == J / (2 * hb) && (I / hb) % 2 == 1 && (J / hb) % 2 == 0;
            if (mode == SI_W || mode == SI_BK) want = I >= nblk;
            const int len = I < nblk ? std::min(kB64, k - I * kB64) : std::min(kSiT, m - k - (I - nblk) * kSiT);
            if (r.second[(size_t)I * nblk + J] != (want ? len : 0))
              return "front " + std::to_string(s) + ", product " + std::to_string(mode) + ": tile (" +
                     std::to_string(I) + ", " + std::to_string(J) + ") not computed once";
          }
      }
    }
  }
  if (info3) {
    info3[0] = nlaunch;
    info3[1] = zmax;
    info3[2] = ctas;
  }
  return std::string();
}

void GpuFactor::selinv(int B, int slot0) {
  if (B < 1 || slot0 < 0 || slot0 + B > max_batch_) throw std::runtime_error("batch size out of range");
  Sg_.alloc((size_t)max_batch_ * ftotal_);  // outside any capture
  launch_cached({4, B, slot0}, [&] { selinv_levels(B, slot0); });
}

void GpuFactor::selinv_levels(int B, int slot0) {
  const int64_t fs = ftotal_;
  const double* Fp = F_.p + (int64_t)slot0 * fs;
  double* Sp = Sg_.p + (int64_t)slot0 * fs;
  const double* Lp = linv_.p + (int64_t)slot0 * ds_.lstride;
  for (int l = (int)levels_.size() - 1; l >= 0; --l) {
    const LevelPlan& P = levels_[l];
    if (band_at_[l] >= 0) {
      const MiniBand& M = bands_[band_at_[l]];
      if (l != M.l0) continue;
      k_selinv_mini<<<dim3(cdiv(M.ntask, kMiniGroups), B), kMiniThreads, 0, stream_>>>(
          ds_, mini_tables(M.off), M.ntask, Fp, Sp, fs);
      ++launches_;
      continue;
    }
    if (!P.si_tiny.empty()) {
      const int nt = (int)P.si_tiny.size();
      k_selinv_tiny<<<dim3(cdiv(nt, kTinySiWarps), B), 32 * kTinySiWarps, 0, stream_>>>(
          ds_, d_lists_.p + P.off_si_tiny, nt, Fp, Sp, fs);
      ++launches_;
    }
    if (!P.si_small.empty()) {
      int mm = P.mmax_si_small;
      k_selinv_small<256><<<dim3((unsigned)P.si_small.size(), B), 256, small_selinv_smem(mm, P.kmax_si_small),
                            stream_>>>(
          ds_, d_lists_.p + P.off_si_small, Fp, Sp, fs);
      ++launches_;
    }
    if (!P.si_large.empty()) {
      const int nl = (int)P.si_large.size();
      const int* lst = d_lists_.p + P.off_si_large;
      if (P.rmax_si_large > 0) {
        k_si_gather8<<<dim3(nl, B, cdiv(P.rmax_si_large, kGatherCols)), 256, 0, stream_>>>(ds_, lst, Sp, fs);
        ++launches_;
      }
      for (const SiLaunch& x : si_launches(P.kmax_si_large, P.rmax_si_large, (int64_t)nl * B, num_sms_)) {
        auto go = [&](auto full, auto half) {
          (x.half ? half : full)<<<dim3(nl, B, x.half ? 2 * x.tiles : x.tiles), 256, kSiGemmSmem, stream_>>>(
              ds_, lst, x.hb > 0 ? x.hb : x.z0, Fp, Sp, fs, Lp);
          ++launches_;
        };
        if (x.mode == SI_T) go(k_si_gemm<SI_T, 64>, k_si_gemm<SI_T, 32>);
        else if (x.mode == SI_X) go(k_si_gemm<SI_X, 64>, k_si_gemm<SI_X, 32>);
        else if (x.mode == SI_W) go(k_si_gemm<SI_W, 64>, k_si_gemm<SI_W, 32>);
        else if (x.mode == SI_BK) go(k_si_gemm<SI_BK, 64>, k_si_gemm<SI_BK, 32>);
        else go(k_si_gemm<SI_KK, 64>, k_si_gemm<SI_KK, 32>);
      }
    }
  }
}

void GpuFactor::extract_diag(double* d_out, int64_t ostride, int B, int slot0) {
  const int n = (int)sym_.n;
  k_extract_diag<<<dim3(std::min(cdiv(n, 256), 1024), B), 256, 0, stream_>>>(ds_, Sg_.p + (int64_t)slot0 * ftotal_,
                                                                              ftotal_, d_out, ostride);
  ++launches_;
  INLA_CUDA(cudaGetLastError());
}

void GpuFactor::sigma_on_pattern(double* d_out, int B, int slot0) {
  k_pattern_values<<<dim3(std::min(cdiv(nnz_, 256), 2048), B), 256, 0, stream_>>>(
      nnz_, spos_.p, Sg_.p + (int64_t)slot0 * ftotal_, ftotal_, d_out);
  ++launches_;
  INLA_CUDA(cudaGetLastError());
}

}  // namespace inla
