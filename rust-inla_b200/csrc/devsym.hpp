// Device view of one symbolic analysis (plain pointers into device arrays).
#pragma once
#include <cstdint>

namespace inla {

// A column of a child's update block: F offset of its first entry (the diagonal one), its rows and the
// offset of their places in relx.
struct alignas(16) GatherCol {
  int64_t src;
  int len, rel;
};

struct DevSym {
  int n = 0, ns = 0;
  const int* first = nullptr;      // ns+1
  const int* rowptr = nullptr;     // ns+1
  const int* rows = nullptr;       // sum m : permuted row indices
  const int* relx = nullptr;       // sum m : position of below-row in parent's structure
  const int64_t* fptr = nullptr;   // ns+1 : front offsets
  const int64_t* lptr = nullptr;   // ns+1 : panel offsets (compact m*k numbering)
  const int* child_ptr = nullptr;  // ns+1
  const int* child_list = nullptr;
  const int* parent = nullptr;     // ns
  const int* uoff = nullptr;       // ns+1 : offsets of the per-supernode update vectors (sum r)
  // children's update entries that add into each front row, in child order: entries
  // rss[rsp[i] .. rsp[i + 1]) of the update vectors for row i of the concatenated structures
  const int* rsp = nullptr;        // sum m + 1
  const int* rss = nullptr;        // sum r
  // the children's columns that add into each column of the large fronts, in child order: rsp's ranges
  // for front s, moved by gptr[s]
  const GatherCol* gcol = nullptr;
  const int64_t* gptr = nullptr;   // ns
  const int64_t* dpos = nullptr;   // n : front offset of D_j
  const int* perm = nullptr;       // n : perm[new] = old
  // 64 x 64 inverse-block cache of the large fronts: block (s, j0 / 64) of
  // problem b at linv + (b * lstride + (lbo[s] + j0 / 64) * 4096); lbo[s] = -1
  // for fronts that have no cached blocks.
  const int* lbo = nullptr;        // ns
  int64_t lstride = 0;
  // Optional (independent models held block-diagonally): the factorization skips the fronts
  // of the (problem, model) pairs whose entry of active ([B][nseg]) is 0; fseg: model of
  // each front. Those fronts keep their previous contents.
  const unsigned char* active = nullptr;
  const int* fseg = nullptr;
  int nseg = 1;
};

// Tables of the bands of small fronts (snode_mini.cuh). A front: its F offset, rows, pivots, first entry in
// the child table, and the F offset and rows of its parent.
struct alignas(16) MiniFront {
  int64_t fptr;
  int rowptr, first;
  int k, m, child0, nch;
  int64_t pptr;
  int pm, uoff;
};
// A child's update block: F offset of its first entry, its place in relx, rows of the child * 16 + rows of
// the block.
struct alignas(16) MiniChild {
  int64_t src;
  int rel, dim;
};
// Task ranges, fronts in task order (children before parents; `list`: their numbers) and their children.
struct MiniTables {
  const int* ptr;
  const int* list;
  const MiniFront* front;
  const MiniChild* child;
};

__host__ __device__ inline bool front_skipped(const DevSym& S, int s, int b) {
  return S.active && !S.active[(int64_t)b * S.nseg + S.fseg[s]];
}

constexpr int kStatusOk = 0;
constexpr int kStatusSingular = 1;
constexpr int kStatusNotFinite = 2;
constexpr int kStatusSchedule = 4;  // the persistent schedule stopped early (a dependency wait ran out)

}  // namespace inla
