// edges.cuh -- passes over the entries of a CSR in tiles of consecutive
// entries, with the row of every entry at hand.
//
// A warp per row leaves a hub row of tens of thousands of entries to one
// warp, and the kernel waits for it (R-MAT 20 directed, writing one 12-byte
// pair per entry: 642 us with a warp per row).  A tile has the same work
// whatever the row lengths: a block finds the rows of its first and last entry
// by a 32-way search of the offsets, marks the position where each row between
// them starts with that row's id, and an inclusive max-scan of the marks gives
// every entry its row.  A tile that spans many more rows than it has entries
// (long runs of empty rows) searches the row of each entry instead: ten million rows of
// 2,000 entries, transposed, 123 us; with every row marked by its tile's one
// block 7,745, a warp per row 380.
#pragma once
#include "common.cuh"

namespace apspie {

constexpr int kEdgeThreads = 256;
constexpr int kEdgeItems = 8;                          // entries per thread
constexpr int kEdgeTile = kEdgeThreads * kEdgeItems;  // entries per tile
constexpr int kEdgeMarkRows = 4 * kEdgeTile;           // rows of a tile that are marked

// A kernel's tiles cover the entries [ptr[0], ptr[m]), whatever count the
// caller gave: offsets may start anywhere in the arrays they index (a slice of
// a larger matrix's rows).

// Largest r with ptr[r] <= k, given ptr[0] <= k < ptr[m] (else some row of the
// matrix).  Warp-collective.  (P: int, or long long for offsets whose total has
// been checked to fit an int.)
template <typename P>
__device__ __forceinline__ int row_of_entry(const P *__restrict__ ptr, int m, int k) {
  const int lane = lane_id();
  int lo = 0, hi = m;  // ptr[lo] <= k < ptr[hi]
  while (hi - lo > 1) {
    const long long span = hi - lo;
    const int piv = lo + (int)(span * lane / 32);
    // lane 0 counts as below: the search stays inside [lo, hi] whatever k is
    const unsigned b = __ballot_sync(kFull, lane == 0 || __ldg(ptr + piv) <= k);
    const int last = 31 - __clz(b);
    const int nlo = lo + (int)(span * last / 32);
    const int nhi = last == 31 ? hi : lo + (int)(span * (last + 1) / 32);
    lo = nlo;
    hi = max(nhi, nlo + 1);
  }
  return lo;
}

// Entries of tile number `tile` (0: none left); *k0: the first of them.
template <typename P>
__device__ __forceinline__ int edge_tile(const P *__restrict__ ptr, int m, unsigned tile, int *k0) {
  const long long first = (long long)__ldg(ptr) + (long long)tile * kEdgeTile;
  const long long left = (long long)__ldg(ptr + m) - first;
  *k0 = (int)first;
  return left <= 0 ? 0 : (int)min((long long)kEdgeTile, left);
}

// Rows of the entries k0 + t, t in [0, n), that lie in rows [r0, r1]: binary
// searches, kSearch of a thread's entries side by side.  (Not inlined, and not
// all of them at once: its registers count for the kernels' ordinary tiles.)
template <typename P>
__device__ __noinline__ void search_rows(const P *__restrict__ ptr, int r0, int r1, int k0,
                                         int n, int *s_row) {
  constexpr int kSearch = 2;
  for (int t0 = (int)threadIdx.x; t0 < n; t0 += kSearch * kEdgeThreads) {
    int lo[kSearch], len[kSearch];  // the row is one of lo .. lo + len - 1
#pragma unroll
    for (int i = 0; i < kSearch; ++i) {
      lo[i] = r0;
      len[i] = r1 - r0 + 1;
    }
#pragma unroll 1
    for (unsigned span = (unsigned)(r1 - r0); span > 0; span >>= 1) {
#pragma unroll
      for (int i = 0; i < kSearch; ++i) {
        const int half = len[i] >> 1;
        const bool up = half > 0 && (int)__ldg(ptr + lo[i] + half) <= k0 + t0 + i * kEdgeThreads;
        lo[i] += up ? half : 0;
        len[i] = up ? len[i] - half : max(half, 1);
      }
    }
#pragma unroll
    for (int i = 0; i < kSearch; ++i) {
      const int t = t0 + i * kEdgeThreads;
      if (t < n) s_row[t] = lo[i];
    }
  }
}

// s_row[t] = row of entry k0 + t for t in [0, n), n <= kEdgeTile.  Called by
// all kEdgeThreads threads; s_row is ready when it returns, and must have been
// read by all of them before the next call.
template <typename P>
__device__ __forceinline__ void edge_tile_rows(const P *__restrict__ ptr, int m, int k0, int n,
                                               int *s_row) {
  __shared__ int s_warp[kEdgeThreads / 32];
  __shared__ int s_end[2];
  const int t = threadIdx.x, lane = lane_id(), w = warp_in_block();
  if (w < 2) {
    const int r = row_of_entry(ptr, m, w == 0 ? k0 : k0 + n - 1);
    if (lane == 0) s_end[w] = r;
  }
  for (int i = t; i < kEdgeTile; i += kEdgeThreads) s_row[i] = -1;
  __syncthreads();
  const int r0 = s_end[0], r1 = s_end[1];
  if (r1 - r0 > kEdgeMarkRows) {
    search_rows(ptr, r0, r1, k0, n, s_row);
    __syncthreads();
    return;
  }
  // empty rows start where the next non-empty one does: the largest id wins
  for (int r = r0 + 1 + t; r <= r1; r += kEdgeThreads) {
    const int at = (int)__ldg(ptr + r) - k0;
    if ((unsigned)at < (unsigned)n) atomicMax(s_row + at, r);
  }
  __syncthreads();
  // inclusive max-scan, kEdgeItems consecutive entries per thread
  int4 *q4 = reinterpret_cast<int4 *>(s_row) + t * (kEdgeItems / 4);
  int v[kEdgeItems];
#pragma unroll
  for (int i = 0; i < kEdgeItems / 4; ++i) {
    const int4 x = q4[i];
    v[4 * i] = x.x, v[4 * i + 1] = x.y, v[4 * i + 2] = x.z, v[4 * i + 3] = x.w;
  }
#pragma unroll
  for (int i = 1; i < kEdgeItems; ++i) v[i] = max(v[i], v[i - 1]);
  int incl = v[kEdgeItems - 1];
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(kFull, incl, o);
    if (lane >= o) incl = max(incl, y);
  }
  if (lane == 31) s_warp[w] = incl;
  int before = __shfl_up_sync(kFull, incl, 1);
  if (lane == 0) before = -1;
  __syncthreads();
  before = max(before, r0);
  for (int x = 0; x < w; ++x) before = max(before, s_warp[x]);
#pragma unroll
  for (int i = 0; i < kEdgeItems / 4; ++i)
    q4[i] = make_int4(max(before, v[4 * i]), max(before, v[4 * i + 1]), max(before, v[4 * i + 2]),
                      max(before, v[4 * i + 3]));
  __syncthreads();
}

// The lanes of a warp that hold entries of this lane's row, for entries in
// CSR order (equal rows are adjacent); leader: the first of them.  Lanes
// past the end pass row -1.  Warp-collective.
__device__ __forceinline__ unsigned row_peers(int row, int *leader) {
  const int lane = lane_id();
  const int prev = __shfl_up_sync(kFull, row, 1);
  const unsigned heads = __ballot_sync(kFull, lane == 0 || row != prev);
  const unsigned upto = lane == 31 ? kFull : (2u << lane) - 1u;
  *leader = 31 - __clz(heads & upto);
  const unsigned after = heads & ~upto;
  const unsigned below_next = after ? (1u << (__ffs(after) - 1)) - 1u : kFull;
  return below_next & ~((1u << *leader) - 1u);
}

// Blocks for nnz entries, at least one.  Kernels that call edge_tile stride
// their tiles by it, so a count below the offsets' leaves no entry out.
inline unsigned edge_tiles(long long nnz) {
  return (unsigned)(nnz > kEdgeTile ? (nnz + kEdgeTile - 1) / kEdgeTile : 1);
}

}  // namespace apspie
