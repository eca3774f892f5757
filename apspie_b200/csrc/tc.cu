// tc.cu -- triangle counting as an L-masked hash SpGEMM with an int64 count,
// and the device-side degree relabelling that builds L.
//
// Replaces the reference's TC path (test/tc/main.cu:139-261): host buildLower
// of the strict lower / upper triangles, cuSPARSE csrgemm U * L materialising
// every wedge (src/tc.cuh:63-165), the ewiseMultTc merge-intersect
// (src/tc.cuh:169-199) and a float mgpu::Reduce.  Here nothing but the count
// is produced.  With U(j) = the rows that have j in L (L's column j), a
// triangle i > k > j is an entry (k, j) of L and an i in both U(j) and U(k),
// so the count is the sum of |U(j) ^ U(k)| over L's entries.  The columns are
// gathered first (tc_scatter; their order does not matter).  An entry belongs
// to the end with the longer column, whose column is a set in shared memory;
// the other end's column, the shorter one, is read and probes it.  Under
// tc_prepare's order by ascending degree the columns are short (R-MAT 18: at
// most 413 entries, rows of L up to 25,224), so the probes are 321 M where
// the products of L's rows are 660 M, and a set is built once per 256
// entries of its end, or by a warp for itself.
//
// Repeated edges: with M the entries of L counted by multiplicity, the result
// is the sum of M * M over L's distinct entries, whichever end an entry belongs
// to.  That needs column j as the set and every entry of column k as a probe, so
// an L with repeats (tc_scatter finds them) is counted by a second kernel whose
// entries all belong to their column's end.
//
// tc_prepare relabels vertices by ascending (degree, id) with the stable
// radix sort and lists the edges with new(col) < new(row) grouped by ascending
// column, so that one stable sort on the row bits leaves every row of L
// ascending; L's offsets come from the row lengths.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstring>

#include "common.cuh"
#include "context.h"
#include "edges.cuh"
#include "gen_common.h"
#include "primitives.cuh"

namespace apspie {
namespace {

// Ends of at most kTcTinyCand entries (row and column together) and a column
// of at most kTcTiny are a quarter warp's (2^20 vertices of mean degree 10:
// 393 us with a warp each); up to kTcWarpCand entries and a column of
// kTcWarpSet they are one warp's; longer ones are cut into units of
// kTcUnit entries, a block each.  A block's set holds kTcPart entries at a
// time (more: the unit's probes are repeated for each part): those among the
// kTcTop largest ids in a bitmap, one shared-memory read per probe, the rest
// in a hash table at most half full.
constexpr int kTcTiny = 8, kTcTinyCand = 24;
constexpr int kTcWarpCand = 128, kTcWarpSet = 128, kTcWarpTableBits = 8;
constexpr int kTcUnit = 256;
constexpr int kTcPart = 1024, kTcTableBits = 11;
constexpr int kTcTop = 1 << 16;
constexpr int kTcThreads = 256;
constexpr int kTcWarps = kTcThreads / 32;
constexpr int kTcLong = 24;  // columns of this many entries are read by the whole warp
constexpr int kNone = INT_MAX;

__device__ __forceinline__ unsigned tc_hash(int j) { return (unsigned)j * 0x9E3779B1u; }

__device__ __forceinline__ void set_insert(int *keys, int bits, int j) {
  unsigned mask = (1u << bits) - 1u, h = tc_hash(j) >> (32 - bits);
  for (unsigned p = 0; p <= mask; ++p) {
    int old = atomicCAS(keys + h, kNone, j);
    if (old == kNone || old == j) return;
    h = (h + 1) & mask;
  }
}

__device__ __forceinline__ bool set_has(const int *keys, int bits, int j) {
  unsigned mask = (1u << bits) - 1u, h = tc_hash(j) >> (32 - bits);
  for (unsigned p = 0; p <= mask; ++p) {
    int k = keys[h];
    if (k == j) return true;
    if (k == kNone) return false;
    h = (h + 1) & mask;
  }
  return false;
}

struct TcBins {
  unsigned n[3];  // tiny ends, warp ends, units
  unsigned grab;  // units handed out
  unsigned long long count;
  unsigned multi;  // some entry of L repeats the one before it in its row
  unsigned pad;
};

// An entry of a column: repeats of a row's entry are stored as ~row.
__device__ __forceinline__ int member(int x) { return x < 0 ? ~x : x; }

// Lengths of L's columns, and each entry's place in its column: the atomics
// that count the columns give it, so the scatter needs none of its own (with a
// cursor per column that each entry advanced, the call on R-MAT 18 took 1,162
// us instead of 1,151).
constexpr int kTcRankItems = 4;

__global__ void __launch_bounds__(kTcThreads)
tc_col_ranks(int m, int lnnz, const int *__restrict__ Lp, const int *__restrict__ Li, int *cnt,
             int *rank) {
  const int *first = Li + __ldg(Lp);
  const int n = min(lnnz, __ldg(Lp + m) - __ldg(Lp));  // rank holds lnnz entries
  constexpr long long kStep = (long long)kTcThreads * kTcRankItems;
  for (long long b = blockIdx.x * kStep; b < n; b += gridDim.x * kStep) {
    int c[kTcRankItems], r[kTcRankItems];
#pragma unroll
    for (int q = 0; q < kTcRankItems; ++q) {
      const long long k = b + q * kTcThreads + threadIdx.x;
      c[q] = k < n ? __ldg(first + k) : -1;
    }
#pragma unroll
    for (int q = 0; q < kTcRankItems; ++q) r[q] = add_if(c[q] >= 0, cnt + c[q], 1, 0);
#pragma unroll
    for (int q = 0; q < kTcRankItems; ++q)
      if (c[q] >= 0) rank[b + q * kTcThreads + threadIdx.x] = r[q];
  }
}

// Every vertex's column as (start, length), and its place among the tiny ends
// (lists from the front), the warp ends (lists from the back) or its units
// (vertex, piece).
__global__ void tc_bin(int m, const int *__restrict__ Lp, const int *__restrict__ Up,
                       int2 *col, int *lists, int2 *units, TcBins *bins) {
  const int lane = lane_id();
  for (int v0 = blockIdx.x * blockDim.x + threadIdx.x - lane; v0 < m; v0 += gridDim.x * blockDim.x) {
    const int v = v0 + lane;
    int cand = 0, d = 0;
    if (v < m) {
      const int us = Up[v];
      d = Up[v + 1] - us;
      cand = Lp[v + 1] - Lp[v] + d;
      col[v] = make_int2(us, d);
    }
    // an entry needs a set to probe and a column no longer than it
    // (an end of one entry has nothing but the entry to its set's member)
    const bool tiny = d > 0 && cand > 1 && cand <= kTcTinyCand && d <= kTcTiny;
    const bool warp = d > 0 && !tiny && cand > 1 && cand <= kTcWarpCand && d <= kTcWarpSet;
    const unsigned at0 = warp_append(tiny, &bins->n[0]);
    if (tiny) lists[at0] = v;
    const unsigned at1 = warp_append(warp, &bins->n[1]);
    if (warp) lists[m - 1 - (int)at1] = v;
    if (d > 0 && cand > kTcTinyCand && !warp) {
      const int pieces = (cand - 1) / kTcUnit + 1;
      const unsigned u = atomicAdd(&bins->n[2], (unsigned)pieces);
      for (int p = 0; p < pieces; ++p) units[u + p] = make_int2(v, p);
    }
  }
}

// L's entries into their columns, in any order within a column; repeats, which
// follow each other in a row of ascending columns, are marked.
__global__ void __launch_bounds__(kEdgeThreads)
tc_scatter(int m, int lnnz, const int *__restrict__ Lp, const int *__restrict__ Li,
           const int *__restrict__ Up, const int *__restrict__ rank, int *Ui, TcBins *bins) {
  __shared__ __align__(16) int s_row[kEdgeTile];
  const int *erank = rank - __ldg(Lp);  // by entry
  int k0;
  const int n = min(edge_tile(Lp, m, blockIdx.x, &k0), lnnz - (int)blockIdx.x * kEdgeTile);
  if (n <= 0) return;
  edge_tile_rows(Lp, m, k0, n, s_row);
  int c[kEdgeItems], at[kEdgeItems];
#pragma unroll
  for (int q = 0; q < kEdgeItems; ++q) {
    const int t = (int)threadIdx.x + q * kEdgeThreads;
    c[q] = t < n ? __ldg(Li + k0 + t) : -1;
  }
#pragma unroll
  for (int q = 0; q < kEdgeItems; ++q) {
    const int t = (int)threadIdx.x + q * kEdgeThreads;
    at[q] = c[q] >= 0 ? __ldg(Up + c[q]) + __ldg(erank + k0 + t) : 0;
  }
  bool repeats = false;
#pragma unroll
  for (int q = 0; q < kEdgeItems; ++q) {
    const int t = (int)threadIdx.x + q * kEdgeThreads;
    int before = __shfl_up_sync(kFull, c[q], 1);
    if (lane_id() == 0) before = t > 0 && t < n ? __ldg(Li + k0 + t - 1) : -1;
    if (c[q] < 0) continue;
    const int row = s_row[t];
    bool again = before == c[q] && t > 0 && s_row[t - 1] == row;
    if (t == 0 && __ldg(Lp + row) < k0) again = __ldg(Li + k0 - 1) == c[q];
    repeats |= again;
    Ui[at[q]] = again ? ~row : row;
  }
  if (__any_sync(kFull, repeats) && lane_id() == 0) bins->multi = 1u;
}

// Members of the set `has` among the columns (start, len) that the lanes
// hold, one each.  Long columns one after the other with 128 entries in
// flight, the entries of the short ones dealt flat over the lanes.
template <bool kMulti, typename Has>
__device__ __forceinline__ unsigned tc_probe(int start, int len, const int *__restrict__ Ui,
                                             Has has) {
  const int lane = lane_id();
  unsigned cnt = 0;
  for (unsigned big = __ballot_sync(kFull, len >= kTcLong); big; big &= big - 1) {
    const int j = __ffs(big) - 1;
    const int a = __shfl_sync(kFull, start, j), n = __shfl_sync(kFull, len, j);
    for (int t = lane; t < n; t += 128) {
      int x[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        x[q] = t + 32 * q < n ? __ldg(Ui + a + t + 32 * q) : -1;
        if (kMulti && t + 32 * q < n) x[q] = member(x[q]);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) cnt += x[q] >= 0 && has(x[q]) ? 1u : 0u;
    }
  }
  const int d = len < kTcLong ? len : 0;
  const int incl = warp_incl_scan(d), excl = incl - d;
  const int total = __shfl_sync(kFull, incl, 31);
  for (int e0 = 0; e0 < total; e0 += 64) {
    int x[2];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int e = e0 + 32 * q + lane;
      const int owner = warp_owner(excl, e);
      const int at = __shfl_sync(kFull, start - excl, owner) + e;
      x[q] = e < total ? __ldg(Ui + at) : -1;
      if (kMulti && e < total) x[q] = member(x[q]);
    }
#pragma unroll
    for (int q = 0; q < 2; ++q) cnt += x[q] >= 0 && has(x[q]) ? 1u : 0u;
  }
  return cnt;
}

// The column that this lane's entry number c of end s reads, (0, 0) when the
// entry belongs to its other end: row entries own columns up to d, column
// entries only shorter ones, so that equal lengths belong to one end.  (With
// repeats: column entries own all columns, row entries none.)
template <bool kMulti>
__device__ __forceinline__ int2 tc_entry(int c, int nc, int la, int ld, int us, int d,
                                         const int *__restrict__ Li, const int *__restrict__ Ui,
                                         const int2 *__restrict__ col) {
  if (c >= nc || (kMulti && c < ld)) return make_int2(0, 0);
  if (kMulti) return __ldg(col + member(__ldg(Ui + us + (c - ld))));
  const int p = c < ld ? __ldg(Li + la + c) : __ldg(Ui + us + (c - ld));
  const int2 x = __ldg(col + p);
  return x.y <= (c < ld ? d : d - 1) ? x : make_int2(0, 0);
}

// A tiny end per eight lanes: its column's members one per lane, an entry per
// lane, and each member of the entry's column compared with the end's by
// eight shuffles.
template <bool kMulti>
__device__ __forceinline__ unsigned tc_tiny_ends(const int *list, const TcBins *bins,
                                                const int *__restrict__ Lp,
                                                const int *__restrict__ Li,
                                                const int2 *__restrict__ col,
                                                const int *__restrict__ Ui) {
  const int lane = lane_id(), sub = lane >> 3, l = lane & 7;
  const unsigned gwarp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned nwarps = (gridDim.x * blockDim.x) >> 5;
  const unsigned n = bins->n[0];
  unsigned cnt = 0;
  for (unsigned r = gwarp * 4; r < n; r += nwarps * 4) {
    int la = 0, ld = 0, us = 0, d = 0, mine = -1;
    if (r + sub < n) {
      const int s = __ldg(list + r + sub);
      la = __ldg(Lp + s);
      ld = __ldg(Lp + s + 1) - la;
      const int2 c = __ldg(col + s);
      us = c.x;
      d = c.y;
      if (l < d) mine = __ldg(Ui + us + l);
      if (kMulti) mine = max(mine, -1);  // the set has one of each
    }
    const int nc = ld + d;
    const int most = (int)__reduce_max_sync(kFull, (unsigned)nc);
    const int dmax = (int)__reduce_max_sync(kFull, (unsigned)d);
    for (int c0 = 0; c0 < most; c0 += 8) {
      const int2 x = tc_entry<kMulti>(c0 + l, nc, la, ld, us, d, Li, Ui, col);
      const int longest = (int)__reduce_max_sync(kFull, (unsigned)x.y);
      for (int t = 0; t < longest; t += 4) {
        int j[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          j[q] = t + q < x.y ? __ldg(Ui + x.x + t + q) : -2;
          if (kMulti && t + q < x.y) j[q] = member(j[q]);
        }
        for (int e = 0; e < dmax; ++e) {
          const int other = __shfl_sync(kFull, mine, e, 8);
#pragma unroll
          for (int q = 0; q < 4; ++q) cnt += j[q] == other ? 1u : 0u;
        }
      }
    }
  }
  return cnt;
}

// A warp end per warp, its set in the warp's part of the block's table.
static_assert(kTcWarps << kTcWarpTableBits == 1 << kTcTableBits, "the warps share the table");

template <bool kMulti>
__device__ __forceinline__ unsigned long long tc_warp_ends(const int *list_end,
                                                           const TcBins *bins, int *s_keys,
                                                           const int *__restrict__ Lp,
                                                           const int *__restrict__ Li,
                                                           const int2 *__restrict__ col,
                                                           const int *__restrict__ Ui) {
  const int w = warp_in_block(), lane = lane_id();
  int *keys = s_keys + (w << kTcWarpTableBits);
  unsigned long long cnt = 0;
  const unsigned n = bins->n[1];
  for (unsigned r = blockIdx.x * kTcWarps + w; r < n; r += gridDim.x * kTcWarps) {
    const int s = list_end[-(int)r];
    const int la = __ldg(Lp + s), ld = __ldg(Lp + s + 1) - la;
    const int2 c = __ldg(col + s);
    int bits = 5;
    while ((1 << bits) < 2 * c.y) ++bits;
    for (int t = lane; t < (1 << bits); t += 32) keys[t] = kNone;
    __syncwarp();
    for (int t = lane; t < c.y; t += 32) {
      const int j = __ldg(Ui + c.x + t);
      if (!kMulti || j >= 0) set_insert(keys, bits, j);
    }
    __syncwarp();
    const int nc = ld + c.y;
    for (int c0 = 0; c0 < nc; c0 += 32) {
      const int2 x = tc_entry<kMulti>(c0 + lane, nc, la, ld, c.x, c.y, Li, Ui, col);
      cnt += tc_probe<kMulti>(x.x, x.y, Ui, [&](int j) { return set_has(keys, bits, j); });
    }
    __syncwarp();
  }
  return cnt;
}

// All ends in one launch: the units first, handed out on demand, then every
// warp its share of the warp ends and of the tiny ends, which fill the time
// that the last units take.
template <bool kMulti>
__global__ void __launch_bounds__(kTcThreads, 8)
tc_count(const int2 *units, const int *lists, TcBins *bins, int m, const int *__restrict__ Lp,
         const int *__restrict__ Li, const int2 *__restrict__ col, const int *__restrict__ Ui) {
  __shared__ unsigned s_bits[kTcTop / 32];
  __shared__ int s_keys[1 << kTcTableBits];
  __shared__ unsigned s_unit;
  __shared__ int s_hashed;
  const int t0 = threadIdx.x, w = warp_in_block(), lane = lane_id();
  unsigned long long cnt = 0;
  if (!kMulti && bins->multi) return;  // left to the other kernel
  const unsigned nunits = bins->n[2];
  const int top = max(0, m - kTcTop);
  for (int t = t0; t < kTcTop / 32; t += kTcThreads) s_bits[t] = 0u;
  for (int t = t0; t < (1 << kTcTableBits); t += kTcThreads) s_keys[t] = kNone;
  if (t0 == 0) s_hashed = 0;
  for (;;) {
    if (t0 == 0) s_unit = atomicAdd(&bins->grab, 1u);
    __syncthreads();
    const unsigned u = s_unit;
    if (u >= nunits) break;
    const int2 un = units[u];
    const int s = un.x;
    const int la = __ldg(Lp + s), ld = __ldg(Lp + s + 1) - la;
    const int2 c = __ldg(col + s);
    const int us = c.x, d = c.y;
    const int c_beg = un.y * kTcUnit, nc = min(ld + d, c_beg + kTcUnit);
    for (int part = 0; part < d; part += kTcPart) {
      const int pe = min(d, part + kTcPart);
      for (int t = part + t0; t < pe; t += kTcThreads) {
        const int j = __ldg(Ui + us + t);
        if (kMulti && j < 0) continue;
        if (j >= top) {
          atomicOr(s_bits + ((j - top) >> 5), 1u << ((j - top) & 31));
        } else {
          set_insert(s_keys, kTcTableBits, j);
          s_hashed = 1;
        }
      }
      __syncthreads();
      const bool hashed = s_hashed != 0;
      for (int c0 = c_beg + w * 32; c0 < nc; c0 += kTcThreads) {
        const int2 x = tc_entry<kMulti>(c0 + lane, nc, la, ld, us, d, Li, Ui, col);
        cnt += tc_probe<kMulti>(x.x, x.y, Ui, [&](int j) -> bool {
          if (j >= top) return (s_bits[(j - top) >> 5] >> ((j - top) & 31)) & 1u;
          return hashed && set_has(s_keys, kTcTableBits, j);
        });
      }
      __syncthreads();
      for (int t = part + t0; t < pe; t += kTcThreads) {
        const int j = __ldg(Ui + us + t);
        if (j >= top) s_bits[(j - top) >> 5] = 0u;
      }
      if (hashed)
        for (int t = t0; t < (1 << kTcTableBits); t += kTcThreads) s_keys[t] = kNone;
      if (t0 == 0) s_hashed = 0;
      __syncthreads();
    }
  }
  cnt += tc_warp_ends<kMulti>(lists + (m - 1), bins, s_keys, Lp, Li, col, Ui);
  cnt += tc_tiny_ends<kMulti>(lists, bins, Lp, Li, col, Ui);
  cnt = warp_sum(cnt);
  if (lane == 0 && cnt) atomicAdd(&bins->count, cnt);
}

// ------------------------------------------------------------- prepare ---
__global__ void degree_keys(int m, const int *__restrict__ ptr, unsigned *keys, int *ids,
                            unsigned *maxdeg) {
  unsigned mx = 0;
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x) {
    unsigned d = (unsigned)(__ldg(ptr + v + 1) - __ldg(ptr + v));
    keys[v] = d;
    ids[v] = v;
    mx = max(mx, d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(kFull, mx, o));
  if (lane_id() == 0) atomicMax(maxdeg, mx);
}

__global__ void rank_to_perm(int m, const int *order, int *perm) {
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < m; r += gridDim.x * blockDim.x)
    perm[order[r]] = r;
}

constexpr int kSplit = 4;  // entries per thread in flight in the two passes over the edges

// Per vertex v of new id r: how many neighbours rank below r (the length
// of L's row r) and how many above (v's entries in L's columns), added to
// zeroed lcnt / ucnt by warp and row from one pass over the edges in tiles of
// equal size (a warp per vertex waited for the hubs' warps: R-MAT 18, 7.6 M
// edges, 221 us).  The same pass sums a
// 64-bit hash of every edge (v, u) and of its reverse (u, v) into hsum[0] and
// hsum[1] (wrapping): the edge multiset equals its transpose -- the graph is
// symmetric -- exactly when the multisets of hashed pairs agree, which the two
// sums confirm up to a 2^-64 chance.
__global__ void __launch_bounds__(kEdgeThreads)
split_counts(int m, const int *__restrict__ ptr, const int *__restrict__ ind,
             const int *__restrict__ perm, int *lcnt, int *ucnt, unsigned long long *hsum) {
  __shared__ __align__(16) int s_row[kEdgeTile];
  const int lane = lane_id();
  unsigned long long h_fwd = 0, h_rev = 0;
  for (unsigned tile = blockIdx.x;; tile += gridDim.x) {
    int k0;
    const int n = edge_tile(ptr, m, tile, &k0);
    if (n == 0) break;
    edge_tile_rows(ptr, m, k0, n, s_row);
    for (int t0 = (int)threadIdx.x; t0 - lane < n; t0 += kSplit * kEdgeThreads) {
      int v[kSplit], u[kSplit], r[kSplit], pu[kSplit];
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        const int t = t0 + q * kEdgeThreads;
        v[q] = t < n ? s_row[t] : -1;
        u[q] = t < n ? __ldg(ind + k0 + t) : 0;
      }
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        r[q] = v[q] >= 0 ? __ldg(perm + v[q]) : 0;
        pu[q] = v[q] >= 0 ? __ldg(perm + u[q]) : 0;
      }
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        if (v[q] >= 0) {
          h_fwd += apspie_gen::mix64(((unsigned long long)(unsigned)v[q] << 32) | (unsigned)u[q]);
          h_rev += apspie_gen::mix64(((unsigned long long)(unsigned)u[q] << 32) | (unsigned)v[q]);
        }
        const unsigned below = __ballot_sync(kFull, pu[q] < r[q]);
        const unsigned above = __ballot_sync(kFull, pu[q] > r[q]);
        int leader;
        const unsigned peers = row_peers(v[q], &leader);
        if (lane == leader && v[q] >= 0) {
          const int lo = __popc(below & peers), hi = __popc(above & peers);
          if (lo) atomicAdd(lcnt + r[q], lo);
          if (hi) atomicAdd(ucnt + r[q], hi);
        }
      }
    }
    __syncthreads();
  }
  h_fwd = warp_sum(h_fwd);
  h_rev = warp_sum(h_rev);
  if (lane == 0 && (h_fwd | h_rev)) {
    atomicAdd(hsum, h_fwd);
    atomicAdd(hsum + 1, h_rev);
  }
}

// L's entries as (row new(u), column r) pairs, grouped by column r in
// ascending order (segment uoff[r], which counts up as the pairs are
// written): a stable sort by row then leaves each row's columns ascending.
// Within a column the pairs may come in any order, since their rows differ
// (equal pairs are the same pair), so a warp reserves its places in a
// column with one add.
__global__ void __launch_bounds__(kEdgeThreads)
upper_pairs(int m, const int *__restrict__ ptr, const int *__restrict__ ind,
            const int *__restrict__ perm, int *uoff, unsigned *rows, int *cols) {
  __shared__ __align__(16) int s_row[kEdgeTile];
  const int lane = lane_id();
  for (unsigned tile = blockIdx.x;; tile += gridDim.x) {
    int k0;
    const int n = edge_tile(ptr, m, tile, &k0);
    if (n == 0) break;
    edge_tile_rows(ptr, m, k0, n, s_row);
    for (int t0 = (int)threadIdx.x; t0 - lane < n; t0 += kSplit * kEdgeThreads) {
      int v[kSplit], u[kSplit], r[kSplit], pu[kSplit], base[kSplit], leader[kSplit];
      unsigned mine[kSplit];
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        const int t = t0 + q * kEdgeThreads;
        v[q] = t < n ? s_row[t] : -1;
        u[q] = t < n ? __ldg(ind + k0 + t) : 0;
      }
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        r[q] = v[q] >= 0 ? __ldg(perm + v[q]) : 0;
        pu[q] = v[q] >= 0 ? __ldg(perm + u[q]) : 0;
      }
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        mine[q] = row_peers(v[q], &leader[q]) & __ballot_sync(kFull, pu[q] > r[q]);
        base[q] = add_if(lane == leader[q] && mine[q] != 0u, uoff + r[q], __popc(mine[q]), 0);
      }
#pragma unroll
      for (int q = 0; q < kSplit; ++q) {
        base[q] = __shfl_sync(kFull, base[q], leader[q]);
        if (pu[q] > r[q]) {
          const int at = base[q] + __popc(mine[q] & ((1u << lane) - 1u));
          rows[at] = (unsigned)pu[q];
          cols[at] = r[q];
        }
      }
    }
    __syncthreads();
  }
}

int tgrid(apspie_context *ctx, long long n, int threads, int per_sm = 16) {
  long long g = (n + threads - 1) / threads;
  return (int)std::max(1ll, std::min(g, (long long)ctx->num_sms * per_sm));
}

}  // namespace
}  // namespace apspie

using namespace apspie;

extern "C" {

int apspie_tc_prepare(apspie_ctx ctx, int64_t nnz, int m, const int *d_ptr, const int *d_ind,
                      int *d_perm, int *d_Lptr, int *d_Lind, int64_t *h_lnnz) {
  APSPIE_CHECK_CTX(ctx);
  if (m <= 0 || nnz < 0 || nnz >= (int64_t)INT32_MAX || !d_ptr || !d_perm || !d_Lptr ||
      (nnz > 0 && (!d_ind || !d_Lind)) || !h_lnnz)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_tc_prepare: bad arguments");
  cudaStream_t st = ctx->stream;
  const int cbits = bits_for(m);
  if (2 * cbits > 62) return set_error(ctx, APSPIE_ERR_OVERFLOW, "apspie_tc_prepare: m too large");
  // 1. order by (degree, id): stable radix sort of degree keys over ids
  auto *dk = (unsigned *)workspace(ctx, kSlotSortKeysA, sizeof(unsigned) * (size_t)m);
  auto *dk2 = (unsigned *)workspace(ctx, kSlotSortKeysB, sizeof(unsigned) * (size_t)m);
  auto *ids = (int *)workspace(ctx, kSlotSortValsA, sizeof(int) * (size_t)m);
  auto *ids2 = (int *)workspace(ctx, kSlotSortValsB, sizeof(int) * (size_t)m);
  auto *small = (unsigned *)workspace(ctx, kSlotSmall, 64);
  if (!dk || !dk2 || !ids || !ids2 || !small) return APSPIE_ERR_OOM;
  cudaMemsetAsync(small, 0, 64, st);
  degree_keys<<<tgrid(ctx, m, 256), 256, 0, st>>>(m, d_ptr, dk, ids, small);
  int rc = check_launch(ctx, "degree_keys");
  if (rc) return rc;
  unsigned *hs = (unsigned *)pinned(ctx, 64);
  if (!hs) return APSPIE_ERR_OOM;
  cudaMemcpyAsync(hs, small, 8, cudaMemcpyDeviceToHost, st);
  rc = check_cuda(ctx, cudaStreamSynchronize(st), "tc_prepare maxdeg");
  if (rc) return rc;
  const int dbits = std::max(1, bits_for((long long)hs[0] + 1));
  bool in_b = false;
  rc = device_radix_sort<unsigned, int>(ctx, dk, ids, dk2, ids2, m, dbits, &in_b);
  if (rc) return rc;
  // before the sorted ids index anything (one tile never waits)
  rc = m > kSortTile ? radix_sort_check(ctx) : APSPIE_OK;
  if (rc) return rc;
  rank_to_perm<<<tgrid(ctx, m, 256), 256, 0, st>>>(m, in_b ? ids2 : ids, d_perm);
  // 2. row lengths of L (indexed by new id) and each vertex's count above it
  auto *lcnt = d_Lptr;
  auto *uoff = (int *)workspace(ctx, kSlotMisc0, sizeof(int) * ((size_t)m + 1));
  if (!uoff) return APSPIE_ERR_OOM;
  cudaMemsetAsync(lcnt, 0, sizeof(int) * ((size_t)m + 1), st);
  cudaMemsetAsync(uoff, 0, sizeof(int) * ((size_t)m + 1), st);
  // small[0]: the largest degree; small + 8 bytes .. + 24: the two edge hashes
  auto *hsum = reinterpret_cast<unsigned long long *>(small) + 1;
  if (nnz > 0) {
    split_counts<<<edge_tiles(nnz), kEdgeThreads, 0, st>>>(m, d_ptr, d_ind, d_perm, lcnt, uoff,
                                                           hsum);
    rc = check_launch(ctx, "split_counts");
    if (rc) return rc;
  }
  // exclusive scans of the m + 1 entries (entry m is 0): offsets + totals
  rc = device_exclusive_scan<int>(ctx, lcnt, d_Lptr, (long long)m + 1, nullptr);
  if (rc) return rc;
  rc = device_exclusive_scan<int>(ctx, uoff, uoff, (long long)m + 1, nullptr);
  if (rc) return rc;
  rc = check_cuda(ctx, cudaMemcpyAsync(hs, d_Lptr + m, 4, cudaMemcpyDeviceToHost, st),
                  "tc_prepare counts");
  if (rc) return rc;
  rc = check_cuda(ctx, cudaMemcpyAsync(hs + 1, uoff + m, 4, cudaMemcpyDeviceToHost, st),
                  "tc_prepare counts");
  if (rc) return rc;
  rc = check_cuda(ctx, cudaMemcpyAsync(hs + 2, hsum, 16, cudaMemcpyDeviceToHost, st),
                  "tc_prepare counts");
  if (rc) return rc;
  rc = check_cuda(ctx, cudaStreamSynchronize(st), "tc_prepare counts");
  if (rc) return rc;
  const long long lnnz = hs[0];
  unsigned long long hh[2];
  std::memcpy(hh, hs + 2, sizeof(hh));
  // L is read from both ends of every edge: the graph must be symmetric
  if (hh[0] != hh[1] || hs[1] != hs[0] || lnnz > nnz / 2)
    return set_error(ctx, APSPIE_ERR_INVALID,
                     "apspie_tc_prepare: the graph is not symmetric (%u entries below, %u above, "
                     "edge hashes %s)",
                     hs[0], hs[1], hh[0] == hh[1] ? "equal" : "differ");
  if (lnnz > 0) {
    // 3. (row, column) pairs grouped by ascending column, stable-sorted by row:
    //    the columns come out in d_Lind (or in the other buffer, then copied)
    auto *ka = (unsigned *)workspace(ctx, kSlotMisc1, sizeof(unsigned) * (size_t)lnnz);
    auto *kb = (unsigned *)workspace(ctx, kSlotMisc2, sizeof(unsigned) * (size_t)lnnz);
    auto *va = (int *)workspace(ctx, kSlotMisc3, sizeof(int) * (size_t)lnnz);
    if (!ka || !kb || !va) return APSPIE_ERR_OOM;
    upper_pairs<<<edge_tiles(nnz), kEdgeThreads, 0, st>>>(m, d_ptr, d_ind, d_perm, uoff, ka, va);
    rc = check_launch(ctx, "upper_pairs");
    if (rc) return rc;
    in_b = false;
    rc = device_radix_sort<unsigned, int>(ctx, ka, va, kb, d_Lind, lnnz, cbits, &in_b);
    if (rc) return rc;
    rc = lnnz > kSortTile ? radix_sort_check(ctx) : APSPIE_OK;
    if (rc) return rc;
    if (!in_b) {
      rc = check_cuda(ctx, cudaMemcpyAsync(d_Lind, va, sizeof(int) * (size_t)lnnz,
                                           cudaMemcpyDeviceToDevice, st),
                      "tc_prepare copy");
      if (rc) return rc;
    }
  }
  *h_lnnz = lnnz;
  return APSPIE_OK;
}

int apspie_tc(apspie_ctx ctx, int m, int64_t lnnz, const int *d_Lptr, const int *d_Lind,
              int64_t *h_count) {
  APSPIE_CHECK_CTX(ctx);
  if (m <= 0 || lnnz < 0 || !d_Lptr || (lnnz > 0 && !d_Lind) || !h_count)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_tc: bad arguments");
  *h_count = 0;
  if (lnnz == 0) return APSPIE_OK;
  cudaStream_t st = ctx->stream;
  if (lnnz >= (int64_t)INT32_MAX) {
    // more than int32 offsets can name (the size of a buffer, say): the
    // offsets tell the entries
    auto *h = (int *)pinned(ctx, 2 * sizeof(int));
    if (!h) return APSPIE_ERR_OOM;
    cudaMemcpyAsync(h, d_Lptr, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaMemcpyAsync(h + 1, d_Lptr + m, sizeof(int), cudaMemcpyDeviceToHost, st);
    const int rc = check_cuda(ctx, cudaStreamSynchronize(st), "apspie_tc");
    if (rc) return rc;
    lnnz = h[1] - h[0];
    if (lnnz <= 0) return APSPIE_OK;
  }
  auto *lists = (int *)workspace(ctx, kSlotMisc0, sizeof(int) * (size_t)m);
  // an end with units has more than kTcWarpSet entries, or a column that is
  // longer: at most 2 lnnz / kTcWarpSet such ends, 2 lnnz / kTcUnit full units
  auto *units = (int2 *)workspace(
      ctx, kSlotMisc1,
      sizeof(int2) * (2 * (size_t)lnnz / kTcUnit + 2 * (size_t)lnnz / kTcWarpSet + 2));
  static_assert(sizeof(TcBins) % sizeof(int) == 0, "the counters precede the column offsets");
  auto *bins = (TcBins *)workspace(ctx, kSlotMisc2, sizeof(TcBins) + sizeof(int) * ((size_t)m + 1));
  auto *Up = bins ? (int *)(bins + 1) : nullptr;
  auto *rank = (int *)workspace(ctx, kSlotSortKeysB, sizeof(int) * (size_t)lnnz);
  auto *col = (int2 *)workspace(ctx, kSlotSortValsA, sizeof(int2) * (size_t)m);
  auto *Ui = (int *)workspace(ctx, kSlotSortKeysA, sizeof(int) * (size_t)lnnz);
  if (!lists || !units || !Up || !rank || !col || !Ui || !bins) return APSPIE_ERR_OOM;
  cudaMemsetAsync(bins, 0, sizeof(TcBins) + sizeof(int) * ((size_t)m + 1), st);
  tc_col_ranks<<<tgrid(ctx, (lnnz + kTcRankItems - 1) / kTcRankItems, kTcThreads), kTcThreads, 0,
                 st>>>(m, (int)lnnz, d_Lptr, d_Lind, Up, rank);
  int rc = check_launch(ctx, "tc_col_ranks");
  if (rc) return rc;
  rc = device_exclusive_scan<int>(ctx, Up, Up, (long long)m + 1, nullptr);
  if (rc) return rc;
  tc_bin<<<tgrid(ctx, m, 256), 256, 0, st>>>(m, d_Lptr, Up, col, lists, units, bins);
  tc_scatter<<<edge_tiles(lnnz), kEdgeThreads, 0, st>>>(m, (int)lnnz, d_Lptr, d_Lind, Up, rank, Ui,
                                                        bins);
  tc_count<false><<<ctx->num_sms * 8, kTcThreads, 0, st>>>(units, lists, bins, m, d_Lptr, d_Lind,
                                                           col, Ui);
  rc = check_launch(ctx, "apspie_tc", 3);
  if (rc) return rc;
  auto *h = (TcBins *)pinned(ctx, sizeof(TcBins));
  if (!h) return APSPIE_ERR_OOM;
  for (int pass = 0; pass < 2; ++pass) {
    cudaMemcpyAsync(h, bins, sizeof(TcBins), cudaMemcpyDeviceToHost, st);
    rc = check_cuda(ctx, cudaStreamSynchronize(st), "apspie_tc");
    if (rc) return rc;
    if (!h->multi || pass == 1) break;
    tc_count<true><<<ctx->num_sms * 8, kTcThreads, 0, st>>>(units, lists, bins, m, d_Lptr, d_Lind,
                                                            col, Ui);
    rc = check_launch(ctx, "apspie_tc");
    if (rc) return rc;
  }
  *h_count = (int64_t)h->count;
  return APSPIE_OK;
}

}  // extern "C"
