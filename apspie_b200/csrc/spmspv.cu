// spmspv.cu -- generic semiring SpMSpV: sparse x times A (column lists),
// sparse sorted y, plus the dense-in/dense-out form.
//
// Replaces both mXv<T>() overloads (src/mXv.cuh:111-247 dense, :250-389
// sparse) and the min-plus spmspvSssp (src/spmspvSssp.cuh:92-291).  The
// reference gathers column segments with four IntervalGathers and an
// IntervalExpand, multiplies, cub-radix-sorts all (row, value) pairs on 32
// key bits and reduces by key.  Here:
// the frontier's columns are laid end to end by a scan of their lengths and
// walked in tiles of equal size (edges.cuh), so a hub column costs no more
// than its entries.
//   * bitmap path: products are combined with atomics into a dense
//     accumulator, and the touched rows' bitmap, then y, are compacted from it
//     in index order -- no sort, and nothing that the host has to know before
//     the end, so the call waits for the device once;
//   * sort path: the tiles write (row, x (x) a) pairs, the pairs are
//     radix-sorted on only ceil(log2 m) key bits, and a segmented reduce emits
//     sorted y.
// The sort path is for frontiers that are sparse against a long y: its cost
// grows with the expanded size E, the bitmap path's with m (clearing and
// reading the accumulator, about 7 us per 2^20 rows), and the sort's launches
// alone outlast that up to kBitmapRows rows.  Beyond, E * factor is compared
// with m (threshold settable, picked by the autotuner; 0 always sorts).  Both
// give y sorted by row with one entry per touched row; PLUS_TIMES accumulates
// in double and rounds once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstddef>

#include "common.cuh"
#include "context.h"
#include "edges.cuh"
#include "primitives.cuh"

namespace apspie {
namespace {

constexpr int kPlusTimes = 0, kMinPlus = 1, kMaxTimes = 2, kOrAnd = 3;

struct SpmspvSmall {  // device-side scalars of one call
  long long total;    // expanded size E
  int ynnz;           // nnz(y)
  unsigned cnt;       // frontier size of the dense form
};

// Path rule.  PLUS_TIMES: the bitmap path when E * factor > m, else the sort
// path, whose sums run in the frontier's order and have the same bits in every
// run (the bitmap path's double atomics add in any order).  The other semirings'
// results do not depend on the order: up to kBitmapRows rows of y they take the
// bitmap path at any density (8 entries a column, 2^22 rows: 63 us against 69
// sorted at 32 products, 75 against 132 at 65,536; 2^20 rows: 51 against 67).
//
// Up to kBitmapRows rows the bitmap path starts before the host knows E (the
// expansion checks the rule for PLUS_TIMES; frontiers that turn out sparse are
// sorted after the read-back): for PLUS_TIMES when the frontier has at least
// 1 / kDenseGuess of the entries that the rule asks for at the mean column
// length.  A frontier of longer columns that was guessed sparse costs a wait,
// 10 us; one guessed dense that is sparse costs 10 us at 2^20 rows and 25 at
// 2^22 (launches and the cleared accumulator).
constexpr int kBitmapRows = 1 << 22;
constexpr double kDenseGuess = 1.25;

bool spmspv_dense(long long E, double factor, int m) { return (double)E * factor > (double)m; }

// The least E that the rule calls dense, an integer for the kernels to compare
// with (the rule's doubles cost the expansion 1.5 us).
long long dense_from(double factor, int m) {
  long long E = (long long)std::min((double)m / factor, 4e18);
  while (E > 0 && spmspv_dense(E - 1, factor, m)) --E;
  while (E < (long long)INT_MAX && !spmspv_dense(E, factor, m)) ++E;
  return E;
}

__device__ __forceinline__ float sr_term(int sr, float a, float x) {
  switch (sr) {
    case kMinPlus: return __fadd_rn(a, x);
    case kOrAnd: return 1.0f;
    default: return __fmul_rn(a, x);  // PLUS_TIMES, MAX_TIMES
  }
}

// ---- the accumulator of the bitmap path ----
// One accumulator word per row, which also tells whether the row was touched:
// a bitmap beside it costs a second random L2 access per product (the expansion
// of 5.6 M products, 1 M rows: 73 us with one, 44 us without).
//   PLUS_TIMES  a double that starts at -0.0, which no sum reaches: a term of
//               -0.0 is added as +0.0, and x + -x is +0.0
//   MIN_PLUS,   32 bits that order as the float does, so that the atomics are
//   MAX_TIMES   native; they start beyond every float's word, and a NaN's word
//               loses to every number's (fminf and fmaxf leave NaN out)
//   OR_AND      0, then 1
constexpr unsigned long long kNoSum = 0x8000000000000000ull;

__device__ __forceinline__ unsigned ordered_bits(float f) {
  const unsigned b = __float_as_uint(f);
  return (b >> 31) ? ~b : b | 0x80000000u;
}
__device__ __forceinline__ float ordered_float(unsigned u) {
  return __uint_as_float((u >> 31) ? u & 0x7fffffffu : ~u);
}
__device__ __forceinline__ unsigned untouched_word(int sr) { return sr == kMinPlus ? ~0u : 0u; }
__device__ __forceinline__ unsigned nan_word(int sr) { return sr == kMinPlus ? ~1u : 1u; }

__device__ __forceinline__ void clear_acc(int sr, int m, unsigned long long *acc) {
  const unsigned w = untouched_word(sr);
  const unsigned long long v = sr == kPlusTimes ? kNoSum : (unsigned long long)w << 32 | w;
  const unsigned n = sr == kPlusTimes ? (unsigned)m : ((unsigned)m + 1u) / 2u;
  const unsigned stride = gridDim.x * blockDim.x;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) acc[i] = v;
}

__global__ void acc_init(int sr, int m, unsigned long long *acc) { clear_acc(sr, m, acc); }

// ---- the frontier's columns ----
// Lengths, and (first entry, x value) side by side for the tiles.  With acc,
// the accumulator of the bitmap path is cleared in the same launch, and the
// call's scalars are read back in one copy: a launch and a copy less took 16,384
// columns of a 1 M-row graph from 119 to 112 us.
__global__ void frontier_columns(int xnnz, const int *__restrict__ xind,
                                 const float *__restrict__ xval, const int *__restrict__ ptr,
                                 long long *deg, int2 *col, int sr, int m,
                                 unsigned long long *acc) {
  for (int j = blockIdx.x * blockDim.x + threadIdx.x; j < xnnz; j += gridDim.x * blockDim.x) {
    const int c = xind[j];
    const int s = __ldg(ptr + c);
    deg[j] = (long long)(__ldg(ptr + c + 1) - s);
    col[j] = make_int2(s, __float_as_int(xval ? xval[j] : 1.0f));
  }
  if (acc) clear_acc(sr, m, acc);
}

// Calls f(e[], row[], term[], on[]) for the entries e of the frontier's columns
// laid end to end (offs: their exclusive scan, offs[xnnz] = *total), each
// thread's kEdgeItems of a tile in flight together.  Blocks stride the tiles.
// Nothing is done when the total does not fit an int (the caller reports it) or
// is below `least`.
template <typename F>
__device__ __forceinline__ void for_each_entry(int sr, int xnnz, const long long *__restrict__ offs,
                                               const long long *total, long long least,
                                               const int2 *__restrict__ col,
                                               const int *__restrict__ ind,
                                               const float *__restrict__ val, F f) {
  __shared__ __align__(16) int s_row[kEdgeTile];
  const long long E = __ldcg(total);
  if (E >= (long long)INT_MAX || E < least) return;
  const unsigned tiles = (unsigned)((E + kEdgeTile - 1) / kEdgeTile);
  for (unsigned tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int k0 = (int)(tile * kEdgeTile);
    const int n = (int)min((long long)kEdgeTile, E - k0);
    edge_tile_rows(offs, xnnz, k0, n, s_row);
    int e[kEdgeItems], row[kEdgeItems];
    float term[kEdgeItems], x[kEdgeItems];
    bool on[kEdgeItems];
    int k[kEdgeItems];
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q) {
      const int t = (int)threadIdx.x + q * kEdgeThreads;
      on[q] = t < n;
      e[q] = k0 + t;
      const int j = on[q] ? s_row[t] : 0;
      const int2 c = __ldg(col + j);
      k[q] = c.x + (int)(e[q] - __ldg(offs + j));
      x[q] = __int_as_float(c.y);
    }
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q) {
      row[q] = on[q] ? __ldg(ind + k[q]) : 0;
      term[q] = on[q] && val ? __ldg(val + k[q]) : 1.0f;
    }
#pragma unroll
    for (int q = 0; q < kEdgeItems; ++q) term[q] = sr_term(sr, term[q], x[q]);
    f(e, row, term, on);
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kEdgeThreads)
expand_pairs(int sr, int xnnz, const long long *__restrict__ offs, const long long *total,
             const int2 *__restrict__ col, const int *__restrict__ ind,
             const float *__restrict__ val, int *keys, float *vals) {
  for_each_entry(sr, xnnz, offs, total, 0, col, ind, val,
                 [&](const int (&e)[kEdgeItems], const int (&row)[kEdgeItems],
                     const float (&term)[kEdgeItems], const bool (&on)[kEdgeItems]) {
#pragma unroll
                   for (int q = 0; q < kEdgeItems; ++q)
                     if (on[q]) {
                       keys[e[q]] = row[q];
                       vals[e[q]] = term[q];
                     }
                 });
}

// ---- segmented reduce of sorted pairs ----
__global__ void head_flags(const int *keys, long long n, unsigned *flags) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1u : 0u;
}

__global__ void reduce_segments(int sr, const int *keys, const float *vals, long long n,
                                const unsigned *segid, int *yind, float *yval, int ycap) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    int k = keys[i];
    if (i > 0 && keys[i - 1] == k) continue;
    double accd = 0.0;
    float accf = vals[i];
    long long j = i;
    for (; j < n && keys[j] == k; ++j) {
      float t = vals[j];
      switch (sr) {
        case kPlusTimes: accd += (double)t; break;
        case kMinPlus: accf = fminf(accf, t); break;
        case kMaxTimes: accf = fmaxf(accf, t); break;
        default: accf = 1.0f; break;
      }
    }
    // at most m distinct rows from a sorted run; more only from a sort that
    // gave up (reported by the caller), whose extra segments are dropped
    unsigned s = segid[i];
    if (s >= (unsigned)ycap) continue;
    yind[s] = k;
    yval[s] = sr == kPlusTimes ? (float)accd : accf;
  }
}

// ---- bitmap path ----
__global__ void __launch_bounds__(kEdgeThreads)
expand_accumulate(int sr, long long least, int xnnz, const long long *__restrict__ offs,
                  const long long *total, const int2 *__restrict__ col,
                  const int *__restrict__ ind, const float *__restrict__ val, void *acc) {
  for_each_entry(sr, xnnz, offs, total, least, col, ind, val,
                 [&](const int (&)[kEdgeItems], const int (&row)[kEdgeItems],
                     const float (&term)[kEdgeItems], const bool (&on)[kEdgeItems]) {
#pragma unroll
                   for (int q = 0; q < kEdgeItems; ++q) {
                     if (!on[q]) continue;
                     if (sr == kPlusTimes) {
                       atomicAdd((double *)acc + row[q], (double)__fadd_rn(term[q], 0.0f));
                       continue;
                     }
                     unsigned *a = (unsigned *)acc + row[q];
                     const unsigned o = term[q] == term[q] ? ordered_bits(term[q]) : nan_word(sr);
                     if (sr == kMinPlus) atomicMin(a, o);
                     else if (sr == kMaxTimes) atomicMax(a, o);
                     else __stcg(a, 1u);
                   }
                 });
}

// y from the accumulator, in two launches: the touched rows become a bitmap
// and every block's are counted (sums), then each block adds up the counts
// before its own and writes its rows in order, a warp per 32 of them; the last
// one leaves nnz(y).
constexpr int kEmitThreads = 256;
constexpr int kEmitBlocks = 2048;  // at most
constexpr int kEmitWords = 64;     // bitmap words per block, at least

__global__ void __launch_bounds__(kEmitThreads)
touched_rows(int sr, int m, const void *__restrict__ acc, int words, int per_block,
             unsigned *bits, unsigned *sums) {
  __shared__ unsigned sw[33];
  const int w0 = blockIdx.x * per_block, w1 = min(words, w0 + per_block);
  const unsigned none = untouched_word(sr);
  unsigned c = 0;
#pragma unroll 4
  for (int w = w0 + warp_in_block(); w < w1; w += kEmitThreads / 32) {
    const unsigned r = (unsigned)w * 32u + lane_id();
    bool on = r < (unsigned)m;
    if (on)
      on = sr == kPlusTimes ? __ldcg((const unsigned long long *)acc + r) != kNoSum
                            : __ldcg((const unsigned *)acc + r) != none;
    const unsigned b = __ballot_sync(kFull, on);
    if (lane_id() == 0) {
      bits[w] = b;
      c += __popc(b);
    }
  }
  unsigned tot;
  block_excl_scan(c, sw, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// MIN_PLUS and MAX_TIMES: a row of NaN terms only is NaN for a frontier below
// the threshold (E * factor <= m), as the sorted reduction has it, else the
// infinity that the reduction starts from.
__global__ void __launch_bounds__(kEmitThreads)
touched_emit(int sr, int m, const unsigned *__restrict__ bits, int words, int per_block,
             const unsigned *__restrict__ sums, const void *__restrict__ acc,
             const long long *total, double factor, int *yind, float *yval, int *ynnz) {
  __shared__ unsigned sw[33];
  __shared__ unsigned s_bits[kEmitThreads], s_off[kEmitThreads];
  unsigned before = 0, tot;
  for (unsigned i = threadIdx.x; i < blockIdx.x; i += kEmitThreads) before += sums[i];
  block_excl_scan(before, sw, &tot);
  before = tot;
  const int w0 = blockIdx.x * per_block, w1 = min(words, w0 + per_block);
  for (int base = w0; base < w1; base += kEmitThreads) {
    const int n = min(kEmitThreads, w1 - base);
    const unsigned mine = (int)threadIdx.x < n ? bits[base + threadIdx.x] : 0u;
    s_bits[threadIdx.x] = mine;
    s_off[threadIdx.x] = before + block_excl_scan((unsigned)__popc(mine), sw, &tot);
    before += tot;
    __syncthreads();
#pragma unroll 4
    for (int w = warp_in_block(); w < n; w += kEmitThreads / 32) {
      const unsigned b = s_bits[w];
      if (!(b >> lane_id() & 1u)) continue;
      const unsigned r = (unsigned)(base + w) * 32u + lane_id();
      const unsigned o = s_off[w] + __popc(b & ((1u << lane_id()) - 1u));
      float v = 1.0f;
      if (sr == kPlusTimes) v = (float)__ldcg((const double *)acc + r);
      else if (sr != kOrAnd) {
        const unsigned u = __ldcg((const unsigned *)acc + r);
        v = ordered_float(u);
        if (u == nan_word(sr) && (double)__ldcg(total) * factor > (double)m)
          v = sr == kMinPlus ? INFINITY : -INFINITY;
      }
      yind[o] = (int)r;
      yval[o] = v;
    }
    __syncthreads();
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *ynnz = (int)before;
}

// ---- dense in / dense out helpers (mXv dense form) ----
__global__ void dense_frontier_flags(int sr, int m, const float *x, unsigned *flags) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) {
    float v = x[i];
    bool in;
    if (sr == kMinPlus)
      in = v > -1.0f && v < 1e38f;  // finite distance (src/spmspvSssp.cuh:31-36)
    else if (sr == kPlusTimes)
      in = v > 0.5f;  // bitify (src/mXv.cuh:50-55)
    else
      in = v != 0.0f;
    flags[i] = in ? 1u : 0u;
  }
}

__global__ void dense_compact(int m, const float *x, const unsigned *flags, const unsigned *offs,
                              int *xind, float *xval) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x)
    if (flags[i]) {
      xind[offs[i]] = i;
      xval[offs[i]] = x[i];
    }
}

__global__ void dense_fill(int m, float v, float *y) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m; i += gridDim.x * blockDim.x) y[i] = v;
}

// (a sort that gave up, which the caller reports, may leave any length and any
// row: both are bounds-checked)
__global__ void dense_scatter(const int *nnz, int m, const int *yind, const float *yval, float *y) {
  const int n = min(*nnz, m);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const int r = yind[i];
    if ((unsigned)r < (unsigned)m) y[r] = yval[i];
  }
}

int grid_for(apspie_context *ctx, long long n, int threads) {
  long long g = (n + threads - 1) / threads;
  return (int)std::max(1ll, std::min(g, (long long)ctx->num_sms * 16));
}

int expand_grid(apspie_context *ctx) {
  return ctx->num_sms * 6;  // resident blocks; they stride the tiles
}

// A call's scalars lie behind the radix sort's give-up word: one copy reads both.
struct SpmspvBack {
  int sort_err, pad[3];
  SpmspvSmall s;
};
static_assert(offsetof(SpmspvBack, s) == kSortErrWords * sizeof(int) &&
                  sizeof(SpmspvBack) <= kSortErrBytes, "read back in one copy");

SpmspvSmall *spmspv_scalars(apspie_context *ctx) {
  int *sort_err = radix_sort_err(ctx);
  return sort_err ? (SpmspvSmall *)(sort_err + kSortErrWords) : nullptr;
}

// Waits for a call and reads its scalars back.  A status when the sort path's
// look-back gave up (y is not sorted), or when the expanded size does not fit
// the int32 layout (the kernels did nothing).
int spmspv_read_back(apspie_context *ctx, const char *what, SpmspvSmall *out) {
  int *sort_err = radix_sort_err(ctx);
  auto *h = (SpmspvBack *)pinned(ctx, sizeof(SpmspvBack));
  if (!sort_err || !h) return APSPIE_ERR_OOM;
  int rc = check_cuda(ctx, cudaMemcpyAsync(h, sort_err, sizeof(SpmspvBack), cudaMemcpyDeviceToHost,
                                           ctx->stream), what);
  if (rc) return rc;
  rc = check_cuda(ctx, cudaStreamSynchronize(ctx->stream), what);
  if (rc) return rc;
  if (h->sort_err) {
    rc = check_cuda(ctx, cudaMemsetAsync(sort_err, 0, sizeof(int), ctx->stream), what);
    if (rc) return rc;
    return set_error(ctx, APSPIE_ERR_TIMEOUT, "%s: radix sort look-back gave up", what);
  }
  if (h->s.total >= (long long)INT32_MAX)
    return set_error(ctx, APSPIE_ERR_OVERFLOW, "%s: %lld expanded pairs", what, h->s.total);
  *out = h->s;
  return APSPIE_OK;
}

// The sort path from the scanned column lengths on.
int spmspv_sorted(apspie_context *ctx, int sr, int m, const int *ind, const float *val, int xnnz,
                  const long long *offs, const int2 *col, long long E, int *yind, float *yval,
                  SpmspvSmall *sm) {
  cudaStream_t st = ctx->stream;
  int *ka = (int *)workspace(ctx, kSlotSortKeysA, sizeof(int) * (size_t)E);
  int *kb = (int *)workspace(ctx, kSlotSortKeysB, sizeof(int) * (size_t)E);
  float *va = (float *)workspace(ctx, kSlotSortValsA, sizeof(float) * (size_t)E);
  float *vb = (float *)workspace(ctx, kSlotSortValsB, sizeof(float) * (size_t)E);
  unsigned *flags = (unsigned *)workspace(ctx, kSlotMisc3, sizeof(unsigned) * (size_t)E);
  if (!ka || !kb || !va || !vb || !flags) return APSPIE_ERR_OOM;
  expand_pairs<<<(unsigned)std::min<long long>(edge_tiles(E), expand_grid(ctx)), kEdgeThreads, 0,
                 st>>>(sr, xnnz, offs, &sm->total, col, ind, val, ka, va);
  int rc = check_launch(ctx, "expand_pairs");
  if (rc) return rc;
  bool in_b = false;
  rc = device_radix_sort<int, float>(ctx, ka, va, kb, vb, E, bits_for(m), &in_b);
  if (rc) return rc;
  int *ks = in_b ? kb : ka;
  float *vs = in_b ? vb : va;
  head_flags<<<grid_for(ctx, E, 256), 256, 0, st>>>(ks, E, flags);
  rc = check_launch(ctx, "head_flags");
  if (rc) return rc;
  rc = device_exclusive_scan<unsigned>(ctx, flags, flags, E, (unsigned *)&sm->ynnz);
  if (rc) return rc;
  reduce_segments<<<grid_for(ctx, E, 256), 256, 0, st>>>(sr, ks, vs, E, flags, yind, yval, m);
  return check_launch(ctx, "reduce_segments");
}

// Sparse SpMSpV.  On return y and sm->ynnz (device) are written and *out holds
// the call's scalars: the expanded size, and nnz(y) where the host had to read
// it (out->ynnz -1: it did not; want_ynnz asks for it).  A status when the
// sort path's look-back gave up or E does not fit the int32 layout.
int spmspv_run(apspie_context *ctx, const char *what, int sr, int m, int64_t nnz, const int *ptr,
               const int *ind, const float *val, int xnnz, const int *xind, const float *xval,
               int *yind, float *yval, SpmspvSmall *sm, bool want_ynnz, SpmspvSmall *out) {
  cudaStream_t st = ctx->stream;
  const double factor = ctx->spmspv_sort_factor;
  out->total = 0;
  out->ynnz = -1;
  int rc = APSPIE_OK;
  if (xnnz == 0) {
    rc = check_cuda(ctx, cudaMemsetAsync(sm, 0, sizeof(SpmspvSmall), st), what);
    return rc || !want_ynnz ? rc : spmspv_read_back(ctx, what, out);
  }
  auto *offs = (long long *)workspace(ctx, kSlotMisc0, sizeof(long long) * (size_t)(xnnz + 1));
  auto *col = (int2 *)workspace(ctx, kSlotMisc2, sizeof(int2) * (size_t)xnnz);
  if (!offs || !col) return APSPIE_ERR_OOM;
  // the bitmap path before E is known
  const bool ahead = m <= kBitmapRows && factor > 0.0 &&
                     (sr != kPlusTimes || (double)xnnz * (double)nnz * factor * kDenseGuess >=
                                              (double)m * (double)m);
  void *acc = nullptr;
  if (ahead) {
    acc = workspace(ctx, kSlotDense, sizeof(double) * (size_t)m);
    if (!acc) return APSPIE_ERR_OOM;
  }
  frontier_columns<<<grid_for(ctx, ahead ? std::max(xnnz, m) : xnnz, 256), 256, 0, st>>>(
      xnnz, xind, xval, ptr, offs, col, sr, m, (unsigned long long *)acc);
  rc = check_launch(ctx, "frontier_columns");
  if (rc) return rc;
  rc = device_exclusive_scan<long long>(ctx, offs, offs, xnnz, &sm->total);
  if (rc) return rc;
  bool bitmap = ahead;
  if (!ahead) {
    long long *h = (long long *)pinned(ctx, sizeof(long long));
    if (!h) return APSPIE_ERR_OOM;
    rc = check_cuda(ctx, cudaMemcpyAsync(h, &sm->total, sizeof(long long), cudaMemcpyDeviceToHost,
                                         st), what);
    if (rc) return rc;
    rc = check_cuda(ctx, cudaStreamSynchronize(st), what);
    if (rc) return rc;
    out->total = *h;
    if (out->total >= (long long)INT32_MAX)
      return set_error(ctx, APSPIE_ERR_OVERFLOW, "%s: %lld expanded pairs", what, out->total);
    if (out->total == 0) {
      rc = check_cuda(ctx, cudaMemsetAsync(&sm->ynnz, 0, sizeof(int), st), what);
      return rc || !want_ynnz ? rc : spmspv_read_back(ctx, what, out);
    }
    bitmap = spmspv_dense(out->total, factor, m);
  }
  if (bitmap) {
    const int words = (int)(((long long)m + 31) / 32);
    unsigned *bits = (unsigned *)workspace(ctx, kSlotBitmap,
                                           sizeof(unsigned) * ((size_t)words + kEmitBlocks));
    if (!bits) return APSPIE_ERR_OOM;
    unsigned *sums = bits + words;
    if (!acc) {  // not cleared with the columns
      acc = workspace(ctx, kSlotDense, sizeof(double) * (size_t)m);
      if (!acc) return APSPIE_ERR_OOM;
      acc_init<<<grid_for(ctx, m, 256), 256, 0, st>>>(sr, m, (unsigned long long *)acc);
      rc = check_launch(ctx, "acc_init");
      if (rc) return rc;
    }
    // a sparse PLUS_TIMES frontier is sorted: no row is touched here
    const long long least = sr == kPlusTimes ? dense_from(factor, m) : 0;
    expand_accumulate<<<expand_grid(ctx), kEdgeThreads, 0, st>>>(sr, least, xnnz, offs, &sm->total,
                                                                 col, ind, val, acc);
    const int per_block = std::max(kEmitWords, (words + kEmitBlocks - 1) / kEmitBlocks);
    const int eblocks = (words + per_block - 1) / per_block;
    touched_rows<<<eblocks, kEmitThreads, 0, st>>>(sr, m, acc, words, per_block, bits, sums);
    touched_emit<<<eblocks, kEmitThreads, 0, st>>>(sr, m, bits, words, per_block, sums, acc,
                                                   &sm->total, factor, yind, yval, &sm->ynnz);
    rc = check_launch(ctx, "spmspv bitmap", 3);
    if (rc) return rc;
    if (ahead || want_ynnz) rc = spmspv_read_back(ctx, what, out);
    if (rc || sr != kPlusTimes || out->total == 0 || spmspv_dense(out->total, factor, m)) return rc;
  }
  const long long E = out->total;
  rc = spmspv_sorted(ctx, sr, m, ind, val, xnnz, offs, col, E, yind, yval, sm);
  if (rc) return rc;
  // a sort of one tile waits for no other: nothing to check
  return want_ynnz || E > kSortTile ? spmspv_read_back(ctx, what, out) : APSPIE_OK;
}

}  // namespace
}  // namespace apspie

using namespace apspie;

extern "C" {

int apspie_spmspv(apspie_ctx ctx, int semiring, int m, int64_t nnz, const int *d_ptr,
                  const int *d_ind, const float *d_val, int xnnz, const int *d_xind,
                  const float *d_xval, int *d_yind, float *d_yval, int *h_ynnz,
                  int64_t *h_expanded) {
  APSPIE_CHECK_CTX(ctx);
  if (semiring < 0 || semiring > 3 || m <= 0 || nnz < 0 || xnnz < 0 || xnnz > m || !d_ptr ||
      (nnz > 0 && !d_ind) || (xnnz > 0 && !d_xind) || !d_yind || !d_yval || !h_ynnz)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_spmspv: bad arguments");
  auto *sm = spmspv_scalars(ctx);
  if (!sm) return APSPIE_ERR_OOM;
  SpmspvSmall back;
  const int rc = spmspv_run(ctx, "apspie_spmspv", semiring, m, nnz, d_ptr, d_ind, d_val, xnnz,
                            d_xind, d_xval, d_yind, d_yval, sm, true, &back);
  if (rc) return rc;
  *h_ynnz = back.ynnz;
  if (h_expanded) *h_expanded = back.total;
  return APSPIE_OK;
}

int apspie_mxv_dense(apspie_ctx ctx, int semiring, int m, int64_t nnz, const int *d_ptr,
                     const int *d_ind, const float *d_val, const float *d_x, float *d_y,
                     int64_t *h_expanded) {
  APSPIE_CHECK_CTX(ctx);
  if (semiring < 0 || semiring > 3 || m <= 0 || nnz < 0 || !d_ptr || (nnz > 0 && !d_ind) ||
      !d_x || !d_y)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_mxv_dense: bad arguments");
  cudaStream_t st = ctx->stream;
  unsigned *flags = (unsigned *)workspace(ctx, kSlotMxvFlags, sizeof(unsigned) * ((size_t)m + 1));
  // frontier (xind, xval) and the sparse result share one buffer of 4m words
  int *buf = (int *)workspace(ctx, kSlotMxvBuf, sizeof(int) * 4 * ((size_t)m + 1));
  if (!flags || !buf) return APSPIE_ERR_OOM;
  int *fx = buf;
  float *fv = (float *)(buf + (m + 1));
  int *yi = buf + 2 * (m + 1);
  float *yv = (float *)(buf + 3 * (m + 1));
  auto *sm = spmspv_scalars(ctx);
  if (!sm) return APSPIE_ERR_OOM;
  unsigned *d_cnt = &sm->cnt;
  dense_frontier_flags<<<grid_for(ctx, m, 256), 256, 0, st>>>(semiring, m, d_x, flags);
  int rc = check_launch(ctx, "dense_frontier_flags");
  if (rc) return rc;
  rc = device_exclusive_scan<unsigned>(ctx, flags + 0, flags + 0, m, d_cnt);
  if (rc) return rc;
  // flags were overwritten by their scan; recompute membership in the compaction
  dense_frontier_flags<<<grid_for(ctx, m, 256), 256, 0, st>>>(semiring, m, d_x,
                                                              (unsigned *)yi);
  dense_compact<<<grid_for(ctx, m, 256), 256, 0, st>>>(m, d_x, (unsigned *)yi, flags, fx, fv);
  rc = check_launch(ctx, "dense_compact", 2);
  if (rc) return rc;
  unsigned *h = (unsigned *)pinned(ctx, sizeof(long long));
  if (!h) return APSPIE_ERR_OOM;
  cudaMemcpyAsync(h, d_cnt, sizeof(unsigned), cudaMemcpyDeviceToHost, st);
  rc = check_cuda(ctx, cudaStreamSynchronize(st), "apspie_mxv_dense");
  if (rc) return rc;
  int xnnz = (int)*h;
  // y reset to the semiring's empty value, as preprocessFlag does
  // (0 for mXv, src/mXv.cuh:45; 1.70141e38 for SSSP, src/spmspvSssp.cuh:26)
  float empty = semiring == kMinPlus ? 1.70141e+38f : 0.0f;
  // y is written when the call's status is known: one that fails leaves it
  SpmspvSmall back;
  rc = spmspv_run(ctx, "apspie_mxv_dense", semiring, m, nnz, d_ptr, d_ind, d_val, xnnz, fx, fv,
                  yi, yv, sm, false, &back);
  if (rc) return rc;
  dense_fill<<<grid_for(ctx, m, 256), 256, 0, st>>>(m, empty, d_y);
  dense_scatter<<<grid_for(ctx, m, 256), 256, 0, st>>>(&sm->ynnz, m, yi, yv, d_y);
  rc = check_launch(ctx, "dense_scatter", 2);
  if (rc) return rc;
  if (h_expanded) *h_expanded = back.total;
  return APSPIE_OK;
}

int apspie_spmspv_set_params(apspie_ctx ctx, double sort_factor) {
  if (!ctx || !(sort_factor >= 0.0)) return APSPIE_ERR_INVALID;
  ctx->spmspv_sort_factor = sort_factor;
  return APSPIE_OK;
}

}  // extern "C"
