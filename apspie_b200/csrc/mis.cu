// mis.cu -- Luby-style maximal independent set with fixed priorities, and the
// neighbour-flag SpMSpV used to validate it.
//
// Replaces spmspvMis<V>() (src/spmspvMis.cuh:150-344).  The reference rounds
// are: candidates = undecided vertices with prio > minimum (buildVector :54,
// minimum -= delta per round), expand candidates to neighbours, radix sort,
// ReduceByKey(max) of candidate priorities per neighbour (:289), a candidate
// joins when its priority beats that maximum (updateMis :64), and the
// neighbours of joiners leave (updateNeighbor :71) -- with a full D->H copy of
// the candidate vector every round (:240).  Here one persistent kernel runs
// the rounds, one pass and one bounded grid barrier each.  A word per vertex
// holds its key while it is undecided, and 0 (OUT) or all ones (IN) after.
// Every undecided vertex v scans its neighbours' words (the max-priority
// SpMSpV with the comparison fused in) until one stops it:
//   * a neighbour that is IN: v leaves (OUT);
//   * an undecided neighbour of larger key: v stays, and is compacted into
//     the next round's queue with the position it stopped at;
//   * none left, and v is a candidate of the round: v joins (IN) and at once
//     marks its neighbours OUT (they would leave next round anyway; doing it
//     now lets their other neighbours decide a round earlier; a queued
//     vertex marked OUT meanwhile is dropped next round).
// A neighbour passed over was OUT, or smaller and undecided; the first is
// final and the second cannot join before v is decided, so the next round
// goes on from where this one stopped and a vertex reads each of its edges
// once over all rounds, plus the stopping one once per round.  (Scanning
// every edge of every undecided vertex each round, state and priority apart:
// 188 us on 2^20 vertices of mean degree 8, half of it waiting for loads
// issued one edge at a time.)
// Words change in place during the pass, so a neighbour's word may be read
// before or after its own update in the same pass; the stale value is always
// "undecided" (IN and OUT are final), which only delays a decision.
// v is IN exactly when no neighbour of larger key is IN, so the set is the
// greedy MIS in descending key order for any delta, whatever the timing.
// key(v) = (prio[v] << 32) | (v + 1), so ties in priority go to the larger id
// and every round decides at least the undecided vertex of largest key.
// Self-loops are ignored.  A lane scans its own vertex's next edges four at a
// time; the few scans longer than that are taken by the whole warp, one
// vertex after the other.
#include <cuda_runtime.h>

#include <algorithm>

#include "common.cuh"
#include "context.h"

namespace apspie {
namespace {

constexpr int kMisThreads = 512;
constexpr int kUndecided = -1, kOut = 0, kIn = 1;

struct MisState {
  unsigned q[3];  // queue lengths, rotating
  alignas(8) unsigned bar[2];  // grid-barrier arrival counter (64-bit)
  int err;
  int rounds;
};

constexpr unsigned long long kOutWord = 0ull, kInWord = ~0ull;
constexpr int kLaneScans = 4;  // batches of four edges a lane scans by itself
constexpr unsigned kLaneMarks = 32;  // joiners of more edges are marked by the warp

__global__ void mis_init(int m, const uint32_t *__restrict__ prio, unsigned long long *word,
                         MisState *st) {
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x)
    word[v] = ((unsigned long long)prio[v] << 32) | (unsigned)(v + 1);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->q[0] = (unsigned)m;
    st->q[1] = st->q[2] = 0;
    st->bar[0] = st->bar[1] = 0;
    st->err = 0;
    st->rounds = 0;
  }
}

enum { kScanning = 0, kStopped, kLeaves, kFree };

__global__ void __launch_bounds__(kMisThreads, 3)
mis_persistent(int m, const int *__restrict__ ptr, const int *__restrict__ ind,
               unsigned long long *word, int32_t *out, int2 *qa, int2 *qb, MisState *st,
               double delta, int max_rounds) {
  const int lane = lane_id();
  const int gwarp = spread_warp();
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  __shared__ unsigned s_q;
  int r = 0;
  for (;; ++r) {
    if (threadIdx.x == 0) {
      s_q = __ldcg(&st->q[r % 3]);
      if (blockIdx.x == 0) st->q[(r + 2) % 3] = 0;
    }
    __syncthreads();
    const unsigned nq = s_q;
    if (nq == 0 || (max_rounds > 0 && r >= max_rounds)) break;
    // candidates of this round: prio > threshold (the reference's minimum)
    double level = 1.0 - (double)(r + 1) * delta;
    unsigned long long thr = level <= 0.0 ? 0ull : (unsigned long long)(level * 4294967296.0);
    const int2 *qin = (r & 1) ? qb : qa;
    int2 *qout = (r & 1) ? qa : qb;
    for (unsigned base = (unsigned)gwarp * 32u; base < nq; base += (unsigned)nwarps * 32u) {
      const unsigned idx = base + lane;
      int v = -1;
      unsigned pos = 0, e = 0;  // unsigned: a batch past the last edge of 2^31 does not wrap
      unsigned long long my = kOutWord;
      if (idx < nq) {
        if (r == 0) {  // every vertex, from its first edge
          v = (int)idx;
          pos = (unsigned)__ldg(ptr + v);
        } else {
          const int2 q = __ldcg(qin + idx);
          v = q.x;
          pos = (unsigned)q.y;
        }
        e = (unsigned)__ldg(ptr + v + 1);
        my = __ldcg(word + v);
      }
      int st_v = my == kOutWord ? kLeaves : (pos < e ? kScanning : kFree);
#pragma unroll 1
      for (int b = 0; b < kLaneScans; ++b) {
        if (!__any_sync(kFull, st_v == kScanning)) break;
        int u[4];
        unsigned long long k[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          u[i] = st_v == kScanning && pos + i < e ? __ldg(ind + pos + i) : -1;
#pragma unroll
        for (int i = 0; i < 4; ++i) k[i] = u[i] >= 0 ? __ldcg(word + u[i]) : kOutWord;
        int stop = 4;
#pragma unroll
        for (int i = 3; i >= 0; --i)
          if (k[i] > my && u[i] != v) stop = i;
        if (st_v == kScanning) {
          const unsigned long long ks =
              stop == 0 ? k[0] : (stop == 1 ? k[1] : (stop == 2 ? k[2] : k[3]));
          pos += (unsigned)stop;
          if (stop < 4) st_v = ks == kInWord ? kLeaves : kStopped;
          else if (pos >= e) st_v = kFree;
        }
      }
      // the scans that are not over: the warp, 128 edges at a time
      for (unsigned left = __ballot_sync(kFull, st_v == kScanning); left; left &= left - 1) {
        const int j = __ffs(left) - 1;
        const int vj = __shfl_sync(kFull, v, j);
        const unsigned ej = __shfl_sync(kFull, e, j);
        const unsigned long long mj = __shfl_sync(kFull, my, j);
        unsigned pj = __shfl_sync(kFull, pos, j);
        int sj = kFree;
        for (; pj < ej; pj += 128) {
          int u[4];
          unsigned long long k[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const unsigned p = pj + 32u * i + (unsigned)lane;
            u[i] = p < ej ? __ldg(ind + p) : -1;
          }
#pragma unroll
          for (int i = 0; i < 4; ++i) k[i] = u[i] >= 0 ? __ldcg(word + u[i]) : kOutWord;
          unsigned in = 0, at = 128;
#pragma unroll
          for (int i = 3; i >= 0; --i) {
            const bool big = k[i] > mj && u[i] != vj;
            const unsigned bm = __ballot_sync(kFull, big);
            in |= __ballot_sync(kFull, big && k[i] == kInWord);
            if (bm) at = 32u * i + (unsigned)__ffs(bm) - 1u;
          }
          if (at < 128u) {
            pj += at;
            sj = in ? kLeaves : kStopped;
            break;
          }
        }
        if (lane == j) {
          st_v = sj;
          pos = pj;
        }
      }
      const bool joins = v >= 0 && st_v == kFree && (my >> 32) >= thr;
      // (v + 1 keeps an undecided word above kOutWord; a vertex marked OUT
      // while it scanned keeps that word: it cannot have come out free)
      if (v >= 0 && st_v == kLeaves && my != kOutWord) word[v] = kOutWord;
      unsigned s = 0;
      if (joins) {
        word[v] = kInWord;
        s = (unsigned)__ldg(ptr + v);
        if (e - s <= kLaneMarks)
          for (unsigned p = s; p < e; p += 4) {
            int u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) u[i] = p + i < e ? __ldg(ind + p + i) : v;
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (u[i] != v) word[u[i]] = kOutWord;
          }
      }
      for (unsigned wide = __ballot_sync(kFull, joins && e - s > kLaneMarks); wide;
           wide &= wide - 1) {
        const int j = __ffs(wide) - 1;
        const int vj = __shfl_sync(kFull, v, j);
        const unsigned ej = __shfl_sync(kFull, e, j);
        for (unsigned p = __shfl_sync(kFull, s, j) + (unsigned)lane; p < ej; p += 32) {
          const int u = __ldg(ind + p);
          if (u != vj) word[u] = kOutWord;
        }
      }
      const bool stays = v >= 0 && (st_v == kStopped || (st_v == kFree && !joins));
      const unsigned slot = warp_append(stays, &st->q[(r + 1) % 3]);
      if (stays) qout[slot] = make_int2(v, (int)pos);
    }
    if (!grid_barrier(st->bar, &st->err)) return;
  }
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < m; v += gridDim.x * blockDim.x) {
    const unsigned long long k = __ldcg(word + v);
    out[v] = k == kInWord ? kIn : (k == kOutWord ? kOut : kUndecided);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) st->rounds = r;
}

__global__ void neighbor_flags_kernel(int m, const int *__restrict__ ptr,
                                      const int *__restrict__ ind, const int32_t *in,
                                      int32_t *out) {
  // one warp per flagged vertex, coalesced over its out-edges
  const int lane = lane_id();
  const int gwarp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int nwarps = (int)((gridDim.x * blockDim.x) >> 5);
  for (int base = gwarp * 32; base < m; base += nwarps * 32) {
    int v = base + lane;
    bool f = v < m && in[v] != 0;
    unsigned mask = __ballot_sync(kFull, f);
    while (mask) {
      int j = __ffs(mask) - 1;
      mask &= mask - 1;
      int vj = base + j;
      int s = __ldg(ptr + vj), e = __ldg(ptr + vj + 1);
      for (int k = s + lane; k < e; k += 32) out[__ldg(ind + k)] = 1;
    }
  }
}

__global__ void zero_i32(int n, int32_t *p) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) p[i] = 0;
}

int mis_grid(apspie_context *ctx) {
  return occupancy_grid(ctx, (const void *)mis_persistent, kMisThreads);
}

// One piece of workspace: the state, a word per vertex, two queues.  (A slot
// each: four allocations in a context's first call, 1.43 ms of it on 2^20
// vertices against 0.50 so.)
constexpr size_t kMisHead = 256;
static_assert(sizeof(MisState) <= kMisHead, "the state precedes the words");

}  // namespace

size_t mis_scratch_bytes(size_t m) {
  return kMisHead + (sizeof(unsigned long long) + 2 * sizeof(int2)) * m;
}

}  // namespace apspie

using namespace apspie;

extern "C" {

int apspie_mis(apspie_ctx ctx, int64_t nnz, int m, const int *d_ptr, const int *d_ind,
               const uint32_t *d_prio, int32_t *d_mis, float delta) {
  APSPIE_CHECK_CTX(ctx);
  if (m <= 0 || nnz < 0 || nnz >= (int64_t)INT32_MAX)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_mis: bad sizes m=%d nnz=%lld", m,
                     (long long)nnz);
  if (!d_ptr || !d_prio || !d_mis || (nnz > 0 && !d_ind))
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_mis: null pointer");
  if (!(delta > 0.0f)) delta = 1.0f;
  auto *st = (MisState *)workspace(ctx, kSlotMis, mis_scratch_bytes((size_t)m));
  if (!st) return APSPIE_ERR_OOM;
  auto *word = (unsigned long long *)((unsigned char *)st + kMisHead);
  auto *qa = (int2 *)(word + m), *qb = qa + m;
  ctx->mis_state = st;
  int grid = clamp_grid(ctx, mis_grid(ctx));
  if (grid <= 0) return set_error(ctx, APSPIE_ERR_CUDA, "apspie_mis: occupancy query failed");
  int init_grid = std::min((m + 255) / 256, ctx->num_sms * 8);
  mis_init<<<init_grid, 256, 0, ctx->stream>>>(m, d_prio, word, st);
  int rc = check_launch(ctx, "mis_init");
  if (rc) return rc;
  double dd = (double)delta;
  // the round cap only guards against a stalled device loop: every round
  // decides at least one vertex, so m + 1 rounds always suffice
  int max_rounds = (int)std::min(2.0e9, (double)m + 1.0 + 1.0 / dd);
  void *args[] = {&m, (void *)&d_ptr, (void *)&d_ind, &word, &d_mis, &qa, &qb, &st, &dd,
                  &max_rounds};
  cudaError_t e = cudaLaunchCooperativeKernel((const void *)mis_persistent, dim3(grid),
                                              dim3(kMisThreads), args, 0, ctx->stream);
  if (e != cudaSuccess) return check_cuda(ctx, e, "mis_persistent");
  ctx->launches += 1;
  return APSPIE_OK;
}

int apspie_mis_get_rounds(apspie_ctx ctx, int *rounds) {
  APSPIE_CHECK_CTX(ctx);
  if (!rounds || !ctx->mis_state)
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_mis_get_rounds: no MIS has run");
  auto *h = (MisState *)pinned(ctx, sizeof(MisState));
  if (!h) return APSPIE_ERR_OOM;
  cudaError_t e = cudaMemcpyAsync(h, ctx->mis_state, sizeof(MisState), cudaMemcpyDeviceToHost,
                                  ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return check_cuda(ctx, e, "apspie_mis_get_rounds");
  *rounds = h->rounds;
  if (h->err) return set_error(ctx, APSPIE_ERR_TIMEOUT, "apspie_mis: grid barrier timed out");
  return APSPIE_OK;
}

int apspie_neighbor_flags(apspie_ctx ctx, int64_t nnz, int m, const int *d_ptr,
                          const int *d_ind, const int32_t *d_in, int32_t *d_out) {
  APSPIE_CHECK_CTX(ctx);
  if (m <= 0 || nnz < 0 || !d_ptr || !d_in || !d_out || (nnz > 0 && !d_ind))
    return set_error(ctx, APSPIE_ERR_INVALID, "apspie_neighbor_flags: bad arguments");
  int grid = std::min((m + 255) / 256, ctx->num_sms * 8);
  zero_i32<<<grid, 256, 0, ctx->stream>>>(m, d_out);
  neighbor_flags_kernel<<<ctx->num_sms * 4, 512, 0, ctx->stream>>>(m, d_ptr, d_ind, d_in, d_out);
  return check_launch(ctx, "neighbor_flags", 2);
}

}  // extern "C"
