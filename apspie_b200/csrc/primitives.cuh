// primitives.cuh -- device-wide scan and a stable LSD radix sort of
// (key, value) pairs, written for this library (the reference uses moderngpu
// Scan and cub::DeviceRadixSort, src/mXv.cuh:142,191-193).
//
// Scan: reduce-then-scan: tile sums, then tile scans that each add up the
// sums before them; from kScanFewTiles tiles on the sums are scanned by one
// block in between; short inputs take one launch.  No inter-block waits.
//
// Radix sort: 8-bit digits, only as many passes as the key's significant
// bits need (ceil(log2 m) bits for row indices), in the onesweep form: one
// read of the keys counts every pass's digits (radix_histograms), then one
// kernel per pass (radix_onesweep) whose tiles of 256 threads x 16 keys
//   * rank their keys: inside a warp, __match_any_sync groups lanes with the
//     same digit, and a per-warp shared histogram carries the running count
//     across rounds; a per-digit prefix over the warps of the tile orders
//     the warps;
//   * find each digit's output offset by decoupled look-back over the tiles
//     before them (bounded waits);
//   * write each digit's run contiguously from a shared-memory copy of the
//     tile, the values copied in by cp.async while the keys were ranked.
// Every key keeps its input order among equal digits, so the LSD passes
// sort stably.
#pragma once
#include <cstdint>

#include "common.cuh"
#include "context.h"

namespace apspie {

constexpr int kScanThreads = 512;
constexpr int kScanItems = 8;
constexpr int kScanTile = kScanThreads * kScanItems;

// Block-wide exclusive scan of one value per thread; returns the prefix and
// writes the block total to *total (all threads).
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T *smem_warp, T *total) {
  const int lane = lane_id(), w = warp_in_block(), nw = blockDim.x >> 5;
  T incl = warp_incl_scan(v);
  if (lane == 31) smem_warp[w] = incl;
  __syncthreads();
  if (w == 0) {
    T x = lane < nw ? smem_warp[lane] : T(0);
    T xi = warp_incl_scan(x);
    if (lane < nw) smem_warp[lane] = xi - x;
    if (lane == nw - 1) smem_warp[32] = xi;
  }
  __syncthreads();
  T res = smem_warp[w] + incl - v;
  *total = smem_warp[32];
  __syncthreads();
  return res;
}

template <typename T>
__global__ void scan_tile_sums(const T *in, long long n, T *sums) {
  __shared__ T sw[33];
  long long base = (long long)blockIdx.x * kScanTile;
  T acc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    long long idx = base + (long long)i * kScanThreads + threadIdx.x;
    if (idx < n) acc += in[idx];
  }
  T tot;
  block_excl_scan(acc, sw, &tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = tot;
}

// Exclusive scan of sums[0..n) in one block, blockDim.x values per pass;
// writes the grand total to *total.
template <typename T>
__global__ void scan_single_block(T *sums, int n, T *total) {
  __shared__ T sw[33];
  __shared__ T carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int base = 0; base < n; base += blockDim.x) {
    int i = base + threadIdx.x;
    T v = i < n ? sums[i] : T(0);
    T tot;
    T ex = block_excl_scan(v, sw, &tot);
    if (i < n) sums[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

// kSumsScanned: sums are exclusive prefixes already; else every tile adds up
// the plain sums before it (at most kScanFewTiles, a coalesced read from L2
// instead of a launch) and the last one writes the total.
constexpr int kScanFewTiles = 1024;

template <typename T, bool kSumsScanned>
__global__ void scan_tiles(const T *in, long long n, const T *sums, T *out, T *total) {
  __shared__ T sw[33];
  T before = 0;
  if (kSumsScanned) {
    before = sums[blockIdx.x];
  } else {
    for (unsigned i = threadIdx.x; i < blockIdx.x; i += kScanThreads) before += sums[i];
    T all;
    block_excl_scan(before, sw, &all);
    before = all;
  }
  long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
  T v[kScanItems];
  T acc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    long long idx = base + i;
    v[i] = idx < n ? in[idx] : T(0);
    acc += v[i];
  }
  T tot;
  T run = block_excl_scan(acc, sw, &tot) + before;
  if (!kSumsScanned && total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0)
    *total = before + tot;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    long long idx = base + i;
    if (idx < n) out[idx] = run;
    run += v[i];
  }
}

// A short scan in one launch instead of three (about 2 us each): one block,
// kScanItems values per thread.  (Twice the values in two steps: no faster
// than the three launches.)
constexpr int kSmallScanThreads = 1024;
constexpr int kSmallScanMax = kSmallScanThreads * kScanItems;

template <typename T>
__global__ void __launch_bounds__(kSmallScanThreads)
scan_small(const T *in, int n, T *out, T *total) {
  __shared__ T sw[33];
  const int first = (int)threadIdx.x * kScanItems;
  T v[kScanItems];
  T acc = 0;
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    v[i] = first + i < n ? in[first + i] : T(0);
    acc += v[i];
  }
  T tot;
  T run = block_excl_scan(acc, sw, &tot);
#pragma unroll
  for (int i = 0; i < kScanItems; ++i) {
    if (first + i < n) out[first + i] = run;
    run += v[i];
  }
  if (threadIdx.x == 0 && total) *total = tot;
}

// Exclusive scan in[0..n) -> out[0..n) (may alias); *d_total gets the sum.
// Scratch: slot kSlotScan.  Returns a status.
template <typename T>
int device_exclusive_scan(apspie_context *ctx, const T *in, T *out, long long n, T *d_total) {
  if (n <= kSmallScanMax) {
    scan_small<T><<<1, kSmallScanThreads, 0, ctx->stream>>>(in, (int)n, out, d_total);
    return check_launch(ctx, "scan_small");
  }
  long long tiles = (n + kScanTile - 1) / kScanTile;
  // the tile sums are scanned by one block in a loop: fine up to 2^20 tiles
  // (2^32 elements); T must hold the total
  if (tiles > (1ll << 20))
    return set_error(ctx, APSPIE_ERR_OVERFLOW, "device scan: %lld elements too many", n);
  T *sums = (T *)workspace(ctx, kSlotScan, sizeof(T) * (size_t)(tiles + 1));
  if (!sums) return APSPIE_ERR_OOM;
  // tile sums are computed from `in` before `out` is written, so in == out works
  scan_tile_sums<T><<<(unsigned)tiles, kScanThreads, 0, ctx->stream>>>(in, n, sums);
  if (tiles <= kScanFewTiles) {
    scan_tiles<T, false><<<(unsigned)tiles, kScanThreads, 0, ctx->stream>>>(in, n, sums, out,
                                                                            d_total);
    return check_launch(ctx, "device_exclusive_scan", 2);
  }
  scan_single_block<T><<<1, kScanThreads, 0, ctx->stream>>>(sums, (int)tiles, d_total);
  scan_tiles<T, true><<<(unsigned)tiles, kScanThreads, 0, ctx->stream>>>(in, n, sums, out,
                                                                         nullptr);
  return check_launch(ctx, "device_exclusive_scan", 3);
}

// ------------------------------------------------------------ radix sort ---
// Onesweep LSD radix sort (Adinets & Merrill, "Onesweep: A Faster Least
// Significant Digit Radix Sort for GPUs", 2022): one read of the keys
// counts every pass's digits, then one kernel per 8-bit pass.  A pass's
// tiles take ids from a counter (so a tile only waits on tiles that are
// already running), rank their keys locally (match_any per warp, a prefix
// over the warps), publish their per-digit counts, and find their digit
// offsets by decoupled look-back over the tiles before them: each status
// word holds a flag (aggregate of this tile / inclusive of all before and
// this one), the pass's tag and the count.  Stable.
constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;
constexpr int kSortTile = kSortThreads * kSortItems;
constexpr int kRadixBits = 8;
constexpr int kRadix = 1 << kRadixBits;
constexpr int kMaxPasses = 8;

// Status words.  32 bits for sorts of fewer than 2^27 keys: flag 2 bits, pass
// tag 3 bits, count 27 bits; else 64 bits (flag 2, tag 22, count 40).  The
// tag tells a pass's words from those an earlier pass left, so all passes
// share one zeroed array.  A tile loads kWindow predecessors' words at once,
// so the look-back moves on by that many tiles per L2 round trip (about
// 0.35 us).  It does not bound a pass: windows of 4 and of 16 words take the
// same time (and the wider one spills registers).
template <typename S>
struct SortStatus;
template <>
struct SortStatus<unsigned> {
  static constexpr unsigned kAgg = 1u << 30, kIncl = 2u << 30, kFlags = 3u << 30;
  static constexpr unsigned kTag = 7u << 27, kCount = (1u << 27) - 1u;
  static constexpr int kWindow = 4;
  __device__ __forceinline__ static unsigned tag(int pass) { return (unsigned)pass << 27; }
  __device__ __forceinline__ static unsigned load(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
  }
};
template <>
struct SortStatus<unsigned long long> {
  static constexpr unsigned long long kAgg = 1ull << 62, kIncl = 2ull << 62, kFlags = 3ull << 62;
  static constexpr unsigned long long kTag = 0x3FFFFFull << 40, kCount = (1ull << 40) - 1ull;
  static constexpr int kWindow = 4;
  __device__ __forceinline__ static unsigned long long tag(int pass) {
    return (unsigned long long)pass << 40;
  }
  __device__ __forceinline__ static unsigned long long load(const unsigned long long *p) {
    return ld_relaxed64(p);
  }
};

// All passes' digit counts in one read of the keys, kHistKeys loads in
// flight per thread (one at a time the kernel waited for each: 64 us for
// 16 M 4-byte keys).
constexpr int kHistKeys = 8;

template <typename K>
__global__ void __launch_bounds__(kSortThreads)
radix_histograms(const K *keys, long long n, int npass, unsigned long long *ghist) {
  __shared__ unsigned hist[kMaxPasses][kRadix];
  for (int t = threadIdx.x; t < kMaxPasses * kRadix; t += blockDim.x) hist[t / kRadix][t % kRadix] = 0;
  __syncthreads();
  constexpr long long kStep = (long long)kSortThreads * kHistKeys;
  for (long long b = blockIdx.x * kStep; b < n; b += gridDim.x * kStep) {
    K k[kHistKeys];
#pragma unroll
    for (int q = 0; q < kHistKeys; ++q) {
      const long long i = b + q * kSortThreads + threadIdx.x;
      k[q] = i < n ? keys[i] : K(0);
    }
    const int cnt = (int)min((long long)kHistKeys,
                             (n - b - threadIdx.x + kSortThreads - 1) / kSortThreads);
    for (int p = 0; p < npass; ++p)
#pragma unroll
      for (int q = 0; q < kHistKeys; ++q)
        if (q < cnt) atomicAdd(&hist[p][(unsigned)(k[q] >> (p * kRadixBits)) & (kRadix - 1)], 1u);
  }
  __syncthreads();
  for (int t = threadIdx.x; t < npass * kRadix; t += blockDim.x) {
    const unsigned c = hist[t / kRadix][t % kRadix];
    if (c) atomicAdd(ghist + t, (unsigned long long)c);
  }
}

// per pass, exclusive prefix of the digit counts (one block of kRadix)
template <int R = kRadix>
__global__ void radix_digit_offsets(unsigned long long *ghist, int npass) {
  __shared__ unsigned long long sw[33];
  for (int p = 0; p < npass; ++p) {
    const unsigned long long c = ghist[p * R + threadIdx.x];
    unsigned long long total;
    const unsigned long long ex = block_excl_scan(c, sw, &total);
    ghist[p * R + threadIdx.x] = ex;
    __syncthreads();
  }
}

// Polls of a look-back wait before it gives up (a predecessor normally
// publishes within microseconds; about half a second with the back-off).
constexpr unsigned kLookbackSpinLimit = 1u << 20;

// A pass over 16 M pairs of 4-byte keys and values takes 151 us, 1.7 TB/s of
// the 256 MB it reads and writes: its bound is the instructions of ranking
// and placing a key (issue slots 43 % busy, the rest mostly waits for shared
// memory, three blocks of 80 registers per SM), not the bytes -- 12-byte
// pairs took as long.  So such pairs go through shared memory side by side:
// one store, one load and one look-up of the digit's run per pair (keys and
// values apart: 167 us).
template <typename K, typename V>
constexpr bool kSortPairs = sizeof(K) == 4 && sizeof(V) == 4;

template <typename K, typename V, typename S>
__global__ void __launch_bounds__(kSortThreads, 3)
radix_onesweep(const K *keys_in, const V *vals_in, K *keys_out, V *vals_out, long long n,
               int pass, const unsigned long long *goff, S *status,
               unsigned *tile_counter, int *err, int *gaveup) {
  constexpr int kWarps = kSortThreads / 32;
  static_assert(sizeof(V) <= sizeof(K), "values are staged in the keys' shared array");
  constexpr bool kPair = kSortPairs<K, V>;
  // the tile in digit order (pairs, or keys and then values), each key's
  // digit, per-warp digit counts, and per digit the output position of the
  // tile's run minus its start within the tile
  __shared__ __align__(16) K skeys[kPair ? 2 * kSortTile : kSortTile];
  __shared__ unsigned char sdig[kPair ? 1 : kSortTile];
  __shared__ unsigned whist[kWarps][kRadix];
  __shared__ unsigned long long gbase[kRadix];
  __shared__ unsigned s_scan[33];
  __shared__ unsigned s_tile;
  __shared__ int s_withhold;
  // the tile's values, copied in by cp.async while the keys are ranked
  // (dynamic: kSortTile values when the sort has values, else none)
  extern __shared__ __align__(16) unsigned char sort_dyn[];
  V *svin = reinterpret_cast<V *>(sort_dyn);
  const int lane = lane_id(), w = warp_in_block();
  const int shift = pass * kRadixBits;
  using St = SortStatus<S>;
  constexpr int kWindow = St::kWindow;
  const S tag = St::tag(pass);
  if (threadIdx.x == 0) {
    s_tile = atomicAdd(tile_counter, 1u);
    // test hook (apspie_debug_inject): err[1] set makes tile 0 of the next
    // pass withhold its status, so that its successors' bounded look-back
    // waits run out; one-shot
    s_withhold = (s_tile == 0u && n > kSortTile) ? atomicExch(err + 1, 0) : 0;
  }
  for (int d = lane; d < kRadix; d += 32) whist[w][d] = 0;
  __syncthreads();
  const unsigned tile = s_tile;
  const long long tbase = (long long)tile * kSortTile;
  const int tlen = (int)min((long long)kSortTile, n - tbase);
  // Values [0, vdone) of the tile are copied to shared memory in the
  // background, 16 bytes a copy, when they start on a 16-byte boundary; the
  // rest (a ragged end, or an unaligned array) are loaded when placed.
  int vdone = 0;
  if (vals_in && (reinterpret_cast<uintptr_t>(vals_in + tbase) & 15u) == 0) {
    constexpr int kPer = 16 / (int)sizeof(V);
    const int nchunk = tlen / kPer;
    vdone = nchunk * kPer;
    const unsigned sbase = (unsigned)__cvta_generic_to_shared(svin);
    for (int c = threadIdx.x; c < nchunk; c += kSortThreads)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sbase + 16u * c),
                   "l"(vals_in + tbase + (long long)c * kPer)
                   : "memory");
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  // this warp's slice of the tile: kSortItems rounds of 32 consecutive keys
  const int wofs = w * 32 * kSortItems;
  // per key its rank (then its tile position); its digit is recomputed
  // from the key where needed (registers for three blocks per SM)
  unsigned pos[kSortItems];
  K kv[kSortItems];
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const int t = wofs + i * 32 + lane;
    kv[i] = t < tlen ? keys_in[tbase + t] : K(0);
  }
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    const bool valid = wofs + i * 32 + lane < tlen;
    const unsigned d = valid ? (unsigned)(kv[i] >> shift) & (kRadix - 1) : (unsigned)kRadix;
    const unsigned peers = __match_any_sync(kFull, d);
    const int leader = __ffs(peers) - 1;
    unsigned prev = 0;
    if (valid && lane == leader) {
      prev = whist[w][d];
      whist[w][d] = prev + __popc(peers);
    }
    prev = __shfl_sync(kFull, prev, leader);
    pos[i] = prev + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  // per digit (one per thread): prefix over the warps, the tile's count,
  // its start within the tile, then the look-back for its output offset
  const int d = threadIdx.x;
  unsigned run = 0;
  for (int ww = 0; ww < kWarps; ++ww) {
    const unsigned c = whist[ww][d];
    whist[ww][d] = run;
    run += c;
  }
  unsigned tot;
  const unsigned loc = block_excl_scan(run, s_scan, &tot);
  S *mine = status + (size_t)tile * kRadix + d;
  S excl = 0;
  if (tile == 0) {
    if (!s_withhold) __stcg(mine, St::kIncl | tag | (S)run);
  } else {
    __stcg(mine, St::kAgg | tag | (S)run);
    // Look back kWindow predecessors at a time (their status words loaded
    // together, relaxed: a word's count is all that is read), adding counts
    // from the nearest one back until an inclusive word; a word not yet
    // published stops the window and is polled again.
    long long t = (long long)tile - 1;
    unsigned spins = 0;
    while (t >= 0) {
      S sv[kWindow];
#pragma unroll
      for (int k = 0; k < kWindow; ++k)
        sv[k] = t - k >= 0 ? St::load(status + (size_t)(t - k) * kRadix + d) : S(0);
      bool done = false, stalled = false;
      int adv = 0;
#pragma unroll
      for (int k = 0; k < kWindow; ++k) {
        if (done || stalled) continue;
        const S x = sv[k];
        if ((x & St::kFlags) == 0 || (x & St::kTag) != tag) {
          stalled = true;  // not published (or before tile 0, when t < k)
          continue;
        }
        excl += x & St::kCount;
        ++adv;
        if ((x & St::kFlags) == St::kIncl) done = true;  // everything before is in it
      }
      if (done) break;
      t -= adv;
      if (stalled && t >= 0) {
        // a predecessor has not published: give up after kLookbackSpinLimit
        // polls, or at once when another tile of this sort already gave up
        // (checked every 256; *gaveup is zeroed with the sort's status words)
        if (++spins > kLookbackSpinLimit ||
            ((spins & 255u) == 0u && *(volatile int *)gaveup != 0)) {
          atomicExch(err, 1);
          atomicExch(gaveup, 1);
          break;
        }
        if ((spins & 15u) == 0u) __nanosleep(64);
      }
    }
    __stcg(mine, St::kIncl | tag | (S)(excl + run));
  }
  gbase[d] = goff[pass * kRadix + d] + (unsigned long long)excl - loc;
  for (int ww = 0; ww < kWarps; ++ww) whist[ww][d] += loc;
  if (kPair && vdone > 0) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // tile position of every key: its digit's start + the warps before it + its rank
#pragma unroll
  for (int i = 0; i < kSortItems; ++i) {
    if (wofs + i * 32 + lane < tlen) {
      const unsigned dd = (unsigned)(kv[i] >> shift) & (kRadix - 1);
      pos[i] += whist[w][dd];
      if constexpr (kPair) {
        union { V v; unsigned u; } bits;
        const int t = wofs + i * 32 + lane;
        bits.v = t < vdone ? svin[t] : (vals_in ? vals_in[tbase + t] : (V)(tbase + t));
        reinterpret_cast<uint2 *>(skeys)[pos[i]] = make_uint2((unsigned)kv[i], bits.u);
      } else {
        skeys[pos[i]] = kv[i];
        sdig[pos[i]] = (unsigned char)dd;
      }
    }
  }
  __syncthreads();
  // The bound (at < n) holds for every sorted pass; it guards a pass after a
  // look-back give-up, whose input then holds keys the histograms did not
  // count.
  if constexpr (kPair) {
#pragma unroll 4
    for (int t = threadIdx.x; t < tlen; t += kSortThreads) {
      const uint2 x = reinterpret_cast<const uint2 *>(skeys)[t];
      const unsigned long long at = gbase[(x.x >> shift) & (kRadix - 1)] + t;
      if (at < (unsigned long long)n) {
        union { unsigned u; V v; } bits;
        bits.u = x.y;
        keys_out[at] = (K)x.x;
        if (vals_out) vals_out[at] = bits.v;
      }
    }
  } else {
    for (int t = threadIdx.x; t < tlen; t += kSortThreads) {
      const unsigned long long at = gbase[sdig[t]] + t;
      if (at < (unsigned long long)n) keys_out[at] = skeys[t];
    }
    if (vals_out) {  // keys-only sorts pass no values
      if (vdone > 0) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
      V *svals = reinterpret_cast<V *>(skeys);
#pragma unroll
      for (int i = 0; i < kSortItems; ++i) {
        const int t = wofs + i * 32 + lane;
        if (t < tlen)
          svals[pos[i]] = t < vdone ? svin[t] : (vals_in ? vals_in[tbase + t] : (V)(tbase + t));
      }
      __syncthreads();
      for (int t = threadIdx.x; t < tlen; t += kSortThreads) {
        const unsigned long long at = gbase[sdig[t]] + t;
        if (at < (unsigned long long)n) vals_out[at] = svals[t];
      }
    }
  }
}

// A sort of at most kSmallSortItems<K> x kSortThreads keys: one block, every
// pass in shared memory (in one launch; a pass of one tile and its status
// words take 9 us, the histograms, offsets and the memset 7 us more).  The
// ranking is radix_onesweep's.
template <typename K>
constexpr int kSmallSortItems = sizeof(K) <= 4 ? 16 : 8;

template <typename K, typename V>
__global__ void __launch_bounds__(kSortThreads)
radix_small(const K *keys_in, const V *vals_in, K *keys_out, V *vals_out, int n, int npass) {
  constexpr int kWarps = kSortThreads / 32;
  constexpr int kItems = kSmallSortItems<K>;
  constexpr int kTile = kItems * kSortThreads;
  __shared__ __align__(16) K skeys[kTile];
  __shared__ __align__(16) V svals[kTile];
  __shared__ unsigned whist[kWarps][kRadix];
  __shared__ unsigned s_scan[33];
  const int lane = lane_id(), w = warp_in_block();
  const int wofs = w * 32 * kItems;
  K kv[kItems];
  V vv[kItems];
  unsigned pos[kItems];
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int t = wofs + i * 32 + lane;
    kv[i] = t < n ? keys_in[t] : K(0);
    vv[i] = t < n && vals_in ? vals_in[t] : (V)t;
  }
  for (int p = 0; p < npass; ++p) {
    const int shift = p * kRadixBits;
    for (int d = lane; d < kRadix; d += 32) whist[w][d] = 0;
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const bool valid = wofs + i * 32 + lane < n;
      const unsigned d = valid ? (unsigned)(kv[i] >> shift) & (kRadix - 1) : (unsigned)kRadix;
      const unsigned peers = __match_any_sync(kFull, d);
      const int leader = __ffs(peers) - 1;
      unsigned prev = 0;
      if (valid && lane == leader) {
        prev = whist[w][d];
        whist[w][d] = prev + __popc(peers);
      }
      prev = __shfl_sync(kFull, prev, leader);
      pos[i] = prev + __popc(peers & ((1u << lane) - 1u));
      __syncwarp();
    }
    __syncthreads();
    unsigned run = 0, tot;
    for (int ww = 0; ww < kWarps; ++ww) {
      const unsigned c = whist[ww][threadIdx.x];
      whist[ww][threadIdx.x] = run;
      run += c;
    }
    const unsigned loc = block_excl_scan(run, s_scan, &tot);
    for (int ww = 0; ww < kWarps; ++ww) whist[ww][threadIdx.x] += loc;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i)
      if (wofs + i * 32 + lane < n) {
        const unsigned at = pos[i] + whist[w][(unsigned)(kv[i] >> shift) & (kRadix - 1)];
        skeys[at] = kv[i];
        svals[at] = vv[i];
      }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int t = wofs + i * 32 + lane;
      if (t < n) {
        kv[i] = skeys[t];
        vv[i] = svals[t];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const int t = wofs + i * 32 + lane;
    if (t < n) {
      keys_out[t] = kv[i];
      if (vals_out) vals_out[t] = vv[i];
    }
  }
}

// The context's radix-sort give-up word: set by a tile whose look-back
// waited kLookbackSpinLimit polls for a predecessor (the output is then in
// bounds but neither sorted nor a permutation of the input: some slots keep
// stale contents).  A caller that uses sorted keys or values as indices must
// therefore check it (radix_sort_check) before doing so, or bounds-check what
// it indexes and check the word at its end (apspie_spmspv, apspie_mxv_dense,
// apspie_csr_transpose, which all wait for the device there).  Sticky: zeroed
// when first allocated and by the check, not by each sort, so a caller sees a
// give-up of any sort it ran.
// kSortErrWords words (give-up, test hook, two unused); the rest of the slot's
// kSortErrBytes is a caller's that wants to read them back with its own.
constexpr int kSortErrWords = 4;
constexpr size_t kSortErrBytes = 64;
inline int *radix_sort_err(apspie_context *ctx) {
  auto *e = (int *)workspace(ctx, kSlotSortErr, kSortErrBytes);
  if (e && ctx->sort_err_zeroed != e) {
    cudaMemsetAsync(e, 0, 16, ctx->stream);
    ctx->sort_err_zeroed = e;
  }
  return e;
}

// Reads the give-up word back (synchronises the stream): APSPIE_ERR_TIMEOUT
// when a sort since the last check gave up, clearing the word.
inline int radix_sort_check(apspie_context *ctx) {
  int *e = radix_sort_err(ctx);
  int *h = (int *)pinned(ctx, sizeof(int));
  if (!e || !h) return APSPIE_ERR_OOM;
  cudaMemcpyAsync(h, e, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  const cudaError_t ce = cudaStreamSynchronize(ctx->stream);
  if (ce != cudaSuccess) return check_cuda(ctx, ce, "radix sort check");
  if (*h == 0) return APSPIE_OK;
  cudaMemsetAsync(e, 0, sizeof(int), ctx->stream);
  return set_error(ctx, APSPIE_ERR_TIMEOUT, "radix sort: a look-back wait gave up");
}

// Stable sort of n (key, value) pairs on the low `bits` bits of the key
// (va == vb == nullptr sorts keys only).  Ping-pongs between (ka, va) and
// (kb, vb); *result_in_b tells where the sorted data ended up.  With kfirst
// the first pass reads its keys there instead (an array that must stay as it
// is) and each key's value is its index, so neither is copied first; va and
// vb must be given.  Scratch: slot kSlotSortHist (histograms, tile counters,
// status words).
template <typename K, typename V>
int device_radix_sort(apspie_context *ctx, K *ka, V *va, K *kb, V *vb, long long n, int bits,
                      bool *result_in_b, const K *kfirst = nullptr) {
  *result_in_b = false;
  if (!kfirst && (n <= 1 || bits <= 0)) return APSPIE_OK;
  if (kfirst && (n < 1 || bits < 1))
    return set_error(ctx, APSPIE_ERR_INVALID, "radix sort: %lld keys of %d bits", n, bits);
  const int npass = (bits + kRadixBits - 1) / kRadixBits;
  if (npass > kMaxPasses || n >= (1ll << 40))
    return set_error(ctx, APSPIE_ERR_OVERFLOW, "radix sort: %lld keys of %d bits", n, bits);
  if (n <= kSmallSortItems<K> * kSortThreads) {
    radix_small<K, V><<<1, kSortThreads, 0, ctx->stream>>>(kfirst ? kfirst : ka,
                                                           kfirst ? nullptr : va, kb, vb, (int)n,
                                                           npass);
    *result_in_b = true;
    return check_launch(ctx, "radix_small");
  }
  const long long tiles = (n + kSortTile - 1) / kSortTile;
  // [histograms: npass x 256 u64][tile counters: 8 x u32, padded; the
  // sort's give-up word at u32 15][status: tiles x 256 words]
  const size_t hist_bytes = sizeof(unsigned long long) * kMaxPasses * kRadix;
  const size_t head = hist_bytes + 64;
  const bool narrow = n < (1ll << 27);
  const size_t bytes = head + (narrow ? 4 : 8) * (size_t)tiles * kRadix;
  int *err = radix_sort_err(ctx);
  auto *ws = (unsigned char *)workspace(ctx, kSlotSortHist, bytes);
  if (!ws || !err) return APSPIE_ERR_OOM;
  auto *ghist = (unsigned long long *)ws;
  auto *counters = (unsigned *)(ws + hist_bytes);
  void *status = ws + head;
  cudaStream_t st = ctx->stream;
  // zero the histograms, counters and every status word
  cudaMemsetAsync(ws, 0, bytes, st);
  const int hgrid = (int)std::max(
      1ll, std::min((n + kSortThreads * kHistKeys - 1) / (kSortThreads * kHistKeys),
                    (long long)ctx->num_sms * 8));
  radix_histograms<K><<<hgrid, kSortThreads, 0, st>>>(kfirst ? kfirst : ka, n, npass, ghist);
  radix_digit_offsets<kRadix><<<1, kRadix, 0, st>>>(ghist, npass);
  int rc = check_launch(ctx, "radix_histograms", 2);
  if (rc) return rc;
  K *kin = ka, *kout = kb;
  V *vin = va, *vout = vb;
  const size_t vdyn = va ? sizeof(V) * kSortTile : 0;
  auto pass32 = radix_onesweep<K, V, unsigned>;
  auto pass64 = radix_onesweep<K, V, unsigned long long>;
  if (vdyn) {
    cudaFuncSetAttribute(pass32, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vdyn);
    cudaFuncSetAttribute(pass64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)vdyn);
  }
  for (int p = 0; p < npass; ++p) {
    const bool first = kfirst && p == 0;
    const K *kp = first ? kfirst : kin;
    const V *vp = first ? nullptr : vin;
    int *gave = (int *)(counters + 15);
    if (narrow)
      pass32<<<(unsigned)tiles, kSortThreads, vdyn, st>>>(kp, vp, kout, vout, n, p, ghist,
                                                          (unsigned *)status, counters + p, err,
                                                          gave);
    else
      pass64<<<(unsigned)tiles, kSortThreads, vdyn, st>>>(kp, vp, kout, vout, n, p, ghist,
                                                          (unsigned long long *)status,
                                                          counters + p, err, gave);
    rc = check_launch(ctx, "radix_onesweep");
    if (rc) return rc;
    std::swap(kin, kout);
    std::swap(vin, vout);
    *result_in_b = !*result_in_b;
  }
  return APSPIE_OK;
}

inline int bits_for(long long m) {
  int b = 0;
  while ((1ll << b) < m) ++b;
  return b;
}

}  // namespace apspie
