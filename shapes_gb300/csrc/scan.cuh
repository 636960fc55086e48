/*
 * The exclusive scan of the step (row, slot and bucket counts), and the first
 * statement of kernels that are launched chained.
 */
#pragma once
#include <cstdint>

namespace shapes {

/* First statement of every kernel that launch_chained launches: nothing before it
 * reads or writes memory.  Waits until the kernels before are complete and their
 * writes visible (at once in a kernel launched plainly); chained_entry also lets
 * the next one's blocks take their places as soon as all of this one's have. */
__device__ __forceinline__ void chained_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void chained_entry() {
  chained_wait();
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

constexpr int kScanThreads = 1024;
constexpr int kScanPerThread = 8;
constexpr int kScanTile = kScanThreads * kScanPerThread;

/* What a scan keeps between launches: a word per tile, {value, epoch << 2 |
 * kind}, and {epoch, tiles taken, tiles done}.  The epoch tells this launch's
 * words from older ones; the last block to finish raises it and clears the
 * counts, so that nothing has to be reset before the next scan (the launches
 * that share a state follow one another on a stream). */
struct ScanState {
  unsigned long long* tile; /* zero (kind 0: no word) to begin with */
  uint32_t* ctl;            /* [3] */
  int tiles;
};
constexpr uint32_t kTileSum = 1, kTilePrefix = 2;
constexpr long long kScanPollLimit = 1ll << 24;

/* A scan's sums stop here.  65,537 bodies on one spot have 2^31 pairs: a wrapped
 * sum would pass for one that fits the buffers, and rows laid out from it would
 * start below zero.  The limit is beyond every buffer's capacity, so a sum that
 * reached it counts as an overflow, and 2^24 below the largest int, so that a
 * row's start plus a position in the row (fewer than 2^20) does not wrap either.
 * Stopping is associative, so the order in which sums are formed does not matter. */
constexpr uint32_t kScanMost = 0x7f000000u;
__host__ __device__ __forceinline__ int32_t scan_sum(int32_t a, int32_t b) { /* neither above kScanMost */
  const uint32_t t = (uint32_t)a + (uint32_t)b;
  return (int32_t)(t < kScanMost ? t : kScanMost);
}

/* The same over the lanes of a warp: 16 bits at a time, whose sums over 32 lanes stay below 2^21. */
__device__ __forceinline__ int32_t scan_sum_lanes(int32_t x) {
  const uint32_t lo = __reduce_add_sync(0xffffffffu, (uint32_t)x & 0xffffu);
  const uint32_t hi = __reduce_add_sync(0xffffffffu, (uint32_t)x >> 16) + (lo >> 16);
  return (int32_t)(hi < kScanMost >> 16 ? hi << 16 | (lo & 0xffffu) : kScanMost);
}

/* out[k] = exclusive prefix of in[0..n), out[n] = total, in one launch (n read
 * from *n_dev when non-null, capped at n_cap), sums stopping at kScanMost;
 * elements below 2^23, so that a warp's fit an int: decoupled look-back (Merrill and
 * Garland, "Single-pass Parallel Prefix Scan with Decoupled Look-back", 2016).
 * Tiles are taken in order from a counter, so a block waits only for blocks
 * that already run; the waits are bounded.  in and out start on 16 bytes.  Tiles
 * of 8192, so that the chain of prefixes is short: a million elements took 37 us
 * in tiles of 2048.  clear: in is left zeroed.  total:
 * gets out[n], and where that exceeds total_cap the overflow counter gets
 * overflow_bit.  As three launches (tile sums, their scan, the prefixes) a scan
 * of 50 to 500 thousand elements took 11 to 13 us. */
__global__ void __launch_bounds__(kScanThreads) k_scan(int32_t* in, int n_cap, const unsigned long long* n_dev,
                                                       ScanState st, int32_t* out, int clear,
                                                       unsigned long long* total, int total_cap,
                                                       unsigned long long* overflow, unsigned overflow_bit,
                                                       unsigned long long* err) {
  chained_entry();
  __shared__ int32_t s_scan[kScanThreads / 32];
  __shared__ int32_t s_prefix, s_tile;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int n = n_dev ? (int)min((unsigned long long)n_cap, *n_dev) : n_cap;
  const int tiles = n / kScanTile + 1; /* the last one also holds out[n] */
  const uint32_t epoch = __ldcg(st.ctl);
  for (;;) {
    if (tid == 0) s_tile = (int)atomicAdd(st.ctl + 1, 1u);
    __syncthreads();
    const int tile = s_tile;
    if (tile >= tiles) break;
    /* per-thread serial over a contiguous run, then block scan of run totals */
    const int r0 = tile * kScanTile + tid * kScanPerThread;
    int32_t v[kScanPerThread] = {};
    if (r0 + kScanPerThread <= n) {
#pragma unroll
      for (int k = 0; k < kScanPerThread; k += 4) {
        const int4 x = *reinterpret_cast<const int4*>(in + r0 + k);
        v[k] = x.x;
        v[k + 1] = x.y;
        v[k + 2] = x.z;
        v[k + 3] = x.w;
        if (clear) *reinterpret_cast<int4*>(in + r0 + k) = make_int4(0, 0, 0, 0);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kScanPerThread; ++k)
        if (r0 + k < n) {
          v[k] = in[r0 + k];
          if (clear) in[r0 + k] = 0;
        }
    }
    int run = 0;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) run += v[k];
    int incl = run;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_scan[wid] = incl;
    __syncthreads();
    if (wid == 0) {
      int ws = s_scan[lane]; /* as many warps as lanes */
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, ws, o);
        if (lane >= o) ws = scan_sum(ws, y);
      }
      const int sum = __shfl_sync(0xffffffffu, ws, 31);
      s_scan[lane] = ws;
      auto publish = [&](int value, uint32_t kind) {
        asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(st.tile + tile),
                     "l"((unsigned long long)(uint32_t)value | (unsigned long long)(epoch << 2 | kind) << 32)
                     : "memory");
      };
      int prefix = 0;
      if (tile > 0) {
        if (lane == 0) publish(sum, kTileSum);
        long long polls = 0;
        for (int at = tile - 1;;) { /* 32 tiles before, nearest first */
          const int q = at - lane;
          unsigned long long word = (unsigned long long)(epoch << 2 | kTilePrefix) << 32; /* before the first: 0 */
          if (q >= 0) asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(word) : "l"(st.tile + q) : "memory");
          const uint32_t tag = (uint32_t)(word >> 32);
          const bool here = tag >> 2 == epoch && (tag & 3u) != 0;
          const unsigned known = __ballot_sync(0xffffffffu, here);
          const unsigned full = __ballot_sync(0xffffffffu, here && (tag & 3u) == kTilePrefix);
          /* the run of known tiles from the nearest on, up to the first with its whole prefix */
          const int usable = known == 0xffffffffu ? 32 : __ffs(~known) - 1;
          const int stop = full ? __ffs(full) - 1 : 32;
          const bool end = stop < usable;
          const int take = end ? stop + 1 : usable;
          prefix = scan_sum(prefix, scan_sum_lanes(lane < take ? (int32_t)(uint32_t)word : 0));
          if (end) break;
          at -= take;
          if (take == 0 && ++polls > kScanPollLimit) {
            if (lane == 0 && err) atomicOr(err, 1ull);
            break;
          }
        }
      }
      if (lane == 0) {
        const int upto = scan_sum(prefix, sum);
        publish(upto, kTilePrefix);
        s_prefix = prefix;
        if (tile == tiles - 1 && total) {
          *total = (unsigned long long)(uint32_t)upto;
          if (upto > total_cap) atomicOr(overflow, (unsigned long long)overflow_bit);
        }
      }
    }
    __syncthreads();
    int prefix = scan_sum(scan_sum(s_prefix, wid > 0 ? s_scan[wid - 1] : 0), incl - run);
    int32_t o[kScanPerThread];
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) {
      o[k] = prefix;
      prefix = scan_sum(prefix, v[k]);
    }
    if (r0 + kScanPerThread <= n) {
#pragma unroll
      for (int k = 0; k < kScanPerThread; k += 4)
        *reinterpret_cast<int4*>(out + r0 + k) = make_int4(o[k], o[k + 1], o[k + 2], o[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < kScanPerThread; ++k)
        if (r0 + k <= n) out[r0 + k] = o[k];
    }
    __syncthreads();
  }
  if (tid == 0 && atomicAdd(st.ctl + 2, 1u) + 1 == gridDim.x) { /* every block is past its last tile */
    st.ctl[1] = 0;
    st.ctl[2] = 0;
    const uint32_t next = (epoch + 1) & 0x3fffffffu;
    if (next == 0) /* the words of 2^30 scans ago would pass for new ones */
      for (int k = 0; k < st.tiles; ++k) st.tile[k] = 0;
    st.ctl[0] = next;
  }
}

}  // namespace shapes
