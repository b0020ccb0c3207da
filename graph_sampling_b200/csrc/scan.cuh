// Block-level exclusive scan + single-pass cross-tile prefix (decoupled look-back).
//
// Every kernel that turns per-item counts into output offsets (column degrees, fanouts,
// first-occurrence flags, surviving-edge flags) does it in ONE launch: a tile's CTA scans its own
// counts in shared memory, publishes the tile total, and warp 0 walks back over the predecessors'
// published words until it meets one that already carries an inclusive prefix.  This replaces the
// reference's "count kernel + cub::DeviceScan (two allocator calls) + blocking read of the total"
// sequence (src/cuda/slicing.cu:133-147, src/cuda/utils.h:17-28).
//
// Tiles are numbered by blockIdx.x and rely on CTAs being dispatched in index order, as every
// single-pass scan does.  The wait on a predecessor is bounded, so a lost predecessor can never hang the GPU: after
// TileState::max_polls polls the CTA marks the words it still waits for as lost (a compare-and-swap, so a word that was
// published meanwhile is used after all), records GSB_ERR_LOOKBACK_TIMEOUT and continues with prefix 0.  Words are published
// with a maximum, which a mark beats, so every tile behind a lost one finds it lost: the last tile, which knows the total and
// posts it to the host, can't take a sum for complete that another tile has given up on.  The kernels that follow see
// CNT_ABORT and CNT_LOST and do not use such a scan.
#pragma once
#include "common.cuh"

namespace gsb {

__device__ __forceinline__ u64 tile_word(uint32_t epoch, uint32_t flag, i64 value) {
  return ((u64)(epoch & kEpochMask) << 42) | ((u64)flag << 40) | ((u64)value & kValueMask);
}

constexpr uint32_t kTileLost = 3;

// A word of an older epoch is smaller, and so is an aggregate (1) than an inclusive prefix (2) and both than a mark (3).
__device__ __forceinline__ void tile_post(const TileState& ts, int tile, u64 word) {
  asm volatile("red.relaxed.gpu.global.max.u64 [%0], %1;" ::"l"(ts.words + tile), "l"(word) : "memory");
}

__device__ __forceinline__ u64 ld_volatile_u64(const u64* p) {
  u64 v;
  asm volatile("ld.volatile.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ void st_volatile_u64(u64* p, u64 v) {
  asm volatile("st.volatile.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

__device__ __forceinline__ void raise_error(i64* counters, int code, i64 info) {
  if (atomicCAS((u64*)&counters[CNT_ERROR], 0ull, (u64)(i64)code) == 0ull) counters[CNT_ERROR_INFO] = info;
  __threadfence();  // recorded before anything this thread publishes afterwards (mail_post reads the flag)
}

// Posts `value` to slot `slot` of a mailbox together with the error flag as it stands.  Called by one thread that knows
// the final value; errors that can still be raised after that point are found by the next status check, as they are
// when nobody waits.
__device__ __forceinline__ void mail_post(const Mail& m, int slot, i64 value, const i64* counters) {
  if (!m.word) return;
  const u64 err = ld_volatile_u64((const u64*)counters + CNT_ERROR) != 0ull ? 1ull : 0ull;
  st_volatile_u64(m.word + slot, m.tag | (err << kMailErrorBit) | ((u64)value & kMailValueMask));
}

// The two halves of tile_exclusive_prefix, for kernels that have independent work to put between them: a tile first
// PUBLISHES its aggregate (its successors can then add it up without waiting for this tile's own prefix), issues
// whatever loads it can, and only then RESOLVES its prefix — the wait for the predecessors overlaps those loads.
__device__ __forceinline__ void tile_publish_aggregate(const TileState& ts, int tile, i64 aggregate) {
  if ((threadIdx.x & 31) == 0) tile_post(ts, tile, tile_word(ts.epoch, tile == 0 ? 2 : 1, aggregate));
}

__device__ __forceinline__ i64 tile_resolve_prefix(const TileState& ts, int tile, i64 aggregate, bool* lost = nullptr);

// Called by all 32 lanes of warp 0 of the CTA that owns `tile`.  Returns the sum of the
// aggregates of tiles [0, tile) and publishes this tile's inclusive prefix.  *lost: a wait was given up, the prefix is 0.
__device__ __forceinline__ i64 tile_exclusive_prefix(const TileState& ts, int tile, i64 aggregate, bool* lost = nullptr) {
  tile_publish_aggregate(ts, tile, aggregate);
  return tile_resolve_prefix(ts, tile, aggregate, lost);
}

// Groups of 32 predecessors that a look-back reads at a time, nearest first.  While nobody has an inclusive prefix yet a tile can
// only add up what it reads, and with n words read per step the first n k^2 / 2 tiles are done after k steps: the last of 4 219
// tiles (135 000 sampled columns) after eight round trips to L2, with one group after sixteen (24.3 -> 22.6 us for the sampler).
// With eight groups it takes 21.3 to 22.8 from run to run, but the 117 000 tiles of 60 M columns by windows are 0.5 % slower; with
// sixteen the reads themselves get in the way (28.2, and 6.5 %).
constexpr int kLookGroups = 4;

__device__ __forceinline__ i64 tile_resolve_prefix(const TileState& ts, int tile, i64 aggregate, bool* lost) {
  const int lane = threadIdx.x & 31;
  if (lost) *lost = false;
  if (tile == 0) return 0;
  i64 exclusive = 0;  // the lane's part of it
  int idx = tile - 1;  // nearest predecessor examined by lane 0
  const uint32_t ep = ts.epoch & kEpochMask;
  auto published = [ep](u64 w) { return ((uint32_t)(w >> 42) == ep) && (((w >> 40) & 3ull) != 0ull); };
  bool found = false;
  while (!found) {
    u64 w[kLookGroups];
    int polls = 0;
    bool ready;
    do {
#pragma unroll
      for (int q = 0; q < kLookGroups; ++q) {
        const int my = idx - q * 32 - lane;
        w[q] = my >= 0 ? ld_volatile_u64(&ts.words[my]) : tile_word(ep, 2, 0);  // before tile 0: inclusive prefix 0
      }
      ready = published(w[0]);
      if (__all_sync(0xffffffffu, ready)) break;
      if (++polls > ts.max_polls && !ready) {  // at most as often as the word changes: three times
        const u64 mark = tile_word(ep, kTileLost, 0);
        if (atomicCAS(&ts.words[idx - lane], w[0], mark) == w[0]) w[0] = mark;
      }
      __nanosleep(20);
    } while (true);
#pragma unroll
    for (int q = 0; q < kLookGroups; ++q) {
      // the groups behind the first are taken as far as they are there
      if (found || (q > 0 && !__all_sync(0xffffffffu, published(w[q])))) break;
      const uint32_t flag = (uint32_t)((w[q] >> 40) & 3ull);
      if (__any_sync(0xffffffffu, flag == kTileLost)) {  // no tile behind a lost one has an inclusive prefix
        if (lane == 0) {
          raise_error(ts.counters, GSB_ERR_LOOKBACK_TIMEOUT, tile);
          ts.counters[CNT_ABORT] = ts.counters[CNT_LOST] = 1;
          tile_post(ts, tile, tile_word(ep, kTileLost, 0));
        }
        if (lost) *lost = true;
        return 0;
      }
      const uint32_t full = __ballot_sync(0xffffffffu, flag == 2u);
      found = full != 0;
      if (!found || lane < __ffs(full)) exclusive += (i64)(w[q] & kValueMask);  // up to the nearest inclusive prefix
      idx -= 32;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) exclusive += __shfl_xor_sync(0xffffffffu, exclusive, o);
  if (lane == 0) tile_post(ts, tile, tile_word(ts.epoch, 2, exclusive + aggregate));
  return exclusive;
}

// Exclusive scan of one value per thread across a CTA of THREADS threads (multiple of 32, <= 1024).
// Returns the thread's exclusive prefix; *total receives the CTA sum (valid in every thread).
// `smem` must hold 33 i64.  Contains __syncthreads: call from all threads.
template <int THREADS>
__device__ __forceinline__ i64 block_exclusive_scan(i64 v, i64* smem, i64* total) {
  constexpr int WARPS = THREADS / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  i64 inc = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const i64 t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  if (lane == 31) smem[warp] = inc;
  __syncthreads();
  if (warp == 0) {
    i64 w = lane < WARPS ? smem[lane] : 0;
    i64 winc = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const i64 t = __shfl_up_sync(0xffffffffu, winc, o);
      if (lane >= o) winc += t;
    }
    if (lane < WARPS) smem[lane] = winc - w;
    if (lane == 31) smem[32] = winc;
  }
  __syncthreads();
  const i64 excl = smem[warp] + inc - v;
  *total = smem[32];
  __syncthreads();  // smem may be reused by the caller
  return excl;
}

}  // namespace gsb
