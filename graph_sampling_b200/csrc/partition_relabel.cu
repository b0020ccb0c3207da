// Batched unique + relabel by partitioning: first occurrences are found in SHARED-MEMORY hash tables.
//
// The hash-region form (batch_relabel.cu) gives every minibatch a table region in global memory and pays two random
// L2 / DRAM accesses per item in its insert pass and one or two more in its compaction, whose look-back chain over
// tens of thousands of tiles is what that kernel mostly waits for.  Measured on a B200 (gsb_selftest_table_atomics),
// random 64-bit atomics on a CTA's own shared memory run at 4.7 G/s per SM (691 G/s on the whole GPU), ten times what
// the L2 path sustains (71 G/s; the hash-region insert reaches 64 G items/s), while atomics on a cluster's distributed
// shared memory reach only 29 - 33 G/s GPU-wide.  So the items of a minibatch are first PARTITIONED by a hash of their
// id into buckets small enough for one CTA's shared memory, and every bucket is resolved by one CTA on its own:
//
//   layout    per minibatch: item offset, number of buckets (items / kBucketTarget = 2 048, rounded up), first bucket;
//   count     a CTA takes 4 096 consecutive items, counts them per bucket in shared memory, adds its counts to the
//             bucket sizes (one global atomic per CTA and bucket).  In the one-call hop (gsb_sage_hop) the uniform
//             sampler does this counting itself while it holds the ids (slice_sample.cu, COUNT) — the buckets are then
//             laid out from the bound seeds x (1 + fanout) before it runs — and this pass is not launched;
//   scan      bucket sizes -> bucket starts (single pass; in the one-call hop part of k_part_after_sampler);
//   scatter   tiles of 2 048 or 8 192 items: sorted by bucket in shared memory, a range reserved per bucket with one global
//             atomic, whole runs of (id << 32 | position inside the minibatch) copied out — the order inside a bucket
//             does not matter, the table keeps the smallest position per id;
//   resolve   one CTA per bucket: the bucket's items stay in registers; position-min insert into a shared-memory
//             table (48 KB: ids and smallest positions as two 32-bit arrays, three slots per item where that fits, two
//             otherwise), then every item reads the first position of its id from the slot it ended in; they are
//             written in the bucket's order; a bucket with more items than the shared-memory table is sized
//             for (many repeats of a few hub ids, or an unlucky hash) uses a table in global memory of its own
//             instead, so nothing depends on luck;
//             With a bound on the ids, buckets can be classes of them instead: see k_part_resolve_classes;
//   rank      the first positions brought back into the order of the items, which the scatter pass told where they went (a
//             tile's share of a bucket is a run, so a CTA that takes the same tile reads whole sectors); bit vector of
//             the first occurrences (ref[item] == own position), prefix counts per 32 items, then one
//             pass that writes the frontier and every neighbour's position in it (see "ranking by bit vectors").
//
// Every pass over the items is coalesced except the 8-byte rank look-ups inside the minibatch's own window.  (While resolve
// wrote ref[item] itself, a sector per item, that scatter was two thirds of its time: 8.3 ms for 320 M items of 500 large
// minibatches, now 2.8 with 0.9 more in the first ranking pass and 0.2 in the scatter pass.)  All of these kernels are bound by instruction issue, not by memory, so their common
// case — a tile or warp whose items lie in ONE minibatch — runs on 32-bit positions with the minibatch's parameters
// in registers; a tile that straddles minibatches takes a general path per item (the counting pass handles the part
// of each minibatch in turn when they are few; doing the same in the scatter pass was measured: 64 instead of 46
// registers, 1.86 instead of 1.62 ms per 1 000 minibatches of the products-scale benchmark, whose tiles rarely straddle).  Results are identical to the other
// forms: first-occurrence order is defined by positions, not by the order in which anything is processed.
#include "batch_table.cuh"
#include "common.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kPartThreads = 256;
constexpr int kPartPerThread = 16;
constexpr int kPartTile = kPartThreads * kPartPerThread;        // items per CTA of the count pass
constexpr int scatter_smem(int tile, int window) { return tile * 8 + window * 8; }  // bytes of the scatter pass
// Buckets of one minibatch that a tile counts in shared memory: 256 serve minibatches of up to 524 288 items; calls with
// larger ones take the instantiations of 1 024 (2 097 152 items), whose arrays cost the narrow calls resident CTAs.
constexpr int kNarrowWindow = 256;
constexpr int kWideWindow = 1024;
constexpr u32 kNoBucket = 0xFFFFFFFFu;
constexpr int kResolveThreads = 256;
constexpr int kResolveAhead = 2;                         // items of a thread whose first probes are in flight together
constexpr int kResolvePer = 12;                          // items per thread of a bucket that fits shared memory
constexpr int kBucketSlots = 6144;                       // shared-memory table of a resolve CTA: 48 KB
constexpr int kBucketSmemItems = kBucketSlots / 2 - 16;  // largest bucket that fits it at two slots per item

struct PartLayout {
  BatchLayout L;       // region_off holds the first bucket of every minibatch ([G + 1], last = bucket count)
  u32* bucket_count;   // [buckets + 1]
  u32* bucket_start;   // [buckets + 1]
  u32* bucket_cursor;  // [buckets]
  u64* bucketed;       // [items]   id << 32 | position inside the minibatch, grouped by bucket
  u32* found;          // [items]   in the same order: position inside the minibatch of the first occurrence of the id
  u32* ref;            // [items]   by item: where it lies in `bucketed`; from k_first_bits on what `found` says there
  u64* spill;          // tables of the buckets that do not fit shared memory: 2 x start + 32 x bucket
  u32 class_parts;     // buckets per minibatch when they are classes of ids (and one for those beyond), 0: buckets by hash
  u32 class_magic;     // see bucket_of_id
};

// Slot inside a bucket's table: a constant other than bucket_of_id's and one xor-shift round, so the ids of one
// bucket — which share the high bits of that product — still spread over the whole table.
__device__ __forceinline__ u32 slot_of_id(u32 id, u32 size) {
  u32 x = id * 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  x ^= x >> 16;
  return __umulhi(x, size);
}

// Parameters of the minibatch that a tile starts in, reduced to what the per-item work needs.
struct TileBatch {
  const i64* seeds;  // seeds[lc] for lc < ns
  const i64* edges;  // edges[lc] for lc >= ns (pointer already shifted by -ns)
  u32 ns;            // seeds of the minibatch
  u32 items;         // items of the minibatch
  u32 bucket0;       // its first bucket
  u32 parts;         // its bucket count
};

__device__ __forceinline__ TileBatch tile_batch(const BatchLayout& L, const BatchUniform& u) {
  TileBatch t;
  t.seeds = L.seeds + u.seeds_begin;
  t.edges = L.indices + u.edges_begin - u.num_seeds;
  t.ns = (u32)u.num_seeds;
  t.items = (u32)(u.next_begin - u.begin);
  const i64 b0 = __ldg(L.region_off + u.batch);
  t.bucket0 = (u32)b0;
  t.parts = (u32)(__ldg(L.region_off + u.batch + 1) - b0);
  return t;
}

__device__ __forceinline__ i64 tile_item(const TileBatch& t, u32 lc) {
  return __ldg(lc < t.ns ? t.seeds + lc : t.edges + lc);
}

// Minibatch of item g, searched by a whole warp (g must be the same in all 32 lanes, which must be converged): every
// round the lanes probe 32 evenly spaced offsets and a ballot narrows the range 32-fold — two rounds for up to 1 024
// minibatches instead of the ten dependent loads of a binary search, which cost the streaming kernels below more
// instructions than a warp's items.
__device__ __forceinline__ i64 batch_of_warp(const i64* __restrict__ off, i64 G, i64 g) {
  const i64 lane = threadIdx.x & 31;
  i64 lo = 0, end = G;  // the answer lies in [lo, end)
  while (end - lo > 1) {
    const i64 step = (end - lo + 31) >> 5;
    const i64 idx = lo + (lane + 1) * step;
    const bool le = idx < end && __ldg(off + idx) <= g;  // offsets do not decrease: true for a prefix of the lanes
    const i64 hits = __popc(__ballot_sync(0xffffffffu, le));
    lo += hits * step;
    end = min(end, lo + step);
  }
  return lo;
}

// General path: item g of the call, wherever it lies.
struct Located {
  i64 node;
  u32 lc;      // position inside its minibatch (seeds first)
  u32 bucket;  // global bucket number
};
__device__ __forceinline__ Located locate(const BatchLayout& L, i64 g, u32 magic) {
  const BatchUniform v = load_batch<false>(L, L.item_off, batch_of(L.item_off, L.G, g));
  const TileBatch t = tile_batch(L, v);
  Located r;
  r.lc = (u32)(g - v.begin);
  r.node = tile_item(t, r.lc);
  r.bucket = t.bucket0 + bucket_of_id((u32)r.node, t.parts, magic);
  return r;
}

constexpr int kMaxSegments = 8;  // minibatches a tile may touch and still be handled segment by segment

template <int kWindow, bool CLASSES>
__global__ void __launch_bounds__(kPartThreads) k_part_count(PartLayout P, i64 n_bound, i64* counters) {
  __shared__ u32 s_cnt[kWindow];
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = P.L;
  const i64 n = min(L.item_off[L.G], n_bound);
  const i64 tile_base = (i64)blockIdx.x * kPartTile;
  if (tile_base >= n) return;
  const i64 tile_end = min(n, tile_base + kPartTile);
  const i64 b_first = batch_of_warp(L.item_off, L.G, tile_base);
  const i64 b_last = batch_of_warp(L.item_off, L.G, tile_end - 1);
  if (b_last - b_first >= kMaxSegments) {  // a tile over many small minibatches: every item on its own
    for (i64 g = tile_base + threadIdx.x; g < tile_end; g += kPartThreads) {
      const Located it = locate(L, g, P.class_magic);
      if (!valid_id(it.node)) continue;  // never bucketed; reported by the scatter pass
      atomicAdd(P.bucket_count + it.bucket, 1u);
    }
    return;
  }
  // the part of every minibatch that lies in the tile, one after the other
  for (i64 b = b_first; b <= b_last; ++b) {
    const BatchUniform u = load_batch<false>(L, L.item_off, b);
    const i64 seg_begin = max(tile_base, u.begin), seg_end = min(tile_end, u.next_begin);
    if (seg_end <= seg_begin) continue;  // an empty minibatch
    const TileBatch t = tile_batch(L, u);
    const u32 lc0 = (u32)(seg_begin - u.begin), here = (u32)(seg_end - seg_begin);
    if (t.parts > (u32)kWindow) {  // more buckets than the shared-memory window holds
      for (u32 i = threadIdx.x; i < here; i += kPartThreads) {
        const i64 node = tile_item(t, lc0 + i);
        if (!valid_id(node)) continue;
        const u32 k = t.bucket0 + bucket_of_id<CLASSES>((u32)node, t.parts, P.class_magic);
        atomicAdd(P.bucket_count + k, 1u);
      }
      continue;
    }
    __syncthreads();  // the previous segment's counts are flushed
    for (int i = threadIdx.x; i < kWindow; i += kPartThreads) s_cnt[i] = 0;
    // ids first (independent loads), then the shared-memory atomics
    i64 node[kPartPerThread];
#pragma unroll
    for (int q = 0; q < kPartPerThread; ++q) {
      const u32 i = q * kPartThreads + threadIdx.x;
      node[q] = i < here ? tile_item(t, lc0 + i) : -1;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kPartPerThread; ++q)
      if (valid_id(node[q])) atomicAdd(&s_cnt[bucket_of_id<CLASSES>((u32)node[q], t.parts, P.class_magic)], 1u);  // the others: scatter pass
    __syncthreads();
    for (u32 i = threadIdx.x; i < t.parts; i += kPartThreads) {
      if (s_cnt[i] != 0) atomicAdd(P.bucket_count + t.bucket0 + i, s_cnt[i]);
    }
  }
}

// bucket sizes -> bucket starts, cursors cleared: single pass with look-back over tiles of 2 048 buckets (one CTA that walked
// all buckets took 250 us for the 130 000 of 500 large minibatches)
constexpr int kScanThreads = 256;
constexpr int kScanPer = 8;
constexpr int kScanTile = kScanThreads * kScanPer;
// Up to here the one CTA that runs between sampler and scatter pass scans the buckets too (43 000 took it 58 us; k_part_scan 9).
constexpr i64 kScanAlongBuckets = 8192;

__global__ void __launch_bounds__(kScanThreads) k_part_scan(PartLayout P, i64* counters, TileState ts) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  if (counters[CNT_ABORT] != 0) return;
  const i64 buckets = P.L.region_off[P.L.G];
  const int tile = blockIdx.x;
  const i64 first = (i64)tile * kScanTile + (i64)threadIdx.x * kScanPer;
  if ((i64)tile * kScanTile >= buckets && !(buckets == 0 && tile == 0)) return;
  u32 c[kScanPer];
  i64 sum = 0;
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    c[j] = first + j < buckets ? P.bucket_count[first + j] : 0u;
    sum += c[j];
  }
  i64 total;
  const i64 excl = block_exclusive_scan<kScanThreads>(sum, s_scan, &total);
  if (threadIdx.x < 32) {
    const i64 prefix = tile_exclusive_prefix(ts, tile, total);
    if (threadIdx.x == 0) s_base = prefix;
  }
  __syncthreads();
  i64 run = s_base + excl;
#pragma unroll
  for (int j = 0; j < kScanPer; ++j) {
    if (first + j < buckets) {
      P.bucket_start[first + j] = (u32)run;
      P.bucket_cursor[first + j] = 0u;
    }
    run += c[j];
  }
  if ((i64)(tile + 1) * kScanTile >= buckets && threadIdx.x == 0) P.bucket_start[buckets] = (u32)(s_base + total);
}

// The one-call hop, between its sampler and the scatter pass — one CTA does what three small launches did: the edge
// offset of every minibatch (the sampled block's offset at the minibatch's first seed), the item offsets, the abort
// check against the caller's bounds, and the scan of the bucket sizes that the sampler counted.
__global__ void __launch_bounds__(1024) k_part_after_sampler(PartLayout P, const i64* __restrict__ sub_indptr, i64 S,
                                                             i64 edges_bound, i64* indices_ptr, int scan, i64* counters) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_carry;
  __shared__ int s_abort;
  const BatchLayout& L = P.L;
  const i64 G = L.G;
  if (threadIdx.x == 0) {
    const i64 ns = L.seeds_ptr[G];
    const i64 ne = sub_indptr[max((i64)0, min(ns, S))];
    const bool over = ns > S || ne > edges_bound || ns < 0 || ne < 0;
    if (over) {
      counters[CNT_ABORT] = 1;
      raise_error(counters, GSB_ERR_CAPACITY, ns > S ? ns : ne);
    }
    s_abort = counters[CNT_ABORT] != 0;
    s_carry = 0;
  }
  __syncthreads();
  for (i64 b = threadIdx.x; b <= G; b += 1024) {
    const i64 sp = L.seeds_ptr[b];
    const i64 ip = sub_indptr[max((i64)0, min(sp, S))];
    indices_ptr[b] = ip;
    L.item_off[b] = sp + ip;
  }
  if (s_abort || !scan) return;
  const i64 buckets = L.region_off[G];
  constexpr int kPer = 8;
  for (i64 base = 0; base < buckets; base += 1024 * kPer) {
    const i64 first = base + (i64)threadIdx.x * kPer;
    u32 c[kPer];
    i64 sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      c[j] = first + j < buckets ? P.bucket_count[first + j] : 0u;
      sum += c[j];
    }
    i64 total;
    i64 run = s_carry + block_exclusive_scan<1024>(sum, s_scan, &total);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      if (first + j < buckets) {
        P.bucket_start[first + j] = (u32)run;
        P.bucket_cursor[first + j] = 0u;
      }
      run += c[j];
    }
    __syncthreads();
    if (threadIdx.x == 0) s_carry += total;
    __syncthreads();
  }
  if (threadIdx.x == 0) P.bucket_start[buckets] = (u32)s_carry;
}

// A tile's items are first sorted by bucket in shared memory (their rank inside the tile's share of a bucket is what
// the counting atomic returned), so the copy to global memory writes whole runs of consecutive words.  The bucket of a
// staged item is computed from its id again instead of being kept beside it.
// THREADS x PER items per tile.  Tiles of 2 048 suit minibatches of some ten thousand items (a tile that straddles
// minibatches takes the per-item path); with hundreds of buckets per minibatch such a tile reserves a range — a global
// atomic, on a cursor that every other tile of the minibatch wants too — for every five items, so large minibatches take
// tiles of 8 192, two of whose CTAs are resident per SM.  That costs 68 bytes of spilled registers a thread (with the 83
// registers the compiler takes of its own accord one CTA is resident, and its barriers leave the SM idle: 3.1 against 2.1 ms for
// 270 M items; 1 024 threads with half the items each 2.8, tiles of 4 096 2.7).
template <int WINDOW, int THREADS, int PER, bool CLASSES>
__global__ void __launch_bounds__(THREADS, THREADS == 512 ? 2 : 1) k_part_scatter(PartLayout P, i64 n_bound, i64* counters) {
  constexpr int kTile = THREADS * PER;
  constexpr int kPer = WINDOW / THREADS > 0 ? WINDOW / THREADS : 1;  // consecutive window entries per thread in the scan
  extern __shared__ __align__(16) u64 s_stage[];                     // [kTile] items, then [WINDOW] two arrays
  u32* s_cnt = reinterpret_cast<u32*>(s_stage + kTile);              // counts, then where the bucket's run starts in the tile
  u32* s_delta = s_cnt + WINDOW;                                     // where it starts in the bucket array minus that
  __shared__ i64 s_scan[33];
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = P.L;
  const i64 n = min(L.item_off[L.G], n_bound);
  const i64 tile_base = (i64)blockIdx.x * kTile;
  if (tile_base >= n) return;
  for (int i = threadIdx.x; i < WINDOW; i += THREADS) s_cnt[i] = 0;
  const BatchUniform u = load_batch<false>(L, L.item_off, batch_of_warp(L.item_off, L.G, tile_base));
  const TileBatch t = tile_batch(L, u);
  const u32 lc0 = (u32)(tile_base - u.begin);
  const u32 here = (u32)min((i64)kTile, n - tile_base);
  const bool uniform = (u64)lc0 + here <= (u64)t.items && t.parts <= (u32)WINDOW;
  if (!uniform) {  // a tile over several minibatches: every item straight to its place
    for (u32 i = threadIdx.x; i < here; i += THREADS) {
      const Located it = locate(L, tile_base + i, P.class_magic);
      if (!valid_id(it.node)) {  // never bucketed: marked for the ranking passes
        raise_error(counters, GSB_ERR_INDEX_RANGE, tile_base + i);
        P.ref[tile_base + i] = 0xFFFFFFFFu;
        continue;
      }
      const u32 at = __ldg(P.bucket_start + it.bucket) + atomicAdd(P.bucket_cursor + it.bucket, 1u);
      P.bucketed[at] = ((u64)it.node << 32) | (u64)it.lc;
      P.ref[tile_base + i] = at;
    }
    return;
  }
  i64 node[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const u32 i = q * THREADS + threadIdx.x;
    node[q] = i < here ? tile_item(t, lc0 + i) : -1;
  }
  __syncthreads();
  u32 id[PER], where[PER];  // where: bucket (inside the minibatch) << 16 | rank inside the tile's share of it
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    where[q] = kNoBucket;
    id[q] = (u32)node[q];
    if (!valid_id(node[q])) {
      if (q * THREADS + threadIdx.x < here) {  // never bucketed: marked for the ranking passes
        raise_error(counters, GSB_ERR_INDEX_RANGE, tile_base + q * THREADS + threadIdx.x);
        P.ref[tile_base + q * THREADS + threadIdx.x] = 0xFFFFFFFFu;
      }
      continue;
    }
    const u32 w = bucket_of_id<CLASSES>(id[q], t.parts, P.class_magic);
    where[q] = (w << 16) | atomicAdd(&s_cnt[w], 1u);  // at most 8 192 items per tile: the rank fits 16 bits
  }
  __syncthreads();
  u32 staged;
  {
    u32 c[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int w = threadIdx.x * kPer + j;
      c[j] = w < WINDOW ? s_cnt[w] : 0;
      sum += c[j];
    }
    // the reservations are in flight during the scan
    u32 base[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const u32 w = t.bucket0 + threadIdx.x * kPer + j;
      base[j] = 0;
      if (c[j] != 0) base[j] = __ldg(P.bucket_start + w) + atomicAdd(P.bucket_cursor + w, c[j]);
    }
    i64 total;
    u32 run = (u32)block_exclusive_scan<THREADS>((i64)sum, s_scan, &total);
    staged = (u32)total;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int w = threadIdx.x * kPer + j;
      if (w < WINDOW) {
        s_cnt[w] = run;
        s_delta[w] = base[j] - run;
      }
      run += c[j];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (where[q] == kNoBucket) continue;
    const u32 i = q * THREADS + threadIdx.x, staged_at = s_cnt[where[q] >> 16] + (where[q] & 0xFFFFu);
    s_stage[staged_at] = ((u64)id[q] << 32) | (u64)(lc0 + i);
    P.ref[tile_base + i] = s_delta[where[q] >> 16] + staged_at;
  }
  __syncthreads();
  for (u32 i = threadIdx.x; i < staged; i += THREADS) {
    const u64 w = s_stage[i];
    P.bucketed[s_delta[bucket_of_id<CLASSES>((u32)(w >> 32), t.parts, P.class_magic)] + i] = w;
  }
}

// ---- one CTA per bucket ---------------------------------------------------------------------------------------
// Position-min insert; returns the slot the id lives in.  `table` may be shared or global memory.
__device__ __forceinline__ u32 table_insert_min(u64* table, u32 size, u32 h, u64 mine) {
  const u32 id = (u32)(mine >> 32);
  for (u32 probe = 0; probe < size; ++probe) {
    u64 w = *(volatile u64*)(table + h);
    if (w == kEmptyWord) {
      const u64 old = atomicCAS(table + h, kEmptyWord, mine);
      if (old == kEmptyWord) return h;
      w = old;
    }
    if ((u32)(w >> 32) == id) {
      if (w > mine) atomicMin(table + h, mine);
      return h;
    }
    h = h + 1 == size ? 0 : h + 1;
  }
  return 0;  // cannot happen: the table has more slots than the bucket has items
}

// A bucket that does not fit shared memory: a table of its own in global memory, by a whole CTA.
__device__ __noinline__ void resolve_in_memory(const u64* items, u32 n, u64* table, u32* found) {
  const u32 size = 2 * n + 32;
  __syncthreads();
  for (u32 i = threadIdx.x; i < size; i += blockDim.x) table[i] = kEmptyWord;
  __syncthreads();
  for (u32 j = threadIdx.x; j < n; j += blockDim.x) {
    const u64 w = __ldg(items + j);
    table_insert_min(table, size, slot_of_id((u32)(w >> 32), size), w);
  }
  __syncthreads();
  for (u32 j = threadIdx.x; j < n; j += blockDim.x) {
    const u64 w = __ldg(items + j);
    const u32 id = (u32)(w >> 32);
    u32 h = slot_of_id(id, size), first = 0xFFFFFFFFu;
    for (u32 probe = 0; probe < size; ++probe) {
      const u64 x = __ldcg(table + h);
      if ((u32)(x >> 32) == id) {
        first = (u32)x;
        break;
      }
      if (x == kEmptyWord) break;
      h = h + 1 == size ? 0 : h + 1;
    }
    found[j] = first;
  }
}

// Shared-memory table as two 32-bit arrays, ids and smallest positions: the probe loop is a 32-bit load and two compares per
// step, and both atomics are native 32-bit shared-memory operations.
// Probing costs a tenth of the kernel and the position minimum nothing that can be measured.  All twelve items of a thread probing side by side with a compare-and-swap per round was slower (3.8 against
// 2.4 ms per launch of an earlier form): without the read in front of it every repeat of a frequent id is an atomic on the same word.
// Measured and not kept: five CTAs per SM instead of four (40 KB tables of 2.5 slots per item, 48 registers): 2.61
// against 2.62 ms per 1 000 minibatches — the kernel is not short of resident warps.
__global__ void __launch_bounds__(kResolveThreads, 4) k_part_resolve(PartLayout P, i64* counters) {
  extern __shared__ __align__(16) u64 s_table[];
  static_assert(kResolvePer * kResolveThreads >= kBucketSmemItems, "a bucket that fits the table fits the registers");
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = P.L;
  const u32 buckets = (u32)L.region_off[L.G];
  for (u32 k = blockIdx.x; k < buckets; k += gridDim.x) {
    const u32 start = P.bucket_start[k];
    const u32 n = P.bucket_start[k + 1] - start;
    if (n == 0) continue;
    u32* found = P.found + start;
    const u64* items = P.bucketed + start;
    if (n <= (u32)kBucketSmemItems) {
      // three slots per item where the table allows it: the lanes of a warp leave the probe loop together more often
      const u32 size = min(3 * n + 32, (u32)kBucketSlots) & ~1u;
      // the bucket's items stay in registers for both passes; their loads are in flight while the table is cleared
      u64 w[kResolvePer];
#pragma unroll
      for (int q = 0; q < kResolvePer; ++q) {
        const u32 j = q * kResolveThreads + threadIdx.x;
        w[q] = j < n ? __ldg(items + j) : kEmptyWord;
      }
      __syncthreads();  // the previous bucket's look-ups are done
      u32* keys = reinterpret_cast<u32*>(s_table);  // [size] ids, then [size] smallest positions; size is even
      u32* first = keys + size;
      {
        uint4* t4 = reinterpret_cast<uint4*>(s_table);
        const uint4 e = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
        for (u32 i = threadIdx.x; i < size / 2; i += kResolveThreads) t4[i] = e;
      }
      __syncthreads();
      u32 slot[kResolvePer];
#pragma unroll
      for (int q0 = 0; q0 < kResolvePer; q0 += kResolveAhead) {
        if ((u32)(q0 * kResolveThreads) >= n) break;  // uniform
        u32 seen[kResolveAhead];
#pragma unroll
        for (int q = 0; q < kResolveAhead; ++q) {
          slot[q0 + q] = slot_of_id((u32)(w[q0 + q] >> 32), size);
          seen[q] = *(volatile u32*)(keys + slot[q0 + q]);
        }
#pragma unroll
        for (int q = 0; q < kResolveAhead; ++q)
          if (seen[q] == 0xFFFFFFFFu && w[q0 + q] != kEmptyWord)
            seen[q] = atomicCAS(keys + slot[q0 + q], 0xFFFFFFFFu, (u32)(w[q0 + q] >> 32));  // ids are below 2^32 - 1
#pragma unroll
        for (int q = 0; q < kResolveAhead; ++q) {
          if (w[q0 + q] == kEmptyWord) continue;
          const u32 id = (u32)(w[q0 + q] >> 32);
          u32 k = seen[q], h = slot[q0 + q];
          while (k != 0xFFFFFFFFu && k != id) {  // ends: the table has more slots than the bucket has items
            h = h + 1 == size ? 0 : h + 1;
            k = *(volatile u32*)(keys + h);
            if (k == 0xFFFFFFFFu) k = atomicCAS(keys + h, 0xFFFFFFFFu, id);
          }
          slot[q0 + q] = h;
          atomicMin(first + h, (u32)w[q0 + q]);
        }
      }
      __syncthreads();
      u32 ref_of[kResolvePer];
#pragma unroll
      for (int q = 0; q < kResolvePer; ++q)
        if ((u32)(q * kResolveThreads) < n) ref_of[q] = first[slot[q]];
#pragma unroll
      for (int q = 0; q < kResolvePer; ++q)
        if ((u32)(q * kResolveThreads) < n && w[q] != kEmptyWord) found[q * kResolveThreads + threadIdx.x] = ref_of[q];
      continue;
    }
    resolve_in_memory(items, n, P.spill + 2 * (u64)start + 32 * (u64)k, found);  // many repeats of a few ids
  }
}

// Buckets that are classes of ids, those with the same remainder by a prime: the table is addressed by the quotient, so an item is
// one reduction and one read in shared memory, without ids to compare and without probes.  Classes and not ranges of neighbouring
// ids, because a graph numbered by degree, or as a crawler met it, has most neighbours in a few ranges, and the CTA with such a range
// kept the others waiting: 6 M items of 7 minibatches over 2.45 M nodes by a power law, whole call, hashed buckets 196 us, ranges 343
// numbered by degree and 164 scattered, classes 166 either way.
// Between HBM (12 bytes an item; half of the copy bandwidth) and the latency of a bucket's load, clear, reduce and read, of which an
// SM has three in flight: 500 M items of 500 minibatches in three hops, hashed / classes: this pass 2.82 / 1.50 ms, the scatter
// pass, whose runs are longer, 2.64 / 2.45, counting 0.67 / 0.72.
constexpr int kClassThreads = 512;
constexpr int kClassPer = 12;  // items of a thread that stay in registers

__global__ void __launch_bounds__(kClassThreads, 3) k_part_resolve_classes(PartLayout P, i64* counters) {
  extern __shared__ __align__(16) u32 s_first[];  // [kClassSlots] smallest position of every id
  if (counters[CNT_ABORT] != 0) return;
  const u32 buckets = (u32)P.L.region_off[P.L.G];
  for (u32 k = blockIdx.x; k < buckets; k += gridDim.x) {
    const u32 start = P.bucket_start[k], n = P.bucket_start[k + 1] - start;
    if (n == 0) continue;
    if (k % P.class_parts == P.class_parts - 1) {  // ids beyond the bound
      resolve_in_memory(P.bucketed + start, n, P.spill + 2 * (u64)start + 32 * (u64)k, P.found + start);
      continue;
    }
    const u64* items = P.bucketed + start;
    u32* found = P.found + start;
    if (k + gridDim.x < buckets) {  // the next bucket's items on their way to L2
      const u32 at = P.bucket_start[k + gridDim.x], end = P.bucket_start[k + gridDim.x + 1];
      for (u32 i = at + threadIdx.x * 16; i < end; i += kClassThreads * 16)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P.bucketed + i));
    }
    u64 w[kClassPer];  // their loads are in flight while the table is cleared
#pragma unroll
    for (int q = 0; q < kClassPer; ++q) {
      const u32 j = q * kClassThreads + threadIdx.x;
      w[q] = j < n ? __ldg(items + j) : kEmptyWord;
    }
    __syncthreads();  // the previous bucket's look-ups are done
    const uint4 e = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu);
    for (u32 i = threadIdx.x; i < kClassSlots / 4; i += kClassThreads) reinterpret_cast<uint4*>(s_first)[i] = e;
    __syncthreads();
    auto slot = [&](u64 item) { return __umulhi((u32)(item >> 32), P.class_magic); };
    u32 at[kClassPer];
#pragma unroll
    for (int q = 0; q < kClassPer; ++q) {
      at[q] = slot(w[q]);  // (beyond the table where there is no item)
      if (at[q] < kClassSlots) atomicMin(s_first + at[q], (u32)w[q]);
    }
    for (u32 j = kClassPer * kClassThreads + threadIdx.x; j < n; j += kClassThreads) {
      const u64 item = __ldg(items + j);
      atomicMin(s_first + slot(item), (u32)item);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kClassPer; ++q)
      if (at[q] < kClassSlots) found[q * kClassThreads + threadIdx.x] = s_first[at[q]];
    for (u32 j = kClassPer * kClassThreads + threadIdx.x; j < n; j += kClassThreads) found[j] = s_first[slot(__ldg(items + j))];
  }
}

// ---- ranking by bit vectors -----------------------------------------------------------------------------------------
// An item is a first occurrence iff ref[item] is its own position.  k_first_bits fills ref in and leaves one bit per item (a 32-bit word
// per 32 consecutive items of the call); k_rank_prefix scans the words' population counts (single pass, look-back over
// tiles of 2 048 words = 65 536 items, so the chain is a few hundred tiles at most) and packs, per word,
// [ number of first occurrences before the word : 32 | bits : 32 ].  The frontier rank of ANY item p is then
// prefix(word of p) + popcount(bits below p): k_rank_emit writes the frontier, the per-minibatch frontier offsets and,
// for every sampled neighbour, the rank of the first occurrence of its id minus its minibatch's frontier offset — one
// 8-byte look-up in an array of 8 bytes per 32 items (62 KB for a minibatch of 250 000 items) instead of a fix-up pass
// over a rank array.  None of the three kernels waits for anything but the short chain of k_rank_prefix.
constexpr int kBitsThreads = 256;
constexpr int kBitsGroups = 8;                                     // 32-item groups per warp
constexpr int kEmitGroups = 4;
constexpr int kEmitTile = (kBitsThreads / 32) * kEmitGroups * 32;
constexpr int kPrefixThreads = 256;
constexpr int kPrefixPer = 8;
constexpr int kPrefixTile = kPrefixThreads * kPrefixPer;  // words per CTA

struct RankArrays {
  const u32* found;
  u32* ref;
  u32* bits;    // [ceil(items / 32)]
  u64* packed;  // [ceil(items / 32) + 1]
};

__global__ void __launch_bounds__(1024) k_first_bits(BatchLayout L, RankArrays R, i64 n_bound, i64* counters) {
  if (counters[CNT_ABORT] != 0) return;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const i64 n = min(L.item_off[L.G], n_bound);
  const i64 base = (i64)blockIdx.x * (blockDim.x * kBitsGroups) + (i64)warp * (kBitsGroups * 32);
  if (base >= n) return;
  const u32 here = (u32)min((i64)(kBitsGroups * 32), n - base);  // items of this warp
  u32* ref = R.ref + base;
  u32 r[kBitsGroups];
#pragma unroll
  for (int q = 0; q < kBitsGroups; ++q) {
    const u32 i = q * 32 + lane;
    r[q] = i < here ? ref[i] : 0xFFFFFFFFu;  // an id that was never bucketed is marked so, too
  }
#pragma unroll
  for (int q = 0; q < kBitsGroups; ++q)
    if (r[q] != 0xFFFFFFFFu) r[q] = __ldg(R.found + r[q]);
#pragma unroll
  for (int q = 0; q < kBitsGroups; ++q) {
    const u32 i = q * 32 + lane;
    if (i < here) ref[i] = r[q];
  }
  const i64 b = batch_of_warp(L.item_off, L.G, base);
  const i64 begin = __ldg(L.item_off + b), next_begin = __ldg(L.item_off + b + 1);
  u32* bits = R.bits + (base >> 5);
  if (base + here <= next_begin) {
    const u32 lc0 = (u32)(base - begin) + lane;
#pragma unroll
    for (int q = 0; q < kBitsGroups; ++q) {
      if ((u32)(q * 32) >= here) break;  // uniform
      const unsigned bal = __ballot_sync(0xffffffffu, r[q] == lc0 + q * 32);  // lanes beyond `here` hold 0xFFFFFFFF
      if (lane == 0) bits[q] = bal;
    }
    return;
  }
#pragma unroll 1
  for (int q = 0; q < kBitsGroups; ++q) {
    if ((u32)(q * 32) >= here) break;
    const u32 i = q * 32 + lane;
    bool first = false;
    if (i < here) {
      const i64 g = base + i;
      first = r[q] == (u32)(g - __ldg(L.item_off + batch_of(L.item_off, L.G, g)));
    }
    const unsigned bal = __ballot_sync(0xffffffffu, first);
    if (lane == 0) bits[q] = bal;
  }
}

__global__ void __launch_bounds__(kPrefixThreads) k_rank_prefix(BatchLayout L, RankArrays R, i64 n_bound, CompactOut out,
                                                                i64* counters, TileState ts) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  if (counters[CNT_ABORT] != 0) return;
  const i64 n = min(L.item_off[L.G], n_bound);
  const i64 words = (n + 31) >> 5;
  const int tile = blockIdx.x;
  const i64 first = (i64)tile * kPrefixTile + (i64)threadIdx.x * kPrefixPer;
  if ((i64)tile * kPrefixTile >= words && !(words == 0 && tile == 0)) return;
  u32 b[kPrefixPer];
  i64 sum = 0;
#pragma unroll
  for (int j = 0; j < kPrefixPer; ++j) {
    b[j] = first + j < words ? R.bits[first + j] : 0u;
    sum += __popc(b[j]);
  }
  i64 total;
  const i64 excl = block_exclusive_scan<kPrefixThreads>(sum, s_scan, &total);
  if (threadIdx.x < 32) {
    const i64 prefix = tile_exclusive_prefix(ts, tile, total);
    if (threadIdx.x == 0) s_base = prefix;
  }
  __syncthreads();
  i64 run = s_base + excl;
#pragma unroll
  for (int j = 0; j < kPrefixPer; ++j) {
    if (first + j < words) R.packed[first + j] = ((u64)run << 32) | (u64)b[j];
    run += __popc(b[j]);
  }
  if ((i64)(tile + 1) * kPrefixTile >= words && threadIdx.x == 0) {
    const i64 all = s_base + total;
    R.packed[words] = (u64)all << 32;  // rank of the position one past the last item
    out.unique_ptr[L.G] = all;
    for (i64 e = L.G - 1; e >= 0 && L.item_off[e] == n; --e) out.unique_ptr[e] = all;
    counters[CNT_UNIQUE] = all;
    counters[CNT_NNZ] = L.indices_ptr[L.G];
    mail_post(out.mail, 0, all, counters);
    mail_post(out.mail, 1, L.indices_ptr[L.G], counters);
  }
}

__device__ __forceinline__ u32 rank_in_word(u64 w, u32 bit) { return (u32)(w >> 32) + __popc((u32)w & ((1u << bit) - 1u)); }
__device__ __forceinline__ i64 rank_before(const u64* __restrict__ packed, i64 item) {
  return (i64)rank_in_word(__ldg(packed + (item >> 5)), (u32)item & 31u);
}

__global__ void __launch_bounds__(kBitsThreads) k_rank_emit(BatchLayout L, RankArrays R, i64 n_bound, CompactOut out,
                                                            i64* __restrict__ out_relabeled, i64* counters) {
  if (counters[CNT_ABORT] != 0) return;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const i64 n = min(L.item_off[L.G], n_bound);
  const i64 base = (i64)blockIdx.x * kEmitTile + (i64)warp * (kEmitGroups * 32);
  if (base >= n) return;
  const u32 here = (u32)min((i64)(kEmitGroups * 32), n - base);
  // loads that depend on nothing first: the refs of the warp's items and the packed words of their own groups
  const u32* ref = R.ref + base;
  const u64* own_words = R.packed + (base >> 5);
  u32 r[kEmitGroups];
  u64 own[kEmitGroups];
#pragma unroll
  for (int q = 0; q < kEmitGroups; ++q) {
    const u32 i = q * 32 + lane;
    r[q] = i < here ? __ldg(ref + i) : 0xFFFFFFFFu;
    own[q] = (u32)(q * 32) < here ? __ldg(own_words + q) : 0ull;
  }
  const BatchUniform u = load_batch<false>(L, L.item_off, batch_of_warp(L.item_off, L.G, base));
  if (base + here <= u.next_begin) {
    // every item of the warp lies in minibatch u: positions are 32-bit, the look-ups of all groups are issued before
    // anything is written
    const u32 items = (u32)(u.next_begin - u.begin), ns = (u32)u.num_seeds;
    const u32 lc0 = (u32)(base - u.begin) + lane;
    const u64* win = R.packed + (u.begin >> 5);  // the minibatch's window of packed words
    const u32 shift = (u32)u.begin & 31u;        // bit of the minibatch's first item inside win[0]
    const u32 front = rank_in_word(__ldg(win), shift);
    const i64* seeds = L.seeds + u.seeds_begin;
    const i64* edges = L.indices + u.edges_begin - ns;
    i64* rel = out_relabeled ? out_relabeled + u.edges_begin - ns : nullptr;
    u64 wref[kEmitGroups];
    i64 node[kEmitGroups];
#pragma unroll
    for (int q = 0; q < kEmitGroups; ++q) {
      const u32 lc = lc0 + q * 32;
      wref[q] = 0;
      node[q] = 0;
      if (q * 32 + lane >= here) continue;
      if (lc >= ns && r[q] < items) wref[q] = __ldg(win + ((r[q] + shift) >> 5));
      if (r[q] == lc) node[q] = __ldg(lc < ns ? seeds + lc : edges + lc);
    }
#pragma unroll
    for (int q = 0; q < kEmitGroups; ++q) {
      const u32 lc = lc0 + q * 32;
      if (q * 32 + lane >= here) continue;
      const u32 pos = rank_in_word(own[q], lane);
      if (r[q] == lc) __stcs(out.unique + pos, node[q]);  // (see k_class_emit)
      if (lc == 0) {  // the frontier of the minibatch starts here; empty minibatches before it start here too
        out.unique_ptr[u.batch] = pos;
        for (i64 e = u.batch - 1; e >= 0 && __ldg(L.item_off + e) == u.begin; --e) out.unique_ptr[e] = pos;
      }
      // an id outside the accepted range was never bucketed and its ref says so; any value that is not a position of
      // this minibatch is treated alike, so no look-up can leave the rank array
      if (lc >= ns && rel)
        __stcs(rel + lc, r[q] < items ? (i64)(rank_in_word(wref[q], (r[q] + shift) & 31u) - front) : (i64)-1);
    }
    return;
  }
#pragma unroll 1
  for (int q = 0; q < kEmitGroups; ++q) {  // the warp straddles minibatches: every item finds its own
    const i64 g = base + q * 32 + lane;
    if (g >= n) continue;
    BatchUniform v = u;
    if (g >= u.next_begin) v = load_batch<false>(L, L.item_off, batch_of(L.item_off, L.G, g));
    const i64 front = rank_before(R.packed, v.begin);
    const i64 lc = g - v.begin;
    const bool first = r[q] == (u32)lc;
    if (first || g == v.begin) {
      const i64 pos = rank_before(R.packed, g);
      if (first) out.unique[pos] = lc < v.num_seeds ? __ldg(L.seeds + v.seeds_begin + lc)
                                                    : __ldg(L.indices + v.edges_begin + (lc - v.num_seeds));
      if (g == v.begin) {
        out.unique_ptr[v.batch] = pos;
        for (i64 e = v.batch - 1; e >= 0 && __ldg(L.item_off + e) == g; --e) out.unique_ptr[e] = pos;
      }
    }
    if (lc >= v.num_seeds && out_relabeled)
      out_relabeled[v.edges_begin + (lc - v.num_seeds)] =
          (i64)r[q] >= v.next_begin - v.begin ? -1 : rank_before(R.packed, v.begin + (i64)r[q]) - front;
  }
}

// ---- host sequence ----------------------------------------------------------------------------------------------------
static inline size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

// Where classes are ahead of hashed buckets, us of a whole call hashed / classes.  40 M items over 2.45 M nodes, ids scattered evenly (in
// brackets: all of them within 16 384 neighbours, which suits hashing best): 1 000 items a class 929 / 954 (784 / 923), 1 400 917 / 880
// (772 / 847), 1 600 910 / 854 (763 / 816), 2 000 909 / 821 (771 / 786), 3 000 905 / 780 (771 / 738), 12 200 900 / 772 (785 / 714);
// numbered by degree, or crowding as squares and fourth powers, 909 / 851, 950 / 853 and 971 / 859 at 1 600.  (Fewer than a hundred
// buckets in all would be no faster, 1.2 M items in 60 of them 84 / 86, but a call with less than 256 has small tables that are
// addressed by the id.)
i64 partition_class_parts(i64 num_nodes, i64 items_per_minibatch, bool forced) {
  if (num_nodes <= 0 || num_nodes > (i64)(kNarrowWindow - 1) * kClassSlots) return 0;
  const i64 needed = max((i64)11, (num_nodes + kClassSlots - 1) / kClassSlots);
  // A prime from 11 on, so that ids that are multiples of something do not crowd in a few classes (multiples of ten in five of them:
  // 92 us hashed, 149 us); 252 to 255, behind the last prime of that size, as they are.
  i64 classes = needed;
  for (i64 d = 2; d * d <= classes && needed <= 251; ++d)
    if (classes % d == 0) ++classes, d = 1;
  const i64 parts = classes + 1;
  return forced || items_per_minibatch >= 1600 * parts ? parts : 0;
}

i64 partition_bucket_capacity(i64 items_bound, i64 G, i64 parts) { return parts > 0 ? G * parts : items_bound / kBucketTarget + G + 1; }

size_t partition_count_bytes(i64 bucket_cap) { return al256(sizeof(u32) * 3 * (size_t)(bucket_cap + 1)); }

size_t partition_workspace_bytes(i64 n_cap, i64 bucket_cap) {
  const size_t words = (size_t)((n_cap + 31) / 32) + 2;
  return partition_count_bytes(bucket_cap) + al256(8 * (size_t)n_cap) + 2 * al256(4 * (size_t)n_cap) +
         al256(4 * words) + al256(8 * words) + al256(8 * (2 * (size_t)n_cap + 32 * (size_t)bucket_cap + 64));
}

uint32_t* partition_bucket_counts(void* ws) { return (u32*)ws; }

struct PartArrays {
  PartLayout P;
  RankArrays R;
};

static PartArrays carve(const BatchLayout& L, i64 n_cap, i64 bucket_cap, void* ws) {
  const size_t words = (size_t)((n_cap + 31) / 32) + 2;
  char* at = (char*)ws;
  PartArrays a;
  PartLayout& P = a.P;
  P.L = L;
  P.bucket_count = (u32*)at;
  P.bucket_start = P.bucket_count + (bucket_cap + 1);
  P.bucket_cursor = P.bucket_count + 2 * (bucket_cap + 1);
  at += partition_count_bytes(bucket_cap);
  P.bucketed = (u64*)at;
  at += al256(8 * (size_t)n_cap);
  P.found = (u32*)at;
  at += al256(4 * (size_t)n_cap);
  P.ref = (u32*)at;
  at += al256(4 * (size_t)n_cap);
  a.R.found = P.found;
  a.R.ref = P.ref;
  a.R.bits = (u32*)at;
  at += al256(4 * words);
  a.R.packed = (u64*)at;
  at += al256(8 * words);
  P.spill = (u64*)at;
  return a;
}

int partition_after_sampler(gsb_ctx* ctx, cudaStream_t stream, BatchLayout L, i64 n_cap, i64 bucket_cap, void* ws,
                            const i64* sub_indptr, i64 S, i64 edges_bound, i64* out_indices_ptr) {
  const PartArrays a = carve(L, n_cap, bucket_cap, ws);
  {
    ScopedKernelTimer timer(ctx, KID_OTHER, stream);
    k_part_after_sampler<<<1, 1024, 0, stream>>>(a.P, sub_indptr, S, edges_bound, out_indices_ptr,
                                                 bucket_cap <= kScanAlongBuckets, ctx_counters(ctx));
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int partition_unique_relabel(gsb_ctx* ctx, cudaStream_t stream, BatchLayout L, i64 n_cap, i64 bucket_cap, void* ws,
                             i64 parts, bool counted, i64* out_unique, i64* out_unique_ptr, i64* out_relabeled, Mail mail) {
  i64* counters = ctx_counters(ctx);
  PartArrays arrays = carve(L, n_cap, bucket_cap, ws);
  arrays.P.class_parts = (u32)parts;
  arrays.P.class_magic = class_magic(parts);
  const PartLayout& P = arrays.P;
  const RankArrays& R = arrays.R;
  const bool wide = n_cap / L.G > (i64)kNarrowWindow * kBucketTarget * 3 / 4;  // the larger minibatches of a ragged call count
  static bool attr_set[64] = {};
  const int dev = ctx_device(ctx);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GSB_CUDA_OK(cudaFuncSetAttribute(k_part_resolve, cudaFuncAttributeMaxDynamicSharedMemorySize, kBucketSlots * 8));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_part_scatter<kWideWindow, 512, 16, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     scatter_smem(8192, kWideWindow)));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_part_resolve_classes, cudaFuncAttributeMaxDynamicSharedMemorySize, kClassSlots * 4));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_part_scatter<kNarrowWindow, 512, 16, true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     scatter_smem(8192, kNarrowWindow)));
    attr_set[dev] = true;
  }
  if (!counted) {
    GSB_CUDA_OK(cudaMemsetAsync(P.bucket_count, 0, sizeof(u32) * (size_t)(bucket_cap + 1), stream));
    {
      ScopedKernelTimer timer(ctx, KID_PART_COUNT, stream);
      const int grid = grid_for(n_cap, kPartTile);
      if (parts > 0) k_part_count<kNarrowWindow, true><<<grid, kPartThreads, 0, stream>>>(P, n_cap, counters);
      else if (wide) k_part_count<kWideWindow, false><<<grid, kPartThreads, 0, stream>>>(P, n_cap, counters);
      else k_part_count<kNarrowWindow, false><<<grid, kPartThreads, 0, stream>>>(P, n_cap, counters);
    }
    GSB_LAUNCH_OK();
  }
  if (!counted || bucket_cap > kScanAlongBuckets) {
    const int scan_tiles = grid_for(bucket_cap, kScanTile);
    TileState scan_ts;
    const int st = ctx_tile_state(ctx, scan_tiles, stream, &scan_ts);
    if (st != GSB_OK) return st;
    {
      ScopedKernelTimer timer(ctx, KID_OTHER, stream);
      k_part_scan<<<scan_tiles, kScanThreads, 0, stream>>>(P, counters, scan_ts);
    }
    GSB_LAUNCH_OK();
  }
  {
    ScopedKernelTimer timer(ctx, KID_PART_SCATTER, stream);
    if (wide && parts > 0)
      k_part_scatter<kNarrowWindow, 512, 16, true><<<grid_for(n_cap, 8192), 512, scatter_smem(8192, kNarrowWindow), stream>>>(
          P, n_cap, counters);
    else if (wide)
      k_part_scatter<kWideWindow, 512, 16, false><<<grid_for(n_cap, 8192), 512, scatter_smem(8192, kWideWindow), stream>>>(
          P, n_cap, counters);
    else if (parts > 0)
      k_part_scatter<kNarrowWindow, 256, 8, true><<<grid_for(n_cap, 2048), 256, scatter_smem(2048, kNarrowWindow), stream>>>(
          P, n_cap, counters);
    else
      k_part_scatter<kNarrowWindow, 256, 8, false><<<grid_for(n_cap, 2048), 256, scatter_smem(2048, kNarrowWindow), stream>>>(
          P, n_cap, counters);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_PART_RESOLVE, stream);
    if (parts > 0)
      k_part_resolve_classes<<<(int)min(bucket_cap, (i64)kNumSMs * 3 * 4), kClassThreads, kClassSlots * 4, stream>>>(P, counters);
    else
      k_part_resolve<<<(int)min(bucket_cap, (i64)kNumSMs * 4 * 4), kResolveThreads, kBucketSlots * 8, stream>>>(P, counters);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_FIRST_BITS, stream);
    // a CTA takes the tile that the scatter pass took
    const int threads = wide ? 1024 : 256;
    k_first_bits<<<grid_for(n_cap, threads * kBitsGroups), threads, 0, stream>>>(L, R, n_cap, counters);
  }
  GSB_LAUNCH_OK();
  const int prefix_tiles = grid_for((n_cap + 31) / 32, kPrefixTile);
  TileState ts;
  int st = ctx_tile_state(ctx, prefix_tiles, stream, &ts);
  if (st != GSB_OK) return st;
  CompactOut out{out_unique, out_unique_ptr, mail};
  {
    ScopedKernelTimer timer(ctx, KID_OTHER, stream);
    k_rank_prefix<<<prefix_tiles, kPrefixThreads, 0, stream>>>(L, R, n_cap, out, counters, ts);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_RANK_EMIT, stream);
    k_rank_emit<<<grid_for(n_cap, kEmitTile), kBitsThreads, 0, stream>>>(L, R, n_cap, out, out_relabeled, counters);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // namespace gsb
