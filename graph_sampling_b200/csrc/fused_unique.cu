// Unique + relabel of an ordinary call in ONE launch.
//
// A minibatch relabelled on its own (or a few of them) is 10^4 to 10^6 items: each pass over them is a few microseconds of
// work, and the multi-launch forms (batch_relabel.cu, partition_relabel.cu) spend more time between their five to nine
// launches than in them.  Here the grid is launched cooperatively, small enough to be resident as a whole, the items of a
// thread stay in registers, and two grid-wide barriers separate the phases:
//
//   insert   every item claims a slot of an L2-resident hash table for its id and lowers the slot's position to its own;
//            a slot is one word, [epoch : 11 | id : 32 | position : 21], and a word of an older epoch counts as empty, so
//            the table is never cleared between calls (once per 2 047 calls, when the epoch wraps).  Slots come in
//            buckets of four, one 32-byte sector that is read in one go, three slots per item: the longest chain of
//            dependent reads of a call sets the pace of its insert, and it is a handful of buckets here where linear
//            probing over single slots at load 0.5 had chains of fifty (813 000 items: 92 -> 52 us);
//   ------   barrier
//   flag     the item whose position the slot kept is the first occurrence of its id: one bit per item and a running
//            count per 32 items inside the CTA, one total per CTA;
//   ------   barrier
//   emit     the rank of any position is its CTA's prefix (a scan of at most a few hundred totals, done by every CTA for
//            itself) + its word's prefix + the bits below it: the frontier is written at those ranks, and every item to
//            relabel writes the rank of the first occurrence of its id.
//
// DIRECT: when the ids are known to be below a bound and the table of one 4-byte word per id and minibatch stays small, the
// table is addressed by the id itself, [2047 - epoch : 11 | position : 21], and an insertion is one fire-and-forget
// reduction: no reads, no chains, no answers to wait for.  An id beyond the bound makes the call report
// GSB_ERR_INDEX_RANGE, and the caller repeats it with the hash table.
//
// BATCHED: the items belong to G minibatches (numbered batch-major, as in batch_table.cuh), each with a region of the
// table of its own; ranks are then relative to the minibatch's first item.
//
// GPU time of a call, five launches (without the gaps between them) / hash table / direct table: 16 000 items
// 26 / 11 / 7 us, 813 000 items 86 / 49 / 26 us.  What bounds the hash table (813 000 items): bucket reads and
// compare-and-swaps at the rate of the L2's atomics, 107 G/s each, and the rounds of the slowest lanes behind them.
// Two CTAs per SM leave 64 registers a thread: five and six items per thread partly live in local memory in some forms (up to 84
// bytes stored per thread), eight, twelve and sixteen in all (76 to 616).
#include "batch_table.cuh"
#include "common.cuh"
#include "grid_sync.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kFuThreads = 512;
constexpr int kFuWarps = kFuThreads / 32;
constexpr int kFuPosBits = 21;
constexpr u64 kFuPosMask = (1ull << kFuPosBits) - 1;
constexpr u32 kFuEpochs = 1u << (64 - 32 - kFuPosBits);  // epochs 1 .. kFuEpochs - 1
constexpr u32 kFuNone = 0xFFFFFFFFu;
constexpr int kFuWindow = 512;  // minibatches whose offsets a CTA keeps in shared memory

struct FusedParams {
  const i64* first;   // S ids
  const i64* second;  // E ids, relabelled into out_second (may be null)
  i64 S, E;           // BATCHED: bounds of the device-side totals
  i64* out_unique;
  i64* out_second;
  const i64* col_index;  // E positions in `first`; out_col receives the rank of the id found there (may be null)
  i64* out_col;
  const i64* copy_src;  // an array to copy along the way (may be null)
  i64* copy_dst;
  i64 copy_n;
  float* ones;  // ones_n floats set to 1 along the way
  i64 ones_n;
  // BATCHED
  const i64* seeds_ptr;    // [G + 1]
  const i64* indices_ptr;  // [G + 1], or null: the offsets are sub_indptr[seeds_ptr[b]] and are written to out_indices_ptr
  const i64* sub_indptr;   // [S + 1]
  i64* out_indices_ptr;
  i64* out_unique_ptr;  // [G + 1]
  i64 G;
  // scratch
  u64* table;
  u64 epoch;  // already shifted
  u32* direct;       // DIRECT: [minibatches][id_bound]
  u32 direct_epoch;  // already inverted and shifted
  u32 id_bound;
  u64* packed;    // [items / 32 + 1]  first occurrences of the CTA before the word << 32 | bits
  u32* totals;    // [CTAs]
  u32* seed_ref;  // [S] first position of every id of `first` (only with col_index)
  GridSync sync;
  i64* counters;
  Mail mail;
};

// Buckets of a region: minibatch b, whose items are [begin, next), has the buckets [bucket0(begin, b), bucket0(next, b + 1)),
// at least 0.75 per item.
__host__ __device__ __forceinline__ u32 fused_bucket0(u32 begin, u32 b) { return begin - (begin >> 2) + 2 * b; }

__device__ __forceinline__ u32 fused_home(u32 id, u32 size) {
  u32 x = id * 0x9E3779B1u;
  x ^= x >> 15;
  x *= 0x85EBCA6Bu;
  return __umulhi(x, size);
}

// Offsets of minibatch b: first seed, first edge.
__device__ __forceinline__ i64 fused_edges_begin(const FusedParams& p, i64 b, i64 seeds_begin) {
  return p.indices_ptr ? __ldg(p.indices_ptr + b) : __ldg(p.sub_indptr + max((i64)0, min(seeds_begin, p.S)));
}
__device__ __forceinline__ i64 fused_item_off(const FusedParams& p, i64 b) {
  const i64 s = __ldg(p.seeds_ptr + b);
  return s + fused_edges_begin(p, b, s);
}

__device__ __forceinline__ void load_bucket(const u64* table, u32 bucket, u64 (&w)[4]) {
  const ulonglong2* p = reinterpret_cast<const ulonglong2*>(table + 4ull * bucket);
  const ulonglong2 a = __ldcg(p), b = __ldcg(p + 1);
  w[0] = a.x;
  w[1] = a.y;
  w[2] = b.x;
  w[3] = b.y;
}

// The first slot of a bucket, in the order start, start + 1, ... (mod 4), that is free or holds mine's id; 4 if none does.
// Starting places differ from id to id: with everybody trying slot 0 first, the ids of a bucket queued up behind each
// other's compare-and-swaps.
__device__ __forceinline__ u32 pick_slot(const u64 (&w)[4], u32 start, u64 mine, u64 epoch, u64* word) {
  u32 best = 4;
#pragma unroll
  for (u32 j = 0; j < 4; ++j) {
    const u32 turn = (j - start) & 3u;
    const bool usable = ((w[j] ^ epoch) >> (32 + kFuPosBits)) != 0 || ((w[j] ^ mine) >> kFuPosBits) == 0;
    if (usable && turn < best) {
      best = turn;
      *word = w[j];
    }
  }
  return best == 4 ? 4 : (best + start) & 3u;
}

template <int R, bool BATCHED, bool DIRECT>
__global__ void __launch_bounds__(kFuThreads, 2) k_fused_unique(const __grid_constant__ FusedParams p) {
  constexpr u32 kItems = kFuThreads * R;  // of a CTA
  __shared__ u32 s_group[kFuWarps * R];   // counts per 32 items, then their exclusive prefixes
  __shared__ u32 s_prefix[kFuThreads];    // first occurrences before every CTA
  __shared__ u32 s_warp[kFuWarps];
  __shared__ u32 s_off[BATCHED ? kFuWindow + 1 : 1];    // item offsets of the CTA's minibatches
  __shared__ u32 s_seeds[BATCHED ? kFuWindow + 1 : 1];  // their first seeds
  __shared__ i64 s_range[2];
  const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const u32 base = blockIdx.x * kItems;
  i64 ns = p.S, ne = p.E;
  if (BATCHED) {
    ns = __ldg(p.seeds_ptr + p.G);
    ne = fused_edges_begin(p, p.G, ns);
    if (ns > p.S || ne > p.E || ns < 0 || ne < 0) {  // every CTA sees the same: nobody waits for anybody
      grid_arrive(p.sync, 2);
      if (tid == 0) {
        raise_error(p.counters, GSB_ERR_CAPACITY, ns > p.S ? ns : ne);
        if (blockIdx.x == 0) {
          p.counters[CNT_ABORT] = 1;
          mail_post(p.mail, 0, 0, p.counters);
          mail_post(p.mail, 1, ne, p.counters);
        }
      }
      return;
    }
    if (blockIdx.x == 0 && tid == 0) p.counters[CNT_ABORT] = 0;
  }
  const u32 n = (u32)(ns + ne);

  // ---- the minibatches of the CTA's items
  i64 b_first = 0, b_count = 1;
  if (BATCHED && base < n) {
    const u32 last = min(n, base + kItems) - 1;
    if (warp < 2) {  // two warp-wide searches side by side: 32 pivots a round
      const i64 g = warp == 0 ? base : last;
      i64 lo = 0, end = p.G;
      while (end - lo > 1) {
        const i64 step = (end - lo + 31) >> 5, idx = lo + (i64)(lane + 1) * step;
        const bool le = idx < end && fused_item_off(p, idx) <= g;
        const i64 hits = __popc(__ballot_sync(0xffffffffu, le));
        lo += hits * step;
        end = min(end, lo + step);
      }
      if (lane == 0) s_range[warp] = lo;
    }
    __syncthreads();
    b_first = s_range[0];
    b_count = s_range[1] - b_first + 1;
    if (b_count <= kFuWindow) {
      for (u32 j = tid; j <= b_count; j += kFuThreads) {
        const i64 s = __ldg(p.seeds_ptr + b_first + j);
        s_seeds[j] = (u32)s;
        s_off[j] = (u32)(s + fused_edges_begin(p, b_first + j, s));
      }
    }
    __syncthreads();
  }
  const bool windowed = b_count <= kFuWindow;
  // minibatch of item g: its item offset, first seed and the offset of the next one's seeds
  struct Where {
    i64 batch;
    u32 begin, seeds, next_seeds, next_begin;
    bool ok;  // the offsets are those of a minibatch (they come from the caller): nothing is accessed otherwise
  };
  auto where = [&](u32 g) {
    Where w;
    if (windowed) {
      u32 lo = 0, hi = (u32)b_count;
      while (hi - lo > 1) {
        const u32 mid = (lo + hi) >> 1;
        if (s_off[mid] <= g) lo = mid;
        else hi = mid;
      }
      w.batch = b_first + lo;
      w.begin = s_off[lo];
      w.seeds = s_seeds[lo];
      w.next_seeds = s_seeds[lo + 1];
      w.next_begin = s_off[lo + 1];
    } else {
      i64 lo = b_first, hi = b_first + b_count;
      while (hi - lo > 1) {
        const i64 mid = (lo + hi) >> 1;
        if (fused_item_off(p, mid) <= (i64)g) lo = mid;
        else hi = mid;
      }
      w.batch = lo;
      w.seeds = (u32)__ldg(p.seeds_ptr + lo);
      w.next_seeds = (u32)__ldg(p.seeds_ptr + lo + 1);
      w.begin = (u32)fused_item_off(p, lo);
      w.next_begin = (u32)fused_item_off(p, lo + 1);
    }
    w.ok = w.begin <= g && g < w.next_begin && w.next_begin <= n && w.seeds <= w.begin && w.seeds <= w.next_seeds &&
           w.next_seeds <= (u32)ns && w.next_seeds - w.seeds <= w.next_begin - w.begin;
    return w;
  };

  // ---- insert
  auto in_range = [&](i64 v) { return DIRECT ? (u64)v < (u64)p.id_bound : valid_id(v); };
  u32 id[R], slot[R], batch0[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 g = base + r * kFuThreads + tid;
    i64 v = -1;
    u32 region = 0, size = fused_bucket0(n, 1);
    batch0[r] = 0;
    if (g < n) {
      if (BATCHED) {
        const Where w = where(g);
        const u32 lc = g - w.begin, seeds = w.next_seeds - w.seeds;
        if (w.ok) v = lc < seeds ? __ldg(p.first + w.seeds + lc) : __ldg(p.second + (g - w.next_seeds));
        region = DIRECT ? (u32)w.batch * p.id_bound : fused_bucket0(w.begin, (u32)w.batch);
        size = DIRECT ? 0 : fused_bucket0(w.next_begin, (u32)w.batch + 1) - region;
        batch0[r] = w.begin;
      } else {
        v = g < (u32)p.S ? __ldg(p.first + g) : __ldg(p.second + (g - (u32)p.S));
      }
      if (!in_range(v)) raise_error(p.counters, GSB_ERR_INDEX_RANGE, g);
    }
    id[r] = in_range(v) ? (u32)v : kFuNone;
    slot[r] = kFuNone;
    if (id[r] != kFuNone) slot[r] = region + (DIRECT ? id[r] : fused_home(id[r], size));
  }
  if (DIRECT) {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (slot[r] != kFuNone)
        asm volatile("red.relaxed.gpu.global.min.u32 [%0], %1;" ::"l"(p.direct + slot[r]),
                     "r"(p.direct_epoch | (base + r * kFuThreads + tid))
                     : "memory");
  } else {
  // A round reads the buckets of up to four unsettled items, then issues their compare-and-swaps, then looks at the
  // answers: the two round trips are paid per round, not per item.  An id always takes the first usable slot of its own
  // order, and slots are never given up, so nobody misses a copy of it.
  constexpr int kAhead = R % 4 == 0 ? 4 : R % 3 == 0 ? 3 : R;
#pragma unroll
  for (int r0 = 0; r0 < R; r0 += kAhead) {
    u32 bucket[kAhead], probes = 0;
    unsigned open = 0;
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      bucket[q] = slot[r0 + q];
      if (slot[r0 + q] != kFuNone) open |= 1u << q;
    }
    while (open) {
      u64 expect[kAhead], found[kAhead];
      u32 at[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        at[q] = 4;
        if (!((open >> q) & 1u)) continue;
        u64 w[4];
        load_bucket(p.table, bucket[q], w);
        const u64 mine = p.epoch | ((u64)id[r0 + q] << kFuPosBits) | (u64)(base + (r0 + q) * kFuThreads + tid);
        at[q] = pick_slot(w, id[r0 + q] & 3u, mine, p.epoch, &expect[q]);
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        found[q] = 0;
        if (!((open >> q) & 1u) || at[q] == 4) continue;
        const u64 mine = p.epoch | ((u64)id[r0 + q] << kFuPosBits) | (u64)(base + (r0 + q) * kFuThreads + tid);
        found[q] = expect[q];
        if ((expect[q] ^ p.epoch) >> (32 + kFuPosBits)) found[q] = atomicCAS(p.table + 4ull * bucket[q] + at[q], expect[q], mine);
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        if (!((open >> q) & 1u)) continue;
        const u32 g = base + (r0 + q) * kFuThreads + tid;
        const u64 mine = p.epoch | ((u64)id[r0 + q] << kFuPosBits) | (u64)g;
        if (at[q] == 4) {  // full of other ids: the next bucket of the item's region
          u32 lo = 0, end = fused_bucket0(n, 1);
          if (BATCHED) {
            const Where w = where(g);
            lo = fused_bucket0(w.begin, (u32)w.batch);
            end = fused_bucket0(w.next_begin, (u32)w.batch + 1);
          }
          bucket[q] = bucket[q] + 1 == end ? lo : bucket[q] + 1;
          if (++probes > 4 * (end - lo)) {  // more slots than items: cannot happen
            raise_error(p.counters, GSB_ERR_TABLE_FULL, g);
            slot[r0 + q] = kFuNone;
            open &= ~(1u << q);
          }
          continue;
        }
        const bool claimed = found[q] == expect[q] && ((expect[q] ^ p.epoch) >> (32 + kFuPosBits)) != 0;
        if (!claimed && ((found[q] ^ mine) >> kFuPosBits) != 0) continue;  // somebody else's id came first: look again
        if (!claimed && found[q] > mine) atomicMin(p.table + 4ull * bucket[q] + at[q], mine);
        slot[r0 + q] = 4 * bucket[q] + at[q];
        open &= ~(1u << q);
      }
    }
  }
  }
  for (i64 j = (i64)blockIdx.x * kFuThreads + tid; j < p.copy_n; j += (i64)gridDim.x * kFuThreads)
    p.copy_dst[j] = __ldg(p.copy_src + j);
  for (i64 j = (i64)blockIdx.x * kFuThreads + tid; j < p.ones_n; j += (i64)gridDim.x * kFuThreads) p.ones[j] = 1.0f;
  // The results of a call that was given up, for the super-batch hops that run on without the host: empty frontiers.
  auto give_up = [&] {
    if (!BATCHED) return;
    grid_share(p.G + 1, [&](i64 b) {
      if (p.out_indices_ptr) p.out_indices_ptr[b] = fused_edges_begin(p, b, __ldg(p.seeds_ptr + b));
      p.out_unique_ptr[b] = 0;
    });
    grid_share(p.out_second ? ne : 0, [&](i64 e) { p.out_second[e] = -1; });
    if (blockIdx.x == 0) {
      p.counters[CNT_UNIQUE] = 0;
      p.counters[CNT_NNZ] = ne;
    }
  };
  grid_barrier(p.sync, 1, give_up);

  // ---- flag
  unsigned bits[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 g = base + r * kFuThreads + tid;
    u32 ref = kFuNone;
    if (slot[r] != kFuNone)
      ref = DIRECT ? __ldcg(p.direct + slot[r]) & (u32)kFuPosMask : (u32)(__ldcg(p.table + slot[r]) & kFuPosMask);
    if (!BATCHED && p.col_index && g < (u32)p.S) p.seed_ref[g] = ref;
    slot[r] = ref;  // from here on: the first position of the item's id
    bits[r] = __ballot_sync(0xffffffffu, ref == g);
    if (lane == 0) s_group[r * kFuWarps + warp] = __popc(bits[r]);
  }
  __syncthreads();
  if (warp == 0) {
    u32 carry = 0;
#pragma unroll
    for (int q = 0; q < kFuWarps * R; q += 32) {
      const u32 at = q + lane;
      const u32 c = at < kFuWarps * R ? s_group[at] : 0;
      u32 inc = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
      }
      if (at < kFuWarps * R) s_group[at] = carry + inc - c;
      carry += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) p.totals[blockIdx.x] = carry;
  }
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const u32 g = base + r * kFuThreads + warp * 32;
      if (g < n) p.packed[g >> 5] = ((u64)s_group[r * kFuWarps + warp] << 32) | (u64)bits[r];
    }
  }
  grid_barrier(p.sync, 2, give_up);

  // ---- emit
  u32 all;
  {
    const u32 t = tid < gridDim.x ? __ldcg(p.totals + tid) : 0;
    u32 inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    u32 before = 0;
    all = 0;
#pragma unroll
    for (int w = 0; w < kFuWarps; ++w) {
      if (w < (int)warp) before += s_warp[w];
      all += s_warp[w];
    }
    s_prefix[tid] = before + inc - t;
    __syncthreads();
  }
  if (blockIdx.x == 0 && tid == 0) {
    p.counters[CNT_UNIQUE] = all;
    if (BATCHED) p.counters[CNT_NNZ] = ne;
    mail_post(p.mail, 0, all, p.counters);
    if (BATCHED) mail_post(p.mail, 1, ne, p.counters);
  }
  auto rank_of = [&](u32 pos) {
    const u64 w = __ldcg(p.packed + (pos >> 5));
    return s_prefix[pos / kItems] + (u32)(w >> 32) + __popc((u32)w & ((1u << (pos & 31)) - 1u));
  };
  u64 of_ref[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 g = base + r * kFuThreads + tid;
    of_ref[r] = 0;
    if (g < n && slot[r] < n) of_ref[r] = __ldcg(p.packed + (slot[r] >> 5));
  }
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const u32 g = base + r * kFuThreads + tid;
    if (g >= n) continue;
    i64 rank = -1;
    const u32 ref = slot[r];
    if (ref < n) rank = s_prefix[ref / kItems] + (u32)(of_ref[r] >> 32) + __popc((u32)of_ref[r] & ((1u << (ref & 31)) - 1u));
    if (ref == g) p.out_unique[rank] = (i64)id[r];
    if (BATCHED) {
      if (p.out_second) {
        const Where w = where(g);
        const u32 lc = g - w.begin;
        if (w.ok && lc >= w.next_seeds - w.seeds)
          p.out_second[g - w.next_seeds] = rank < 0 ? -1 : rank - (i64)rank_of(batch0[r]);
      }
    } else if (g >= (u32)p.S) {
      if (p.out_second) p.out_second[g - (u32)p.S] = rank;
    }
  }
  // Three reads that depend on each other: those of up to eight items go together (one item after the other, behind the stores
  // above, 1.1 M items spent 17 of the call's 39 us here; 13 now, most of it the three output arrays).
  if (!BATCHED && p.out_col) {
    constexpr int kAhead = R <= 8 ? R : R / 2;
#pragma unroll
    for (int r0 = 0; r0 < R; r0 += kAhead) {
      u32 ref[kAhead];
      u64 word[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const u32 g = base + (r0 + q) * kFuThreads + tid;
        const i64 c = r0 + q < R && g < n && g >= (u32)p.S ? __ldg(p.col_index + (g - (u32)p.S)) : -1;
        ref[q] = (u64)c < (u64)p.S ? (u32)c : kFuNone;
      }
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (ref[q] != kFuNone) ref[q] = __ldcg(p.seed_ref + ref[q]);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) word[q] = ref[q] < n ? __ldcg(p.packed + (ref[q] >> 5)) : 0;
#pragma unroll
      for (int q = 0; q < kAhead; ++q) {
        const u32 g = base + (r0 + q) * kFuThreads + tid;
        if (r0 + q < R && g < n && g >= (u32)p.S)
          p.out_col[g - (u32)p.S] = ref[q] < n ? (i64)(s_prefix[ref[q] / kItems] + (u32)(word[q] >> 32) +
                                                       __popc((u32)word[q] & ((1u << (ref[q] & 31)) - 1u)))
                                               : (i64)-1;
      }
    }
  }
  if (BATCHED) {
    for (i64 b = (i64)blockIdx.x * kFuThreads + tid; b <= p.G; b += (i64)gridDim.x * kFuThreads) {
      const i64 s = __ldg(p.seeds_ptr + b), e = fused_edges_begin(p, b, s);
      if (p.out_indices_ptr) p.out_indices_ptr[b] = e;
      p.out_unique_ptr[b] = (u64)(s + e) < (u64)n ? (i64)rank_of((u32)(s + e)) : (i64)all;
    }
  }
}

// ---- host side ------------------------------------------------------------------------------------------------------
// Items per thread: the fewest whose CTAs are resident together.  A finer list than powers of two leaves fewer SMs with one CTA
// where others have two: 700 000 items, direct / hash table, five a thread 24.3 / 48.1 us, eight 27.9 / 55.6; 340 000, three
// 20.6 / 36.0, four 21.7 / 38.7.  With the hash table fewer CTAs of more items are never ahead, not even where that evens out the SMs:
// 200 000 items, two a thread 30.6, three 32.6, of 20 minibatches 25.1 and 27.4.  With the direct table they sometimes are, by less
// than a microsecond (200 000 items 19.1 and 18.4, 120 000 with one and two 17.7 and 17.3, but 260 000 with two and three 18.9
// and 20.8), and the rule is the same for both.
constexpr int kFuItems[] = {1, 2, 3, 4, 5, 6, 8, 12, 16};

static int items_per_thread(i64 n, int max_ctas) {
  for (int r : kFuItems)
    if (n <= (i64)max_ctas * kFuThreads * r) return r;
  return 16;
}

template <bool BATCHED, bool DIRECT>
static const void* fused_kernel(int r) {
  switch (r) {
    case 1: return (const void*)k_fused_unique<1, BATCHED, DIRECT>;
    case 2: return (const void*)k_fused_unique<2, BATCHED, DIRECT>;
    case 3: return (const void*)k_fused_unique<3, BATCHED, DIRECT>;
    case 4: return (const void*)k_fused_unique<4, BATCHED, DIRECT>;
    case 5: return (const void*)k_fused_unique<5, BATCHED, DIRECT>;
    case 6: return (const void*)k_fused_unique<6, BATCHED, DIRECT>;
    case 8: return (const void*)k_fused_unique<8, BATCHED, DIRECT>;
    case 12: return (const void*)k_fused_unique<12, BATCHED, DIRECT>;
    default: return (const void*)k_fused_unique<16, BATCHED, DIRECT>;
  }
}

// All instantiations are compiled for two CTAs per SM; the largest of each kind is asked.
static int resident_ctas(gsb_ctx* ctx) {
  static int known[4][64];
  int ctas = kFuThreads;  // one thread per CTA total in the scan
  ctas = min(ctas, ctx_resident_ctas(ctx, fused_kernel<false, false>(16), kFuThreads, 0, known[0]));
  ctas = min(ctas, ctx_resident_ctas(ctx, fused_kernel<true, false>(16), kFuThreads, 0, known[1]));
  ctas = min(ctas, ctx_resident_ctas(ctx, fused_kernel<false, true>(16), kFuThreads, 0, known[2]));
  return min(ctas, ctx_resident_ctas(ctx, fused_kernel<true, true>(16), kFuThreads, 0, known[3]));
}

bool fused_unique_suits(gsb_ctx* ctx, i64 n, i64 G) {
  // Several minibatches share the hash table's L2, and from a million items on the passes of the partitioned form are worth
  // their launches: 40 minibatches with 1.3 M items in the second hop 207 against 180 us for the call, 8 large ones with 1.8 M
  // 550 against 497; at half a million the single launch is still ahead (470 against 484).
  if (G > 1 && n > kFusedUniqueMaxItems / 2) return false;
  return n > 0 && n <= kFusedUniqueMaxItems && G <= kFusedUniqueMaxBatches &&
         n <= (i64)resident_ctas(ctx) * kFuThreads * 16;
}

// The direct-address table: 4 bytes per id and minibatch.  Up to 32 MB it lives in L2 beside what the call reads.
bool fused_unique_direct(i64 G, i64 id_bound) { return id_bound > 0 && (double)G * (double)id_bound * 4.0 <= (double)(32 << 20); }

template <bool BATCHED>
static int launch_fused(gsb_ctx* ctx, cudaStream_t stream, FusedParams p, i64 n, i64 id_bound) {
  const int r = items_per_thread(n, resident_ctas(ctx));
  const int grid = grid_for(n, kFuThreads * r);
  const i64 G = BATCHED ? p.G : 1;
  const bool direct = fused_unique_direct(G, id_bound);
  void* ws;
  const size_t packed_bytes = ((size_t)n / 32 + 2) * 8;
  int st = ctx_reserve_workspace(ctx, stream, packed_bytes + sizeof(u32) * (size_t)(kFuThreads + (p.col_index ? p.S : 0)), &ws);
  if (st != GSB_OK) return st;
  p.packed = (u64*)ws;
  p.totals = (u32*)((char*)ws + packed_bytes);
  p.seed_ref = p.totals + kFuThreads;
  void* table;
  u32 epoch;
  if (direct) st = ctx_epoch_table(ctx, 1, sizeof(u32) * (size_t)(G * id_bound), 0xFF, kFuEpochs, stream, &table, &epoch);
  else st = ctx_epoch_table(ctx, 0, 32 * (size_t)fused_bucket0((u32)n, (u32)G), 0, kFuEpochs, stream, &table, &epoch);
  if (st != GSB_OK) return st;
  p.table = (u64*)table;
  p.epoch = (u64)epoch << (32 + kFuPosBits);
  p.direct = (u32*)table;
  p.direct_epoch = (kFuEpochs - 1 - epoch) << kFuPosBits;
  p.id_bound = (u32)id_bound;
  p.counters = ctx_counters(ctx);
  p.sync = ctx_grid_sync(ctx, grid, 2);
  ScopedKernelTimer timer(ctx, KID_RELABEL, stream);
  void* args[] = {&p};
  return launch_cooperative(ctx, stream, direct ? fused_kernel<BATCHED, true>(r) : fused_kernel<BATCHED, false>(r), grid,
                            kFuThreads, 0, args, p.sync);
}

int fused_unique_single(gsb_ctx* ctx, cudaStream_t stream, const i64* first, i64 S, const i64* second, i64 E,
                        const i64* col_index, i64* out_unique, i64* out_second, i64* out_col, const i64* copy_src,
                        i64* copy_dst, i64 copy_n, float* ones, i64 id_bound, Mail mail) {
  FusedParams p{};
  p.first = first;
  p.second = second;
  p.S = S;
  p.E = E;
  p.out_unique = out_unique;
  p.out_second = out_second;
  p.col_index = out_col ? col_index : nullptr;
  p.out_col = out_col;
  p.copy_src = copy_src;
  p.copy_dst = copy_dst;
  p.copy_n = copy_src && copy_dst ? copy_n : 0;
  p.ones = ones;
  p.ones_n = ones ? E : 0;
  p.mail = mail;
  return launch_fused<false>(ctx, stream, p, S + E, id_bound);
}

int fused_unique_batched(gsb_ctx* ctx, cudaStream_t stream, const BatchLayout& L, i64 seeds_bound, i64 edges_bound,
                         const i64* sub_indptr, i64* out_indices_ptr, i64* out_unique, i64* out_unique_ptr,
                         i64* out_relabeled, i64 id_bound, Mail mail) {
  FusedParams p{};
  p.first = L.seeds;
  p.second = L.indices;
  p.S = seeds_bound;
  p.E = edges_bound;
  p.out_unique = out_unique;
  p.out_second = out_relabeled;
  p.seeds_ptr = L.seeds_ptr;
  p.indices_ptr = sub_indptr ? nullptr : L.indices_ptr;
  p.sub_indptr = sub_indptr;
  p.out_indices_ptr = sub_indptr ? out_indices_ptr : nullptr;
  p.out_unique_ptr = out_unique_ptr;
  p.G = L.G;
  p.mail = mail;
  return launch_fused<true>(ctx, stream, p, seeds_bound + edges_bound, id_bound);
}

}  // namespace gsb
