// Batched unique + relabel by classes of ids (see k_part_resolve_classes), for minibatches of 36 000 items and more.
//
// An item is the quotient of its id and its number in a tile of 16 384 items of one minibatch: one 32-bit word, half of what the
// partitioned form moves.  A tile sorts its own stretch by class, so nothing is counted before and nothing reserved across tiles:
//
//   scatter  words of a tile by class; per tile where every class starts, per item where its word went (16 bits);
//   resolve  a CTA per minibatch and class goes through the class's runs in all tiles of the minibatch (a hundred words each):
//            position minimum in shared memory, barrier, every word becomes the position of the first item with its id;
//   bits     the first positions back in the order of the items (a tile's words are read by the CTA that takes the tile), a bit per
//            item that is its own first one;
//   prefix   population counts of the bit words, one pass;
//   emit     frontier ids at their ranks, and for every neighbour the rank of the first item with its id.
//
// Items are numbered by tile throughout, so every minibatch begins at a tile, with bit words of its own.
//
// 500 minibatches of 813 000 items over 2.45 M nodes, ms, partitioned form / this: count 0.73 / none, scatter 1.94 / 1.29 (instruction
// issue and shared memory; tiles of 8 192 1.34), resolve 0.88 / 0.86 (1.52 out of tiles of 8 192, whose runs are shorter), bits
// 1.12 / 0.72, emit 2.20 / 1.78 (HBM).
#include "batch_table.cuh"
#include "common.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kTileThreads = 512;
constexpr u32 kClassThreads = 512;
constexpr int kTilePer = kClassTile / kTileThreads;
constexpr int kScatterBytes = 6 * kClassTile;  // a word and a rank per item
constexpr int kNumberBits = 14;  // of an item in its tile
constexpr u32 kNumberMask = (1u << kNumberBits) - 1;
static_assert(kClassTile == 1 << kNumberBits && (u64)kClassSlots * kClassTile < (1ull << 32), "quotient and number share a word");
constexpr int kMaxParts = 256;
constexpr int kTileWords = kClassTile / 32;
constexpr uint16_t kNoPlace = 0xFFFFu;
constexpr u32 kNoFirst = 0xFFFFFFFFu;

// Where a tile's items are: its minibatch and what the passes need of that.
struct __align__(16) TileOwner {
  u32 batch, tile0;        // the minibatch and its first tile
  u32 num_seeds, items;    // seeds first, then sampled neighbours
  i64 seeds, edges;        // the first of them; that of the neighbours minus num_seeds
};

struct ClassLayout {
  BatchLayout L;    // region_off: first tile of every minibatch
  TileOwner* owner; // [tiles]
  u32* words;       // [tiles][kClassTile] quotient : number, by class; then position in the minibatch of the id's first item
  uint16_t* place;  // [tiles][kClassTile] by item: where its word is
  uint16_t* start;  // [tiles][parts + 1]
  u32* ref;         // [tiles][kClassTile] by item: first position
  u32* bits;        // [tiles][kTileWords]
  u64* packed;      // [tiles][kTileWords], and one: first items before the word : 32 | bits : 32
  u64* spill;       // tables of the ids beyond the bound: 2 x kClassTile x first tile + 32 x minibatch
  u32 parts, magic;
  u32 chunks, chunk_magic;  // pieces that the runs of a class are dealt out in, and the factor that divides by them
};

// Minibatch of a tile, searched by a whole warp: 32 pivots a round.
__device__ __forceinline__ i64 minibatch_of_tile(const BatchLayout& L, i64 tile) {
  const i64 lane = threadIdx.x & 31;
  i64 lo = 0, end = L.G;  // the answer lies in [lo, end)
  while (end - lo > 1) {
    const i64 step = (end - lo + 31) >> 5;
    const i64 idx = lo + (lane + 1) * step;
    const bool le = idx < end && __ldg(L.region_off + idx) <= tile;
    const i64 hits = __popc(__ballot_sync(0xffffffffu, le));
    lo += hits * step;
    end = min(end, lo + step);
  }
  return lo;
}

__device__ __forceinline__ TileOwner owner_of(const BatchLayout& L, i64 b) {
  TileOwner t;
  t.batch = (u32)b;
  t.tile0 = (u32)__ldg(L.region_off + b);
  t.seeds = __ldg(L.seeds_ptr + b);
  t.num_seeds = (u32)(__ldg(L.seeds_ptr + b + 1) - t.seeds);
  const i64 edges = __ldg(L.indices_ptr + b);
  t.items = t.num_seeds + (u32)(__ldg(L.indices_ptr + b + 1) - edges);
  t.edges = edges - t.num_seeds;
  return t;
}
__device__ __forceinline__ TileOwner owner_of_tile(const ClassLayout& C, i64 tile) {
  TileOwner t;
  const uint4* from = reinterpret_cast<const uint4*>(C.owner + tile);
  uint4* to = reinterpret_cast<uint4*>(&t);
  to[0] = __ldg(from);
  to[1] = __ldg(from + 1);
  return t;
}
__device__ __forceinline__ i64 item_id(const BatchLayout& L, const TileOwner& t, u32 i) {
  return __ldg(i < t.num_seeds ? L.seeds + t.seeds + i : L.indices + t.edges + i);
}

// A thread keeps its 32 ids in registers between counting and placing, the next eight always on their way, and their ranks in shared
// memory.  Ranks in registers and ids read again (out of L2) took 1.45 ms for 407 M items and 0.38 for 82 M; this 1.29 and 0.31.  Without the second
// set of eight 1.36 and 0.33; 16 at once 1.35, four and four 1.35, 1 024 threads 1.36 and 0.31.
__global__ void __launch_bounds__(kTileThreads, 2) k_class_scatter(ClassLayout C, i64* counters) {
  extern __shared__ __align__(16) u32 s_words[];
  __shared__ u32 s_cnt[kMaxParts];
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = C.L;
  const i64 tile = blockIdx.x;
  if (tile >= L.region_off[L.G]) return;
  const u32 tid = threadIdx.x, lane = tid & 31;
  if (tid < kMaxParts) s_cnt[tid] = 0;
  const TileOwner t = owner_of(L, minibatch_of_tile(L, tile));
  if (tid == 0) C.owner[tile] = t;
  const u32 first = ((u32)tile - t.tile0) * kClassTile, here = min((u32)kClassTile, t.items - first);
  uint16_t* place = C.place + tile * kClassTile + tid;
  constexpr int kAhead = 8;
  const bool mixed = first < t.num_seeds && first + here > t.num_seeds;
  const i64* from = (first >= t.num_seeds ? L.indices + t.edges : L.seeds + t.seeds) + first + tid;
  auto load = [&](int q0, i64 (&node)[kAhead]) {
    if (!mixed) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) node[q] = (q0 + q) * kTileThreads + tid < here ? __ldg(from + (q0 + q) * kTileThreads) : -1;
    } else {
#pragma unroll 1
      for (int q = 0; q < kAhead; ++q) {
        const u32 i = (q0 + q) * kTileThreads + tid;
        const i64 v = i < here ? item_id(L, t, first + i) : -1;
#pragma unroll
        for (int z = 0; z < kAhead; ++z)
          if (z == q) node[z] = v;
      }
    }
  };
  struct Split {
    u32 c, quotient;
  };
  auto split = [&](u32 id) {
    const u32 q = __umulhi(id, C.magic);
    return q < kClassSlots ? Split{id - q * (C.parts - 1), q} : Split{C.parts - 1, 0};  // beyond the bound: looked up again
  };
  __syncthreads();
  constexpr u32 kNoId = 0xFFFFFFFFu;
  uint16_t* s_rank = reinterpret_cast<uint16_t*>(s_words + kClassTile) + tid;  // by item: its rank in the tile's share of the class
  u32 ids[kTilePer];
  i64 node[2][kAhead];
  load(0, node[0]);
#pragma unroll
  for (int q0 = 0; q0 < kTilePer; q0 += kAhead) {
    i64(&now)[kAhead] = node[q0 / kAhead % 2];
    if (q0 + kAhead < kTilePer) load(q0 + kAhead, node[(q0 / kAhead + 1) % 2]);
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      u32 own = 0;
      ids[q0 + q] = valid_id(now[q]) ? (u32)now[q] : kNoId;
      if (valid_id(now[q])) own = atomicAdd(&s_cnt[split((u32)now[q]).c], 1u);
      s_rank[(q0 + q) * kTileThreads] = (uint16_t)own;
    }
  }
  __syncthreads();
  if (tid < 32) {
    constexpr int kPer = kMaxParts / 32;
    u32 c[kPer], sum = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) sum += c[j] = s_cnt[lane * kPer + j];
    u32 run = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, run, o);
      if (lane >= o) run += x;
    }
    run -= sum;
    uint16_t* start = C.start + tile * (C.parts + 1);
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const u32 k = lane * kPer + j;
      s_cnt[k] = run;
      if (k <= C.parts) start[k] = (uint16_t)run;
      run += c[j];
    }
    if (lane == 31 && C.parts == kMaxParts) start[kMaxParts] = (uint16_t)run;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kTilePer; ++q) {
    const u32 i = q * kTileThreads + tid;
    if (i >= here) break;
    u32 to = kNoPlace;
    if (ids[q] != kNoId) {
      const Split s = split(ids[q]);
      to = s_cnt[s.c] + s_rank[q * kTileThreads];
      s_words[to] = s.quotient << kNumberBits | i;
    } else {
      raise_error(counters, GSB_ERR_INDEX_RANGE, (i64)first + i);
    }
    place[q * kTileThreads] = (uint16_t)to;
  }
  __syncthreads();
  uint4* out = reinterpret_cast<uint4*>(C.words + tile * kClassTile);
  for (u32 i = tid; i < (here + 3) / 4; i += kTileThreads) out[i] = reinterpret_cast<const uint4*>(s_words)[i];
}

// Ids beyond the bound: a table of their own in global memory, by a whole CTA.
__device__ __noinline__ void resolve_beyond(const ClassLayout& C, i64 b, u32 tile_end, u64* table) {
  const TileOwner t = owner_of(C.L, b);
  const u32 c = C.parts - 1;
  u32 n = 0;
  for (u32 tile = t.tile0; tile < tile_end; ++tile) {
    const uint16_t* start = C.start + (i64)tile * (C.parts + 1) + c;
    n += start[1] - start[0];
  }
  if (n == 0) return;
  const u32 size = 2 * n + 32;
  auto home = [size](u32 id) {
    u32 x = id * 0x85EBCA6Bu;
    x ^= x >> 13;
    x *= 0xC2B2AE35u;
    x ^= x >> 16;
    return __umulhi(x, size);
  };
  auto each = [&](auto f) {  // f(word, id, position)
    for (u32 tile = t.tile0; tile < tile_end; ++tile) {
      const uint16_t* start = C.start + (i64)tile * (C.parts + 1) + c;
      u32* words = C.words + (i64)tile * kClassTile;
      for (u32 j = start[0] + threadIdx.x; j < start[1]; j += kClassThreads) {
        const u32 at = (tile - t.tile0) * kClassTile + words[j];
        f(words + j, (u32)item_id(C.L, t, at), at);
      }
    }
  };
  __syncthreads();
  for (u32 i = threadIdx.x; i < size; i += kClassThreads) table[i] = kEmptyWord;
  __syncthreads();
  each([&](u32*, u32 id, u32 at) {
    const u64 mine = ((u64)id << 32) | at;
    u32 h = home(id);
    for (u32 probe = 0; probe < size; ++probe) {  // more slots than items: ends at one of them
      u64 w = *(volatile u64*)(table + h);
      if (w == kEmptyWord) w = atomicCAS(table + h, kEmptyWord, mine);
      if (w == kEmptyWord) break;
      if ((u32)(w >> 32) == id) {
        if (w > mine) atomicMin(table + h, mine);
        break;
      }
      h = h + 1 == size ? 0 : h + 1;
    }
  });
  __syncthreads();
  each([&](u32* word, u32 id, u32) {
    u32 h = home(id), found = kNoFirst;
    for (u32 probe = 0; probe < size; ++probe) {
      const u64 x = __ldcg(table + h);
      if (x == kEmptyWord) break;
      if ((u32)(x >> 32) == id) {
        found = (u32)x;
        break;
      }
      h = h + 1 == size ? 0 : h + 1;
    }
    *word = found;
  });
  __syncthreads();
}

// A bucket of a minibatch whose positions take more than 20 bits (see below), by a whole CTA with a table that it clears and leaves
// as it is.
__device__ __noinline__ void resolve_wide(const ClassLayout& C, u32 tile0, u32 tiles, u32 c, u32* s_first) {
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto each = [&](auto f) {  // f(word, position of the tile)
    for (u32 t = warp; t < tiles; t += kClassThreads / 32) {
      const uint16_t* start = C.start + ((size_t)(tile0 + t) * (C.parts + 1) + c);
      u32* words = C.words + (size_t)(tile0 + t) * kClassTile;
      for (u32 j = start[0] + lane; j < start[1]; j += 32) f(words + j, t * kClassTile);
    }
  };
  __syncthreads();  // the previous bucket's look-ups are done
  for (u32 i = threadIdx.x; i < kClassSlots; i += kClassThreads) s_first[i] = kNoFirst;
  __syncthreads();
  each([&](u32* word, u32 before) { atomicMin(s_first + (*word >> kNumberBits), before + (*word & kNumberMask)); });
  __syncthreads();
  each([&](u32* word, u32) { *word = s_first[*word >> kNumberBits]; });
}

constexpr int kSlots = kClassTile / 4096;  // loads of a warp for a run
constexpr int kPositionBits = 20;
constexpr u32 kFirstEpoch = (1u << (32 - kPositionBits)) - 1;
constexpr u32 kEpochTiles = ((1u << kPositionBits) - 1) / kClassTile;
constexpr int kKept = 4;  // pieces of a warp that stay in registers
constexpr u32 kMaxChunks = 8;  // no more than 32 pieces to a warp
static_assert(kEpochTiles * kMaxChunks <= 32 * kClassThreads / 32, "a lane to each");

// CUT: the runs are long enough to be cut into pieces.
// Two CTAs per SM, with registers for the pieces and the look-ahead: 843 us for 500 minibatches of 813 000 items; three, which spill 76
// bytes a thread, 1 088; clearing the table for every bucket 1 200.
template <bool CUT>
__global__ void __launch_bounds__(kClassThreads, 2) k_class_resolve(const __grid_constant__ ClassLayout C, i64* counters) {
  extern __shared__ __align__(16) u32 s_first[];  // [kClassSlots] smallest position of every id
  if (counters[CNT_ABORT] != 0) return;
  constexpr u32 kWarps = kClassThreads / 32;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5, parts = C.parts, G = (u32)C.L.G;
  // The runs of a bucket are cut into `chunks` pieces each, all but the last of 32 kSlots words, and the warp's are number `warp` and
  // every kWarps-th from there on; lane m knows number m.  kBeyond: the bucket is that of the ids beyond the bound.
  constexpr u32 kBeyond = 1u << 31;
  const u32 buckets = G * parts, magic = 0xFFFFFFFFu / parts + 1;
  const u32 chunks = CUT ? C.chunks : 1;
  const u32 piece = warp + lane * kWarps, own_tile = CUT ? __umulhi(piece, C.chunk_magic) : piece;
  const u32 own_first = (piece - own_tile * chunks) * (32 * kSlots);  // word of the run, and whether the piece is the run's last
  const bool own_last = !CUT || piece + 1 == (own_tile + 1) * chunks;
  u32 next_tile0 = 0, next_tiles = 0;
  u32 next_begin = 0, next_end = 0;  // put together where they are used: in here that would wait for them
  auto look_ahead = [&](u32 k) {
    if (k >= buckets) return;
    u32 b = __umulhi(k, magic);  // k / parts, or one more
    u32 c = k - b * parts;
    if (c >= parts) --b, c += parts;
    next_tile0 = (u32)__ldg(C.L.region_off + b);
    next_tiles = (u32)__ldg(C.L.region_off + b + 1) - next_tile0;
    next_begin = next_end = 0;
    if (own_tile < next_tiles) {
      const uint16_t* start = C.start + ((size_t)(next_tile0 + own_tile) * (parts + 1) + c);
      next_begin = __ldg(start);
      next_end = __ldg(start + 1);
    }
    if (c == parts - 1) next_tiles |= kBeyond;
  };
  look_ahead(blockIdx.x);
  // A table word is [epoch : 12 | position : 20]: every bucket takes a smaller epoch than the one before, so that its positions beat
  // what that left behind and the table is not cleared in between.
  u32 epoch = 0;
  for (u32 k = blockIdx.x; k < buckets; k += gridDim.x) {
    const u32 tile0 = next_tile0, all = next_tiles;
    const u32 from_word = min(next_begin + own_first, next_end);
    const u32 run = from_word | (own_last ? next_end : min(from_word + 32 * kSlots, next_end)) << 16;  // [end : 16 | begin : 16]
    if (all == 0 || all >= kBeyond) {
      if (all > kBeyond) resolve_beyond(C, k / parts, tile0 + all - kBeyond, C.spill + 2ull * kClassTile * tile0 + 32ull * (k / parts));
      look_ahead(k + gridDim.x);
      continue;
    }
    if (all > kEpochTiles) {
      resolve_wide(C, tile0, all, k % parts, s_first);
      epoch = 0;
      look_ahead(k + gridDim.x);
      continue;
    }
    const u32 pieces = all * chunks > warp ? (all * chunks - warp + kWarps - 1) / kWarps : 0;
    u32* words = C.words + ((size_t)tile0 * kClassTile + lane);
    u32 w[kSlots * kKept], at[kKept];  // their loads are in flight while the next runs are looked up
#pragma unroll
    for (int m = 0; m < kKept; ++m) {
#pragma unroll
      for (int h = 0; h < kSlots; ++h) w[kSlots * m + h] = kNoFirst;
      if (m >= pieces) continue;  // uniform
      const u32 r = __shfl_sync(0xffffffffu, run, m), begin = r & 0xFFFFu, n = (r >> 16) - begin;
      at[m] = (CUT ? __shfl_sync(0xffffffffu, own_tile, m) : warp + m * kWarps) * kClassTile;
      const u32* from = words + (at[m] + begin);
#pragma unroll
      for (int h = 0; h < kSlots; ++h)
        if (lane + 32 * h < n) w[kSlots * m + h] = from[32 * h];
    }
    // what does not stay: f(word, position of the tile) for the rest of long runs and the pieces behind
    const bool more = pieces > kKept || __any_sync(0xffffffffu, (run >> 16) - (run & 0xFFFFu) > 32 * kSlots);
    auto rest = [&](auto f) {
#pragma unroll 1
      for (u32 m = 0; m < pieces; ++m) {  // uniform
        const u32 r = __shfl_sync(0xffffffffu, run, m), tile = __shfl_sync(0xffffffffu, own_tile, m) * kClassTile;
#pragma unroll 1
        for (u32 j = (r & 0xFFFFu) + (m < kKept ? 32 * kSlots : 0); j + lane < r >> 16; j += 32) f(words + (tile + j), tile);
      }
    };
    look_ahead(k + gridDim.x);
    __syncthreads();  // the previous bucket's look-ups are done
    if (epoch == 0) {
      const uint4 e = make_uint4(kNoFirst, kNoFirst, kNoFirst, kNoFirst);
      for (u32 i = threadIdx.x; i < kClassSlots / 4; i += kClassThreads) reinterpret_cast<uint4*>(s_first)[i] = e;
      epoch = kFirstEpoch + 1;
      __syncthreads();
    }
    --epoch;
    const u32 tag = epoch << kPositionBits;
    constexpr u32 kMask = (1u << kPositionBits) - 1;
#pragma unroll
    for (int m = 0; m < kKept; ++m) {
      if (m >= pieces) continue;
#pragma unroll
      for (int h = 0; h < kSlots; ++h) {
        const u32 x = w[kSlots * m + h];
        if (x != kNoFirst) atomicMin(s_first + (x >> kNumberBits), tag + at[m] + (x & kNumberMask));
      }
    }
    if (more) rest([&](u32* word, u32 before) { atomicMin(s_first + (*word >> kNumberBits), tag + before + (*word & kNumberMask)); });
    if (own_last && next_begin < next_end) {  // the next bucket's words on their way to L2
      const u32* from = C.words + (size_t)(next_tile0 + own_tile) * kClassTile;
      for (u32 j = next_begin; j < next_end + 31; j += 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(from + min(j, next_end - 1)));
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kKept; ++m) {
      if (m >= pieces) continue;
      u32* to = words + (at[m] + (__shfl_sync(0xffffffffu, run, m) & 0xFFFFu));
#pragma unroll
      for (int h = 0; h < kSlots; ++h)
        if (w[kSlots * m + h] != kNoFirst) to[32 * h] = s_first[w[kSlots * m + h] >> kNumberBits] & kMask;
    }
    if (more) rest([&](u32* word, u32) { *word = s_first[*word >> kNumberBits] & kMask; });
  }
}

// A lane takes eight consecutive items at a time.
constexpr int kBitsThreads = 1024;

__global__ void __launch_bounds__(kBitsThreads) k_class_bits(ClassLayout C, i64* counters) {
  extern __shared__ __align__(16) u32 s_words[];
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = C.L;
  const i64 tile = blockIdx.x;
  if (tile >= L.region_off[L.G]) return;
  const TileOwner t = owner_of_tile(C, tile);
  const u32 first = ((u32)tile - t.tile0) * kClassTile, here = min((u32)kClassTile, t.items - first);
  union Places {
    uint4 v;
    uint16_t at[8];
  } place[kClassTile / 8 / kBitsThreads];
#pragma unroll
  for (int h = 0; h < kClassTile / 8 / kBitsThreads; ++h) {
    const u32 i0 = (h * kBitsThreads + threadIdx.x) * 8;
    place[h].v = i0 < here ? __ldg(reinterpret_cast<const uint4*>(C.place + tile * kClassTile + i0)) : make_uint4(0, 0, 0, 0);
  }
  const uint4* words = reinterpret_cast<const uint4*>(C.words + tile * kClassTile);
  for (u32 i = threadIdx.x; i < (here + 3) / 4; i += kBitsThreads) reinterpret_cast<uint4*>(s_words)[i] = __ldg(words + i);
  __syncthreads();
#pragma unroll
  for (int h = 0; h < kClassTile / 8 / kBitsThreads; ++h) {
    const u32 i0 = (h * kBitsThreads + threadIdx.x) * 8;
    u32 r[8], own = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = i0 + j < here && place[h].at[j] != kNoPlace ? s_words[place[h].at[j]] : kNoFirst;
#pragma unroll
    for (int j = 0; j < 8; ++j) own |= (r[j] == first + i0 + j ? 1u : 0u) << j;
    if (i0 < here) {
      uint4* ref = reinterpret_cast<uint4*>(C.ref + tile * kClassTile + i0);
      ref[0] = make_uint4(r[0], r[1], r[2], r[3]);
      ref[1] = make_uint4(r[4], r[5], r[6], r[7]);
    }
    own <<= 8 * (threadIdx.x & 3);
    own |= __shfl_xor_sync(0xffffffffu, own, 1);
    own |= __shfl_xor_sync(0xffffffffu, own, 2);
    if ((threadIdx.x & 3) == 0) C.bits[tile * kTileWords + i0 / 32] = own;
  }
}

constexpr int kPrefixThreads = 256;
constexpr int kPrefixPer = 8;
constexpr int kPrefixTile = kPrefixThreads * kPrefixPer;  // words per CTA

__global__ void __launch_bounds__(kPrefixThreads) k_class_prefix(ClassLayout C, CompactOut out, i64* counters, TileState ts) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = C.L;
  const i64 words = L.region_off[L.G] * kTileWords;
  const int tile = blockIdx.x;
  const i64 first = (i64)tile * kPrefixTile + (i64)threadIdx.x * kPrefixPer;
  if ((i64)tile * kPrefixTile >= words && !(words == 0 && tile == 0)) return;
  u32 b[kPrefixPer];
  i64 sum = 0;
#pragma unroll
  for (int j = 0; j < kPrefixPer; ++j) {
    b[j] = first + j < words ? C.bits[first + j] : 0u;
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
    if (first + j < words) C.packed[first + j] = ((u64)run << 32) | (u64)b[j];
    run += __popc(b[j]);
  }
  if ((i64)(tile + 1) * kPrefixTile >= words && threadIdx.x == 0) {
    const i64 all = s_base + total;
    out.unique_ptr[L.G] = all;
    for (i64 e = L.G - 1; e >= 0 && L.region_off[e] * kTileWords == words; --e) out.unique_ptr[e] = all;
    counters[CNT_UNIQUE] = all;
    counters[CNT_NNZ] = L.indices_ptr[L.G];
    mail_post(out.mail, 0, all, counters);
    mail_post(out.mail, 1, L.indices_ptr[L.G], counters);
  }
}

constexpr int kEmitThreads = 256;
constexpr int kEmitGroups = 4;
constexpr int kEmitItems = kEmitThreads * kEmitGroups;

__device__ __forceinline__ u32 rank_in(u64 w, u32 bit) { return (u32)(w >> 32) + __popc((u32)w & ((1u << bit) - 1u)); }

// The outputs are stored as what nobody reads soon: they are most of the traffic, and what the pass looks up stays in L2 (400 M items
// 1.95 -> 1.78 ms; in k_rank_emit 7.2 M 44.5 -> 41.4 us; the sampling passes, the row copy and the other passes here are no faster
// with it).  Two / eight groups a warp 2.16 / 2.93 ms, six CTAs an SM 2.35.
__global__ void __launch_bounds__(kEmitThreads) k_class_emit(ClassLayout C, CompactOut out, i64* __restrict__ out_relabeled,
                                                             i64* counters) {
  if (counters[CNT_ABORT] != 0) return;
  const BatchLayout& L = C.L;
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const i64 tile = blockIdx.x / (kClassTile / kEmitItems);
  if (tile >= L.region_off[L.G]) return;
  const i64 at = (i64)blockIdx.x * kEmitItems + warp * (kEmitGroups * 32);  // of the warp's first item
  // loads that depend on nothing first
  u32 r[kEmitGroups];
  u64 own[kEmitGroups];
#pragma unroll
  for (int q = 0; q < kEmitGroups; ++q) {
    r[q] = __ldg(C.ref + at + q * 32 + lane);
    own[q] = __ldg(C.packed + (at >> 5) + q);
  }
  const TileOwner t = owner_of_tile(C, tile);
  const u32 first = (u32)(at - (i64)t.tile0 * kClassTile) + lane;
  const u64* win = C.packed + (i64)t.tile0 * kTileWords;
  const u32 front = (u32)(__ldg(win) >> 32);
  i64* rel = out_relabeled ? out_relabeled + t.edges : nullptr;
  const i64 *seeds = L.seeds + t.seeds, *edges = L.indices + t.edges;
  const u32 items = t.items, ns = t.num_seeds;
  u64 of_first[kEmitGroups];
  i64 node[kEmitGroups];
#pragma unroll
  for (int q = 0; q < kEmitGroups; ++q) {
    const u32 i = first + q * 32;
    of_first[q] = i < items && i >= ns && r[q] < items ? __ldg(win + (r[q] >> 5)) : 0;
    node[q] = i < items && r[q] == i ? __ldg(i < ns ? seeds + i : edges + i) : 0;
  }
#pragma unroll
  for (int q = 0; q < kEmitGroups; ++q) {
    const u32 i = first + q * 32;
    if (i >= items) continue;
    const u32 pos = rank_in(own[q], lane);
    if (r[q] == i) __stcs(out.unique + pos, node[q]);
    // an id outside the accepted range has no word and its ref says so
    if (i >= ns && rel) __stcs(rel + i, r[q] < items ? (i64)(rank_in(of_first[q], r[q] & 31u) - front) : (i64)-1);
  }
  if (first == 0) {  // the frontier of the minibatch starts here; empty minibatches before it start here too
    out.unique_ptr[t.batch] = front;
    for (i64 e = (i64)t.batch - 1; e >= 0 && __ldg(L.region_off + e) == (i64)t.tile0; --e) out.unique_ptr[e] = front;
  }
}

// ---- host ---------------------------------------------------------------------------------------------------------------
static inline size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

// us of a whole call, hashed buckets / the partitioned form with classes / this (ids scattered evenly; in brackets: by a power law
// numbered by degree), by nodes and items of a minibatch:
//   40 M items, 2.45 M nodes    76 000 959 / 1173 / 892 (977 / 1172 / 962)    106 400 960 / 1029 / 768 (962 / 1032 / 825)
//                               243 200 945 / 828 / 617 (950 / 830 / 643)      760 000 929 / 730 / 526 (999 / 740 / 562)
//               1 M nodes       34 000 992 / 1196 / 1034 (951 / 1198 / 1106)   47 600 958 / 1033 / 843 (1044 / 1033 / 899)
//                               108 800 934 / 827 / 643 (941 / 827 / 673)      340 000 916 / 721 / 539 (952 / 727 / 582)
//               700 000         30 800 992 / 1063 / 869 (955 / 1067 / 930)     70 400 938 / 826 / 674 (941 / 829 / 719)
//               500 000         38 400 970 / 900 / 756 (994 / 902 / 913)       51 200 936 / 811 / 697 (942 / 812 / 815)
//               180 000         19 200 996 / 888 / 1291 (943 / 883 / 1420)     60 000 916 / 746 / 893 (929 / 750 / 1004)
//   1.4 M items, 2.45 M nodes   136 800 91 / 86 / 67 (129 / 89 / 72)           760 000 (one) 73 / 60 / 58 (171 / 73 / 71)
// With few classes a tile's run is longer than the pieces it is cut into; with few tiles SMs are left idle.  Few large minibatches gain
// or lose by how their ids crowd, partitioned with classes / this, evenly and (as fourth powers): 700 000 nodes, 4.1 M items in 6
// 121 / 97 (134 / 152), 8 M in 8 194 / 184 (218 / 261), in 24 189 / 154 (197 / 180); 2.45 M nodes, 4.1 M in 2 113 / 110 (142 / 158), in 4
// 118 / 86 (131 / 113).
bool class_tiled(i64 path, i64 num_nodes, i64 items, i64 G) {
  const i64 parts = path == 0 || path == 5 ? partition_class_parts(num_nodes, items / G, true) : 0;
  if (parts <= 0 || parts > kMaxParts || G > items / (kClassTile / 2) + 4096) return false;
  if (path == 5) return true;
  const i64 minibatch = items / G;
  return parts >= 40 && minibatch >= max(700 * parts, (i64)36'000) && (items >= 4'000'000 || minibatch < 1600 * parts);
}

i64 class_tiles(i64 n_cap, i64 G) { return n_cap / kClassTile + G; }

size_t class_workspace_bytes(i64 n_cap, i64 G, i64 parts) {
  const size_t tiles = (size_t)class_tiles(n_cap, G), items = tiles * kClassTile;
  return al256(sizeof(TileOwner) * tiles) + al256(4 * items) + al256(2 * items) + al256(2 * tiles * (size_t)(parts + 1)) + al256(4 * items) + al256(4 * tiles * kTileWords) +
         al256(8 * (tiles * kTileWords + 1)) + al256(8 * (2 * items + 32 * (size_t)G));
}

int class_unique_relabel(gsb_ctx* ctx, cudaStream_t stream, const BatchLayout& L, i64 n_cap, void* ws, i64 parts, i64* out_unique,
                         i64* out_unique_ptr, i64* out_relabeled, Mail mail) {
  i64* counters = ctx_counters(ctx);
  const i64 tiles = class_tiles(n_cap, L.G), items = tiles * kClassTile;
  ClassLayout C;
  C.L = L;
  C.parts = (u32)parts;
  C.magic = class_magic(parts);
  C.chunks = (u32)min((i64)kMaxChunks, (kClassTile / (parts - 1) + 12 + 32 * kSlots - 1) / (32 * kSlots));  // most runs of the mean's size fit
  C.chunk_magic = 0xFFFFFFFFu / C.chunks + 1;
  char* at = (char*)ws;
  auto take = [&](size_t bytes) {
    char* p = at;
    at += al256(bytes);
    return p;
  };
  C.owner = (TileOwner*)take(sizeof(TileOwner) * (size_t)tiles);
  C.words = (u32*)take(4 * (size_t)items);
  C.place = (uint16_t*)take(2 * (size_t)items);
  C.start = (uint16_t*)take(2 * (size_t)tiles * (size_t)(parts + 1));
  C.ref = (u32*)take(4 * (size_t)items);
  C.bits = (u32*)take(4 * (size_t)tiles * kTileWords);
  C.packed = (u64*)take(8 * ((size_t)tiles * kTileWords + 1));
  C.spill = (u64*)at;
  static bool attr_set[64] = {};
  const int dev = ctx_device(ctx);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    GSB_CUDA_OK(cudaFuncSetAttribute(k_class_resolve<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kClassSlots * 4));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_class_resolve<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kClassSlots * 4));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_class_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, kScatterBytes));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_class_bits, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * kClassTile));
    attr_set[dev] = true;
  }
  {
    ScopedKernelTimer timer(ctx, KID_PART_SCATTER, stream);
    k_class_scatter<<<(int)tiles, kTileThreads, kScatterBytes, stream>>>(C, counters);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_PART_RESOLVE, stream);
    const int grid = (int)min(L.G * parts, (i64)kNumSMs * 2);
    if (C.chunks > 1) k_class_resolve<true><<<grid, kClassThreads, kClassSlots * 4, stream>>>(C, counters);
    else k_class_resolve<false><<<grid, kClassThreads, kClassSlots * 4, stream>>>(C, counters);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_FIRST_BITS, stream);
    k_class_bits<<<(int)tiles, kBitsThreads, 4 * kClassTile, stream>>>(C, counters);
  }
  GSB_LAUNCH_OK();
  const int prefix_tiles = grid_for(tiles * kTileWords, kPrefixTile);
  TileState ts;
  const int st = ctx_tile_state(ctx, prefix_tiles, stream, &ts);
  if (st != GSB_OK) return st;
  const CompactOut out{out_unique, out_unique_ptr, mail};
  {
    ScopedKernelTimer timer(ctx, KID_OTHER, stream);
    k_class_prefix<<<prefix_tiles, kPrefixThreads, 0, stream>>>(C, out, counters, ts);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_RANK_EMIT, stream);
    k_class_emit<<<grid_for(items, kEmitItems), kEmitThreads, 0, stream>>>(C, out, out_relabeled, counters);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // namespace gsb
