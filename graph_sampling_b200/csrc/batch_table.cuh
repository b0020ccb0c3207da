// Per-minibatch hash-table regions of the batched unique + relabel: one 64-bit word per slot
// (id << 32 | position), empty = all ones, multiplicative hashing, linear probing inside the region.
#pragma once
#include "common.cuh"

namespace gsb {

constexpr u64 kEmptyWord = 0xFFFFFFFFFFFFFFFFull;
constexpr uint32_t kFinalBit = 0x80000000u;

// Slots of a table region for `items` insertions: load <= 0.5.  Denser tables (load 0.8 was tried) cost more than
// the memset they save: linear probing then has probe runs of hundreds of slots, which set the duration of a
// small call outright (one warp walks them with dependent loads) and still cost 7 % on a 256-batch call.
__host__ __device__ __forceinline__ i64 region_size_for(i64 items) { return 2 * items + 32; }

__device__ __forceinline__ i64 home_slot(i64 node, i64 size) {
  const uint32_t h = (uint32_t)(((u64)node * 0x9E3779B97F4A7C15ull) >> 32);
  return (i64)(((u64)h * (u64)size) >> 32);
}

__device__ __forceinline__ bool valid_id(i64 node) { return node >= 0 && node < 0xFFFFFFFFll; }

// Insert with the home slot's current word already loaded (`w`): plain loads suffice when the id is
// present with a smaller position; otherwise CAS / atomicMin, then linear probing.
__device__ __forceinline__ bool insert_from(u64* region, i64 size, i64 h, u64 w, i64 node, u64 mine) {
  for (i64 probe = 0; probe < size; ++probe) {
    u64* s = region + h;
    if (probe > 0) w = __ldcg(s);
    if (w == kEmptyWord) {
      const u64 old = atomicCAS(s, kEmptyWord, mine);
      if (old == kEmptyWord) return true;
      w = old;
    }
    if ((w >> 32) == (u64)node) {
      if ((uint32_t)w > (uint32_t)mine) atomicMin(s, mine);
      return true;
    }
    h = (h + 1 == size) ? 0 : h + 1;
  }
  return false;
}

// Lookup with the home slot's word already loaded.  Returns the slot or nullptr; *word receives its value.
__device__ __forceinline__ u64* find_from(u64* region, i64 size, i64 h, u64 w, i64 node, u64* word) {
  for (i64 probe = 0; probe < size; ++probe) {
    u64* s = region + h;
    if (probe > 0) w = *s;
    if ((w >> 32) == (u64)node) {
      *word = w;
      return s;
    }
    if (w == kEmptyWord) return nullptr;
    h = (h + 1 == size) ? 0 : h + 1;
  }
  return nullptr;
}

// Largest b with off[b] <= g  (off has G + 1 non-decreasing entries, off[0] <= g < off[G]).
__device__ __forceinline__ i64 batch_of(const i64* __restrict__ off, i64 G, i64 g) {
  i64 lo = 0, hi = G;
  while (hi - lo > 1) {
    const i64 mid = (lo + hi) >> 1;
    if (__ldg(off + mid) <= g) lo = mid;
    else hi = mid;
  }
  return lo;
}

// Calls f(i, b) for every item i in [0, n) with b = its batch (off: G + 1 offsets).  A warp takes 256 consecutive
// items: one binary search for the first of them, then the batch number only walks forward — one search per 256
// items instead of one per item (a search is 8 dependent loads whichever lanes take part).
template <class F>
__device__ __forceinline__ void for_each_item_with_batch(const i64* __restrict__ off, i64 G, i64 n, F f) {
  constexpr int kPerLane = 8;
  const int lane = threadIdx.x & 31;
  const i64 warps = (i64)gridDim.x * (blockDim.x >> 5);
  for (i64 base = ((i64)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * (32 * kPerLane); base < n;
       base += warps * (32 * kPerLane)) {
    i64 b = batch_of(off, G, base);
    i64 next = __ldg(off + b + 1);
#pragma unroll
    for (int q = 0; q < kPerLane; ++q) {
      const i64 i = base + q * 32 + lane;
      if (i >= n) break;
      while (i >= next && b + 1 < G) {  // (the bound only matters for offsets that do not cover n)
        ++b;
        next = __ldg(off + b + 1);
      }
      f(i, b);
    }
  }
}

// ---- layout of a super-batch call (shared by the hash-table and the direct-address kernels) ----------------
constexpr int kBThreads = 256;
constexpr int kBPerThread = 4;
constexpr int kBTile = kBThreads * kBPerThread;

struct BatchLayout {
  const i64* seeds;
  const i64* seeds_ptr;    // [G + 1]
  const i64* indices;
  const i64* indices_ptr;  // [G + 1]
  i64 G;
  i64* item_off;    // [G + 1]  seeds_ptr[b] + indices_ptr[b]
  i64* region_off;  // [G + 1]  slot offsets
  u64* slots;
  i64 slot_capacity;
};


// ---- traversal by warp tiles ------------------------------------------------------------------------
// A warp owns kWarpItems consecutive items, lane-strided so that loads coalesce.  Items are batch-major,
// so almost every tile lies inside ONE batch: the batch is found once per tile (one binary search per
// 128 items instead of one per item) and its parameters stay in warp-uniform registers.  The rare tile
// that straddles a batch boundary resolves each item on its own (resolve_item).  Each lane first issues
// the loads of its four ids, then the four home-slot probes, so four independent memory round trips are
// in flight per lane; only a collision enters the probing loop.
constexpr int kLaneItems = 4;
constexpr int kWarpItems = 32 * kLaneItems;

struct BatchUniform {
  i64 batch, begin, next_begin, seeds_begin, num_seeds, edges_begin;
  u64* region;
  i64 size;
};

template <bool WITH_REGION = true>
__device__ __forceinline__ BatchUniform load_batch(const BatchLayout& L, const i64* __restrict__ off, i64 b) {
  BatchUniform u;
  u.batch = b;
  u.begin = __ldg(off + b);
  u.next_begin = __ldg(off + b + 1);
  u.seeds_begin = __ldg(L.seeds_ptr + b);
  u.num_seeds = __ldg(L.seeds_ptr + b + 1) - u.seeds_begin;
  u.edges_begin = __ldg(L.indices_ptr + b);
  u.region = nullptr;
  u.size = 0;
  if (WITH_REGION) {
    const i64 ro = __ldg(L.region_off + b);
    u.region = L.slots + ro;
    u.size = __ldg(L.region_off + b + 1) - ro;
  }
  return u;
}

// Direct-address tables of a super-batch call: table b (num_nodes words) belongs to minibatch b.  A word is
// [~epoch : 32 | key : 32]; atomicMin keeps, per node id, the smallest key of the CURRENT call (a larger epoch gives
// a smaller upper half, so entries of earlier calls lose against any entry of this one and the tables are never
// cleared).  Keys grow with the position of an item inside its minibatch: a seed's key is its index among the
// minibatch's seeds, a sampled neighbour's key is kEdgeKeyBit | its position in the call's edge array.
struct DirectTables {
  u64* words;
  i64 num_nodes;
  u64 epoch_hi;            // (u64)(~epoch) << 32
  uint32_t* rank_of_item;  // [items of the call]: frontier position of an item that is a first occurrence
  int seeds_distinct;      // the caller promises that no id repeats among the seeds of a minibatch
};
constexpr uint32_t kEdgeKeyBit = 0x80000000u;

// insert -> first-occurrence compaction -> relabel with direct-address tables (defined in direct_relabel.cu).
// L.item_off must be valid (k_batch_layout); n_cap / e_cap bound the items / edges of the call.
int direct_unique_relabel_launch(gsb_ctx* ctx, cudaStream_t stream, const BatchLayout& L, const DirectTables& T,
                                 i64 n_cap, i64 e_cap, i64* out_unique, i64* out_unique_ptr, i64* out_relabeled,
                                 Mail mail);
// Partitioned form of the batched unique + relabel (defined in partition_relabel.cu): shared-memory tables per bucket of
// items, bit-vector ranking, no fix-up pass.  L carries seeds / seeds_ptr / indices / indices_ptr / G; item_off and
// region_off (first bucket of every minibatch) must be filled by k_batch_layout; `ws` is scratch of
// partition_workspace_bytes(n_cap, bucket_cap) bytes and begins with the per-bucket item counts.  counted = true: the
// counts and bucket starts are already there (the sampler of the same hop counted, partition_after_sampler did the
// rest) and the counting and scan passes are skipped.
// parts > 0: buckets are the parts - 1 classes of ids with the same remainder by that number (partition_class_parts), and one more
// that takes the ids from the bound on; parts = 0: buckets by a hash of the id.
constexpr uint32_t kClassSlots = 1u << 14;  // ids of a class at most, a word of shared memory each
i64 partition_class_parts(i64 num_nodes, i64 items_per_minibatch, bool forced);
// m = ceil(2^32 / classes): __umulhi(id, m) is the quotient for every id below kClassSlots x classes, because there
// id x (m x classes - 2^32) < id x classes < 2^32, which is what may be added to the remainder without reaching the next quotient; the
// error is upwards, so an id from there on gives kClassSlots at least.
inline uint32_t class_magic(i64 parts) { return parts > 0 ? (uint32_t)((((u64)1 << 32) + (u64)parts - 2) / (u64)(parts - 1)) : 0u; }
i64 partition_bucket_capacity(i64 items_bound, i64 G, i64 parts);
size_t partition_workspace_bytes(i64 n_cap, i64 bucket_cap);
uint32_t* partition_bucket_counts(void* ws);
size_t partition_count_bytes(i64 bucket_cap);  // what the counts, starts and cursors of the buckets take of it, at its head
int partition_unique_relabel(gsb_ctx* ctx, cudaStream_t stream, BatchLayout L, i64 n_cap, i64 bucket_cap, void* ws,
                             i64 parts, bool counted, i64* out_unique, i64* out_unique_ptr, i64* out_relabeled, Mail mail);
// The one-call hop, after its counting sampler: edge offsets of the minibatches (from the sampled block's offsets),
// item offsets, bound check, bucket starts — everything partition_unique_relabel(counted = true) expects, one launch.
int partition_after_sampler(gsb_ctx* ctx, cudaStream_t stream, BatchLayout L, i64 n_cap, i64 bucket_cap, void* ws,
                            const i64* sub_indptr, i64 S, i64 edges_bound, i64* out_indices_ptr);
// Classes of ids where minibatches have some tiles of kClassTile items: the tiles sort themselves (defined in
// class_relabel.cu).  class_tiled: whether a call takes that form, by the option GSB_OPT_RELABEL_PATH and its sizes.  L.item_off and
// L.region_off (first tile of every minibatch; class_tiles bounds the tiles) must be filled by k_batch_layout; `ws` is scratch of
// class_workspace_bytes.
constexpr int kClassTile = 1 << 14;
bool class_tiled(i64 path, i64 num_nodes, i64 items, i64 G);
i64 class_tiles(i64 n_cap, i64 G);
size_t class_workspace_bytes(i64 n_cap, i64 G, i64 parts);
int class_unique_relabel(gsb_ctx* ctx, cudaStream_t stream, const BatchLayout& L, i64 n_cap, void* ws, i64 parts, i64* out_unique,
                         i64* out_unique_ptr, i64* out_relabeled, Mail mail);
// Bucket of an id among the `parts` buckets of its minibatch: its class (magic != 0; the last bucket takes all ids beyond), or
// Fibonacci hashing (the high bits of id x odd constant), scaled to the bucket count by a multiply-high.  Ids are below 2^32 - 1
// wherever this is used.
template <bool CLASSES>
__device__ __forceinline__ uint32_t bucket_of_id(uint32_t id, uint32_t parts, uint32_t magic) {
  if (!CLASSES) return __umulhi(id * 0x9E3779B1u, parts);
  const uint32_t q = __umulhi(id, magic);
  return q < kClassSlots ? id - q * (parts - 1) : parts - 1;
}
__device__ __forceinline__ uint32_t bucket_of_id(uint32_t id, uint32_t parts, uint32_t magic) {
  return magic != 0 ? bucket_of_id<true>(id, parts, magic) : bucket_of_id<false>(id, parts, 0);
}
// What the uniform sampler needs to count, per bucket, the seeds and the ids it samples (fan-outs up to 16).
struct SamplerCount {
  uint32_t* bucket_count;  // [buckets]
  const i64* bucket_base;  // [G + 1] first bucket of every minibatch
  uint32_t magic;          // of the classes of ids that are the buckets, 0: hashed
  void* scratch;           // of window_sample_bytes, or null: the call does not sample by windows
};
// Sampling by windows of the edges (defined in window_sample.cu): whether S columns of k picks out of a graph of num_edges take it,
// and the scratch it needs then.
bool window_sample_suits(gsb_ctx* ctx, i64 S, i64 k, i64 num_edges);
size_t window_sample_bytes(gsb_ctx* ctx, i64 S, i64 k, i64 num_edges);
constexpr int kBucketTarget = 2048;  // mean items per bucket

struct CompactOut {
  i64* unique;      // all frontiers back to back
  i64* unique_ptr;  // [G + 1]
  Mail mail;        // slots 0, 1: frontier and edge totals, for a caller that waits for them
};

// Single-launch unique + relabel (defined in fused_unique.cu).  Ids below 2^32 - 1; a larger or negative one makes the
// kernel record GSB_ERR_INDEX_RANGE.  fused_unique_suits: whether a call of n items in G minibatches fits its registers,
// its table and one resident grid.
//   single   unique(cat(first, second)) -> out_unique, ranks of `second` -> out_second (may be null), and with col_index
//            (positions in `first`, one per entry of `second`) the ranks of first[col_index[e]] -> out_col; copies
//            copy_n words from copy_src to copy_dst and sets E floats of `ones` (may be null) along the way.  mail slot 0:
//            distinct ids.
// id_bound > 0: ids are expected below it, which allows the direct-address table when fused_unique_direct says so; an id
// beyond it is then reported as GSB_ERR_INDEX_RANGE too.
//   batched  as gsb_batch_unique_relabel; with sub_indptr the edge offsets of the minibatches are sub_indptr[seeds_ptr[b]]
//            and are written to out_indices_ptr.  mail slots 0, 1: frontier and edge totals.
constexpr i64 kFusedUniqueMaxItems = 1ll << 21;
constexpr i64 kFusedUniqueMaxBatches = 1ll << 16;
bool fused_unique_suits(gsb_ctx* ctx, i64 n, i64 G);
bool fused_unique_direct(i64 G, i64 id_bound);
int fused_unique_single(gsb_ctx* ctx, cudaStream_t stream, const i64* first, i64 S, const i64* second, i64 E,
                        const i64* col_index, i64* out_unique, i64* out_second, i64* out_col, const i64* copy_src,
                        i64* copy_dst, i64 copy_n, float* ones, i64 id_bound, Mail mail);
int fused_unique_batched(gsb_ctx* ctx, cudaStream_t stream, const BatchLayout& L, i64 seeds_bound, i64 edges_bound,
                         const i64* sub_indptr, i64* out_indices_ptr, i64* out_unique, i64* out_unique_ptr,
                         i64* out_relabeled, i64 id_bound, Mail mail);

// Single-batch unique + relabel through the packed-slot batched kernels (defined in batch_relabel.cu).
int unique_relabel_packed(gsb_ctx* ctx, cudaStream_t stream, const i64* first, i64 S, const i64* second, i64 E,
                          i64* out_unique, i64* out_relabeled, i64* unique_host);

// Uniform sampler shared by gsb_sample_uniform and the batched hop (defined in slice_sample.cu).  With S_dev the
// exact seed count is read on the device and S is an upper bound that sizes the grid.  num_edges: entries of `indices`, 0: not
// known (a large call is then sampled in one pass whatever the graph).
int sample_uniform_launch(gsb_ctx* ctx, cudaStream_t stream, const i64* indptr, const i64* indices, i64 num_cols,
                          const i64* seeds, i64 S, i64 k, int replace, u64 seed, i64* out_indptr, i64* out_indices,
                          i64* out_select, i64* out_coo_col, const float* data, const i64* e_ids, float* out_data,
                          i64 capacity, const i64* S_dev = nullptr, const i64* batch_ptr = nullptr,
                          const i64* batch_ids = nullptr, i64 G = 0, const SamplerCount* count = nullptr,
                          Mail mail = Mail{nullptr, 0}, i64 num_edges = 0);

}  // namespace gsb
