// Probability-weighted per-column sampling.
//
// Without replacement: Efraimidis-Spirakis A-Res.  Every edge of a column gets the key
// log2(u) / w (a monotone transform of the reference's u^(1/w), src/cuda/sampling_probs.cu:70-72)
// from the Philox word keyed by (seed, column position, edge position); the k largest keys win.
// A column of at most 128 edges is sorted: four edges per lane, so that 8, 16 or 32 lanes hold a column and a warp takes four,
// two or one of them at a time: through a register sorting network, or, where k is small beside the lanes, behind a bound that few
// edges reach.  In a longer column the warp keeps the running top-k as
// a sorted list, one entry per lane (k <= 32, the reference's own limit: sampling_probs.cu:32).  A new key enters the list
// only if it beats the current k-th entry, which after the first few dozen edges is rare, so a hub column costs one key
// evaluation per edge plus O(k log(deg/k)) list insertions.  Ties rank the smaller edge position first; the output is in
// descending key order.
//
// With replacement: k inverse-CDF draws over max(w, 0), the CDF being the fp32 running sum in
// edge order (sampling_probs.cu:137-186 builds it with a warp scan into a temporary buffer; here
// a warp adds the column up once and keeps at most 128 points of the sum, between which each draw walks).
//
// One cooperative launch: the CTAs count their ranges of columns and sort them into lists by the kind of work they are
// (first barrier: everyone knows every count, so output offsets and list positions follow), then all warps of the GPU take
// work from the lists, the longest first.  What bounds the sampler is latency — a column is three dependent reads, a draw, a
// sort or a scan, a gather — so what counts is that no warp waits for another one's columns.  With a tile of columns per CTA
// a CTA lived as long as its slowest column and hubs were scanned one after the other: 65 537 columns of 50 edges, fan-out
// 16: 112 us, 2 048 hub columns with 1.2 M edges 82 us; now 64 and 42 us.
#include "common.cuh"
#include "philox.cuh"
#include "grid_sync.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kWThreads = 256;
constexpr int kWarps = kWThreads / 32;

struct WeightedParams {
  const i64* indptr;
  const i64* indices;
  const float* probs;
  i64 num_cols;
  const i64* seeds;
  i64 S;
  i64 k;
  int replace;
  u64 seed;
  i64* out_indptr;
  i64* out_indices;
  i64* out_select;
  i64* out_coo_col;
  const float* data;
  const i64* e_ids;
  float* out_data;
  i64 capacity;
  i64* counters;
  Mail mail;  // the edge total, for a caller that waits for it
  // workspace
  i64* partial;          // [CTA][NUM_SUMS]
  u64* queue;            // [NUM_QUEUES]
  i64* lists;            // [S]: column positions, one region per kind
  struct WeightedSlice* slices;  // [kMaxSlices]
  u64* slice_lists;      // [kMaxSlices][32]: key bits : 32 | position : 32
  unsigned* slice_done;  // [kMaxSlices], counted at a column's first slice
  unsigned* slice_floor;
  GridSync sync;
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// A list entry / candidate is (key, edge position inside its column).  Positions are 32-bit: a column of more than
// kMaxScanEnd edges is refused by the kernel (kNoIdx marks an empty entry and ranks after every real position).
constexpr u32 kNoIdx = 0xffffffffu;
constexpr u32 kMaxScanEnd = 0xffffff00u;

__device__ __forceinline__ bool ranks_before(float ka, u32 ia, float kb, u32 ib) {
  return ka > kb || (ka == kb && ia < ib);
}

__device__ __forceinline__ void emit_weighted(const WeightedParams& p, i64 out_pos, i64 in_pos, i64 col_pos) {
  p.out_indices[out_pos] = __ldg(p.indices + in_pos);
  if (p.out_select) p.out_select[out_pos] = in_pos;
  if (p.out_coo_col) p.out_coo_col[out_pos] = col_pos;
  if (p.out_data) p.out_data[out_pos] = p.data[p.e_ids ? p.e_ids[in_pos] : in_pos];
}

// Warp-collective: every lane offers one candidate; the running top-k list (lane j holds the j-th best, empty
// entries rank last) absorbs the candidates that beat its k-th entry, one at a time.  The warp's shuffle unit is
// what bounds this kernel, so an insertion costs four shuffles (candidate key + position, shift of key + position):
// whether a queued candidate still makes the list is read off its insertion rank, and the k-th entry is broadcast
// once per call, not once per insertion.
__device__ __forceinline__ void topk_offer(float ck, u32 ci, bool valid, int k, unsigned kmask, float& my_key,
                                           u32& my_idx, float& thr_key, u32& thr_idx) {
  const bool want = valid && ranks_before(ck, ci, thr_key, thr_idx);
  unsigned pending = __ballot_sync(0xffffffffu, want);
  if (!pending) return;
  while (pending) {
    const int src = __ffs(pending) - 1;
    pending &= pending - 1;
    const float nk = __shfl_sync(0xffffffffu, ck, src);
    const u32 ni = __shfl_sync(0xffffffffu, ci, src);
    const bool mine_first = ranks_before(my_key, my_idx, nk, ni);
    const int pos = __popc(__ballot_sync(0xffffffffu, mine_first) & kmask);
    if (pos >= k) continue;  // k entries rank before it by now
    const float up_key = __shfl_up_sync(0xffffffffu, my_key, 1);
    const u32 up_idx = __shfl_up_sync(0xffffffffu, my_idx, 1);
    if (lane_id() > pos) {
      my_key = up_key;
      my_idx = up_idx;
    } else if (lane_id() == pos) {
      my_key = nk;
      my_idx = ni;
    }
  }
  thr_key = __shfl_sync(0xffffffffu, my_key, k - 1);
  thr_idx = __shfl_sync(0xffffffffu, my_idx, k - 1);
}

// The ranking key of an edge, or -inf when the key surely ranks after `thr_key` (the list's current k-th key; -inf
// while the list is not full, which rejects nothing).  Once a long column has filled its list almost every edge
// fails, and this test spares it the logarithm and the division: log2(u) <= (u - 1)·log2(e) for every u in (0, 1],
// so key = log2(u) / w <= (u - 1)·log2(e) / w.  The two 1e-4 margins (the bound is pulled towards zero, the
// threshold pushed away from it) are far wider than the rounding of the key's own arithmetic (< 1e-6 relative), so a
// key that would tie with or beat thr_key is always evaluated exactly and results do not depend on this shortcut.
__device__ __forceinline__ float ares_key_if_above(uint32_t r, float w, float thr_key) {
  const float neg_inf = __uint_as_float(0xFF800000u);
  if (!(w > 0.0f)) return neg_inf;
  const float bound = (uniform01(r) - 1.0f) * (1.44269504f * 0.9999f);
  const float limit = thr_key * w * 1.0001f;
  if (bound < limit) return neg_inf;
  return ares_key(r, w);
}

__device__ __forceinline__ u32 sortable_key(float key) {
  const u32 u = __float_as_uint(key + 0.0f);  // -0 becomes +0: the comparison the list uses cannot tell them apart
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_of_sortable(u32 u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Code that a warp runs once per column has to be short: the kernel's instructions are read from L2 by every SM of every
// launch, and with the parts below unrolled and inlined where they are used one short column took a warp 10 us.  So what is
// used in several places is a function, and the network is a loop.

// Keys of four consecutive edges of a column, which are one Philox block (edge e draws word e & 3 of block e >> 2).
__device__ __noinline__ float4 four_keys(u64 seed, i64 col_pos, u32 block, float4 w, float thr_key) {
  const U32x4 r = rand_block(seed, (u64)col_pos, (u64)block, STREAM_WEIGHTED);
  return make_float4(ares_key_if_above(r.v[0], w.x, thr_key), ares_key_if_above(r.v[1], w.y, thr_key),
                     ares_key_if_above(r.v[2], w.z, thr_key), ares_key_if_above(r.v[3], w.w, thr_key));
}

// Weights of edges e .. e+3; 0 from `end` on.
__device__ __forceinline__ float4 four_weights(const float* probs, u32 e, u32 end) {
  float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
  if (e < end) w.x = __ldg(probs + e);
  if (e + 1 < end) w.y = __ldg(probs + e + 1);
  if (e + 2 < end) w.z = __ldg(probs + e + 2);
  if (e + 3 < end) w.w = __ldg(probs + e + 3);
  return w;
}

// Edges e_begin .. min(e_end, e_begin + 4 lanes) - 1 of one column, in descending order, by `lanes` lanes (8, 16 or 32: a warp
// does 32 / lanes columns in step): lane g holds the composites (order-preserving image of the key : 32 | ~position : 32) of
// edges 4g .. 4g+3 and a bitonic network — steps below 4 inside a lane, the others by exchange — orders them.  Leaves the
// composites in `s_order`, which is the warp's: position 4 lanes x group + rank, the first k of them at least; 0, which ranks last,
// where there is no edge.
// Where k is no more than half the lanes the k best are nearly always among few: the k-th largest of the lanes' own best keys is a
// bound that k entries reach, and what reaches it (20 of 128 for k = 16) is ranked by counting, one entry per lane.  With a larger k
// more entries than lanes would reach it, so the network stays; it also stays for the group of columns of which one has that many.
// 300 000 columns of 50 edges, network / bound: k = 2 241 / 196 us, 5 247 / 213, 10 257 / 234, 16 253 / 237.
__device__ __noinline__ void sort_edges(u64 seed, const float* probs, i64 col_pos, u32 e_begin, u32 e_end, u32 lanes, u32 k,
                                        u64* s_order) {
  const u32 g = (u32)lane_id() & (lanes - 1), e = e_begin + 4 * g;
  u64 c0 = 0, c1 = 0, c2 = 0, c3 = 0;
  if (e < e_end) {
    const float4 key = four_keys(seed, col_pos, e >> 2, four_weights(probs, e, e_end), __uint_as_float(0xFF800000u));
    c0 = ((u64)sortable_key(key.x) << 32) | (u64)~e;
    if (e + 1 < e_end) c1 = ((u64)sortable_key(key.y) << 32) | (u64)~(e + 1);
    if (e + 2 < e_end) c2 = ((u64)sortable_key(key.z) << 32) | (u64)~(e + 2);
    if (e + 3 < e_end) c3 = ((u64)sortable_key(key.w) << 32) | (u64)~(e + 3);
  }
  if (2 * k <= lanes) {
    const unsigned group = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1u) << (lane_id() - g), lt = (1u << lane_id()) - 1u;
    u32 bound = (u32)(max(max(c0, c1), max(c2, c3)) >> 32);
#pragma unroll 1
    for (u32 size = 2; size <= lanes; size <<= 1) {
#pragma unroll 1
      for (u32 step = size >> 1; step > 0; step >>= 1) {
        const u32 other = __shfl_xor_sync(0xffffffffu, bound, step);
        bound = ((g & step) == 0) == ((g & size) == 0) ? max(bound, other) : min(bound, other);
      }
    }
    bound = __shfl_sync(0xffffffffu, bound, k - 1, lanes);
    auto reaches = [&](u64 c) { return c != 0 && (u32)(c >> 32) >= bound; };
    const unsigned b0 = __ballot_sync(0xffffffffu, reaches(c0)) & group, b1 = __ballot_sync(0xffffffffu, reaches(c1)) & group,
                   b2 = __ballot_sync(0xffffffffu, reaches(c2)) & group, b3 = __ballot_sync(0xffffffffu, reaches(c3)) & group;
    const u32 n0 = __popc(b0), n1 = n0 + __popc(b1), n2 = n1 + __popc(b2), n = n2 + __popc(b3);
    if (__all_sync(0xffffffffu, n <= lanes)) {
      u64* s_group = s_order + 4 * (lane_id() - g);
      __syncwarp();  // the last readers of s_order are done
      if (reaches(c0)) s_group[__popc(b0 & lt)] = c0;
      if (reaches(c1)) s_group[n0 + __popc(b1 & lt)] = c1;
      if (reaches(c2)) s_group[n1 + __popc(b2 & lt)] = c2;
      if (reaches(c3)) s_group[n2 + __popc(b3 & lt)] = c3;
      if (g >= n) s_group[g] = 0;
      __syncwarp();
      const u64 own = s_group[g];
      const u32 most = __reduce_max_sync(0xffffffffu, n);
      u32 rank = 0;
#pragma unroll 4
      for (u32 j = 0; j < most; ++j) rank += s_group[j] > own;  // (most <= lanes)
      __syncwarp();
      if (g < n) s_group[rank] = own;
      __syncwarp();
      return;
    }
  }
  auto order = [](u64& x, u64& y, bool descending) {
    const bool swap = (x < y) == descending;
    const u64 t = swap ? y : x;
    y = swap ? x : y;
    x = t;
  };
  order(c0, c1, true);
  order(c2, c3, false);
#pragma unroll 1
  for (u32 size = 4; size <= 4 * lanes; size <<= 1) {
    const bool descending = ((4 * g) & size) == 0;
#pragma unroll 1
    for (u32 step = size >> 3; step > 0; step >>= 1) {
      const bool keep_max = ((g & step) == 0) == descending;
      auto exchange = [&](u64& c) {
        const u64 other = __shfl_xor_sync(0xffffffffu, c, step);
        if ((c < other) == keep_max) c = other;
      };
      exchange(c0);
      exchange(c1);
      exchange(c2);
      exchange(c3);
    }
    order(c0, c2, descending);
    order(c1, c3, descending);
    order(c0, c1, descending);
    order(c2, c3, descending);
  }
  __syncwarp();  // the last readers of s_order are done
  u64* out = s_order + 4 * lane_id();
  out[0] = c0;
  out[1] = c1;
  out[2] = c2;
  out[3] = c3;
  __syncwarp();
}

// Top-k of the edges [e_begin, e_end) of one column (e_begin a multiple of 4, e_end <= kMaxScanEnd), k <= 32, scanned by one
// warp, 128 edges per iteration.  The first 128 are sorted, which fills the list; the keys of a later iteration are transposed
// through shared memory so that each offer round holds 32 CONSECUTIVE edges, and what is inserted, one at a time, is only the
// few that still beat the k-th entry (about k ln(d / 128) for a column of d edges).  An iteration without any such candidate —
// most of them, far into a hub — ends at one vote.  Weights are loaded an iteration ahead.
// With several warps on slices of one column `floor_word` is the best k-th key (its sortable image) that any of them has
// reached: what ranks strictly below it cannot be among the column's k best.
struct ListEntry {
  float key;
  u32 idx;
};

__device__ __noinline__ ListEntry topk_scan(u64 seed, const float* probs, i64 col_pos, u32 e_begin, u32 e_end, int k,
                                            u64* s_order, u32* floor_word) {
  const float neg_inf = __uint_as_float(0xFF800000u);
  const u32 lane = (u32)lane_id();
  const unsigned kmask = k >= 32 ? 0xffffffffu : ((1u << k) - 1u);
  float4 ahead = four_weights(probs, e_begin + 128 + 4 * lane, e_end);
  sort_edges(seed, probs, col_pos, e_begin, e_end, 32, (u32)k, s_order);
  const u64 own = (int)lane < k ? s_order[lane] : 0;
  float my_key = own ? key_of_sortable((u32)(own >> 32)) : neg_inf;
  u32 my_idx = own ? ~(u32)own : kNoIdx;
  float thr_key = __shfl_sync(0xffffffffu, my_key, k - 1);
  u32 thr_idx = __shfl_sync(0xffffffffu, my_idx, k - 1);
  float* s_keys = reinterpret_cast<float*>(s_order);
  u32 floor_ahead = 0;
  if (floor_word) {
    if (lane == 0 && thr_key > neg_inf) atomicMax(floor_word, sortable_key(thr_key));
    floor_ahead = *(volatile u32*)floor_word;
  }
  for (u32 e0 = e_begin + 128; e0 < e_end; e0 += 128) {  // e_end <= kMaxScanEnd: e0 + 128 does not wrap
    const u32 e4 = e0 + 4 * lane;
    const float4 w = ahead;
    ahead = e4 < e_end ? four_weights(probs, e4 + 128, e_end) : make_float4(0.f, 0.f, 0.f, 0.f);
    float floor_key = thr_key;
    if (floor_word) {
      floor_key = fmaxf(floor_key, key_of_sortable(floor_ahead));
      floor_ahead = *(volatile u32*)floor_word;
    }
    float4 kq = make_float4(neg_inf, neg_inf, neg_inf, neg_inf);
    // an edge past the end has weight 0 here and its key is not offered below
    if (e4 < e_end) kq = four_keys(seed, col_pos, e4 >> 2, w, floor_key);
    if (!__any_sync(0xffffffffu, fmaxf(fmaxf(kq.x, kq.y), fmaxf(kq.z, kq.w)) >= floor_key)) continue;
    __syncwarp();  // the previous iteration's reads are done
    reinterpret_cast<float4*>(s_keys)[lane] = kq;
    __syncwarp();
#pragma unroll 1
    for (u32 q = 0; q < 128 && e0 + q < e_end; q += 32) {
      const u32 e = e0 + q + lane;
      topk_offer(s_keys[q + lane], e, e < e_end, k, kmask, my_key, my_idx, thr_key, thr_idx);
    }
    if (floor_word && lane == 0 && thr_key > neg_inf) atomicMax(floor_word, sortable_key(thr_key));
  }
  return ListEntry{my_key, my_idx};
}

// k draws with replacement from one column, by one warp.  The running sum over the column is a chain of d additions in edge
// order: the warp loads 128 weights ahead, goes through the chain once (every lane the same, the weights from shared memory:
// with shuffles the shuffle unit of a busy SM was four times slower than the chain) and keeps the sum at the end of each block
// of edges, at most 128 of them.  A draw then finds the first block whose sum exceeds it — sums never fall — and walks that
// block with the same additions.  (Before, every draw walked the column twice, one dependent load per edge: 65 537 columns of
// 50 edges 1 100 us, 5 000 columns with hubs among them 1 670 us; now 124 and 80.)
__device__ __forceinline__ void draw_with_replacement(const WeightedParams& p, i64 b, i64 d, i64 o, i64 col_pos, float* s_warp) {
  const int lane = lane_id();
  const float* probs = p.probs + b;
  float* s_weights = s_warp;       // [128]
  float* s_sums = s_warp + 128;    // [128]
  const i64 chunks = (d + 31) >> 5, per_block = (chunks + 127) >> 7;
  const int blocks = (int)((chunks + per_block - 1) / per_block);
  float run = 0.f, ahead[4];
  auto load = [&](i64 e0) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // 0 past the end of the column: adds nothing
      const i64 e = e0 + q * 32 + lane;
      ahead[q] = e < d ? fmaxf(__ldg(probs + e), 0.f) : 0.f;
    }
  };
  load(0);
  i64 until = per_block - 1;
  int block = 0;
#pragma unroll 1
  for (i64 q0 = 0; q0 < chunks; q0 += 4) {
    __syncwarp();  // everyone is done with what is overwritten
#pragma unroll
    for (int q = 0; q < 4; ++q) s_weights[q * 32 + lane] = ahead[q];
    __syncwarp();
    load((q0 + 4) * 32);
#pragma unroll 1
    for (i64 q = q0; q < min(q0 + 4, chunks); ++q) {
      const float4* w = reinterpret_cast<const float4*>(s_weights + (q - q0) * 32);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 v = w[j];
        run = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(run, v.x), v.y), v.z), v.w);
      }
      if (q == until || q == chunks - 1) {
        if (lane == 0) s_sums[block] = run;
        ++block;
        until += per_block;
      }
    }
  }
  __syncwarp();
  for (i64 j = lane; j < p.k; j += 32) {
    const float r = __fmul_rn(uniform01(rand_u32(p.seed, (u64)col_pos, (u64)j, STREAM_WEIGHTED)), run);
    int lo = 0, hi = blocks;  // first block whose sum exceeds r, or `blocks`
    while (lo < hi) {
      const int mid = (lo + hi) >> 1;
      if (s_sums[mid] > r) hi = mid;
      else lo = mid + 1;
    }
    i64 pos = d - 1;
    if (lo < blocks) {
      float acc = lo > 0 ? s_sums[lo - 1] : 0.f;
      const i64 end = min(d, (i64)(lo + 1) * per_block * 32);
      bool found = false;
      for (i64 e0 = (i64)lo * per_block * 32; e0 < end && !found; e0 += 8) {
        float w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) w[q] = e0 + q < end ? fmaxf(__ldg(probs + e0 + q), 0.f) : 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          acc = __fadd_rn(acc, w[q]);
          if (!found && acc > r) {
            pos = e0 + q;
            found = true;
          }
        }
      }
    }
    emit_weighted(p, o + j, b + pos, col_pos);
  }
}

// Kinds of columns, the longest first.
enum ColumnKind { KIND_HUGE, KIND_SCAN, KIND_SORT128, KIND_SORT64, KIND_SORT32, KIND_COPY, NUM_KINDS };
enum { SUM_EDGES = NUM_KINDS, SUM_HUGE_DEGREE, NUM_SUMS };
enum { QUEUE_SLICES, QUEUE_HUGE, QUEUE_NEXT, NUM_QUEUES };
constexpr int kSortedColumn = 128;
// A scan of more edges than this is cut into slices.  16 iterations of 128 cost about as much as the draw, sort and gather of a
// short column four times over; at 512 no column keeps one warp much longer than another.
constexpr i64 kSlice = 512;
constexpr int kMaxSlices = 32768;

struct WeightedSlice {
  i64 column;
  unsigned index, first;  // which slice of the column, and where the column's slices start
};

struct Column {
  i64 b, d;
};

__device__ __forceinline__ Column column_of(const WeightedParams& p, i64 col_pos, bool report) {
  const i64 col = p.seeds ? __ldg(p.seeds + col_pos) : col_pos;
  Column c{0, 0};  // a seed outside the graph counts as an empty column and is never dereferenced
  if ((u64)col < (u64)p.num_cols) {
    c.b = __ldg(p.indptr + col);
    c.d = __ldg(p.indptr + col + 1) - c.b;
  } else if (report) {
    raise_error(p.counters, GSB_ERR_INDEX_RANGE, col_pos);
  }
  return c;
}

__device__ __forceinline__ i64 picks_of(const WeightedParams& p, i64 d) {
  return p.replace ? (d > 0 ? p.k : 0) : min(d, p.k);
}

__device__ __forceinline__ int kind_of(const WeightedParams& p, i64 d) {
  if (d == 0 || p.k == 0) return -1;
  if (!p.replace) {
    if (d <= p.k) return KIND_COPY;
    if (d > (i64)kMaxScanEnd) return -1;  // positions are 32-bit here
    if (d <= 32) return KIND_SORT32;
    if (d <= 64) return KIND_SORT64;
    if (d <= kSortedColumn) return KIND_SORT128;
  }
  return d <= kSlice ? KIND_SCAN : KIND_HUGE;
}

// Warp-collective: a unit of copies (columns no longer than the fan-out) or sorts, as many columns as fit a warp.
__device__ __forceinline__ void short_columns(const WeightedParams& p, int kind, i64 list, i64 first, i64 count, u64* s_order) {
  const int lanes = kind == KIND_SORT128 ? 32 : kind == KIND_SORT64 ? 16 : 8;
  const int lane = lane_id(), g = lane & (lanes - 1);
  const i64 at = first + lane / lanes;
  const i64 c = at < count ? __ldcg(p.lists + list + at) : -1;
  i64 o = 0;
  Column column{0, 0};
  if (c >= 0) {
    column = column_of(p, c, false);
    o = __ldcg(p.out_indptr + c);
  }
  if (kind != KIND_COPY) sort_edges(p.seed, p.probs + column.b, c, 0, (u32)column.d, lanes, (u32)p.k, s_order);
  const u64* order = s_order + 4 * (lane - g);
#pragma unroll 1
  for (i64 j = g; j < min(p.k, column.d); j += lanes)
    emit_weighted(p, o + j, column.b + (kind == KIND_COPY ? j : (i64)(u32)~(u32)order[j]), c);
}

// Warp-collective: the whole of a column or one slice of it.  The warp that finishes a column's last slice merges their lists.
__device__ __forceinline__ void scan_column(const WeightedParams& p, i64 c, bool sliced, unsigned unit, i64 slice, u64* s_order) {
  const int lane = lane_id(), k = (int)p.k;
  unsigned index = 0, first = 0, slices = 1;
  if (sliced) {
    c = __ldcg(&p.slices[unit].column);
    index = __ldcg(&p.slices[unit].index);
    first = __ldcg(&p.slices[unit].first);
  }
  const Column column = column_of(p, c, false);
  const i64 o = __ldcg(p.out_indptr + c);
  u32 e_begin = 0, e_end = (u32)column.d;
  if (sliced) {
    slices = (unsigned)((column.d + slice - 1) / slice);
    e_begin = (u32)(index * slice);
    e_end = (u32)min(column.d, (i64)(index + 1) * slice);
  }
  const ListEntry best = topk_scan(p.seed, p.probs + column.b, c, e_begin, e_end, k, s_order, sliced ? p.slice_floor + first : nullptr);
  float my_key = best.key;
  u32 my_idx = best.idx;
  if (sliced) {
    __stcg(p.slice_lists + (size_t)unit * 32 + lane, ((u64)__float_as_uint(my_key) << 32) | my_idx);
    __threadfence();
    __syncwarp();
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(p.slice_done + first, 1u);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before != slices - 1) return;
    __threadfence();
    const unsigned kmask = k >= 32 ? 0xffffffffu : ((1u << k) - 1u);
    float thr_key = __shfl_sync(0xffffffffu, my_key, k - 1);
    u32 thr_idx = __shfl_sync(0xffffffffu, my_idx, k - 1);
    u64 ahead = __ldcg(p.slice_lists + (size_t)first * 32 + lane);
#pragma unroll 1
    for (unsigned w = 0; w < slices; ++w) {
      const u64 other = ahead;
      if (w + 1 < slices) ahead = __ldcg(p.slice_lists + (size_t)(first + w + 1) * 32 + lane);
      if (w == index) continue;  // that is where the merge started
      topk_offer(__uint_as_float((u32)(other >> 32)), (u32)other, lane < k && (u32)other != kNoIdx, k, kmask, my_key, my_idx,
                 thr_key, thr_idx);
    }
  }
  if (lane < k) emit_weighted(p, o + lane, column.b + (i64)my_idx, c);
}

// ---- fan-outs above 32 (the reference stops at 32: src/cuda/sampling_probs.cu:32) -----------------------------
// Columns of more than 128 edges and more than the fan-out take a CTA each.  It finds the fan-out-th best entry by a
// most-significant-digit radix select over the 64-bit composite (order-preserving image of the key : 32 | ~position : 32) —
// composites are distinct, larger = ranks first, so "the k best" is "composite >= threshold" with no tie handling — then
// gathers the winners into shared memory, sorts them (bitonic, descending) and emits them in the order the list kernel uses.
// The select stops as soon as a digit's bin is taken whole, which without ties is after the four key digits.  Keys of
// columns up to kWideCache entries are evaluated once and kept in shared memory, longer columns evaluate them again
// in every pass.  Fan-out 40 of 65 537 columns of 50 edges: 535 us when every column, however short, had the CTA to itself,
// 129 us now.
constexpr int kWideMaxK = 1024;
constexpr int kWideCache = 6144;

struct WideShared {
  u32 cache[kWideCache];
  u64 win[kWideMaxK];
  u32 hist[256];
  u64 prefix;
  u32 need;
  int done;
  u32 count;
};

__device__ __forceinline__ void select_wide(const WeightedParams& p, WideShared& s, i64 col_pos) {
  const int tid = threadIdx.x, k = (int)p.k;
  const Column column = column_of(p, col_pos, false);
  const i64 b = column.b, o = __ldcg(p.out_indptr + col_pos);
  const u32 n = (u32)column.d;
  const bool cached = n <= (u32)kWideCache;
  const float* probs = p.probs + b;
  auto key_of = [&](u32 e) -> u32 {
    const U32x4 r = rand_block(p.seed, (u64)col_pos, (u64)(e >> 2), STREAM_WEIGHTED);
    return sortable_key(ares_key(r.v[e & 3], __ldg(probs + e)));
  };
  __syncthreads();  // the previous column is done with the shared arrays
  if (cached) {
    for (u32 e4 = 4 * tid; e4 < n; e4 += 4 * kWThreads) {
      const U32x4 r = rand_block(p.seed, (u64)col_pos, (u64)(e4 >> 2), STREAM_WEIGHTED);
#pragma unroll
      for (u32 q = 0; q < 4; ++q)
        if (e4 + q < n) s.cache[e4 + q] = sortable_key(ares_key(r.v[q], __ldg(probs + e4 + q)));
    }
  }
  if (tid == 0) {
    s.prefix = 0;
    s.need = (u32)k;
    s.done = 0;
    s.count = 0;
  }
  u64 mask = 0;
  for (int shift = 56; shift >= 0; shift -= 8) {
    s.hist[tid] = 0;
    __syncthreads();
    if (s.done) break;  // uniform: written before the barrier of the previous round
    const u64 prefix = s.prefix;
    for (u32 e = tid; e < n; e += kWThreads) {
      const u64 comp = ((u64)(cached ? s.cache[e] : key_of(e)) << 32) | (u64)(~e);
      if ((comp & mask) == prefix) atomicAdd(&s.hist[(comp >> shift) & 255u], 1u);
    }
    __syncthreads();
    if (tid < 32) {  // the bin that holds the need-th entry from the top: eight bins per lane, the highest in lane 0
      const u32 need = s.need;
      u32 own = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) own += s.hist[255 - 8 * tid - q];
      u32 upto = own;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const u32 x = __shfl_up_sync(0xffffffffu, upto, d);
        if (tid >= d) upto += x;
      }
      u32 above = upto - own;
      if (above < need && need <= upto) {
        int bin = 255 - 8 * tid;
        for (; above + s.hist[bin] < need; --bin) above += s.hist[bin];
        s.prefix = prefix | ((u64)bin << shift);
        if (above + s.hist[bin] == need) s.done = 1;  // the bin is taken whole: nothing below this digit matters
        s.need = need - above;
      }
    }
    mask |= (u64)255u << shift;
    __syncthreads();
  }
  const u64 threshold = s.prefix;  // digits below the last decided one are zero
  for (u32 e = tid; e < n; e += kWThreads) {
    const u64 comp = ((u64)(cached ? s.cache[e] : key_of(e)) << 32) | (u64)(~e);
    if (comp >= threshold) {
      const u32 at = atomicAdd(&s.count, 1u);
      if (at < (u32)kWideMaxK) s.win[at] = comp;
    }
  }
  __syncthreads();
  int width = 32;
  while (width < k) width <<= 1;
  for (int j = k + tid; j < width; j += kWThreads) s.win[j] = 0;  // ranks after every real composite
  __syncthreads();
  for (int size = 2; size <= width; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int t = tid; t < width / 2; t += kWThreads) {
        const int lo = 2 * t - (t & (stride - 1)), hi = lo + stride;
        const bool descending = (lo & size) == 0;
        const u64 a = s.win[lo], c = s.win[hi];
        if ((a < c) == descending) {
          s.win[lo] = c;
          s.win[hi] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int j = tid; j < k; j += kWThreads) emit_weighted(p, o + j, b + (i64)(u32)(~(u32)s.win[j]), col_pos);
}

// ---- the kernel ---------------------------------------------------------------------------------------------------------
constexpr int kWeightedBarriers = 2;

template <bool WIDE>
__global__ void __launch_bounds__(kWThreads, 4) k_sample_weighted(WeightedParams p) {
  __shared__ i64 s_scan[33];
  __shared__ u64 s_before[NUM_SUMS], s_total[NUM_SUMS], s_at[NUM_KINDS];
  __shared__ i64 s_unit;
  __shared__ unsigned s_taken;
  __shared__ __align__(16) u64 s_order[kWarps][128];
  __shared__ u64 s_part[kWarps][NUM_SUMS][2];
  __shared__ unsigned s_listed[NUM_KINDS];
  extern __shared__ __align__(16) char s_dynamic[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const i64 S = p.S, k = p.k;
  const i64 per = (S + gridDim.x - 1) / gridDim.x;
  const i64 lo = min(S, (i64)blockIdx.x * per), hi = min(S, lo + per);

  // what this CTA's columns add up to
  if (blockIdx.x == 0 && tid < NUM_QUEUES) p.queue[tid] = 0;
  if (tid < NUM_KINDS) s_listed[tid] = 0;
  if (tid == NUM_KINDS) s_taken = 0;
  u64 sums[NUM_SUMS] = {};
  for (i64 c0 = lo; c0 < hi; c0 += kWThreads) {
    const i64 c = c0 + tid;
    i64 d = 0;
    if (c < hi) {
      d = column_of(p, c, true).d;
      if (!p.replace && d > k && d > (i64)kMaxScanEnd) raise_error(p.counters, GSB_ERR_UNSUPPORTED, d);
    }
    const int kind = kind_of(p, d);
#pragma unroll
    for (int v = 0; v < NUM_KINDS; ++v) sums[v] += __popc(__ballot_sync(0xffffffffu, kind == v));
    sums[SUM_EDGES] += (u64)picks_of(p, d);
    if (kind == KIND_HUGE) sums[SUM_HUGE_DEGREE] += (u64)d;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sums[SUM_EDGES] += __shfl_xor_sync(0xffffffffu, sums[SUM_EDGES], o);
    sums[SUM_HUGE_DEGREE] += __shfl_xor_sync(0xffffffffu, sums[SUM_HUGE_DEGREE], o);
  }
  if (lane == 0) {
#pragma unroll
    for (int v = 0; v < NUM_SUMS; ++v) s_part[warp][v][0] = sums[v];
  }
  __syncthreads();
  if (tid < NUM_SUMS) {
    u64 sum = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) sum += s_part[w][tid][0];
    p.partial[(i64)blockIdx.x * NUM_SUMS + tid] = (i64)sum;
  }
  // The result of a call that was given up: an empty sample.
  auto give_up = [&] {
    grid_share(p.S, [&](i64 c) { p.out_indptr[c] = 0; });  // the CTA's columns
    if (blockIdx.x == 0) p.out_indptr[p.S] = p.counters[CNT_NNZ] = 0;
  };
  grid_barrier(p.sync, 1, give_up);

  // every CTA adds up what comes before it and the totals
  static_assert(NUM_SUMS == 8, "eight threads take one CTA's sums");
  {
    u64 before = 0, total = 0;
#pragma unroll 8
    for (int b = tid >> 3; b < (int)gridDim.x; b += kWThreads / 8) {
      const u64 x = (u64)__ldcg(p.partial + b * NUM_SUMS + (tid & 7));
      total += x;
      if (b < (int)blockIdx.x) before += x;
    }
#pragma unroll
    for (int o = 8; o < 32; o <<= 1) {
      before += __shfl_xor_sync(0xffffffffu, before, o);
      total += __shfl_xor_sync(0xffffffffu, total, o);
    }
    if (lane < NUM_SUMS) {
      s_part[warp][lane][0] = before;
      s_part[warp][lane][1] = total;
    }
  }
  __syncthreads();
  if (tid < NUM_SUMS) {
    u64 before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      before += s_part[w][tid][0];
      total += s_part[w][tid][1];
    }
    s_before[tid] = before;
    s_total[tid] = total;
  }
  __syncthreads();
  const i64 edges = (i64)s_total[SUM_EDGES];
  const bool overflow = edges > p.capacity;
  if (blockIdx.x == 0 && tid == 0) {
    p.out_indptr[S] = edges;
    p.counters[CNT_NNZ] = edges;
    if (overflow) {
      raise_error(p.counters, GSB_ERR_CAPACITY, edges);
      mail_post(p.mail, 0, edges, p.counters);
    }
  }
  // slices so long that there is room for them: no more than kMaxSlices / 2 columns are longer than one, and what is left over
  // of each adds one more at most
  i64 slice = kSlice;
  while (slice < (1ll << 32) && (i64)s_total[SUM_HUGE_DEGREE] > slice * (kMaxSlices / 2)) slice <<= 1;
  if (tid < NUM_KINDS) {
    u64 at = s_before[tid];
    for (int v = 0; v < tid; ++v) at += s_total[v];
    s_at[tid] = at;
  }
  __syncthreads();

  // output offsets, and the columns by kind
  i64 next = (i64)s_before[SUM_EDGES];
  for (i64 c0 = lo; c0 < hi; c0 += kWThreads) {
    const i64 c = c0 + tid;
    const i64 d = c < hi ? column_of(p, c, false).d : 0;
    i64 sum;
    const i64 before = block_exclusive_scan<kWThreads>(picks_of(p, d), s_scan, &sum);
    if (c < hi) p.out_indptr[c] = next + before;
    next += sum;
    const int kind = kind_of(p, d);
#pragma unroll
    for (int v = KIND_HUGE + 1; v < NUM_KINDS; ++v) {
      const unsigned who = __ballot_sync(0xffffffffu, kind == v);
      if (!who) continue;
      unsigned at = 0;
      if (lane == 0) at = atomicAdd(&s_listed[v], (unsigned)__popc(who));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (kind == v) p.lists[s_at[v] + at + __popc(who & ((1u << lane) - 1u))] = c;
    }
    if (kind == KIND_HUGE) {
      if (WIDE || p.replace || d <= slice) {
        p.lists[atomicAdd(p.queue + QUEUE_HUGE, 1ull)] = c;  // the first region
      } else {
        const unsigned slices = (unsigned)((d + slice - 1) / slice);
        const u64 first = atomicAdd(p.queue + QUEUE_SLICES, (u64)slices);
        if (first + slices <= kMaxSlices) {
          p.slice_done[first] = 0;
          p.slice_floor[first] = 0;
          for (unsigned i = 0; i < slices; ++i) p.slices[first + i] = WeightedSlice{c, i, (unsigned)first};
        }
      }
    }
  }
  if (overflow) {  // the same in every CTA
    grid_arrive(p.sync, 1);
    return;
  }
  grid_barrier(p.sync, 2, give_up);
  if (blockIdx.x == 0 && tid == 0) mail_post(p.mail, 0, edges, p.counters);  // nothing can go wrong from here on

  // Every CTA does each gridDim-th unit of work, the long ones first, and its warps take them as they become free: a counter
  // for the whole grid is what the grid would wait for (one word takes about one atomic per nanosecond).
  const i64 slices = min((i64)__ldcg(p.queue + QUEUE_SLICES), (i64)kMaxSlices), huge = (i64)__ldcg(p.queue + QUEUE_HUGE);
  const i64 scans = (i64)s_total[KIND_SCAN], scan_list = (i64)s_total[KIND_HUGE];
  const i64 heavy = slices + huge + scans;
  auto heavy_column = [&](i64 unit) {
    unit -= slices;
    return __ldcg(p.lists + (unit < huge ? unit : scan_list + unit - huge));
  };
  i64 first = blockIdx.x;  // of the CTA's units
  if (WIDE) {
    WideShared& s_wide = *reinterpret_cast<WideShared*>(s_dynamic);
    for (;;) {  // these differ too much to be dealt out: the next free CTA takes the next one
      if (tid == 0) s_unit = (i64)atomicAdd(p.queue + QUEUE_NEXT, 1ull);
      __syncthreads();
      const i64 unit = s_unit;
      if (unit >= heavy) break;
      select_wide(p, s_wide, heavy_column(unit));
      __syncthreads();
    }
    first += heavy;
  }
  for (;;) {
    i64 unit = 0;
    if (lane == 0) unit = first + (i64)atomicAdd(&s_taken, 1u) * gridDim.x;
    unit = __shfl_sync(0xffffffffu, unit, 0);
    if (!WIDE && unit < heavy) {
      const bool sliced = unit < slices;
      const i64 c = sliced ? 0 : heavy_column(unit);
      if (p.replace) {
        const Column column = column_of(p, c, false);
        draw_with_replacement(p, column.b, column.d, __ldcg(p.out_indptr + c), c, reinterpret_cast<float*>(s_order[warp]));
      } else {
        scan_column(p, c, sliced, (unsigned)unit, slice, s_order[warp]);
      }
      continue;
    }
    unit -= heavy;
    i64 list = scan_list + scans;
    int kind = KIND_SORT128;
#pragma unroll 1
    for (; kind < NUM_KINDS; ++kind) {
      const int columns = kind == KIND_SORT128 ? 1 : kind == KIND_SORT64 ? 2 : 4;  // in a unit
      const i64 count = (i64)s_total[kind], units = (count + columns - 1) / columns;
      if (unit < units) {
        short_columns(p, kind, list, unit * columns, count, s_order[warp]);
        break;
      }
      list += count;
      unit -= units;
    }
    if (kind == NUM_KINDS) break;
  }
}

}  // namespace gsb

using namespace gsb;

extern "C" int gsb_sample_weighted(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices,
                                   int64_t num_cols, const float* probs, const int64_t* seeds, int64_t S, int64_t k, int replace,
                                   uint64_t seed, int64_t* out_indptr, int64_t* out_indices, int64_t* out_select,
                                   int64_t* out_coo_col, const float* data, const int64_t* e_ids, float* out_data,
                                   int64_t capacity, int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && S >= 0 && k >= 0 && num_cols >= 0 && (seeds || S <= num_cols),
              GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(out_indices || capacity == 0, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(replace || k <= kWideMaxK, GSB_ERR_UNSUPPORTED);
  cudaStream_t stream = (cudaStream_t)stream_;
  const bool wide = !replace && k > 32;
  const void* kernel = wide ? (const void*)k_sample_weighted<true> : (const void*)k_sample_weighted<false>;
  const size_t smem = wide ? sizeof(WideShared) : 0;
  static int resident[2][64];
  const int ctas = ctx_resident_ctas(ctx, kernel, kWThreads, smem, resident[wide]);
  GSB_REQUIRE(ctas > 0, GSB_ERR_UNSUPPORTED);
  // a small call gets few CTAs, whose barriers are cheaper; 32 of them share the slices of its hubs
  const int grid = (int)min((i64)ctas, 32 + S / 4);
  auto bytes = [](size_t n) { return (n + 255) & ~(size_t)255; };
  const size_t sizes[] = {bytes(sizeof(i64) * NUM_SUMS * (size_t)ctas), bytes(sizeof(u64) * NUM_QUEUES),
                          bytes(sizeof(i64) * (size_t)S), wide ? 0 : bytes(sizeof(WeightedSlice) * kMaxSlices),
                          wide ? 0 : bytes(sizeof(u64) * 32 * kMaxSlices), wide ? 0 : bytes(sizeof(unsigned) * kMaxSlices),
                          wide ? 0 : bytes(sizeof(unsigned) * kMaxSlices)};
  char* at[7];
  size_t total_bytes = 0;
  for (size_t n : sizes) total_bytes += n;
  void* ws;
  int st = ctx_reserve_workspace(ctx, stream, total_bytes, &ws);
  if (st != GSB_OK) return st;
  at[0] = (char*)ws;
  for (int i = 1; i < 7; ++i) at[i] = at[i - 1] + sizes[i - 1];
  WeightedParams p{indptr,      indices, probs, num_cols, seeds,    S,        k,                 replace,
                   (u64)seed,   out_indptr, out_indices, out_select, out_coo_col, data, e_ids,   out_data,
                   capacity,    ctx_counters(ctx), nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0},
                   (i64*)at[0], (u64*)at[1], (i64*)at[2], (WeightedSlice*)at[3], (u64*)at[4], (unsigned*)at[5],
                   (unsigned*)at[6], ctx_grid_sync(ctx, grid, kWeightedBarriers)};
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_WEIGHTED, stream);
    void* args[] = {&p};
    st = launch_cooperative(ctx, stream, kernel, grid, kWThreads, smem, args, p.sync);
    if (st != GSB_OK) return st;
  }
  if (!nnz_host) return GSB_OK;
  i64 total = 0;
  st = ctx_mail_result(ctx, stream, p.mail, 1, &total);
  *nnz_host = total;
  return st;
}
