// Row slicing by membership: keep the edges whose row id is in `row_ids`, renumber the kept row id
// to its position in `row_ids`, preserve edge order.
//
// pass 1  k_build_row_table   row id -> position (largest position for a repeated id)
// pass 2  k_row_filter        edge-parallel: probe, flag, block scan + look-back, stable compaction;
//                             also stores each edge's exclusive prefix so that
// pass 3  k_row_indptr        out_indptr[c] = prefix at indptr[c]  (offsets over ALL operand columns)
//
// The reference probes every edge with a warp per column, writes a dense mask, then compacts with
// torch::nonzero and two or three torch index gathers (src/cuda/slicing.cu:416-526); the COO form
// (:543-563, 727-771) is the same without offsets.
#include "batch_table.cuh"
#include "column_walk.cuh"
#include "common.cuh"
#include "grid_sync.cuh"
#include "hash_table.cuh"
#include "radix_sort.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kRowThreads = 256;
constexpr int kRowPerThread = 4;
constexpr int kRowTile = kRowThreads * kRowPerThread;
constexpr u64 kMaxFlip = 0x7fffffffffffffffull;  // val = kMaxFlip - position, so atomicMin keeps the LARGEST position

// Membership filter in front of the row table: one bit per hashed id, kept INVERTED (0 = some row id hashes here) so that
// one 0xFF fill clears table and filter together.  It is small enough for shared memory, and most edges of a slice miss:
// they never reach the table, whose random 32-byte reads were what the filter kernels waited for.
struct RowBloom {
  u32* words;  // null: no filter
  int shift;   // 32 - log2(bits)
};
// Of the id's low half: a filter may take two ids for one, and the 64-bit product was six instructions more per edge.
__device__ __forceinline__ u32 bloom_bit(const RowBloom& b, i64 key) { return ((u32)key * 0x9E3779B1u) >> b.shift; }

__global__ void __launch_bounds__(kRowThreads) k_build_row_table(const i64* __restrict__ row_ids, i64 R, Table table,
                                                                 RowBloom bloom, i64* counters) {
  for (i64 i = (i64)blockIdx.x * kRowThreads + threadIdx.x; i < R; i += (i64)gridDim.x * kRowThreads) {
    const i64 key = row_ids[i];
    if (key < 0) {
      raise_error(counters, GSB_ERR_INDEX_RANGE, i);
      continue;
    }
    if (!table_insert_min(table, key, kMaxFlip - (u64)i)) raise_error(counters, GSB_ERR_TABLE_FULL, i);
    if (bloom.words) {
      const u32 bit = bloom_bit(bloom, key);
      atomicAnd(bloom.words + (bit >> 5), ~(1u << (bit & 31)));
    }
  }
}

struct RowFilterParams {
  const i64* rows;      // row id per edge (CSC indices or COO row)
  const i64* coo_col;   // COO: column per edge (copied through); CSC: null
  i64 E;
  Table table;
  i64* out_rows;        // renumbered row per kept edge
  i64* out_cols;        // COO: column of kept edge; CSC with_coo: filled by k_row_indptr pass; may be null
  i64* out_select;      // kept edge positions
  i64* edge_prefix;     // [E + 1] exclusive prefix of the keep flags (CSC form), may be null
  i64* counters;
  TileState ts;
  Mail mail;
};

__global__ void __launch_bounds__(kRowThreads) k_row_filter(RowFilterParams p) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  const int tile = blockIdx.x;
  const i64 base = (i64)tile * kRowTile;
  if (base >= p.E && !(p.E == 0 && tile == 0)) return;
  i64 newid[kRowPerThread];
  int keep[kRowPerThread];
  int mine = 0;
#pragma unroll
  for (int q = 0; q < kRowPerThread; ++q) {
    const i64 e = base + (i64)threadIdx.x * kRowPerThread + q;
    keep[q] = 0;
    newid[q] = -1;
    if (e < p.E) {
      const i64 r = p.rows[e];
      const Slot* s = r >= 0 ? table_find(p.table, r) : nullptr;
      if (s) {
        keep[q] = 1;
        newid[q] = (i64)(kMaxFlip - s->val);
      }
    }
    mine += keep[q];
  }
  i64 total;
  const i64 excl = block_exclusive_scan<kRowThreads>((i64)mine, s_scan, &total);
  if (threadIdx.x < 32) {
    const i64 prefix = tile_exclusive_prefix(p.ts, tile, total);
    if (threadIdx.x == 0) s_base = prefix;
  }
  __syncthreads();
  i64 pos = s_base + excl;
#pragma unroll
  for (int q = 0; q < kRowPerThread; ++q) {
    const i64 e = base + (i64)threadIdx.x * kRowPerThread + q;
    if (e < p.E) {
      if (p.edge_prefix) p.edge_prefix[e] = pos;
      if (keep[q]) {
        p.out_rows[pos] = newid[q];
        p.out_select[pos] = e;
        if (p.coo_col) p.out_cols[pos] = p.coo_col[e];
        ++pos;
      }
    }
  }
  if (base + kRowTile >= p.E && threadIdx.x == kRowThreads - 1) {
    if (p.edge_prefix) p.edge_prefix[p.E] = s_base + total;
    p.counters[CNT_NNZ] = s_base + total;
    mail_post(p.mail, 0, s_base + total, p.counters);
  }
}

// out_indptr[c] = number of kept edges before column c; optionally the column id of every kept edge.
__global__ void __launch_bounds__(kRowThreads) k_row_indptr(const i64* __restrict__ indptr, i64 num_cols,
                                                            const i64* __restrict__ edge_prefix,
                                                            i64* __restrict__ out_indptr, i64* __restrict__ out_cols) {
  const int lane = threadIdx.x & 31;
  const i64 warp_global = ((i64)blockIdx.x * kRowThreads + threadIdx.x) >> 5;
  const i64 num_warps = ((i64)gridDim.x * kRowThreads) >> 5;
  for (i64 c = warp_global; c <= num_cols; c += num_warps) {
    const i64 lo = edge_prefix[indptr[c]];
    if (lane == 0) out_indptr[c] = lo;
    if (out_cols && c < num_cols) {
      const i64 hi = edge_prefix[indptr[c + 1]];
      for (i64 j = lo + lane; j < hi; j += 32) out_cols[j] = c;
    }
  }
}

// ---- fused column + row slicing (induced subgraph) ---------------------------------------------------
// For the seed columns only: keep the edges whose row id is in `row_ids` (src/cuda/fusion/column_row_slicing.cu:
// 101-217).  Super-batch form (:218-365): column c of batch b keeps rows that are in batch b's row list; the
// table key is id + b * encoding_size, as in the reference.
//
// Edge-parallel, so that a hub column costs what its edges cost: the D edges of the seed columns form one
// virtual list (sub_indptr = exclusive scan of the seed degrees); a CTA takes 1024 consecutive positions,
// finds their columns by a search restricted to the tile's column range, probes the row table and compacts
// the survivors with ballots + one look-back; the thread that owns the first edge of a column also writes
// that column's output offset.  (One warp per column was measured 6x slower on a power-law graph: the
// warp that gets a 17 000-edge column runs 540 dependent rounds while the rest of the grid is idle.)
struct ColRowParams {
  const i64* indptr;
  const i64* indices;
  i64 num_cols;
  const i64* seeds;
  i64 S;
  const i64* sub_indptr;  // [S + 1]
  i64 D;
  const i64* col_ptr;  // [G + 1] or null (one batch)
  i64 G;
  i64 encoding_size;
  Table table;
  int renumber;  // 1: write the position in row_ids; 0: keep the row id
  i64* out_indptr;
  i64* out_indices;
  i64* out_select;
  const float* data;
  const i64* e_ids;
  float* out_data;
  i64* counters;
  TileState ts;
  Mail mail;
};

__global__ void __launch_bounds__(kRowThreads) k_build_batch_row_table(const i64* __restrict__ row_ids, i64 R,
                                                                       const i64* __restrict__ row_ptr, i64 G,
                                                                       i64 encoding_size, Table table,
                                                                       i64* counters) {
  for (i64 i = (i64)blockIdx.x * kRowThreads + threadIdx.x; i < R; i += (i64)gridDim.x * kRowThreads) {
    const i64 id = row_ids[i];
    if (id < 0) {
      raise_error(counters, GSB_ERR_INDEX_RANGE, i);
      continue;
    }
    const i64 key = id + batch_of(row_ptr, G, i) * encoding_size;
    if (!table_insert_min(table, key, kMaxFlip - (u64)i)) raise_error(counters, GSB_ERR_TABLE_FULL, i);
  }
}

constexpr int kCrLane = 4;
constexpr int kCrWarp = 32 * kCrLane;                      // positions per warp
constexpr int kCrTile = (kRowThreads / 32) * kCrWarp;      // positions per CTA

// largest c in [lo, hi] with sub_indptr[c] <= pos  (sub_indptr[lo] <= pos is given)
__device__ __forceinline__ i64 column_at(const i64* __restrict__ sub_indptr, i64 lo, i64 hi, i64 pos) {
  while (lo < hi) {
    const i64 mid = (lo + hi + 1) >> 1;
    if (__ldg(sub_indptr + mid) <= pos) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

__global__ void __launch_bounds__(kRowThreads) k_col_row_filter(ColRowParams p) {
  __shared__ i64 s_warp_total[kRowThreads / 32];
  __shared__ i64 s_base, s_clo, s_chi;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tile = blockIdx.x;
  const i64 tile_base = (i64)tile * kCrTile;
  const i64 tile_end = min(p.D, tile_base + kCrTile);
  // the tile's column range: two warp-wide searches side by side (one thread doing both binary searches over the
  // global offsets was 36 dependent loads with the rest of the CTA waiting at the barrier — most of the kernel's time)
  if (warp < 2) {
    const i64 c = warp_column_search(p.sub_indptr, p.S, warp == 0 ? tile_base : tile_end - 1);
    if (lane == 0) (warp == 0 ? s_clo : s_chi) = c;
  }
  __syncthreads();
  const i64 clo = s_clo, chi = s_chi;
  const i64 base = tile_base + (i64)warp * kCrWarp;
  bool keep[kCrLane];
  i64 col_of[kCrLane], edge[kCrLane], value[kCrLane];
  // the warp's 128 positions are consecutive: search for the first one, then the column only walks forward.
  // Phases (column -> edge position -> row id -> table probe) run for all four positions of a lane before the next
  // phase starts, so that four independent loads are in flight per lane in every phase.
  i64 c = base < tile_end ? column_at(p.sub_indptr, clo, chi, base) : clo;
  i64 start_of[kCrLane], row_of[kCrLane];
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    keep[q] = false;
    col_of[q] = -1;
    const i64 pos = base + q * 32 + lane;
    if (pos < tile_end) {
      while (c < chi && __ldg(p.sub_indptr + c + 1) <= pos) ++c;
      col_of[q] = c;
    }
  }
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    if (col_of[q] >= 0) {
      const i64 col = p.seeds ? __ldg(p.seeds + col_of[q]) : col_of[q];
      if ((u64)col < (u64)p.num_cols) {
        start_of[q] = __ldg(p.indptr + col);
      } else {  // only reachable when sub_indptr was not counted for these seeds: drop the position
        raise_error(p.counters, GSB_ERR_INDEX_RANGE, col_of[q]);
        col_of[q] = -1;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    row_of[q] = -1;
    if (col_of[q] >= 0) {
      const i64 pos = base + q * 32 + lane;
      edge[q] = start_of[q] + (pos - __ldg(p.sub_indptr + col_of[q]));
      row_of[q] = __ldg(p.indices + edge[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    if (row_of[q] >= 0) {
      const i64 shift = p.col_ptr ? batch_of(p.col_ptr, p.G, col_of[q]) * p.encoding_size : 0;
      const Slot* s = table_find(p.table, row_of[q] + shift);
      if (s) {
        keep[q] = true;
        value[q] = p.renumber ? (i64)(kMaxFlip - s->val) : row_of[q];
      }
    }
  }
  const unsigned lt = (1u << lane) - 1u;
  unsigned rank[kCrLane];
  unsigned run = 0;
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    const unsigned bal = __ballot_sync(0xffffffffu, keep[q]);
    rank[q] = run + __popc(bal & lt);
    run += __popc(bal);
  }
  if (lane == 0) s_warp_total[warp] = run;
  __syncthreads();
  i64 warp_excl = 0, tile_total = 0;
#pragma unroll
  for (int x = 0; x < kRowThreads / 32; ++x) {
    const i64 t = s_warp_total[x];
    if (x < warp) warp_excl += t;
    tile_total += t;
  }
  if (warp == 0) {
    const i64 prefix = tile_exclusive_prefix(p.ts, tile, tile_total);
    if (lane == 0) s_base = prefix;
  }
  __syncthreads();
  const i64 warp_pos = s_base + warp_excl;
#pragma unroll
  for (int q = 0; q < kCrLane; ++q) {
    const i64 pos = base + q * 32 + lane;
    if (pos < tile_end) {
      const i64 out = warp_pos + rank[q];
      const i64 c = col_of[q];
      if (pos == __ldg(p.sub_indptr + c)) {
        // first edge of column c: its output offset, and that of the empty columns right in front of it
        p.out_indptr[c] = out;
        for (i64 e = c - 1; e >= 0 && __ldg(p.sub_indptr + e) == pos; --e) p.out_indptr[e] = out;
      }
      if (keep[q]) {
        p.out_indices[out] = value[q];
        if (p.out_select) p.out_select[out] = edge[q];
        if (p.out_data) p.out_data[out] = p.data[p.e_ids ? p.e_ids[edge[q]] : edge[q]];
      }
    }
  }
  if (tile_end == p.D && threadIdx.x == 0) {
    const i64 total = s_base + tile_total;
    p.out_indptr[p.S] = total;
    for (i64 e = p.S - 1; e >= 0 && __ldg(p.sub_indptr + e) == p.D; --e) p.out_indptr[e] = total;
    p.counters[CNT_NNZ] = total;
    mail_post(p.mail, 0, total, p.counters);
  }
}

// ---- induced subgraph of one node set in one launch -----------------------------------------------------------------
// The single-batch form of k_col_row_filter as a cooperative kernel: a warp owns one stretch of the virtual edge list.
//   filter   128 positions at a time, columns found without barriers (column_walk.cuh); an edge is looked up in the table only
//            when the shared-memory filter lets it pass; survivors go to scratch in order, with their positions;
//   barrier
//   emit     every CTA scans the CTAs' totals, copies its survivors to their places (and gathers their edge data), and a
//            share of the columns finds its offset by a binary search among the survivors of the warp that had the column's
//            first position (seven reads in the case below, instead of a word per 32 positions that all groups have to leave).
// Bounded by instruction issue, then by the reads a warp waits for.  20 000 columns with 7.1 M edges, 20 000 rows: 178 us with a
// table probe per edge and a look-back chain of 6 400 tiles, 84 with a stretch per CTA (six tiles of two searches and four
// barriers each), 67 with one per warp, 51 with pieces of columns, one read per table slot and the edge data on their way to L2
// before the barrier.  One column after the other, 128 positions a step, has fewer instructions (20 M for 24 M), but a warp
// whose columns are short takes 80 such steps: half the warps were done after 25 us, the last after 43.
constexpr int kInThreads = 512;
constexpr int kInPer = 4;
constexpr u32 kInQueue = 128;  // edges of a warp that wait for their look-up: 31 left over and 64 more at most
constexpr int kInWarps = kInThreads / 32;
constexpr int kBloomMaxBits = 1 << 19;  // 64 KB: two CTAs per SM
constexpr i64 kBloomMaxRows = 1 << 18;  // beyond, most edges would pass
// Edges per column from which pieces of columns are the faster way: 4 M edges, 20 000 rows, positions against pieces: columns of 4
// 106 / 149 us for the call, 12 92 / 95, 16 86.5 / 85.9, 24 87 / 81, 64 69 / 65; a heavy tail of mean 16 78 / 83, of mean 32 75 / 72.
constexpr i64 kInPieces = 20;
constexpr i64 kInducedMaxEdges = 1 << 27;  // its scratch is 12 bytes per edge
constexpr int kInAtBits = 16;              // of a position in a warp's stretch (28 400 at most with two CTAs on each SM)

struct InducedParams {
  ColRowParams c;
  RowBloom bloom;
  i64 range;        // positions per warp
  u32* totals;      // [CTAs]
  u32* warp_before;  // [CTAs][kInWarps] survivors of the CTA's warps before this one
  u32* warp_kept;   // [CTAs][kInWarps] survivors of the warp
  u32* kept_at;     // [D] position in the warp's stretch : 16 | high part of the position in the operand : 16, ascending
  u32* kept_edge;   // [D] its low part
  u32* kept_row;    // [D] position in row_ids
  GridSync sync;
};

// Position in row_ids of a row id of the table, or kNoRow.
constexpr u32 kNoRow = 0xFFFFFFFFu;
__device__ __forceinline__ u32 find_row(const Table& t, i64 id) {
  const u32 mask = (u32)t.mask;
  u32 h = (u32)table_home(t, id);
  for (u32 left = mask;; --left) {
    const longlong2 slot = __ldg(reinterpret_cast<const longlong2*>(t.slots) + h);
    if (slot.x == id) return (u32)(kMaxFlip - (u64)slot.y);
    if (slot.x == kEmptyKey || left == 0) return kNoRow;
    h = (h + 1) & mask;
  }
}

// PIECES: the columns are long enough to be taken in pieces of their own.
template <bool PIECES>
__global__ void __launch_bounds__(kInThreads, 2) k_induced(const __grid_constant__ InducedParams p) {
  extern __shared__ __align__(16) u32 s_bloom[];
  __shared__ u32 s_warp[kInWarps];
  __shared__ u32 s_prefix[kInThreads];
  struct Passed {  // an edge that passed the filter
    i64 edge;      // position in the operand
    u32 id;        // low half of its row id
    u32 at;        // position in the stretch; kWide: the id has a high half, which is read again
  };
  constexpr u32 kWide = 0x80000000u;
  __shared__ __align__(16) Passed s_queue[kInWarps][kInQueue];
  const ColRowParams& c = p.c;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const i64 begin = min(c.D, ((i64)blockIdx.x * kInWarps + warp) * p.range), end = min(c.D, begin + p.range);
  if (p.bloom.words) {
    const int quads = (1 << (32 - p.bloom.shift)) / 128;
    for (int i = tid; i < quads; i += kInThreads)
      reinterpret_cast<uint4*>(s_bloom)[i] = __ldcg(reinterpret_cast<const uint4*>(p.bloom.words) + i);
  }
  ColumnWalk walk;
  walk.off = c.sub_indptr;
  walk.seeds = c.seeds;
  walk.indptr = c.indptr;
  walk.S = c.S;
  walk.num_cols = c.num_cols;
  walk.counters = c.counters;  // a bad seed has positions only when sub_indptr was not counted for these seeds
  if (begin < end) walk.init(begin, (int)(end - begin));
  __syncthreads();  // the filter is loaded
  u32 kept = 0;  // survivors of the warp so far
  u32 head = 0, tail = 0;
  // Few edges pass the filter, but nearly every group of 32 has some: looked up where they stand, each group would wait out a
  // chain of table reads for two or three lanes.  They are queued instead, and looked up 32 at a time; the queue has the order
  // of the edges, so the survivors leave it in theirs.
  auto look_up = [&] {
    __syncwarp();
    u32 row = kNoRow;
    Passed e;
    if (lane < (int)(tail - head)) {
      e = s_queue[warp][(head + lane) % kInQueue];
      row = find_row(c.table, e.at & kWide ? __ldg(c.indices + e.edge) : (i64)e.id);
    }
    const unsigned bits = __ballot_sync(0xffffffffu, row != kNoRow);
    if (row != kNoRow) {
      const i64 to = begin + kept + __popc(bits & lt);
      p.kept_row[to] = row;
      p.kept_edge[to] = (u32)e.edge;
      p.kept_at[to] = (e.at << kInAtBits) | (u32)((u64)e.edge >> 32);  // (which shifts kWide out)
      // random reads that the DRAM serves 43 G of a second: they come while the filter leaves it idle
      if (c.out_data) asm volatile("prefetch.global.L2 [%0];" ::"l"(c.e_ids ? (const void*)(c.e_ids + e.edge) : c.data + e.edge));
    }
    kept += __popc(bits);
    head += min(32u, tail - head);
    __syncwarp();
  };
  auto test = [&](const int (&at)[kInPer], const i64 (&edge)[kInPer]) {
    i64 id[kInPer];
#pragma unroll
    for (int r = 0; r < kInPer; ++r) id[r] = edge[r] >= 0 ? __ldg(c.indices + edge[r]) : -1;
#pragma unroll
    for (int r = 0; r < kInPer; ++r) {
      bool pass = id[r] >= 0;
      if (p.bloom.words) {  // (what lies in the filter's place for no id is read and not used)
        const u32 bit = bloom_bit(p.bloom, id[r]);
        pass = pass && ((s_bloom[bit >> 5] >> (bit & 31u)) & 1u) == 0u;
      }
      const unsigned passing = __ballot_sync(0xffffffffu, pass);
      if (pass) {
        Passed e;
        e.edge = edge[r];
        e.id = (u32)id[r];
        e.at = (u32)at[r] | ((u64)id[r] >> 32 ? kWide : 0u);
        s_queue[warp][(tail + __popc(passing & lt)) % kInQueue] = e;
      }
      tail += __popc(passing);
      if (r % 2 == 1)
        while (tail - head >= 32) look_up();
    }
  };
  if (begin < end) {
    if (PIECES) {
      walk.for_pieces<kInPer>(test);
    } else {
      for (int first = 0; first < walk.len; first += 32 * kInPer) {
        int at[kInPer];
        i64 edge[kInPer];
#pragma unroll
        for (int r = 0; r < kInPer; ++r) {
          at[r] = first + r * 32 + lane;
          edge[r] = first + r * 32 < walk.len ? walk.locate<false>(first + r * 32, nullptr) : -1;  // uniform
        }
        test(at, edge);
      }
    }
  }
  while (tail != head) look_up();
  u32 cta_before = 0;  // of the CTA's warps before this one
  if (lane == 0) s_warp[warp] = kept;
  __syncthreads();
  {
    u32 all = 0;
#pragma unroll
    for (int w = 0; w < kInWarps; ++w) {
      if (w < warp) cta_before += s_warp[w];
      all += s_warp[w];
    }
    if (lane == 0) {
      p.warp_before[blockIdx.x * kInWarps + warp] = cta_before;
      p.warp_kept[blockIdx.x * kInWarps + warp] = kept;
    }
    if (tid == 0) p.totals[blockIdx.x] = all;
  }
  grid_barrier(p.sync, 1, [&] {  // given up: an empty subgraph
    grid_share(c.S + 1, [&](i64 j) { c.out_indptr[j] = 0; });
    if (blockIdx.x == 0) c.counters[CNT_NNZ] = 0;
  });
  // ---- emit
  u32 total;
  {
    const u32 t = tid < (int)gridDim.x ? __ldcg(p.totals + tid) : 0;
    u32 inc = t;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 x = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += x;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    u32 before = 0;
    total = 0;
#pragma unroll
    for (int w = 0; w < kInWarps; ++w) {
      if (w < warp) before += s_warp[w];
      total += s_warp[w];
    }
    s_prefix[tid] = before + inc - t;
    __syncthreads();
  }
  if (blockIdx.x == 0 && tid == 0) {
    c.counters[CNT_NNZ] = total;
    mail_post(c.mail, 0, total, c.counters);
  }
  const i64 out0 = s_prefix[blockIdx.x] + cta_before;
  constexpr int kAhead = 4;  // survivors of a lane whose reads are in flight together
  for (u32 j0 = lane; j0 < kept; j0 += 32 * kAhead) {  // written by this very warp
    i64 e[kAhead], value[kAhead];
    float x[kAhead];
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      const u32 j = j0 + q * 32;
      e[q] = j < kept ? (i64)(((u64)(__ldcg(p.kept_at + begin + j) & 0xFFFFu) << 32) | __ldcg(p.kept_edge + begin + j)) : -1;
    }
#pragma unroll
    for (int q = 0; q < kAhead; ++q)
      if (e[q] >= 0) value[q] = c.renumber ? (i64)__ldcg(p.kept_row + begin + j0 + q * 32) : __ldg(c.indices + e[q]);
    if (c.out_data) {
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (e[q] >= 0) x[q] = __ldg(c.data + (c.e_ids ? __ldg(c.e_ids + e[q]) : e[q]));
    }
#pragma unroll
    for (int q = 0; q < kAhead; ++q) {
      if (e[q] < 0) continue;
      const i64 to = out0 + j0 + q * 32;
      c.out_indices[to] = value[q];
      if (c.out_select) c.out_select[to] = e[q];
      if (c.out_data) c.out_data[to] = x[q];
    }
  }
  for (i64 j = (i64)blockIdx.x * kInThreads + tid; j <= c.S; j += (i64)gridDim.x * kInThreads) {
    const i64 pos = __ldg(c.sub_indptr + j);
    i64 rank = total;
    if (pos < c.D) {
      const u32 owner = (u32)(pos / p.range), at = (u32)(pos - (i64)owner * p.range);
      const u32* list = p.kept_at + (i64)owner * p.range;
      u32 lo = 0, hi = __ldcg(p.warp_kept + owner);  // survivors before the column: the first that lies at or behind it
      while (lo < hi) {
        const u32 mid = (lo + hi) >> 1;
        if (__ldcg(list + mid) < at << kInAtBits) lo = mid + 1;
        else hi = mid;
      }
      rank = s_prefix[owner / kInWarps] + __ldcg(p.warp_before + owner) + lo;
    }
    c.out_indptr[j] = rank;
  }
}

// ---- index search: position of every key in `origin` (largest position for a repeated id), -1 if absent --
__global__ void __launch_bounds__(kRowThreads) k_index_search(const i64* __restrict__ keys, i64 M, Table table,
                                                              i64* __restrict__ out) {
  for (i64 i = (i64)blockIdx.x * kRowThreads + threadIdx.x; i < M; i += (i64)gridDim.x * kRowThreads) {
    const i64 k = __ldg(keys + i);
    const Slot* s = k >= 0 ? table_find(table, k) : nullptr;
    out[i] = s ? (i64)(kMaxFlip - s->val) : -1;
  }
}

}  // namespace gsb

using namespace gsb;

// With `bloom` the filter is built too: 24 bits per row id (a miss passes it one time in 25), at most kBloomMaxBits.
static int build_table(gsb_ctx* ctx, cudaStream_t stream, const int64_t* row_ids, int64_t R, size_t extra_bytes,
                       Table* table, void** extra, RowBloom* bloom = nullptr) {
  u64 cap;
  table_geometry(R, &cap, &table->shift);
  table->mask = cap - 1;
  int bits_log2 = 10;
  while (bloom && (1 << bits_log2) < kBloomMaxBits && ((i64)1 << bits_log2) < 24 * R) ++bits_log2;
  const size_t bloom_bytes = bloom ? ((size_t)1 << bits_log2) / 8 : 0;
  void* ws;
  const size_t table_bytes = cap * sizeof(Slot) + bloom_bytes;
  int st = ctx_reserve_workspace(ctx, stream, table_bytes + extra_bytes + 256, &ws);
  if (st != GSB_OK) return st;
  table->slots = (Slot*)ws;
  *extra = (char*)ws + table_bytes;
  RowBloom filter{nullptr, 0};
  if (bloom) {
    filter.words = (u32*)((char*)ws + cap * sizeof(Slot));
    filter.shift = 32 - bits_log2;
    *bloom = filter;
  }
  GSB_CUDA_OK(cudaMemsetAsync(table->slots, 0xFF, table_bytes, stream));
  if (R > 0) {
    k_build_row_table<<<min(grid_for(R, kRowThreads), kNumSMs * 8), kRowThreads, 0, stream>>>(row_ids, R, *table,
                                                                                              filter, ctx_counters(ctx));
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
  }
  return GSB_OK;
}

static int finish_count(gsb_ctx* ctx, cudaStream_t stream, const Mail& mail, int64_t* nnz_host) {
  if (!nnz_host) return GSB_OK;
  i64 total = 0;
  const int st = ctx_mail_result(ctx, stream, mail, 1, &total);
  *nnz_host = total;
  return st;
}

extern "C" {

int gsb_row_slice_csc(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices, int64_t num_cols,
                      int64_t E, const int64_t* row_ids, int64_t R, int64_t* out_indptr, int64_t* out_indices,
                      int64_t* out_select, int64_t* out_coo_col, int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && num_cols >= 0 && E >= 0 && R >= 0, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(E == 0 || (indices && out_indices && out_select), GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  Table table;
  void* extra;
  int st = build_table(ctx, stream, row_ids, R, sizeof(i64) * (size_t)(E + 1), &table, &extra);
  if (st != GSB_OK) return st;
  i64* edge_prefix = (i64*)extra;
  const int tiles = grid_for(E, kRowTile);
  TileState ts;
  st = ctx_tile_state(ctx, tiles, stream, &ts);
  if (st != GSB_OK) return st;
  RowFilterParams p{indices, nullptr, E, table, out_indices, nullptr, out_select, edge_prefix, ctx_counters(ctx), ts,
                    nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0}};
  k_row_filter<<<tiles, kRowThreads, 0, stream>>>(p);
  GSB_LAUNCH_OK();
  const i64 blocks = ((num_cols + 1) * 32 + kRowThreads - 1) / kRowThreads;
  k_row_indptr<<<(int)min(blocks, (i64)kNumSMs * 16), kRowThreads, 0, stream>>>(indptr, num_cols, edge_prefix,
                                                                                 out_indptr, out_coo_col);
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 2);
  return finish_count(ctx, stream, p.mail, nnz_host);
}

int gsb_row_slice_coo(gsb_ctx* ctx, void* stream_, const int64_t* coo_row, const int64_t* coo_col, int64_t E,
                      const int64_t* row_ids, int64_t R, int64_t* out_row, int64_t* out_col, int64_t* out_select,
                      int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(E >= 0 && R >= 0, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(E == 0 || (coo_row && coo_col && out_row && out_col && out_select), GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  Table table;
  void* extra;
  int st = build_table(ctx, stream, row_ids, R, 0, &table, &extra);
  if (st != GSB_OK) return st;
  const int tiles = grid_for(E, kRowTile);
  TileState ts;
  st = ctx_tile_state(ctx, tiles, stream, &ts);
  if (st != GSB_OK) return st;
  RowFilterParams p{coo_row, coo_col, E, table, out_row, out_col, out_select, nullptr, ctx_counters(ctx), ts,
                    nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0}};
  k_row_filter<<<tiles, kRowThreads, 0, stream>>>(p);
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 1);
  return finish_count(ctx, stream, p.mail, nnz_host);
}

}  // extern "C"

static int col_row_table(gsb_ctx* ctx, cudaStream_t stream, const int64_t* row_ids, int64_t R, const int64_t* row_ptr,
                         int64_t G, int64_t encoding_size, Table* table) {
  void* extra;
  if (!row_ptr) return build_table(ctx, stream, row_ids, R, 0, table, &extra);
  u64 cap;
  table_geometry(R, &cap, &table->shift);
  table->mask = cap - 1;
  void* ws;
  const size_t table_bytes = cap * sizeof(Slot);
  int st = ctx_reserve_workspace(ctx, stream, table_bytes + 256, &ws);
  if (st != GSB_OK) return st;
  table->slots = (Slot*)ws;
  GSB_CUDA_OK(cudaMemsetAsync(table->slots, 0xFF, table_bytes, stream));
  if (R > 0) {
    k_build_batch_row_table<<<min(grid_for(R, kRowThreads), kNumSMs * 8), kRowThreads, 0, stream>>>(
        row_ids, R, row_ptr, G, encoding_size, *table, ctx_counters(ctx));
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
  }
  return GSB_OK;
}

extern "C" {

int gsb_col_row_slice(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices, int64_t num_cols,
                      const int64_t* column_ids, int64_t S, const int64_t* sub_indptr, int64_t D,
                      const int64_t* row_ids, int64_t R, const int64_t* col_ptr, const int64_t* row_ptr, int64_t G,
                      int64_t encoding_size, int renumber, int64_t* out_indptr, int64_t* out_indices,
                      int64_t* out_select, const float* data, const int64_t* e_ids, float* out_data,
                      int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && sub_indptr && out_indptr && S >= 0 && D >= 0 && R >= 0 && num_cols >= 0 &&
                  (column_ids || S <= num_cols),
              GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE((col_ptr == nullptr) == (row_ptr == nullptr) && (!col_ptr || G >= 1), GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(R == 0 || row_ids, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(D == 0 || (indices && out_indices), GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(D < ((i64)1 << 40), GSB_ERR_UNSUPPORTED);
  cudaStream_t stream = (cudaStream_t)stream_;
  if (D == 0 || R == 0) {  // nothing can survive
    GSB_CUDA_OK(cudaMemsetAsync(out_indptr, 0, sizeof(i64) * (size_t)(S + 1), stream));
    if (nnz_host) *nnz_host = 0;
    return GSB_OK;
  }
  Table table;
  if (!col_ptr && column_ids && D <= kInducedMaxEdges && R < (i64)1 << 31) {
    static int resident[2][64];
    static bool attr_set[64];
    const int dev = ctx_device(ctx);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      GSB_CUDA_OK(cudaFuncSetAttribute(k_induced<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBloomMaxBits / 8));
      GSB_CUDA_OK(cudaFuncSetAttribute(k_induced<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kBloomMaxBits / 8));
      attr_set[dev] = true;
    }
    const bool pieces = D >= kInPieces * S;
    const void* kernel = pieces ? (const void*)k_induced<true> : (const void*)k_induced<false>;
    const int ctas = min(kInThreads, ctx_resident_ctas(ctx, kernel, kInThreads, kBloomMaxBits / 8, resident[pieces]));
    const i64 warps = (i64)ctas * kInWarps;
    const i64 range = ctas > 0 ? max((i64)(32 * kInPer), ((D + warps - 1) / warps + 31) / 32 * 32) : 0;
    if (ctas > 0 && range <= 1 << kInAtBits) {
      InducedParams p{};
      p.range = range;
      const int grid = (int)((D + p.range * kInWarps - 1) / (p.range * kInWarps));
      auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
      const size_t part_bytes = al(4 * (size_t)D);
      void* extra;
      int st = build_table(ctx, stream, row_ids, R, 3 * part_bytes + 4 * kInThreads * (1 + 2 * kInWarps), &table, &extra,
                           R <= kBloomMaxRows ? &p.bloom : nullptr);
      if (st != GSB_OK) return st;
      p.kept_at = (u32*)extra;
      p.kept_edge = (u32*)((char*)extra + part_bytes);
      p.kept_row = (u32*)((char*)extra + 2 * part_bytes);
      p.totals = (u32*)((char*)extra + 3 * part_bytes);
      p.warp_before = p.totals + kInThreads;
      p.warp_kept = p.warp_before + kInThreads * kInWarps;
      p.c = ColRowParams{indptr, indices, num_cols, column_ids, S, sub_indptr, D, nullptr, G, encoding_size, table,
                         renumber ? 1 : 0, out_indptr, out_indices, out_select, data, e_ids, out_data, ctx_counters(ctx),
                         TileState{}, nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0}};
      p.sync = ctx_grid_sync(ctx, grid, 1);
      {
        ScopedKernelTimer timer(ctx, KID_ROW_FILTER, stream);
        void* args[] = {&p};
        st = launch_cooperative(ctx, stream, kernel, grid, kInThreads,
                                p.bloom.words ? ((size_t)1 << (32 - p.bloom.shift)) / 8 : 0, args, p.sync);
      }
      if (st != GSB_OK) return st;
      return finish_count(ctx, stream, p.c.mail, nnz_host);
    }
  }
  int st = col_row_table(ctx, stream, row_ids, R, row_ptr, G, encoding_size, &table);
  if (st != GSB_OK) return st;
  const int tiles = grid_for(D, kCrTile);
  TileState ts;
  st = ctx_tile_state(ctx, tiles, stream, &ts);
  if (st != GSB_OK) return st;
  ColRowParams p{indptr, indices, num_cols, column_ids, S, sub_indptr, D, col_ptr, G, encoding_size, table, renumber ? 1 : 0,
                 out_indptr, out_indices, out_select, data, e_ids, out_data, ctx_counters(ctx), ts,
                 nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0}};
  {
    ScopedKernelTimer timer(ctx, KID_ROW_FILTER, stream);
    k_col_row_filter<<<tiles, kRowThreads, 0, stream>>>(p);
  }
  GSB_LAUNCH_OK();
  return finish_count(ctx, stream, p.mail, nnz_host);
}

int gsb_index_search(gsb_ctx* ctx, void* stream_, const int64_t* origin, int64_t n, const int64_t* keys, int64_t m,
                     int64_t* out) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(n >= 0 && m >= 0 && (n == 0 || origin), GSB_ERR_INVALID_ARGUMENT);
  if (m == 0) return GSB_OK;
  GSB_REQUIRE(keys && out, GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  Table table;
  void* extra;
  int st = build_table(ctx, stream, origin, n, 0, &table, &extra);
  if (st != GSB_OK) return st;
  {
    ScopedKernelTimer timer(ctx, KID_OTHER, stream);
    k_index_search<<<min(grid_for(m, kRowThreads), kNumSMs * 8), kRowThreads, 0, stream>>>(keys, m, table, out);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // extern "C"
