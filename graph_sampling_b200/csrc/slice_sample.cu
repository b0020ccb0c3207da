// Column slicing and uniform per-column sampling (plain and fused with slicing).
//
// Data layout: the graph is CSC in HBM (int64 indptr[n+1], int64 indices[nnz]); a call works on a
// list of S seed columns.  Slicing is a counting pass (degrees and their scan by decoupled look-back)
// and a copy by OUTPUT position, a stretch of positions per warp (column_walk.cuh), so hub columns are
// spread over the grid.  Sampling is one launch: counts, their scan and the picks.  Fan-outs up to 16
// give each column a lane and each warp a tile of 32 columns; larger ones group columns into tiles of
// kTileCols per CTA, whose (start, degree, count) triples are staged in shared memory, and give each
// column a group of 32 lanes.  Either needs O(fanout) draws per column whatever its degree (Floyd's
// k-subset), instead of the reference's O(degree) reservoir pass (src/cuda/fusion/slice_sampling.cu:62-75).
#include "column_walk.cuh"
#include "uniform_sample.cuh"

namespace gsb {

constexpr int kThreads = 256;
constexpr int kTileCols = 128;  // columns per CTA of the lane-group sampler

// ---- count + scan only (one column per thread) -------------------------------------------------
// PER consecutive columns per thread: one when the call is small (every column wants a thread of its own, they are all in
// flight at once), four when it is large, where the number of tiles sets the length of the look-back chain.
template <int PER>
__global__ void __launch_bounds__(kThreads) k_count_scan(const i64* __restrict__ indptr, i64 num_cols,
                                                         const i64* __restrict__ seeds, i64 S, i64 k, int mode,
                                                         i64* __restrict__ out_indptr, i64* counters, TileState ts,
                                                         Mail mail) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  constexpr i64 kTile = kThreads * PER;
  const int tile = blockIdx.x;
  const i64 i = (i64)tile * kTile + (i64)threadIdx.x * PER;
  if ((i64)tile * kTile >= S && !(S == 0 && tile == 0)) return;
  i64 col[PER], begin[PER], f[PER], sum = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    col[q] = -1;
    if (i + q < S) {
      col[q] = seeds ? seeds[i + q] : i + q;
      if (!column_in_range(col[q], num_cols, counters, i + q)) col[q] = -1;
    }
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    begin[q] = col[q] >= 0 ? __ldg(indptr + col[q]) : 0;
    f[q] = col[q] >= 0 ? __ldg(indptr + col[q] + 1) : 0;
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    f[q] = column_count(f[q] - begin[q], k, mode);
    sum += f[q];
  }
  i64 total;
  i64 run = block_exclusive_scan<kThreads>(sum, s_scan, &total);
  if (threadIdx.x < 32) {
    bool lost;
    const i64 prefix = tile_exclusive_prefix(ts, tile, total, &lost);
    if (threadIdx.x == 0) s_base = lost ? -1 : prefix;
  }
  __syncthreads();
  i64 tile_base = s_base;
  if (tile_base < 0) {  // given up, and so is every tile behind it: no edges from here on
    tile_base = total = run = 0;
#pragma unroll
    for (int q = 0; q < PER; ++q) f[q] = 0;
  }
  run += tile_base;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (i + q < S) out_indptr[i + q] = run;
    run += f[q];
  }
  if ((i64)(tile + 1) * kTile >= S && threadIdx.x == 0) {
    out_indptr[S] = tile_base + total;
    counters[CNT_NNZ] = tile_base + total;
    mail_post(mail, 0, tile_base + total, counters);
  }
}

// ---- slice fill ---------------------------------------------------------------------------------
struct FillParams {
  const i64* indptr;
  const i64* indices;
  i64 num_cols;
  const i64* seeds;
  i64 S;
  const i64* out_indptr;
  i64* out_indices;
  i64* out_select;
  i64* out_coo_col;
  const float* data;
  const i64* e_ids;
  float* out_data;
  // super-batch form (src/cuda/slicing.cu:184-270): seeds of batch b are seeds[nid_ptr[b] .. nid_ptr[b+1]);
  // with encoding_size > 0 the row id of an edge of batch b is written as id + b * encoding_size
  const i64* nid_ptr;
  i64 G;
  i64 encoding_size;
  i64 D;  // edge total, or -1: it is read on the device
};

// The OUTPUT positions are cut into one stretch per warp, whatever columns they belong to: a hub column is spread over the
// grid, and a call with few, long columns fills it as well as one with many short ones.  A warp finds the columns of 192
// positions at a time (column_walk.cuh) and requests all their ids and data before it writes any.
// What bounds it is HBM and the positions in flight per SM against the registers they take (64 at 8 CTAs per SM; the forms with
// edge ids or batch numbers spill 4 to 36 bytes there):
// 262 144 columns with 13.2 M edges, weights and column ids: 92 us with six positions per lane and 8 CTAs per SM; eight
// positions and 8 / 7 / 9 / 10 CTAs 94 / 99 / 142 / 147, four and 10 CTAs 132.  Tiles of 1 024 positions whose columns a CTA
// keeps in shared memory, two barriers and two searches each: 105 us, and 16 instead of 5 us for the slices of layer-wise
// sampling, whose columns are mostly empty.
constexpr int kFillThreads = 128;
constexpr int kFillCtas = 8;
constexpr int kFillPer = 6;
constexpr int kFillStretch = 1024;

template <bool ENCODE, bool EIDS>
__global__ void __launch_bounds__(kFillThreads, kFillCtas) k_slice_fill(FillParams p) {
  const int lane = threadIdx.x & 31;
  const i64 D = p.D >= 0 ? p.D : __ldg(p.out_indptr + p.S);
  const i64 warps = (i64)gridDim.x * (kFillThreads / 32);
  const i64 per = ((D + warps - 1) / warps + 31) / 32 * 32;
  const i64 begin = ((i64)blockIdx.x * (kFillThreads / 32) + (threadIdx.x >> 5)) * per;
  if (begin >= D) return;
  ColumnWalk walk;
  walk.off = p.out_indptr;
  walk.seeds = p.seeds;
  walk.indptr = p.indptr;
  walk.S = p.S;
  walk.num_cols = p.num_cols;
  walk.counters = nullptr;  // the counting pass reported bad seeds; they have no positions
  walk.init(begin, (int)min(per, D - begin));
  for (int at = 0; at < walk.len; at += 32 * kFillPer) {
    i64 val[kFillPer];
    float x[kFillPer];
    i64 add[ENCODE ? kFillPer : 1];
    unsigned valid = 0;
#pragma unroll
    for (int r = 0; r < kFillPer; ++r) {
      if (at + r * 32 >= walk.len) break;  // uniform
      i64 column = 0;
      const i64 in = walk.locate<true>(at + r * 32, &column);
      if (in < 0) continue;
      valid |= 1u << r;
      const i64 pos = begin + at + r * 32 + lane;
      val[r] = __ldg(p.indices + in);
      if (EIDS) x[r] = __ldg(p.data + __ldg(p.e_ids + in));
      else if (p.out_data) x[r] = __ldg(p.data + in);
      if (p.out_select) p.out_select[pos] = in;
      if (p.out_coo_col) p.out_coo_col[pos] = column;
      if (ENCODE) add[r] = batch_of(p.nid_ptr, p.G, column) * p.encoding_size;
    }
#pragma unroll
    for (int r = 0; r < kFillPer; ++r) {
      if (!((valid >> r) & 1u)) continue;
      const i64 pos = begin + at + r * 32 + lane;
      p.out_indices[pos] = ENCODE ? val[r] + add[r] : val[r];
      if (EIDS || p.out_data) p.out_data[pos] = x[r];
    }
  }
}

// A grid that fills the chip; smaller when the edge total is known to be small, as a warp takes 32 positions at least, and
// larger when it is large, so that the hardware can balance stretches of 1 024 positions (2 048: 102, 512: 99 us for the slice
// above, where the search for a stretch's first column begins to show).
template <bool ENCODE>
static void launch_fill(FillParams p, i64 D, cudaStream_t stream) {
  p.D = D;
  const int full = kNumSMs * kFillCtas;
  const int grid = D >= 0 ? max(min(grid_for(D, kFillThreads), full), grid_for(D, kFillThreads / 32 * kFillStretch)) : full;
  if (p.out_data && p.e_ids) k_slice_fill<ENCODE, true><<<grid, kFillThreads, 0, stream>>>(p);
  else k_slice_fill<ENCODE, false><<<grid, kFillThreads, 0, stream>>>(p);
}

// ---- fused count + scan + uniform sampling -------------------------------------------------------
__device__ __forceinline__ void emit_pick(const SampleParams& p, i64 out_pos, i64 in_pos, i64 column_pos) {
  p.out_indices[out_pos] = __ldg(p.indices + in_pos);
  if (p.out_select) p.out_select[out_pos] = in_pos;
  if (p.out_coo_col) p.out_coo_col[out_pos] = column_pos;
  if (p.out_data) p.out_data[out_pos] = p.data[p.e_ids ? p.e_ids[in_pos] : in_pos];
}

template <int G>
__global__ void __launch_bounds__(kThreads) k_sample_uniform(SampleParams p) {
  __shared__ i64 s_in[kTileCols];
  __shared__ i64 s_deg[kTileCols];
  __shared__ i64 s_off[kTileCols];
  __shared__ u64 s_item[kTileCols];
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  const int tile = blockIdx.x;
  const int tid = threadIdx.x;
  const i64 S = p.S_dev ? min(p.S, __ldg(p.S_dev)) : p.S;
  const i64 base = (i64)tile * kTileCols;
  if (base >= S && !(S == 0 && tile == 0)) return;
  const int ncol = (int)max((i64)0, min((i64)kTileCols, S - base));
  const i64 k = p.k;

  i64 f = 0;
  if (tid < ncol) {
    const i64 col = p.seeds ? p.seeds[base + tid] : base + tid;
    i64 b = 0, d = 0;
    if (column_in_range(col, p.num_cols, p.counters, base + tid)) {
      b = p.indptr[col];
      d = p.indptr[col + 1] - b;
    }
    f = column_count(d, k, p.replace ? COUNT_WR : COUNT_WOR);
    s_in[tid] = b;
    s_deg[tid] = d;
    s_item[tid] = sample_item(p, base + tid, p.batch_ids ? batch_of(p.batch_ptr, p.G, base + tid) : 0);
  }
  i64 total;
  const i64 excl = block_exclusive_scan<kThreads>(f, s_scan, &total);
  if (tid < kTileCols) s_off[tid] = excl;
  if (tid < 32) {
    bool lost;
    const i64 prefix = tile_exclusive_prefix(p.ts, tile, total, &lost);
    if (tid == 0) s_base = lost ? -1 : prefix;
  }
  __syncthreads();
  const i64 tile_base = s_base;
  if (tile_base < 0) {  // given up, and so is every tile behind it: no edges from here on
    if (tid < ncol) p.out_indptr[base + tid] = 0;
    if (base + kTileCols >= S && tid == 0) {
      p.out_indptr[S] = p.counters[CNT_NNZ] = 0;
      mail_post(p.mail, 0, 0, p.counters);
    }
    return;
  }
  if (tid < ncol) p.out_indptr[base + tid] = tile_base + excl;
  if (base + kTileCols >= S && tid == 0) {
    p.out_indptr[S] = tile_base + total;
    p.counters[CNT_NNZ] = tile_base + total;
  }
  const bool overflow = tile_base + total > p.capacity;  // the prefix only grows: the last tile sees it if any tile does
  if (tid == 0) {
    if (overflow) raise_error(p.counters, GSB_ERR_CAPACITY, tile_base + total);
    if (base + kTileCols >= S) mail_post(p.mail, 0, tile_base + total, p.counters);
  }
  if (overflow) return;

  constexpr int kGroups = kThreads / G;
  const int lane = tid % G;
  const int grp = tid / G;
  const unsigned gmask = (G == 32) ? 0xffffffffu : (((1u << G) - 1u) << (((tid & 31) / G) * G));

  for (int c = grp; c < ncol; c += kGroups) {
    const i64 d = s_deg[c];
    const i64 b = s_in[c];
    const i64 o = tile_base + s_off[c];
    const i64 col_pos = base + c;
    const u64 item = s_item[c];
    if (p.replace) {
      if (d == 0) continue;
      for (i64 j = lane; j < k; j += G)
        emit_pick(p, o + j, b + (i64)rand_bounded(p.seed, item, (u64)j, STREAM_UNIFORM, (u64)d), col_pos);
    } else if (d <= k) {
      for (i64 j = lane; j < d; j += G) emit_pick(p, o + j, b + j, col_pos);
    } else if (k <= G) {
      // Floyd's k-subset inside the lane group: lane j draws t_j in [0, d-k+j]; the draws are
      // resolved in slot order (a repeated value is replaced by d-k+j).
      const i64 m = d - k + lane;
      i64 t = 0;
      if (lane < k) t = (i64)rand_bounded(p.seed, item, (u64)lane, STREAM_UNIFORM, (u64)(m + 1));
      i64 pick = -1;
      for (int j = 0; j < (int)k; ++j) {
        const i64 tj = __shfl_sync(gmask, t, j, G);
        const bool dup = (lane < j) && (pick == tj);
        const unsigned any = __ballot_sync(gmask, dup);
        if (lane == j) pick = any ? m : tj;
      }
      if (lane < k) emit_pick(p, o + lane, b + pick, col_pos);
    } else {
      // fanout > 32 (G == 32 here): same procedure with the chosen positions kept in the output
      // buffer; membership is checked by the whole warp.
      for (i64 j = 0; j < k; ++j) {
        const i64 m = d - k + j;
        const i64 tj = b + (i64)rand_bounded(p.seed, item, (u64)j, STREAM_UNIFORM, (u64)(m + 1));
        bool dup = false;
        for (i64 q = lane; q < j; q += G) dup |= (p.out_indices[o + q] == tj);
        const unsigned any = __ballot_sync(gmask, dup);
        if (lane == 0) p.out_indices[o + j] = any ? (b + m) : tj;
        __syncwarp(gmask);
      }
      for (i64 j = lane; j < k; j += G) emit_pick(p, o + j, p.out_indices[o + j], col_pos);
    }
  }
}


// ---- thread-per-column sampler for small fanouts --------------------------------------------------
// One lane owns one column: it draws all k picks itself (Floyd's k-subset in registers, one Philox block per four picks).  A
// warp is a tile of 32 columns: counts are scanned with shuffles and the tile prefix comes from the same look-back chain, so
// the kernel has no CTA-wide barrier at all.  The picks then change hands through shared memory: lane e % 32 reads and writes
// pick e of the tile, with k independent loads in flight.  The picks of a column are so asked for by neighbouring lanes at
// the same time: those in one line are one request, and lines that lie in one DRAM page arrive together, which DRAM serves
// faster than as many anywhere (with every lane reading its own column's picks one after the other, 600 000 columns out of
// 122 M edges, 5 / 10 / 15 picks 82 / 140 / 189 us, now 73 / 101 / 127; with data 117 / 211 / 299, now 108 / 156 / 197; 1 024
// columns out of caches 4.8 / 5.6 / 6.7, now 4.6 / 5.1 / 5.6: what a call of a few columns takes is the instructions that every
// SM has to read first).
constexpr int kTpcThreads = 128;
constexpr int kCountWindow = 256;  // buckets a CTA of the counting sampler keeps in shared memory

// COUNT: the kernel also counts, per bucket of the partitioned unique + relabel, the seeds and sampled ids of its
// columns — in shared memory, flushed with one global atomic per bucket and CTA — so that no pass over the items is
// needed for the counts.  A warp whose tile lies beyond the seeds then stays until the CTA's barriers are passed.
// DATA: edge data in edge order is wanted: its gathers go out with those of the ids, not after the wait for the prefix.
template <int KMAX, bool COUNT, bool DATA>
__global__ void __launch_bounds__(kTpcThreads) k_sample_uniform_tpc(SampleParams p) {
  __shared__ uint32_t s_cnt[COUNT ? kCountWindow : 1];
  __shared__ i64 s_win0;
  __shared__ i64 s_picks[kTpcThreads / 32][32 * KMAX];
  const int lane = threadIdx.x & 31;
  const i64 tile = (i64)blockIdx.x * (kTpcThreads / 32) + (threadIdx.x >> 5);
  const i64 S = p.S_dev ? min(p.S, __ldg(p.S_dev)) : p.S;
  if (COUNT) {
    const i64 first = (i64)blockIdx.x * kTpcThreads;  // first column of the CTA
    if (first >= S && !(S == 0 && blockIdx.x == 0)) return;  // the whole CTA
    for (int t = threadIdx.x; t < kCountWindow; t += kTpcThreads) s_cnt[t] = 0;
    if (threadIdx.x == 0) s_win0 = S > 0 ? __ldg(p.bucket_base + batch_of(p.batch_ptr, p.G, first)) : 0;
    __syncthreads();
    if (tile * 32 >= S && !(S == 0 && tile == 0)) {  // nothing to sample, but the CTA's flush below needs everybody
      __syncthreads();
      for (int t = threadIdx.x; t < kCountWindow; t += kTpcThreads)
        if (s_cnt[t] != 0) atomicAdd(p.bucket_count + s_win0 + t, s_cnt[t]);
      return;
    }
  } else if (tile * 32 >= S && !(S == 0 && tile == 0)) {
    return;
  }
  const i64 i = tile * 32 + lane;
  const bool valid = i < S;
  const int k = (int)p.k;
  i64 b = 0, d = 0, f = 0, col = 0;
  if (valid) {
    col = p.seeds ? __ldg(p.seeds + i) : i;
    if (column_in_range(col, p.num_cols, p.counters, i)) {
      b = __ldg(p.indptr + col);
      d = max(__ldg(p.indptr + col + 1) - b, (i64)0);
      if (d > 0xFFFFFFFFll) {  // positions inside a column are drawn from one 32-bit word
        raise_error(p.counters, GSB_ERR_UNSUPPORTED, i);
        d = 0;
      }
    }
    f = column_count(d, k, p.replace ? COUNT_WR : COUNT_WOR);
  }
  i64 inc = f;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const i64 t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  const i64 total = __shfl_sync(0xffffffffu, inc, 31);
  // The tile's count is published at once; its own prefix is resolved only after the picks are drawn and the gathers
  // issued, so the wait for the predecessors' counts overlaps the k random loads of every lane.
  tile_publish_aggregate(p.ts, (int)tile, total);
  const int n = (int)f;
  // minibatch of the warp's first column by one search; a lane beyond that minibatch's end searches for itself
  i64 bt = 0;
  if (p.batch_ptr && valid) {
    bt = batch_of(p.batch_ptr, p.G, tile * 32);
    if (i >= __ldg(p.batch_ptr + bt + 1)) bt = batch_of(p.batch_ptr, p.G, i);
  }
  // The picks in the order of the output, where they lie in `indices`: lane e % 32 reads pick e, so that the picks of a column are
  // read together and everything is written in whole lines.
  i64* s_where = s_picks[threadIdx.x >> 5];
  i64* s_own = s_where + (int)(inc - f);  // the lane's own picks
  const int have = (int)total;
  {
    uint32_t pick[KMAX];
    if (n > 0) draw_picks<KMAX>(p, i, bt, d, pick);
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      if (j < n) s_own[j] = b + pick[j];
  }
  __syncwarp();
  i64 val[KMAX];
  float x[DATA ? KMAX : 1];
#pragma unroll
  for (int r = 0; r < KMAX; ++r)
    if (r * 32 + lane < have) {
      const i64 w = s_where[r * 32 + lane];
      val[r] = __ldg(p.indices + w);
      if (DATA) x[r] = __ldg(p.data + w);
    }
  bool lost;
  const i64 prefix = __shfl_sync(0xffffffffu, tile_resolve_prefix(p.ts, (int)tile, total, &lost), 0);
  const i64 o = prefix + inc - f;
  if (valid) {
    p.out_indptr[i] = lost ? 0 : o;  // given up, and so is every tile behind it: no edges from here on
    if (i == S - 1) {
      p.out_indptr[S] = lost ? 0 : o + f;
      p.counters[CNT_NNZ] = lost ? 0 : o + f;
    }
  } else if (S == 0 && lane == 0) {
    p.out_indptr[0] = 0;
    p.counters[CNT_NNZ] = 0;
  }
  const bool overflow = lost || prefix + total > p.capacity;  // the prefix only grows: the last tile sees it if any tile does
  if (lane == 0) {
    if (overflow) raise_error(p.counters, GSB_ERR_CAPACITY, prefix + total);  // (behind the error of a wait that was given up)
    if (tile * 32 + 32 >= S) mail_post(p.mail, 0, prefix + total, p.counters);
  }
  if (overflow && !COUNT) return;
  if (!overflow) {
    // one array after the other, each behind one test
#pragma unroll
    for (int r = 0; r < KMAX; ++r)
      if (r * 32 + lane < have) p.out_indices[prefix + r * 32 + lane] = val[r];
    if (DATA) {
#pragma unroll
      for (int r = 0; r < KMAX; ++r)
        if (r * 32 + lane < have) p.out_data[prefix + r * 32 + lane] = x[r];
    } else if (p.out_data) {
      float y[KMAX];
#pragma unroll
      for (int r = 0; r < KMAX; ++r)
        if (r * 32 + lane < have) y[r] = __ldg(p.data + __ldg(p.e_ids + s_where[r * 32 + lane]));
#pragma unroll
      for (int r = 0; r < KMAX; ++r)
        if (r * 32 + lane < have) p.out_data[prefix + r * 32 + lane] = y[r];
    }
    if (p.out_select) {
#pragma unroll
      for (int r = 0; r < KMAX; ++r)
        if (r * 32 + lane < have) p.out_select[prefix + r * 32 + lane] = s_where[r * 32 + lane];
    }
    if (!COUNT && p.out_coo_col) {
      __syncwarp();
      for (int j = 0; j < n; ++j) s_own[j] = i;
      __syncwarp();
      for (int e = lane; e < have; e += 32) p.out_coo_col[prefix + e] = s_where[e];
    }
  }
  if (COUNT) {
    // a call whose device-side sizes exceed the caller's bounds was flagged by the layout kernel: its bucket layout
    // may not fit the count array, so nothing is counted (the passes that would use the counts return at once).  A look-back that is
    // given up elsewhere sets the flag at any time: the warp decides as one, what follows needs all its lanes.
    if (__all_sync(0xffffffffu, !overflow && p.counters[CNT_ABORT] == 0)) {
      const i64 b0 = valid ? __ldg(p.bucket_base + bt) : 0;
      const int win = (int)(b0 - s_win0);  // >= 0: minibatches follow the CTA's first one
      const uint32_t parts = valid ? (uint32_t)(__ldg(p.bucket_base + bt + 1) - b0) : 0;
      auto count_id = [&](i64 id, int first, uint32_t buckets) {
        if (id < 0 || id >= 0xFFFFFFFFll) return;  // never bucketed; reported by the pass that scatters the items
        const int w = first + (int)bucket_of_id((uint32_t)id, buckets, p.bucket_magic);
        if (w < kCountWindow) atomicAdd(&s_cnt[w], 1u);
        else atomicAdd(p.bucket_count + s_win0 + w, 1u);
      };
      if (valid) count_id(col, win, parts);
      const int win_first = __shfl_sync(0xffffffffu, win, 0);
      const uint32_t parts_first = __shfl_sync(0xffffffffu, parts, 0);
      if (__all_sync(0xffffffffu, !valid || win == win_first)) {
#pragma unroll
        for (int r = 0; r < KMAX; ++r)
          if (r * 32 + lane < have) count_id(val[r], win_first, parts_first);
      } else {  // several minibatches: every lane counts its own column's picks
        for (int j = 0; j < n; ++j) count_id(__ldg(p.indices + s_own[j]), win, parts);
      }
    }
    __syncthreads();
    for (int t = threadIdx.x; t < kCountWindow; t += kTpcThreads)
      if (s_cnt[t] != 0) atomicAdd(p.bucket_count + s_win0 + t, s_cnt[t]);
  }
}

__global__ void __launch_bounds__(kThreads) k_sample_one_keepdim(const i64* __restrict__ indptr,
                                                                 const i64* __restrict__ indices, i64 num_cols,
                                                                 const i64* __restrict__ seeds, i64 S, u64 seed,
                                                                 i64* counters,
                                                                 i64* __restrict__ out_indptr,
                                                                 i64* __restrict__ out_indices,
                                                                 i64* __restrict__ out_select) {
  const i64 i = (i64)blockIdx.x * kThreads + threadIdx.x;
  if (i > S) return;
  out_indptr[i] = i;
  if (i == S) return;
  const i64 col = seeds[i];
  // -1 is what this operator itself emits for an isolated seed, so a walk may feed it back: it stays -1 silently
  const bool ok = col == -1 ? false : column_in_range(col, num_cols, counters, i);
  const i64 b = ok ? indptr[col] : 0;
  const i64 d = ok ? indptr[col + 1] - b : 0;
  if (d == 0) {
    out_indices[i] = -1;
    out_select[i] = -1;
  } else {
    const i64 pos = b + (i64)rand_bounded(seed, (u64)i, 0, STREAM_UNIFORM, (u64)d);
    out_indices[i] = indices[pos];
    out_select[i] = pos;
  }
}

// Offsets of a per-column sample (min(degree, k) without replacement, k per non-empty column with) or of the plain
// slice (mode 0) by the counting kernel alone; the total lands in the context's counters.
int count_scan_launch(gsb_ctx* ctx, cudaStream_t stream, const i64* indptr, i64 num_cols, const i64* seeds, i64 S, i64 k,
                      int mode, i64* out_indptr, Mail mail) {
  const bool large = S >= 4ll * kThreads * kNumSMs;  // a full wave of CTAs at four columns per thread
  const int grid = grid_for(S, large ? 4 * kThreads : kThreads);
  TileState ts;
  int st = ctx_tile_state(ctx, grid, stream, &ts);
  if (st != GSB_OK) return st;
  {
    ScopedKernelTimer timer(ctx, KID_COUNT_SCAN, stream);
    if (large)
      k_count_scan<4><<<grid, kThreads, 0, stream>>>(indptr, num_cols, seeds, S, k, mode, out_indptr, ctx_counters(ctx), ts,
                                                     mail);
    else
      k_count_scan<1><<<grid, kThreads, 0, stream>>>(indptr, num_cols, seeds, S, k, mode, out_indptr, ctx_counters(ctx), ts,
                                                     mail);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

template <int G>
static void launch_sample(const SampleParams& p, int grid, cudaStream_t stream) {
  k_sample_uniform<G><<<grid, kThreads, 0, stream>>>(p);
}

// Data in edge order is gathered with the ids: 40 000 columns of ten picks out of 12 M edges 28.4 -> 24.0 us, 600 000 of fifteen
// 130 -> 112, and out of 122 M, where DRAM is the bound, the same (two million columns of five 304 -> 306).
template <int KMAX>
static void launch_tpc(const SampleParams& p, int grid, cudaStream_t stream) {
  if (p.bucket_count) k_sample_uniform_tpc<KMAX, true, false><<<grid, kTpcThreads, 0, stream>>>(p);
  else if (p.out_data && !p.e_ids) k_sample_uniform_tpc<KMAX, false, true><<<grid, kTpcThreads, 0, stream>>>(p);
  else k_sample_uniform_tpc<KMAX, false, false><<<grid, kTpcThreads, 0, stream>>>(p);
}

int sample_uniform_launch(gsb_ctx* ctx, cudaStream_t stream, const i64* indptr, const i64* indices, i64 num_cols,
                          const i64* seeds, i64 S, i64 k, int replace, u64 seed, i64* out_indptr, i64* out_indices,
                          i64* out_select, i64* out_coo_col, const float* data, const i64* e_ids, float* out_data,
                          i64 capacity, const i64* S_dev, const i64* batch_ptr, const i64* batch_ids, i64 G,
                          const SamplerCount* count, Mail mail, i64 num_edges) {
  const bool per_thread = k <= 16;  // small fanouts: one lane per column, one warp per tile of 32 columns
  const int grid = per_thread ? grid_for(S, kTpcThreads) : grid_for(S, kTileCols);
  TileState ts;
  int st = ctx_tile_state(ctx, per_thread ? (S + 31) / 32 + 1 : grid, stream, &ts);
  if (st != GSB_OK) return st;
  SampleParams p{indptr,     indices,     num_cols, seeds, S,        k,        replace, 0,        seed, out_indptr,
                 out_indices, out_select, out_coo_col, data, e_ids, out_data, capacity, ctx_counters(ctx), ts,
                 S_dev,      batch_ptr,  batch_ptr ? batch_ids : nullptr,
                 batch_ptr ? G : 0,      nullptr,    nullptr, mail};
  if (count && count->bucket_count) {
    if (!per_thread || !batch_ptr || G < 1) return GSB_ERR_INVALID_ARGUMENT;
    p.bucket_count = count->bucket_count;
    p.bucket_base = count->bucket_base;
    p.bucket_magic = count->magic;
  }
  if (out_select && !out_coo_col && !out_data && window_sample_suits(ctx, S, k, num_edges)) {
    void* ws = count ? count->scratch : nullptr;
    if (!ws && !ctx_try_workspace(ctx, stream, window_sample_bytes(ctx, S, k, num_edges), 0, &ws)) ws = nullptr;
    if (ws) return window_sample_launch(ctx, stream, p, num_edges, ws);
  }
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_UNIFORM, stream);
    // the register count follows the unrolled pick array (64 / 64 / 72 / 80 / 94 registers, with data up to 126); the usual fan-outs 5 and
    // 10 get instantiations of their own.  A large call runs at the rate at which DRAM serves random 64-byte accesses, not at
    // the limit of its resident lanes: gathers through ld.global.nc.L2::64B (with or without L1::no_allocate) instead of
    // __ldg, to keep the L2 from fetching more than one 64-byte line per gather, changed nothing.
    if (k <= 4) launch_tpc<4>(p, grid, stream);
    else if (k <= 5) launch_tpc<5>(p, grid, stream);
    else if (k <= 8) launch_tpc<8>(p, grid, stream);
    else if (k <= 10) launch_tpc<10>(p, grid, stream);
    else if (k <= 16) launch_tpc<16>(p, grid, stream);
    else launch_sample<32>(p, grid, stream);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // namespace gsb

using namespace gsb;

extern "C" {

int gsb_col_slice_count(gsb_ctx* ctx, void* stream_, const int64_t* indptr, int64_t num_cols, const int64_t* seeds,
                        int64_t S, int64_t* out_indptr, int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && S >= 0 && num_cols >= 0 && (seeds || S <= num_cols), GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  const Mail mail = nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0};
  int st = count_scan_launch(ctx, stream, indptr, num_cols, seeds, S, 0, COUNT_DEGREE, out_indptr, mail);
  if (st != GSB_OK || !nnz_host) return st;
  i64 total = 0;
  st = ctx_mail_result(ctx, stream, mail, 1, &total);
  *nnz_host = total;
  return st;
}

int gsb_col_slice_fill(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices, int64_t num_cols,
                       const int64_t* seeds, int64_t S, const int64_t* out_indptr, int64_t D, int64_t* out_indices,
                       int64_t* out_select, int64_t* out_coo_col, const float* data, const int64_t* e_ids,
                       float* out_data) {
  // out_indices may be null only when the slice is empty (nothing is written then)
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && S >= 0 && num_cols >= 0 && (seeds || S <= num_cols), GSB_ERR_INVALID_ARGUMENT);
  if (S == 0 || D == 0) return GSB_OK;
  GSB_REQUIRE(indices && out_indices, GSB_ERR_INVALID_ARGUMENT);
  FillParams p{indptr, indices, num_cols, seeds, S, out_indptr, out_indices, out_select, out_coo_col, data, e_ids,
               out_data, nullptr, 0, 0, D};
  {
    ScopedKernelTimer timer(ctx, KID_SLICE_FILL, (cudaStream_t)stream_);
    launch_fill<false>(p, D, (cudaStream_t)stream_);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int gsb_batch_col_slice_fill(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices,
                             int64_t num_cols, const int64_t* seeds, int64_t S, const int64_t* nid_ptr, int64_t G,
                             int64_t encoding_size, const int64_t* out_indptr, int64_t* out_indices,
                             int64_t* out_select, int64_t* out_coo_col, int64_t* out_coo_offsets, const float* data,
                             const int64_t* e_ids, float* out_data) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && nid_ptr && S >= 0 && G >= 1 && encoding_size >= 0 && num_cols >= 0 &&
                  (seeds || S <= num_cols),
              GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  if (out_coo_offsets) {
    int st = gsb_batch_edge_offsets(ctx, stream_, out_indptr, nid_ptr, G, out_coo_offsets);
    if (st != GSB_OK) return st;
  }
  if (S == 0) return GSB_OK;
  FillParams p{indptr, indices, num_cols, seeds, S, out_indptr, out_indices, out_select, out_coo_col, data, e_ids,
               out_data, nid_ptr, G, encoding_size, -1};
  {
    ScopedKernelTimer timer(ctx, KID_SLICE_FILL, stream);
    if (encoding_size > 0) launch_fill<true>(p, -1, stream);
    else launch_fill<false>(p, -1, stream);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int gsb_sample_uniform_sized(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices, int64_t num_cols,
                             int64_t num_edges, const int64_t* seeds, int64_t S, int64_t k, int replace, uint64_t seed,
                             int64_t* out_indptr, int64_t* out_indices, int64_t* out_select, int64_t* out_coo_col,
                             const float* data, const int64_t* e_ids, float* out_data, int64_t capacity,
                             int64_t* nnz_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && S >= 0 && k >= 0 && num_cols >= 0 && (seeds || S <= num_cols),
              GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(out_indices || capacity == 0, GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  const Mail mail = nnz_host ? ctx_mail(ctx) : Mail{nullptr, 0};
  int st = sample_uniform_launch(ctx, stream, indptr, indices, num_cols, seeds, S, k, replace, (u64)seed, out_indptr,
                                 out_indices, out_select, out_coo_col, data, e_ids, out_data, capacity, nullptr, nullptr,
                                 nullptr, 0, nullptr, mail, num_edges);
  if (st != GSB_OK || !nnz_host) return st;
  i64 total = 0;
  st = ctx_mail_result(ctx, stream, mail, 1, &total);
  *nnz_host = total;
  return st;
}

int gsb_sample_uniform(gsb_ctx* ctx, void* stream, const int64_t* indptr, const int64_t* indices, int64_t num_cols,
                       const int64_t* seeds, int64_t S, int64_t k, int replace, uint64_t seed, int64_t* out_indptr,
                       int64_t* out_indices, int64_t* out_select, int64_t* out_coo_col, const float* data,
                       const int64_t* e_ids, float* out_data, int64_t capacity, int64_t* nnz_host) {
  return gsb_sample_uniform_sized(ctx, stream, indptr, indices, num_cols, 0, seeds, S, k, replace, seed, out_indptr,
                                  out_indices, out_select, out_coo_col, data, e_ids, out_data, capacity, nnz_host);
}

int gsb_sample_one_keepdim(gsb_ctx* ctx, void* stream_, const int64_t* indptr, const int64_t* indices,
                           int64_t num_cols, const int64_t* seeds, int64_t S, uint64_t seed, int64_t* out_indptr,
                           int64_t* out_indices, int64_t* out_select) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && out_indptr && S >= 0 && num_cols >= 0 && (S == 0 || seeds), GSB_ERR_INVALID_ARGUMENT);
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_KEEPDIM, (cudaStream_t)stream_);
    k_sample_one_keepdim<<<grid_for(S + 1, kThreads), kThreads, 0, (cudaStream_t)stream_>>>(
        indptr, indices, num_cols, seeds, S, (u64)seed, ctx_counters(ctx), out_indptr, out_indices, out_select);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // extern "C"
