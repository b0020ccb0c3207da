// Uniform sampling of many columns out of a graph that is larger than L2: every stretch of the edges is read while it is there.
//
// The last hops of a super-batch visit the columns of a graph tens of times, in an order that has nothing to do with where they
// lie, and the thread-per-column sampler (slice_sample.cu) fetches a 64-byte line from DRAM for nearly every pick, which DRAM
// serves at 50 to 75 G/s.  The edges are therefore cut into WINDOWS of 64 MB, and three passes take the place of one:
//
//   draw   tiles of 512 columns in the order of the call: counts, their scan (look-back), the picks and their positions
//          (out_select); the positions also leave, as 32-bit words, for the tile's own stretch of scratch, sorted by window;
//   read   window after window, all tiles: position -> id, in place.  The reads of a window come out of L2 but for the first
//          one of a line;
//   emit   a tile's words come back into the order of the call and leave as 64-bit ids.
//
// A tile's stretch is its own, so nothing has to be counted across tiles; every pick costs 8 more bytes written and 8 more read,
// in whole lines.  67 M columns of 5 picks and 8.2 M of 10 out of 124 M edges (the last hops of 500 minibatches), ms: one pass 6.30
// and 1.63 (with the counts of buckets), draw 1.41 and 0.31 (instruction issue, barriers), read 1.25 and 0.33 (random reads at
// 264 G/s), emit 0.92 and 0.31 (5.2 TB/s of real traffic), 1.32 with the counts of the larger one.
// Tiles of 1 024 columns: read 1.22, draw 1.57, emit 1.04; of 512 with windows of 32 / 128 MB: read 1.35 / 2.17.  The emit pass spills a
// few words at its eight CTAs an SM (64 bytes stored, 56 loaded a thread); with seven a call of 60 M columns takes the
// same 3.21 ms, with six 3.26.
#include "uniform_sample.cuh"

namespace gsb {

constexpr int kWinThreads = 256;
constexpr int kWinPer = 2;  // columns per thread
constexpr int kWinTile = kWinThreads * kWinPer;
constexpr int kWinWarps = kWinThreads / 32;
constexpr int kMaxWindows = 64;
constexpr int kWindowShift = 23;
constexpr uint32_t kUnstaged = 0xFFFFFFFFu;  // an id that 32 bits don't hold: read again where its position is known
constexpr int kReadThreads = 256;
constexpr int kReadAhead = 6;

struct WindowParams {
  SampleParams p;
  uint32_t* staged;  // [tiles][kWinTile * k] positions, then ids, of a tile's picks by window
  uint16_t* place;   // [tiles][kWinTile] where a column's picks are in there
  uint16_t* start;   // [windows + 2][tiles] first word of a window in a tile, the tile's total, whether it was given up
  i64 tiles;         // bound that the rows of `start` are laid out for
  uint32_t windows;
  int shift;         // log2 of a window's edges
};

__device__ __forceinline__ i64 seed_count(const SampleParams& p) { return p.S_dev ? min(p.S, __ldg(p.S_dev)) : p.S; }

template <int KMAX>
__global__ void __launch_bounds__(kWinThreads, KMAX > 5 ? 4 : 6) k_window_draw(WindowParams w) {
  extern __shared__ uint4 s_raw[];
  __shared__ uint32_t s_count[kMaxWindows], s_start[kMaxWindows], s_warp[kWinWarps];
  __shared__ i64 s_base;
  const SampleParams& p = w.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const i64 tile = blockIdx.x, S = seed_count(p), base = tile * kWinTile;
  if (base >= S && !(S == 0 && tile == 0)) return;
  const int k = (int)p.k;
  uint32_t* s_call = reinterpret_cast<uint32_t*>(s_raw);  // positions of the picks in the order of the call
  uint32_t* s_sorted = s_call + kWinTile * k;             // and by window
  if (threadIdx.x < kMaxWindows) s_count[threadIdx.x] = 0;
  const i64 first = base + warp * (32 * kWinPer) + lane;  // a warp's columns are neighbours
  i64 col[kWinPer];
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    const i64 i = first + q * 32;
    col[q] = i < S ? (p.seeds ? __ldg(p.seeds + i) : i) : 0;
  }
  uint32_t b[kWinPer], d[kWinPer];  // fewer than 2^32 edges
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    const i64 i = first + q * 32;
    b[q] = d[q] = 0;
    if (i < S && column_in_range(col[q], p.num_cols, p.counters, i)) {
      const i64 begin = __ldg(p.indptr + col[q]), degree = __ldg(p.indptr + col[q] + 1) - begin;
      if (degree > 0xFFFFFFFFll) raise_error(p.counters, GSB_ERR_UNSUPPORTED, i);
      else if (degree > 0) b[q] = (uint32_t)begin, d[q] = (uint32_t)degree;
    }
  }
  uint32_t n[kWinPer], inc[kWinPer], window[kWinPer], run = 0;
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    n[q] = (uint32_t)column_count(d[q], k, p.replace ? COUNT_WR : COUNT_WOR);
    window[q] = min(b[q] >> w.shift, w.windows - 1);
    inc[q] = n[q];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, inc[q], o);
      if (lane >= o) inc[q] += t;
    }
    inc[q] += run;
    run = __shfl_sync(0xffffffffu, inc[q], 31);
  }
  if (lane == 31) s_warp[warp] = run;
  __syncthreads();
  uint32_t at[kWinPer];  // inside the window's words
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) at[q] = n[q] > 0 ? atomicAdd(&s_count[window[q]], n[q]) : 0;
  uint32_t before, total;
  {
    const uint32_t t = lane < kWinWarps ? s_warp[lane] : 0;
    before = __reduce_add_sync(0xffffffffu, lane < warp ? t : 0u);
    total = __reduce_add_sync(0xffffffffu, t);
  }
  if (warp == 0) tile_publish_aggregate(p.ts, (int)tile, total);
  __syncthreads();
  if (warp == 1) {  // starts of the windows
    uint32_t c[kMaxWindows / 32], sum = 0;
#pragma unroll
    for (int q = 0; q < kMaxWindows / 32; ++q) sum += c[q] = s_count[lane * (kMaxWindows / 32) + q];
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    x -= sum;
#pragma unroll
    for (int q = 0; q < kMaxWindows / 32; ++q) {
      s_start[lane * (kMaxWindows / 32) + q] = x;
      x += c[q];
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    const i64 i = first + q * 32;
    i64 bt = 0;
    if (p.batch_ids && i < S) {
      bt = batch_of(p.batch_ptr, p.G, base + warp * (32 * kWinPer) + q * 32);
      if (i >= __ldg(p.batch_ptr + bt + 1)) bt = batch_of(p.batch_ptr, p.G, i);
    }
    inc[q] += before - n[q];
    if (n[q] == 0) continue;
    at[q] += s_start[window[q]];
    uint32_t pick[KMAX];
    draw_picks<KMAX>(p, i, bt, d[q], pick);
#pragma unroll
    for (int j = 0; j < KMAX; ++j)
      if (j < n[q]) s_call[inc[q] + j] = s_sorted[at[q] + j] = b[q] + pick[j];
  }
  if (warp == 0) {
    bool lost;
    const i64 prefix = tile_resolve_prefix(p.ts, (int)tile, total, &lost);
    if (lane == 0) {
      // given up, and so is every tile behind it: no edges from here on.  The prefix only grows: the last tile sees it if any
      // tile is beyond the capacity.
      const bool overflow = lost || prefix + total > p.capacity;
      if (overflow) raise_error(p.counters, GSB_ERR_CAPACITY, prefix + total);
      if (base + kWinTile >= S) {
        p.out_indptr[S] = lost ? 0 : prefix + total;
        p.counters[CNT_NNZ] = lost ? 0 : prefix + total;
        mail_post(p.mail, 0, prefix + total, p.counters);
      }
      s_base = lost ? -2 : overflow ? -3 - prefix : prefix;
    }
  }
  __syncthreads();
  const bool lost = s_base == -2, given_up = s_base < 0;
  const i64 prefix = lost ? 0 : given_up ? -3 - s_base : s_base;
#pragma unroll
  for (int q = 0; q < kWinPer; ++q)
    if (first + q * 32 < S) {
      p.out_indptr[first + q * 32] = lost ? 0 : prefix + inc[q];
      w.place[first + q * 32] = (uint16_t)at[q];
    }
  for (uint32_t t = threadIdx.x; t < w.windows + 2; t += kWinThreads)
    w.start[(i64)t * w.tiles + tile] =
        (uint16_t)(t > w.windows ? (given_up ? 1u : 0u) : given_up ? 0u : t < w.windows ? s_start[t] : total);
  if (given_up) return;
  uint4* out = reinterpret_cast<uint4*>(w.staged + tile * (i64)(kWinTile * k));
  const uint4* sorted = reinterpret_cast<const uint4*>(s_sorted);
  for (uint32_t e = threadIdx.x; e < (total + 3) / 4; e += kWinThreads) out[e] = sorted[e];
  for (uint32_t e = threadIdx.x; e < total; e += kWinThreads) p.out_select[prefix + e] = (i64)s_call[e];
}

// A warp per tile and window.
__global__ void __launch_bounds__(kReadThreads) k_window_read(WindowParams w) {
  const SampleParams& p = w.p;
  const int lane = threadIdx.x & 31;
  const i64 tile = (i64)blockIdx.x * (kReadThreads / 32) + (threadIdx.x >> 5);
  if (tile * kWinTile >= seed_count(p)) return;
  const uint16_t* row = w.start + (i64)blockIdx.y * w.tiles + tile;
  const uint32_t begin = __ldg(row), end = __ldg(row + w.tiles);
  uint32_t* words = w.staged + tile * (i64)(kWinTile * (int)p.k);
  for (uint32_t at = begin + lane; at < end; at += 32 * kReadAhead) {
    uint32_t word[kReadAhead];
    i64 id[kReadAhead];
#pragma unroll
    for (int r = 0; r < kReadAhead; ++r) word[r] = at + r * 32 < end ? words[at + r * 32] : 0;
#pragma unroll
    for (int r = 0; r < kReadAhead; ++r)
      if (at + r * 32 < end) id[r] = __ldg(p.indices + word[r]);
#pragma unroll
    for (int r = 0; r < kReadAhead; ++r)
      if (at + r * 32 < end) words[at + r * 32] = (u64)id[r] < kUnstaged ? (uint32_t)id[r] : kUnstaged;
  }
}

// COUNT: as in k_sample_uniform_tpc, the seeds and ids of the columns are counted per bucket of the pass that follows.
constexpr int kWinCountWindow = 512;

template <bool COUNT>
__global__ void __launch_bounds__(kWinThreads, COUNT ? 6 : 8) k_window_emit(WindowParams w) {
  extern __shared__ uint4 s_raw[];
  __shared__ uint32_t s_cnt[COUNT ? kWinCountWindow : 1];
  __shared__ i64 s_win0, s_next;  // of the minibatch that the tile begins in: its first bucket, its end,
  __shared__ uint32_t s_parts;    // its buckets
  const SampleParams& p = w.p;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const i64 tile = blockIdx.x, S = seed_count(p), base = tile * kWinTile;
  if (base >= S) return;
  const int k = (int)p.k;
  const uint32_t* s_sorted = reinterpret_cast<const uint32_t*>(s_raw);
  uint32_t* s_call = reinterpret_cast<uint32_t*>(s_raw) + kWinTile * k;
  const uint32_t total = __ldg(w.start + (i64)w.windows * w.tiles + tile);
  const uint4* in = reinterpret_cast<const uint4*>(w.staged + tile * (i64)(kWinTile * k));
  const i64 first = base + warp * (32 * kWinPer) + lane;
  const i64 prefix = __ldg(p.out_indptr + base);
  uint32_t from[kWinPer], at[kWinPer], n[kWinPer];
  i64 col[kWinPer];
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    const i64 i = first + q * 32;
    from[q] = at[q] = n[q] = 0;
    if (i < S && total > 0) {
      from[q] = __ldg(w.place + i);
      at[q] = (uint32_t)(__ldg(p.out_indptr + i) - prefix);
      n[q] = (i + 1 < min(S, base + kWinTile) ? (uint32_t)(__ldg(p.out_indptr + i + 1) - prefix) : total) - at[q];
    }
    if (COUNT) col[q] = i < S ? (p.seeds ? __ldg(p.seeds + i) : i) : -1;
  }
  for (uint32_t e = threadIdx.x; e < (total + 3) / 4; e += kWinThreads) s_raw[e] = __ldg(in + e);
  if (COUNT) {
    for (int t = threadIdx.x; t < kWinCountWindow; t += kWinThreads) s_cnt[t] = 0;
    if (threadIdx.x == 0) {
      const i64 bt = batch_of(p.batch_ptr, p.G, base);
      s_next = __ldg(p.batch_ptr + bt + 1);
      s_win0 = __ldg(p.bucket_base + bt);
      s_parts = (uint32_t)(__ldg(p.bucket_base + bt + 1) - s_win0);
    }
  }
  __syncthreads();
  // nothing is counted in a call whose sizes exceed the caller's bounds (CNT_ABORT), or that gave up or ran out of room
  const bool counts = COUNT && p.counters[CNT_ABORT] == 0 && __ldg(w.start + (i64)(w.windows + 1) * w.tiles + tile) == 0;
#pragma unroll
  for (int q = 0; q < kWinPer; ++q) {
    const i64 i = first + q * 32;
    if (i >= S) continue;
    if (!counts) {
      for (uint32_t j = 0; j < n[q]; ++j) s_call[at[q] + j] = s_sorted[from[q] + j];
      continue;
    }
    uint32_t parts = s_parts;
    i64 win = 0;
    if (i >= s_next) {
      const i64 bt = batch_of(p.batch_ptr, p.G, i), b0 = __ldg(p.bucket_base + bt);
      parts = (uint32_t)(__ldg(p.bucket_base + bt + 1) - b0);
      win = b0 - s_win0;
    }
    auto count_id = [&](uint32_t v) {
      const i64 t = win + bucket_of_id(v, parts, p.bucket_magic);
      if (t < kWinCountWindow) atomicAdd(&s_cnt[t], 1u);
      else atomicAdd(p.bucket_count + s_win0 + t, 1u);
    };
    // ids beyond 32 bits are never bucketed; the pass that scatters the items reports them
    if ((u64)col[q] < kUnstaged) count_id((uint32_t)col[q]);
    for (uint32_t j = 0; j < n[q]; ++j) {
      const uint32_t v = s_sorted[from[q] + j];
      s_call[at[q] + j] = v;
      if (v != kUnstaged) count_id(v);
    }
  }
  __syncthreads();
  for (uint32_t e = threadIdx.x; e < total; e += kWinThreads) {
    const uint32_t v = s_call[e];
    p.out_indices[prefix + e] = v != kUnstaged ? (i64)v : __ldg(p.indices + p.out_select[prefix + e]);
  }
  if (COUNT)
    for (int t = threadIdx.x; t < kWinCountWindow; t += kWinThreads)
      if (s_cnt[t] != 0) atomicAdd(p.bucket_count + s_win0 + t, s_cnt[t]);
}

// ---- host ---------------------------------------------------------------------------------------------------------------
static i64 window_tiles(i64 S) { return grid_for(S, kWinTile); }

// log2 of a window's edges: 64 MB of them, or as few as 64 windows allow.
static int window_shift(gsb_ctx* ctx, i64 num_edges) {
  if (ctx_option(ctx, GSB_OPT_SAMPLE_PATH) != 2) return kWindowShift;
  int shift = 0;
  while (((num_edges - 1) >> shift) >= kMaxWindows) ++shift;
  return shift;
}
static i64 window_count(gsb_ctx* ctx, i64 num_edges) { return ((num_edges - 1) >> window_shift(ctx, num_edges)) + 1; }

// Windows / one pass, time of a call, the columns being the frontiers of 500 minibatches of 1 024 seeds after a hop of 15 (3 M columns
// out of an R-MAT graph with 50 edges a column | 6 M, power-law degrees, 24 edges | 7 M, 50 edges), by edges and picks a column:
//             2 picks         5 picks         6 picks         8 picks         10 picks        12 picks        15 picks        16 picks
//   17 M      0.90|0.87|0.86  0.96|0.96|0.94  0.99|1.07|1.05  1.05|1.19|1.27  0.96|1.15|1.10  0.99|1.16|1.18  1.03|1.26|1.17  1.14|1.32|1.34
//   20 M      0.94|0.91|0.90  0.95|0.97|0.94  0.97|1.08|1.03  1.03|1.18|1.24  0.92|1.13|1.06  0.95|1.16|1.12  0.98|1.24|1.14  1.11|1.32|1.32
//   25 M      1.01|0.96|0.96  0.93|0.98|0.93  0.95|1.08|1.02  0.98|1.18|1.21  0.87|1.10|1.01  0.89|1.15|1.08  0.91|1.22|1.09  1.06|1.31|1.31
//   31 M      1.10|1.04|1.04  0.92|1.00|0.94  0.94|1.10|1.02  0.95|1.17|1.18  0.84|1.09|0.97  0.85|1.13|1.08  0.86|1.18|1.06  1.01|1.29|1.28
//   40 M      0.97|0.91|0.91  0.83|0.88|0.81  0.86|0.98|0.90  0.86|1.06|1.07  0.77|1.01|0.91  0.80|1.08|1.01  0.81|1.13|1.00  0.97|1.24|1.24
//   60 M      1.09|1.03|1.02  0.85|0.92|0.85  0.87|1.00|0.91  0.86|1.07|1.04  0.76|1.00|0.88  0.79|1.10|1.01  0.77|1.10|0.96  0.92|1.21|1.20
//   124 M     1.11|1.05|0.95  0.88|0.92|0.78  0.90|0.99|0.84  0.88|1.03|0.97  0.78|0.98|0.82  0.82|1.09|0.95  0.77|1.06|0.90  0.90|1.18|1.16
// 250 and 100 minibatches (half and a fifth of the columns) at 124 M edges: 5 picks 1.02|1.01|0.92 and -|1.16|1.10, 10 picks 0.94|1.06|0.92
// and 1.18|1.27|1.12; 10 picks at 31 M 0.89|1.14|1.02 and 1.08|1.25|1.08.
// What windows save depends on how often a window's lines are met, which the rule has the picks for, and on how the columns lie, which
// it doesn't know: it stands where the two kinds of graphs lose about the same (2 % on average of the better form, up to 1.35 before for
// calls that stayed in one pass).  Up to four windows one pass comes out of L2 for the most part, and the smaller the graph the more
// picks it takes; a step of 15 % lies between four windows and five.  8, 12 and 16 picks a column lie in the same banks of shared
// memory column after column, and more than 10 leave fewer CTAs an SM.  Columns that all have the same chance are read whole more
// often and gain least (10 picks 1.1 to 1.4): first hops, which have few picks.  S may be a bound on the columns, which is all that the
// host knows.
bool window_sample_suits(gsb_ctx* ctx, i64 S, i64 k, i64 num_edges) {
  const i64 path = ctx_option(ctx, GSB_OPT_SAMPLE_PATH);
  if (k < 1 || k > 16 || num_edges < 1 || path == 1 || num_edges > ((i64)kMaxWindows << kWindowShift)) return false;
  if (path == 2) return true;
  if (num_edges < (16 << 20) || k == 16) return false;
  const i64 picks = S * k;
  const bool few = num_edges <= ((i64)4 << kWindowShift), wide = k == 8 || k >= 12;
  if (k <= 5) return picks >= (few ? num_edges : max((i64)12'000'000, num_edges * max(k, (i64)4) / 64));
  if (few) return !wide && num_edges >= 20'000'000 && picks >= 127'500'000 - 3 * num_edges;
  return picks >= max((i64)(wide ? 40'000'000 : 20'000'000), num_edges * k / 64);
}

static inline size_t al256(size_t b) { return (b + 255) & ~(size_t)255; }

size_t window_sample_bytes(gsb_ctx* ctx, i64 S, i64 k, i64 num_edges) {
  const i64 tiles = window_tiles(S);
  return al256((size_t)tiles * kWinTile * k * 4) + al256((size_t)tiles * kWinTile * 2) +
         al256((size_t)(window_count(ctx, num_edges) + 2) * tiles * 2);
}

template <int KMAX>
static int launch_window(gsb_ctx* ctx, cudaStream_t stream, const WindowParams& w) {
  const size_t smem = (size_t)kWinTile * w.p.k * 8;
  static bool attr_set[64] = {};
  const int dev = ctx_device(ctx);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const int most = kWinTile * KMAX * 8;
    GSB_CUDA_OK(cudaFuncSetAttribute(k_window_draw<KMAX>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_window_emit<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWinTile * 16 * 8));
    GSB_CUDA_OK(cudaFuncSetAttribute(k_window_emit<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kWinTile * 16 * 8));
    attr_set[dev] = true;
  }
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_UNIFORM, stream);
    k_window_draw<KMAX><<<(int)w.tiles, kWinThreads, smem, stream>>>(w);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_UNIFORM, stream);
    const dim3 grid((unsigned)grid_for(w.tiles, kReadThreads / 32), w.windows);
    k_window_read<<<grid, kReadThreads, 0, stream>>>(w);
  }
  GSB_LAUNCH_OK();
  {
    ScopedKernelTimer timer(ctx, KID_SAMPLE_UNIFORM, stream);
    if (w.p.bucket_count) k_window_emit<true><<<(int)w.tiles, kWinThreads, smem, stream>>>(w);
    else k_window_emit<false><<<(int)w.tiles, kWinThreads, smem, stream>>>(w);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int window_sample_launch(gsb_ctx* ctx, cudaStream_t stream, const SampleParams& p, i64 num_edges, void* ws) {
  WindowParams w;
  w.p = p;
  w.tiles = window_tiles(p.S);
  w.shift = window_shift(ctx, num_edges);
  w.windows = (uint32_t)window_count(ctx, num_edges);
  char* at = (char*)ws;
  w.staged = (uint32_t*)at;
  at += al256((size_t)w.tiles * kWinTile * p.k * 4);
  w.place = (uint16_t*)at;
  at += al256((size_t)w.tiles * kWinTile * 2);
  w.start = (uint16_t*)at;
  if (p.k <= 5) return launch_window<5>(ctx, stream, w);
  if (p.k <= 10) return launch_window<10>(ctx, stream, w);
  return launch_window<16>(ctx, stream, w);
}

}  // namespace gsb
