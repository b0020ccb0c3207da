// List sampling: pick k of the N items of one list (layer-wise samplers: LADIES / FastGCN).
//
// Without replacement every item gets a ranking key — a Philox word for the uniform case, the
// A-Res key log2(u)/w for the weighted case (w <= 0 can never beat a positive weight) — and the k
// best keys win; ties go to the smaller position; the output is in descending key order, which is
// what the reference's descending stable sort yields (src/cuda/list_sampling_probs.cu:56-88).
// Instead of sorting all N keys to take k of them, the k-th best key is found by a most-significant-digit radix SELECT
// over the 64-bit composite (key << 32 | ~position), and only the k winners are sorted: one cooperative launch up to
// k = 4 096 (k_list_select), one launch per pass beyond.  With replacement: k independent draws, uniform
// or by inverse CDF (src/cuda/list_sampling.cu:35-52, list_sampling_probs.cu:28-55).
#include "common.cuh"
#include "grid_sync.cuh"
#include "philox.cuh"
#include "radix_sort.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kListThreads = 256;
constexpr int kListPerThread = 4;
constexpr int kListTile = kListThreads * kListPerThread;
constexpr int kCdfChunk = 1024;

__device__ __forceinline__ uint32_t orderable_f32(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ uint32_t weighted_key(float w, i64 i, u64 seed) {
  if (!(w > 0.0f)) return orderable_f32(ares_key(0, w));  // whatever the draw: most rows of a layer's list have no weight
  return orderable_f32(ares_key(rand_u32(seed, (u64)i, 0, STREAM_LIST_WEIGHTED), w));
}

__device__ __forceinline__ u64 composite_of(uint32_t key, i64 i) { return ((u64)key << 32) | (u64)(0xFFFFFFFFu - (uint32_t)i); }

__device__ __forceinline__ u64 list_composite(const float* __restrict__ probs, i64 i, u64 seed) {
  return composite_of(probs ? weighted_key(__ldg(probs + i), i, seed) : rand_u32(seed, (u64)i, 0, STREAM_LIST), i);
}

// Sampling without replacement of k <= kSelectMaxK items in one launch: composites -> radix select, 11 bits per pass, a
// grid barrier per pass, until the selected bin is needed whole (two or three passes unless keys tie) -> the winners are
// appended in any order -> every warp counts, for one of them after the other, the winners that rank before it, and puts it there
// (with few CTAs for many winners CTA 0 sorts them).  Layer-wise sampling makes one such call per layer on a list of a
// million rows; as thirteen launches it was 140 us, most of it between the launches; with composites read again in every pass
// and a sort in one CTA 31 us for 512 of a million, of which four were a re-reading each and six the sort; 22 now (4 096 of a
// million 70 -> 29).  Its grid barriers, four to eight of them, bound it.
// KEPT: a thread's keys, up to eight, stay in its registers.
constexpr int kSelectThreads = 1024;
constexpr int kSelectBins = 2048;
constexpr int kSelectMaxK = 4096;
constexpr int kSelectPasses = 6;                   // shifts 53, 42, 31, 20, 9 and 0 (the last digit has nine bits)
constexpr int kSelectBarriers = kSelectPasses + 2;

struct SelectParams {
  const float* probs;
  const i64* data;
  i64 N, k;
  u64 seed;
  u64* composite;    // [N]
  unsigned* hist;    // [kSelectPasses][kSelectBins]
  unsigned* found;   // [1]
  u64* winners;      // [kSelectMaxK]
  i64* out_data;
  i64* out_index;
  i64* counters;
  GridSync sync;
};

// Adds the warp's digits to a shared-memory histogram: the lanes that share the first one's digit, and then those that share the
// first of the others', add once (all zero-weight items share one key, and plain atomics on one address would serialise the
// CTA); the rest add one by one (__match_any_sync, which gathers all of them, takes 0.5 us for 32 distinct digits).
__device__ __forceinline__ void select_count(unsigned* s_hist, unsigned digit, bool counts) {
  unsigned rest = __ballot_sync(0xffffffffu, counts);
#pragma unroll
  for (int t = 0; t < 2; ++t) {
    if (rest == 0) return;
    const int first = __ffs(rest) - 1;
    const unsigned same = __ballot_sync(0xffffffffu, digit == __shfl_sync(0xffffffffu, digit, first)) & rest;
    if ((int)(threadIdx.x & 31) == first) atomicAdd(&s_hist[digit], (unsigned)__popc(same));
    rest &= ~same;
  }
  if ((rest >> (threadIdx.x & 31)) & 1u) atomicAdd(&s_hist[digit], 1u);
}

// A thread's keys in registers: 148 CTAs keep the lists of up to 1 212 416 items.  The line lies behind the million rows that layer-wise
// sampling was timed on (22.8 us for 512 of them); beyond it composites go through memory (1 250 000 items 35.2 us, three million 46.7),
// and more keys a thread have not been tried.
constexpr int kSelectKept = 8;
// Winners per CTA up to which all CTAs rank them: a rank is k comparisons by a warp (4 096 winners on 22 CTAs about 16 us, 512 on
// three 2), the sort of one CTA 35 us for 4 096 and 6.5 for 512.
constexpr i64 kSelectRanked = 192;

// (two CTAs per SM are never launched: the bound is for 32 registers, with 45 the passes over ten million items take 170 us
// instead of 160)
template <bool KEPT>
__global__ void __launch_bounds__(kSelectThreads, KEPT ? 1 : 2) k_list_select(const __grid_constant__ SelectParams p) {
  __shared__ __align__(16) u64 s_win[kSelectMaxK];   // the histogram of a pass, later the winners
  __shared__ unsigned s_warp[kSelectThreads / 32];
  __shared__ unsigned s_pick[2];                     // bin, items of it that are needed
  unsigned* s_hist = reinterpret_cast<unsigned*>(s_win);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const i64 stride = (i64)gridDim.x * kSelectThreads;
  const i64 rounds = (p.N + stride - 1) / stride;
  for (i64 i = (i64)blockIdx.x * kSelectThreads + tid; i < kSelectPasses * kSelectBins; i += stride) p.hist[i] = 0;
  if (blockIdx.x == 0 && tid == 0) *p.found = 0;
  for (int i = tid; i < kSelectBins; i += kSelectThreads) s_hist[i] = 0;
  grid_barrier_arrive(p.sync);
  const i64 own = (i64)blockIdx.x * kSelectThreads + tid;  // the thread's items: own, own + stride, ...
  uint32_t key[KEPT ? kSelectKept : 1];
  if (KEPT) {
    float w[kSelectKept];
#pragma unroll
    for (int r = 0; r < kSelectKept; ++r) w[r] = p.probs && own + r * stride < p.N ? __ldg(p.probs + own + r * stride) : 0.0f;
#pragma unroll
    for (int r = 0; r < kSelectKept; ++r) {
      const i64 i = own + r * stride;
      key[r] = 0;
      if (i < p.N) key[r] = p.probs ? weighted_key(w[r], i, p.seed) : rand_u32(p.seed, (u64)i, 0, STREAM_LIST);
    }
#pragma unroll
    for (int r = 0; r < kSelectKept; ++r)
      if (r < rounds) select_count(s_hist, key[r] >> 21, own + r * stride < p.N);
  } else {
    for (i64 r = 0; r < rounds; ++r) {
      const i64 i = r * stride + own;
      const bool valid = i < p.N;
      const u64 c = valid ? list_composite(p.probs, i, p.seed) : 0;
      if (valid) p.composite[i] = c;
      select_count(s_hist, (unsigned)(c >> 53), valid);
    }
  }
  // f(item's composite, whether there is an item) for the thread's items, in all lanes
  auto for_composites = [&](auto f) {
    if (KEPT) {
#pragma unroll
      for (int r = 0; r < kSelectKept; ++r)
        if (r < rounds) f(composite_of(key[r], own + r * stride), own + r * stride < p.N);
    } else {
      for (i64 r = 0; r < rounds; ++r) {
        const i64 i = r * stride + own;
        f(i < p.N ? p.composite[i] : 0ull, i < p.N);  // written by this very thread
      }
    }
  };
  // The result of a call that was given up: the first k items.
  auto give_up = [&] {
    for (i64 i = 0; blockIdx.x == 0 && i < p.k; ++i) {
      p.out_index[i] = i;
      p.out_data[i] = __ldg(p.data + i);
    }
  };
  u32 barrier = 1;
  grid_barrier_wait(p.sync, barrier, give_up);  // the global histograms are clear
  u64 prefix = 0, mask = 0;
  unsigned need = (unsigned)p.k;
  int pass = 0;
  for (int shift = 53;; ++pass) {
    const int bits = pass == kSelectPasses - 1 ? 9 : 11;
    unsigned* hist = p.hist + pass * kSelectBins;
    for (int i = tid; i < kSelectBins; i += kSelectThreads)
      if (s_hist[i]) atomicAdd(hist + i, s_hist[i]);
    grid_barrier(p.sync, ++barrier, give_up);
    // every CTA picks the bin for itself: thread t owns bins 2t, 2t + 1; `above` counts the items in larger bins
    {
      const uint2 h = __ldcg(reinterpret_cast<const uint2*>(hist) + tid);
      unsigned inc = h.x + h.y;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_down_sync(0xffffffffu, inc, o);
        if (lane + o < 32) inc += t;
      }
      if (lane == 0) s_warp[warp] = inc;
      __syncthreads();
      unsigned above = inc - h.x - h.y;
      for (int w = warp + 1; w < kSelectThreads / 32; ++w) above += s_warp[w];
      if (above < need && above + h.y >= need) {
        s_pick[0] = 2 * tid + 1;
        s_pick[1] = need - above;
      }
      above += h.y;
      if (above < need && above + h.x >= need) {
        s_pick[0] = 2 * tid;
        s_pick[1] = need - above;
      }
      __syncthreads();
    }
    const unsigned bin = s_pick[0];
    need = s_pick[1];
    prefix |= (u64)bin << shift;
    mask |= ((1ull << bits) - 1ull) << shift;
    const bool whole = __ldcg(hist + bin) == need;  // all composites >= prefix are exactly the winners
    if (whole || pass == kSelectPasses - 1) break;
    shift = pass == kSelectPasses - 2 ? 0 : shift - 11;
    const unsigned digit_mask = pass == kSelectPasses - 2 ? 511u : 2047u;
    for (int i = tid; i < kSelectBins; i += kSelectThreads) s_hist[i] = 0;
    __syncthreads();
    for_composites([&](u64 c, bool item) {
      select_count(s_hist, (unsigned)(c >> shift) & digit_mask, item && (c & mask) == prefix);
    });
    __syncthreads();
  }
  for_composites([&](u64 c, bool item) {
    if (!item || c < prefix) return;
    const unsigned at = atomicAdd(p.found, 1u);
    if (at < (unsigned)p.k) p.winners[at] = c;
    else raise_error(p.counters, GSB_ERR_CAPACITY, at);  // cannot happen: composites are distinct
  });
  // everybody arrives, also for the passes that were not needed
  const u32 unused = kSelectBarriers - 1 - barrier;
  if (p.k <= (i64)gridDim.x * kSelectRanked) {
    grid_arrive(p.sync, unused);
    grid_barrier(p.sync, kSelectBarriers, give_up);
    const int k = (int)p.k;
    for (int i = tid; i < k; i += kSelectThreads) s_win[i] = __ldcg(p.winners + i);
    __syncthreads();
    const int warps = (int)gridDim.x * (kSelectThreads / 32);
    for (int j = (int)blockIdx.x * (kSelectThreads / 32) + warp; j < k; j += warps) {
      const u64 c = s_win[j];
      unsigned before = 0;
      for (int i = lane; i < k; i += 32) before += s_win[i] > c;
      before = __reduce_add_sync(0xffffffffu, before);
      if (lane == 0) {
        const i64 idx = (i64)(0xFFFFFFFFu - (uint32_t)c);
        p.out_index[before] = idx;
        p.out_data[before] = __ldg(p.data + idx);
      }
    }
    return;
  }
  if (blockIdx.x != 0) {  // only CTA 0 waits: it has the rest to itself
    __syncthreads();
    __threadfence();
    grid_arrive(p.sync, unused + 1);
    return;
  }
  grid_arrive(p.sync, unused);
  grid_barrier(p.sync, kSelectBarriers, give_up);
  int n = 1;
  while (n < (int)p.k) n <<= 1;
  for (int i = tid; i < n; i += kSelectThreads) s_win[i] = i < (int)p.k ? __ldcg(p.winners + i) : 0ull;  // 0 sorts last
  __syncthreads();
  for (int size = 2; size <= n; size <<= 1) {
    for (int j = size >> 1; j > 0; j >>= 1) {
      for (int i = tid; i < n / 2; i += kSelectThreads) {
        const int lo = 2 * i - (i & (j - 1)), hi = lo + j;
        const bool desc = (lo & size) == 0;
        const u64 a = s_win[lo], b = s_win[hi];
        if ((a < b) == desc) {
          s_win[lo] = b;
          s_win[hi] = a;
        }
      }
      __syncthreads();
    }
  }
  for (int i = tid; i < (int)p.k; i += kSelectThreads) {
    const i64 idx = (i64)(0xFFFFFFFFu - (uint32_t)s_win[i]);
    p.out_index[i] = idx;
    p.out_data[i] = __ldg(p.data + idx);
  }
}

struct SelectState {
  u64 prefix;     // bits decided so far (high digits)
  i64 remaining;  // how many winners must still come from the undecided bin
  i64 hist[256];
  unsigned done;      // CTAs that have added their counts in the current pass
  unsigned resolved;  // the selected bin is needed entirely: the threshold is final, later passes have nothing to do
};

__global__ void __launch_bounds__(kListThreads) k_list_keys(const float* __restrict__ probs, i64 N, u64 seed,
                                                            u64* __restrict__ composite) {
  for (i64 i = (i64)blockIdx.x * kListThreads + threadIdx.x; i < N; i += (i64)gridDim.x * kListThreads) {
    composite[i] = list_composite(probs, i, seed);
  }
}

__global__ void k_select_init(SelectState* st, i64 k) {
  if (threadIdx.x == 0) {
    st->prefix = 0;
    st->remaining = k;
    st->done = 0;
    st->resolved = 0;
  }
  st->hist[threadIdx.x] = 0;
}

// One pass of the radix select: every CTA counts, per value of the current digit, the items that still match the
// decided prefix; the CTA that adds its counts last (a ticket from `done`) walks the 256 bins from the top — the
// bin in which the running count reaches `remaining` holds the k-th best item — and clears the state for the next
// pass.  (Counting and picking were two launches per pass; the operator is launch bound.)
__global__ void __launch_bounds__(kListThreads) k_select_pass(const u64* __restrict__ composite, i64 N, int shift,
                                                              SelectState* st) {
  __shared__ unsigned s_hist[256];
  __shared__ bool s_last;
  if (st->resolved) return;  // uniform over the grid: written by the previous launch
  s_hist[threadIdx.x] = 0;
  __syncthreads();
  const u64 prefix = st->prefix;
  const u64 high_mask = shift >= 56 ? 0ull : (~0ull << (shift + 8));
  for (i64 i = (i64)blockIdx.x * kListThreads + threadIdx.x; i < N; i += (i64)gridDim.x * kListThreads) {
    const u64 c = composite[i];
    // lanes that hit the same bin add once: with many equal keys (all zero-weight items share one) plain
    // shared-memory atomics on one address serialise the whole CTA
    const unsigned digit = (c & high_mask) == prefix ? ((unsigned)(c >> shift) & 0xFFu) : 0x100u;
    const unsigned peers = __match_any_sync(__activemask(), digit);
    if (digit < 0x100u && (int)(__ffs(peers) - 1) == (int)(threadIdx.x & 31)) atomicAdd(&s_hist[digit], (unsigned)__popc(peers));
  }
  __syncthreads();
  if (s_hist[threadIdx.x]) atomicAdd((u64*)&st->hist[threadIdx.x], (u64)s_hist[threadIdx.x]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  __shared__ i64 s_h[256];
  s_h[threadIdx.x] = ((volatile i64*)st->hist)[threadIdx.x];
  st->hist[threadIdx.x] = 0;
  __syncthreads();
  if (threadIdx.x == 0) {
    i64 need = st->remaining;
    int bin = 0;
    for (int d = 255; d >= 0; --d) {
      if (s_h[d] >= need) {
        bin = d;
        break;
      }
      need -= s_h[d];
    }
    st->prefix |= (u64)bin << shift;
    st->remaining = need;
    st->done = 0;
    // every item of the selected bin is needed: all composites >= prefix (lower digits zero) are exactly the k
    // winners, so the remaining digits need not be examined (the usual case once the key digits are through:
    // the last passes only split ties)
    if (s_h[bin] == need) st->resolved = 1;
  }
}

__global__ void __launch_bounds__(kListThreads) k_compact_winners(const u64* __restrict__ composite, i64 N,
                                                                  const SelectState* st, u64* __restrict__ winners,
                                                                  i64 k, i64* counters, TileState ts) {
  __shared__ i64 s_scan[33];
  __shared__ i64 s_base;
  const int tile = blockIdx.x;
  const i64 base = (i64)tile * kListTile;
  if (base >= N) return;
  const u64 threshold = st->prefix;
  u64 c[kListPerThread];
  int mine = 0;
#pragma unroll
  for (int q = 0; q < kListPerThread; ++q) {
    const i64 i = base + (i64)threadIdx.x * kListPerThread + q;
    c[q] = i < N ? composite[i] : 0;
    mine += (i < N && c[q] >= threshold) ? 1 : 0;
  }
  i64 total;
  const i64 excl = block_exclusive_scan<kListThreads>((i64)mine, s_scan, &total);
  if (threadIdx.x < 32) {
    const i64 prefix = tile_exclusive_prefix(ts, tile, total);
    if (threadIdx.x == 0) s_base = prefix;
  }
  __syncthreads();
  i64 pos = s_base + excl;
#pragma unroll
  for (int q = 0; q < kListPerThread; ++q) {
    const i64 i = base + (i64)threadIdx.x * kListPerThread + q;
    if (i < N && c[q] >= threshold) {
      if (pos < k) winners[pos] = c[q];
      else raise_error(counters, GSB_ERR_CAPACITY, pos);
      ++pos;
    }
  }
}

__global__ void __launch_bounds__(kListThreads) k_invert_keys(u64* __restrict__ keys, i64* __restrict__ vals, i64 n) {
  for (i64 i = (i64)blockIdx.x * kListThreads + threadIdx.x; i < n; i += (i64)gridDim.x * kListThreads) {
    keys[i] = ~keys[i];
    vals[i] = i;
  }
}

__global__ void __launch_bounds__(kListThreads) k_emit_winners(const u64* __restrict__ winners, i64 k,
                                                               const i64* __restrict__ data, i64* __restrict__ out_data,
                                                               i64* __restrict__ out_index, const i64* counters) {
  const bool lost = counters[CNT_LOST] != 0;  // then the first k items, as k_list_select leaves them
  for (i64 j = (i64)blockIdx.x * kListThreads + threadIdx.x; j < k; j += (i64)gridDim.x * kListThreads) {
    const u64 c = ~winners[j];  // k_invert_keys
    const i64 idx = lost ? j : (i64)(0xFFFFFFFFu - (uint32_t)c);
    out_index[j] = idx;
    out_data[j] = data[idx];
  }
}

__global__ void __launch_bounds__(kListThreads) k_list_identity(const i64* __restrict__ data, i64 N,
                                                                i64* __restrict__ out_data, i64* __restrict__ out_index) {
  for (i64 i = (i64)blockIdx.x * kListThreads + threadIdx.x; i < N; i += (i64)gridDim.x * kListThreads) {
    out_data[i] = data[i];
    out_index[i] = i;
  }
}

__global__ void __launch_bounds__(kListThreads) k_list_uniform_replace(const i64* __restrict__ data, i64 N, i64 k,
                                                                       u64 seed, i64* __restrict__ out_data,
                                                                       i64* __restrict__ out_index) {
  for (i64 j = (i64)blockIdx.x * kListThreads + threadIdx.x; j < k; j += (i64)gridDim.x * kListThreads) {
    const i64 pos = (i64)rand_bounded(seed, 0, (u64)j, STREAM_LIST, (u64)N);
    out_index[j] = pos;
    out_data[j] = data[pos];
  }
}

// Weighted with replacement: chunk totals (double), their prefix, then per draw a binary search
// over chunks and a walk inside one chunk.
__global__ void __launch_bounds__(kListThreads) k_cdf_chunk_sums(const float* __restrict__ probs, i64 N,
                                                                 double* __restrict__ chunk_sum) {
  __shared__ double s_part[kListThreads / 32];
  const i64 base = (i64)blockIdx.x * kCdfChunk;
  double acc = 0.0;
  for (int q = threadIdx.x; q < kCdfChunk; q += kListThreads)
    if (base + q < N) acc += (double)fmaxf(probs[base + q], 0.0f);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kListThreads / 32; ++w) t += s_part[w];
    chunk_sum[blockIdx.x] = t;
  }
}

__global__ void k_cdf_chunk_prefix(double* chunk_sum, i64 num_chunks) {
  // one thread: num_chunks = N / 1024 is small
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double run = 0.0;
    for (i64 c = 0; c < num_chunks; ++c) {
      const double v = chunk_sum[c];
      chunk_sum[c] = run;
      run += v;
    }
    chunk_sum[num_chunks] = run;
  }
}

__global__ void __launch_bounds__(kListThreads) k_list_weighted_replace(const i64* __restrict__ data,
                                                                        const float* __restrict__ probs, i64 N, i64 k,
                                                                        u64 seed, const double* __restrict__ chunk_pre,
                                                                        i64 num_chunks, i64* __restrict__ out_data,
                                                                        i64* __restrict__ out_index) {
  for (i64 j = (i64)blockIdx.x * kListThreads + threadIdx.x; j < k; j += (i64)gridDim.x * kListThreads) {
    const double total = chunk_pre[num_chunks];
    const double r = (double)uniform01(rand_u32(seed, 0, (u64)j, STREAM_LIST_WEIGHTED)) * total;
    i64 lo = 0, hi = num_chunks;  // largest chunk c with chunk_pre[c] <= r
    while (hi - lo > 1) {
      const i64 mid = (lo + hi) >> 1;
      if (chunk_pre[mid] <= r) lo = mid;
      else hi = mid;
    }
    double acc = chunk_pre[lo];
    i64 pos = -1;
    for (i64 c = lo; c < num_chunks && pos < 0; ++c) {
      const i64 end = min(N, (c + 1) * (i64)kCdfChunk);
      for (i64 i = c * (i64)kCdfChunk; i < end; ++i) {
        acc += (double)fmaxf(probs[i], 0.0f);
        if (acc > r) {
          pos = i;
          break;
        }
      }
    }
    if (pos < 0) pos = N - 1;
    out_index[j] = pos;
    out_data[j] = data[pos];
  }
}

}  // namespace gsb

using namespace gsb;

extern "C" int gsb_list_sample(gsb_ctx* ctx, void* stream_, const int64_t* data, const float* probs, int64_t N,
                               int64_t k, int replace, uint64_t seed, int64_t* out_data, int64_t* out_index,
                               int64_t* n_out_host) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(N >= 0 && k >= 0 && n_out_host, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(N < 0xFFFFFFFFll, GSB_ERR_UNSUPPORTED);
  cudaStream_t stream = (cudaStream_t)stream_;
  const int wide = kNumSMs * 8;
  if (!replace && N <= k) {
    *n_out_host = N;
    if (N == 0) return GSB_OK;
    GSB_REQUIRE(data && out_data && out_index, GSB_ERR_INVALID_ARGUMENT);
    k_list_identity<<<min(grid_for(N, kListThreads), wide), kListThreads, 0, stream>>>(data, N, out_data, out_index);
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
    return GSB_OK;
  }
  *n_out_host = (N == 0) ? 0 : k;
  if (N == 0 || k == 0) return GSB_OK;
  GSB_REQUIRE(data && out_data && out_index, GSB_ERR_INVALID_ARGUMENT);
  if (replace && !probs) {
    k_list_uniform_replace<<<min(grid_for(k, kListThreads), wide), kListThreads, 0, stream>>>(data, N, k, (u64)seed,
                                                                                             out_data, out_index);
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
    return GSB_OK;
  }
  if (replace) {
    const i64 chunks = (N + kCdfChunk - 1) / kCdfChunk;
    void* ws;
    int st = ctx_reserve_workspace(ctx, stream, sizeof(double) * (size_t)(chunks + 1), &ws);
    if (st != GSB_OK) return st;
    double* chunk_pre = (double*)ws;
    k_cdf_chunk_sums<<<(int)chunks, kListThreads, 0, stream>>>(probs, N, chunk_pre);
    GSB_LAUNCH_OK();
    k_cdf_chunk_prefix<<<1, 32, 0, stream>>>(chunk_pre, chunks);
    GSB_LAUNCH_OK();
    k_list_weighted_replace<<<min(grid_for(k, kListThreads), wide), kListThreads, 0, stream>>>(
        data, probs, N, k, (u64)seed, chunk_pre, chunks, out_data, out_index);
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 3);
    return GSB_OK;
  }
  static int resident[2][64];
  const int ctas = min(ctx_resident_ctas(ctx, (const void*)k_list_select<false>, kSelectThreads, 0, resident[0]),
                       ctx_resident_ctas(ctx, (const void*)k_list_select<true>, kSelectThreads, 0, resident[1]));
  if (k <= kSelectMaxK && ctas > 0) {
    const size_t bytes = ((size_t)N * 8 + 255) & ~(size_t)255;
    void* ws;
    int st = ctx_reserve_workspace(ctx, stream, bytes + kSelectMaxK * 8 + sizeof(unsigned) * (kSelectPasses * kSelectBins + 64), &ws);
    if (st != GSB_OK) return st;
    SelectParams p{};
    p.probs = probs;
    p.data = data;
    p.N = N;
    p.k = k;
    p.seed = (u64)seed;
    p.composite = (u64*)ws;
    p.winners = (u64*)((char*)ws + bytes);
    p.hist = (unsigned*)(p.winners + kSelectMaxK);
    p.found = p.hist + kSelectPasses * kSelectBins;
    p.out_data = out_data;
    p.out_index = out_index;
    p.counters = ctx_counters(ctx);
    // four items per thread: fewer CTAs make the barriers of a short list cheaper
    const int grid = (int)min((i64)min(ctas, kNumSMs), (N + 4 * kSelectThreads - 1) / (4 * kSelectThreads));
    p.sync = ctx_grid_sync(ctx, grid, kSelectBarriers);
    ScopedKernelTimer timer(ctx, KID_LIST_SAMPLE, stream);
    void* args[] = {&p};
    const bool kept = N <= (i64)grid * kSelectThreads * kSelectKept;
    return launch_cooperative(ctx, stream, kept ? (const void*)k_list_select<true> : (const void*)k_list_select<false>, grid,
                              kSelectThreads, 0, args, p.sync);
  }
  // many winners: keys -> radix select of the k-th best -> compact winners -> order them, one launch per pass
  const size_t comp_bytes = ((size_t)N * 8 + 255) & ~(size_t)255;
  const size_t win_bytes = ((size_t)k * 16 + 255) & ~(size_t)255;  // winners + index payload for the sort
  const size_t sort_bytes = radix_sort_scratch_bytes(k);
  void* ws;
  int st = ctx_reserve_workspace(ctx, stream, comp_bytes + win_bytes + sort_bytes + 4096, &ws);
  if (st != GSB_OK) return st;
  u64* composite = (u64*)ws;
  u64* winners = (u64*)((char*)ws + comp_bytes);
  i64* win_vals = (i64*)(winners + k);
  void* sort_ws = (char*)ws + comp_bytes + win_bytes;
  SelectState* state = (SelectState*)((char*)sort_ws + sort_bytes);
  const int grid_n = min(grid_for(N, kListThreads), wide);
  {
    ScopedKernelTimer timer(ctx, KID_LIST_SAMPLE, stream);
    k_list_keys<<<grid_n, kListThreads, 0, stream>>>(probs, N, (u64)seed, composite);
  }
  GSB_LAUNCH_OK();
  k_select_init<<<1, 256, 0, stream>>>(state, k);
  GSB_LAUNCH_OK();
  // few, long-running CTAs for the select passes: every CTA ends with up to 256 global atomics on the same 256
  // counters and one ticket, and those serialise
  const int grid_sel = max(1, min(grid_for(N, kListThreads * 16), kNumSMs * 2));
  for (int shift = 56; shift >= 0; shift -= 8) {
    ScopedKernelTimer timer(ctx, KID_SORT, stream);
    k_select_pass<<<grid_sel, kListThreads, 0, stream>>>(composite, N, shift, state);
    GSB_LAUNCH_OK();
  }
  const int tiles = grid_for(N, kListTile);
  TileState ts;
  st = ctx_tile_state(ctx, tiles, stream, &ts);
  if (st != GSB_OK) return st;
  {
    ScopedKernelTimer timer(ctx, KID_FIRST_COMPACT, stream);
    k_compact_winners<<<tiles, kListThreads, 0, stream>>>(composite, N, state, winners, k, ctx_counters(ctx), ts);
  }
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 1);
  k_invert_keys<<<min(grid_for(k, kListThreads), wide), kListThreads, 0, stream>>>(winners, win_vals, k);
  GSB_LAUNCH_OK();
  st = radix_sort_pairs(ctx, stream, winners, win_vals, k, 0, 64, sort_ws);
  if (st != GSB_OK) return st;
  ctx_count_launches(ctx, 1);
  k_emit_winners<<<min(grid_for(k, kListThreads), wide), kListThreads, 0, stream>>>(winners, k, data,
                                                                                    out_data, out_index,
                                                                                    ctx_counters(ctx));
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 1);
  return GSB_OK;
}
