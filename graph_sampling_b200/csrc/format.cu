// Sparse-format conversion: CSC -> COO (column id per edge) and COO -> CSC / CSR (stable sort by
// the key coordinate, edge permutation, offsets).
#include "common.cuh"
#include "grid_sync.cuh"
#include "radix_sort.cuh"

namespace gsb {

constexpr int kFmtThreads = 256;
constexpr int kFmtTileCols = 256;

// One CTA per tile of columns; warps walk the tile's contiguous edge range 256 edges at a time and find the
// column of the first edge by binary search in the shared copy of the tile's offsets, then step forward (the
// reference searches the whole indptr in global memory per edge: src/cuda/format_transform.cu:23-33).
__global__ void __launch_bounds__(kFmtThreads) k_csc2coo(const i64* __restrict__ indptr, i64 num_cols,
                                                         i64* __restrict__ out_col) {
  __shared__ i64 s_off[kFmtTileCols + 1];
  const i64 base = (i64)blockIdx.x * kFmtTileCols;
  if (base >= num_cols) return;
  const int ncol = (int)min((i64)kFmtTileCols, num_cols - base);
  for (int q = threadIdx.x; q <= ncol; q += kFmtThreads) s_off[q] = indptr[base + q];
  __syncthreads();
  const i64 lo_e = s_off[0], hi_e = s_off[ncol];
  // a warp writes 256 consecutive edges at a time: one binary search for the first, then the column only walks on
  constexpr int kChunk = 32 * 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (i64 chunk = lo_e + (i64)warp * kChunk; chunk < hi_e; chunk += (i64)(kFmtThreads / 32) * kChunk) {
    int lo = 0, hi = ncol;  // invariant: s_off[lo] <= chunk < s_off[hi]
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_off[mid] <= chunk) lo = mid;
      else hi = mid;
    }
    int c = lo;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const i64 e = chunk + r * 32 + lane;
      if (e >= hi_e) break;
      while (s_off[c + 1] <= e) ++c;
      out_col[e] = base + c;
    }
  }
}

__global__ void __launch_bounds__(kFmtThreads) k_count_keys(const i64* __restrict__ key, i64 E, i64 num_keys,
                                                            i64* __restrict__ counts, i64* counters) {
  for (i64 e = (i64)blockIdx.x * kFmtThreads + threadIdx.x; e < E; e += (i64)gridDim.x * kFmtThreads) {
    const i64 k = key[e];
    if (k < 0 || k >= num_keys) {
      raise_error(counters, GSB_ERR_INDEX_RANGE, e);
      continue;
    }
    atomicAdd((u64*)&counts[k], 1ull);
  }
}

__global__ void __launch_bounds__(kFmtThreads) k_make_sort_input(const i64* __restrict__ key, i64 E,
                                                                 u64* __restrict__ keys, i64* __restrict__ vals) {
  for (i64 e = (i64)blockIdx.x * kFmtThreads + threadIdx.x; e < E; e += (i64)gridDim.x * kFmtThreads) {
    keys[e] = (u64)key[e];
    vals[e] = e;
  }
}

// The other coordinate in key order (perm null: the edges are in that order as they are).  Where a scan was given up the result is
// what k_coo2csc leaves in that case: all edges, in the order of the list, in column 0.
__global__ void __launch_bounds__(kFmtThreads) k_conversion_end(const i64* __restrict__ other, i64* perm, i64 E, i64 num_keys,
                                                                i64* __restrict__ out_indptr, i64* __restrict__ out_other,
                                                                const i64* counters) {
  const i64 first = (i64)blockIdx.x * kFmtThreads + threadIdx.x, step = (i64)gridDim.x * kFmtThreads;
  const bool lost = counters[CNT_LOST] != 0;
  if (lost) {
    for (i64 e = first; e < E && perm; e += step) perm[e] = e;
    for (i64 k = first; k <= num_keys; k += step) out_indptr[k] = k == 0 ? 0 : E;
  }
  for (i64 e = first; e < E; e += step) out_other[e] = other[perm && !lost ? perm[e] : e];
}

// Lanes that hold the same value of up to 2^bits, among the lanes where `valid` holds.  A ballot per bit: __match_any_sync takes
// its time once per DISTINCT value, 0.5 us for 32 of them.
__device__ __forceinline__ unsigned same_digit(u32 d, int bits, bool valid) {
  unsigned peers = __ballot_sync(0xffffffffu, valid);
  for (int b = 0; b < bits; ++b) {
    const bool one = (d >> b) & 1u;
    const unsigned ones = __ballot_sync(0xffffffffu, one);
    peers &= one ? ones : ~ones;
  }
  return peers;
}

// ---- COO -> CSC / CSR of a short list, without a barrier ----------------------------------------------------------------
// The keys of up to 26 624 edges are read from L2 by EVERY CTA (213 KB at most) and stay in its registers, so it needs nothing from
// the others.  Each counts the edges of up to 8 192 bins of neighbouring keys, and from the counts' prefix sums all of them derive the
// same shares: a bin costs E units and an edge as many as there are bins, a share is an equal part of that line, and so holds at
// most twice an equal part of the edges and of the bins, however the keys crowd.  A bin may span several shares; its edges are then
// dealt out by their number within the bin, and a CTA that has not the first of them counts, per key, those that others place before
// its own.
// Counts per key of the share's bins, their scan (the offsets), and a rank per edge among the few hundred of the share: all in
// shared memory.
// Bound by instruction issue, of which reading and counting all keys is the most.  us a call, calls in a row, the cooperative form
// below / a fixed range of keys per CTA, which sorts its edges / this: 25 000 edges over 200 000 keys evenly 33.3 / 14.9 / 17.3, by
// a power law numbered by degree 33.2 / 26.4 / 19.3, all within 1 351 neighbouring keys 32.7 / 92.7 / 23.0, all of one key
// 45.7 / 72.3 / 23.0; over a million keys evenly 41.4 / 15.7 / 18.8, as the sixth power of an even spread 42.1 / 47.7 / 25.0; 700
// edges over a thousand keys 17.0 / 8.9 / 8.8; 26 600 over a thousand, the case with the least to win, 24.9 .. 39.1 / 14.8 .. 47.5 /
// 17.7 .. 25.1.
constexpr int kShortThreads = 1024;
constexpr int kShortWarps = kShortThreads / 32;
constexpr int kShortPer = 26;   // keys of a thread
constexpr int kKeysAhead = 9;   // of them on their way
constexpr i64 kShortMaxEdges = (i64)kShortPer * kShortThreads;  // more keys of a thread would not stay in its 64 registers
constexpr int kShortBins = 8192;
constexpr int kShortBinsPer = kShortBins / kShortThreads;
// The keys of a share, 55 296 then, have a word of shared memory each (222 KB) and a number of 16 bits.  Up to there this is far
// ahead: 26 600 edges over four million keys 67 .. 82 us / 23 .. 31.
constexpr i64 kShortMaxKeys = 4'000'000;

struct ShortShape {
  u32 grid;
  int shift;   // a bin is 2^shift keys
  u32 bins;
  u32 keys;    // of the bins of a share, at most
  u32 edges;   // of a share, at most
};
// A share is at most 2 x E x bins / grid + 1 units long: the bins that start in it, two more that begin before and at its end.
static ShortShape short_shape(i64 E, i64 num_keys) {
  ShortShape s;
  s.grid = kNumSMs;
  s.shift = 0;
  while (((num_keys - 1) >> s.shift) + 1 > kShortBins) ++s.shift;
  s.bins = (u32)(((num_keys - 1) >> s.shift) + 1);
  s.keys = min(s.bins, 2 * s.bins / s.grid + 3) << s.shift;
  s.edges = 2 * (u32)E / s.grid + 2;
  return s;
}
static size_t short_smem(const ShortShape& s) { return 4 * ((size_t)max((u32)kShortBins, s.keys) + ((size_t)1 << s.shift) + s.edges + 7); }

// Exclusive prefix of `mine` over the CTA's threads.
__device__ __forceinline__ u32 short_scan(u32 mine, u32* s_warp) {
  const u32 lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  u32 inc = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += t;
  }
  __syncthreads();  // s_warp may be in use
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  return __reduce_add_sync(0xffffffffu, lane < warp ? s_warp[lane] : 0u) + inc - mine;
}

__global__ void __launch_bounds__(kShortThreads, 1) k_coo2csc_short(const i64* __restrict__ key, const i64* __restrict__ other,
                                                                   u32 E, i64 num_keys, const __grid_constant__ ShortShape shape,
                                                                   i64* __restrict__ out_indptr, i64* __restrict__ out_other,
                                                                   i64* __restrict__ out_perm, i64* counters) {
  extern __shared__ __align__(16) u32 s_start[];  // [bins] edges per bin; later [keys] edges per key, then where the key's begin
  u32* s_mine = s_start + max((u32)kShortBins, (shape.keys + 3) & ~3u);  // [edges] key within the share : 16 | edge : 16, in order
  u32* s_before = s_mine + ((shape.edges + 3) & ~3u);  // [2^shift] per key of the first bin: edges that other CTAs place first
  __shared__ u32 s_warp[3][kShortWarps];
  __shared__ u32 s_share[6];
  const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
  const int shift = shape.shift;
  const u32 per_warp = (E + kShortThreads - 1) / kShortThreads * 32;
  const u32 begin = min(E, warp * per_warp), end = min(E, begin + per_warp);
  const u64 line = 2ull * E * shape.bins;
  const u32 from = (u32)(line * blockIdx.x / gridDim.x), to = (u32)(line * (blockIdx.x + 1) / gridDim.x);
  for (u32 k = tid; k < kShortBins / 4; k += kShortThreads) reinterpret_cast<uint4*>(s_start)[k] = make_uint4(0, 0, 0, 0);
  for (u32 k = tid; k < (1u << shift); k += kShortThreads) s_before[k] = 0;
  __syncthreads();
  constexpr u32 kNoKey = 0xFFFFFFFFu;
  u32 mine[kShortPer];  // the lane's keys, of every 32 edges of the warp one
#pragma unroll
  for (int q0 = 0; q0 < kShortPer; q0 += kKeysAhead) {
    i64 k[kKeysAhead];
#pragma unroll
    for (int q = 0; q < kKeysAhead; ++q) {
      const u32 i = begin + 32 * (q0 + q) + lane;
      k[q] = q0 + q < kShortPer && i < end ? __ldg(key + i) : 0;
    }
#pragma unroll
    for (int q = 0; q < kKeysAhead; ++q) {
      if (q0 + q >= kShortPer) break;
      const u32 i = begin + 32 * (q0 + q) + lane;
      mine[q0 + q] = kNoKey;
      if (i >= end) continue;
      if ((u64)k[q] >= (u64)num_keys) {
        if (blockIdx.x == 0) raise_error(counters, GSB_ERR_INDEX_RANGE, i);
        k[q] = 0;
      }
      mine[q0 + q] = (u32)k[q];
      atomicAdd(s_start + (mine[q0 + q] >> shift), 1u);
    }
  }
  if (blockIdx.x == 0 && tid == 0) out_indptr[num_keys] = (i64)E;
  if (from == to) return;
  __syncthreads();
  // ---- the share: bins first .. last, of the first the edges from `skip` on, of the last those up to `stop`
  {
    u32 count[kShortBinsPer], sum = 0;
    const u32 bin0 = tid * kShortBinsPer;
#pragma unroll
    for (int j = 0; j < kShortBinsPer; j += 4) {
      const uint4 four = reinterpret_cast<const uint4*>(s_start + bin0)[j / 4];
      count[j] = four.x, count[j + 1] = four.y, count[j + 2] = four.z, count[j + 3] = four.w;
      sum += four.x + four.y + four.z + four.w;
    }
    u32 edges = short_scan(sum, s_warp[0]);
#pragma unroll
    for (int j = 0; j < kShortBinsPer; ++j) {
      const u32 bin = bin0 + j;
      if (bin >= shape.bins) break;
      const u32 at = bin * E + edges * shape.bins, its = at + E, next = its + count[j] * shape.bins;
      if (at <= from && from < next) {
        s_share[0] = bin;
        s_share[1] = edges;  // with smaller keys
        s_share[2] = from <= its ? 0 : (from - its + shape.bins - 1) / shape.bins;
        s_share[3] = at == from;  // the offsets of its keys are the CTA's to write
      }
      if (at < to && to <= next) {
        s_share[4] = bin;
        s_share[5] = to <= its ? 0 : (to - its + shape.bins - 1) / shape.bins;
      }
      edges += count[j];
    }
  }
  __syncthreads();
  const u32 first = s_share[0], below = s_share[1], skip = s_share[2], last = s_share[4], stop = s_share[5];
  const u32 key_begin = first << shift, keys = min((u32)num_keys, (last + 1) << shift) - key_begin;
  for (u32 k = tid; k < keys; k += kShortThreads) s_start[k] = 0;
  __syncthreads();
  // ---- count the keys of the share's bins; edges of the warp in the first and in the last bin, and between them
  u32 in_first = 0, in_last = 0, between = 0;
#pragma unroll
  for (int q = 0; q < kShortPer; ++q) {
    if (begin + 32 * q >= end) break;  // uniform
    const u32 rel = mine[q] - key_begin;  // (no key: beyond all)
    const bool in = rel < keys;
    if (!__any_sync(0xffffffffu, in)) continue;
    if (in) atomicAdd(s_start + rel, 1u);
    const u32 bin = mine[q] >> shift;
    in_first += in && bin == first;
    in_last += in && bin == last && last != first;
    between += in && bin != last && bin != first;
  }
  in_first = __reduce_add_sync(0xffffffffu, in_first);
  in_last = __reduce_add_sync(0xffffffffu, in_last);
  between = __reduce_add_sync(0xffffffffu, between);
  if (lane == 0) {
    s_warp[0][warp] = in_first;
    s_warp[1][warp] = in_last;
    s_warp[2][warp] = between;
  }
  __syncthreads();
  // which of the first (last) bin's edges the CTA places: number skip and up, below `stop` (of the last)
  const u32 first_stop = first == last ? stop : 0xFFFFFFFFu;
  auto overlap = [](u32 a0, u32 a1, u32 b0, u32 b1) { return min(a1, b1) > max(a0, b0) ? min(a1, b1) - max(a0, b0) : 0u; };
  u32 at, total, number_first, number_last;
  {  // a warp per lane
    u32 f = s_warp[0][lane], l = s_warp[1][lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 tf = __shfl_up_sync(0xffffffffu, f, o), tl = __shfl_up_sync(0xffffffffu, l, o);
      if (lane >= o) f += tf, l += tl;
    }
    const u32 places = s_warp[2][lane] + overlap(f - s_warp[0][lane], f, skip, first_stop) + overlap(l - s_warp[1][lane], l, 0, stop);
    total = __reduce_add_sync(0xffffffffu, places);
    at = __reduce_add_sync(0xffffffffu, lane < warp ? places : 0u);
    number_first = __shfl_sync(0xffffffffu, f, warp) - in_first;
    number_last = __shfl_sync(0xffffffffu, l, warp) - in_last;
  }
  // ---- the share's edges, in order
  if (in_first + in_last + between > 0) {
#pragma unroll
    for (int q = 0; q < kShortPer; ++q) {
      if (begin + 32 * q >= end) break;
      const u32 rel = mine[q] - key_begin, bin = mine[q] >> shift;
      const bool in = rel < keys, of_first = in && bin == first, of_last = in && bin == last && last != first;
      if (!__any_sync(0xffffffffu, in)) continue;
      const unsigned firsts = __ballot_sync(0xffffffffu, of_first), lasts = __ballot_sync(0xffffffffu, of_last);
      const u32 number = of_first ? number_first + __popc(firsts & lt) : number_last + __popc(lasts & lt);
      const bool take = in && (of_first ? number >= skip && number < first_stop : of_last ? number < stop : true);
      if (of_first && number < skip) atomicAdd(s_before + rel, 1u);
      const unsigned taken = __ballot_sync(0xffffffffu, take);
      if (take) s_mine[at + __popc(taken & lt)] = (rel << 16) | (begin + 32 * q + lane);
      at += __popc(taken);
      number_first += __popc(firsts);
      number_last += __popc(lasts);
    }
  }
  if (tid < (-total & 3u)) s_mine[total + tid] = 0xFFFFFFFFu;
  // ---- offsets: a stretch of keys per thread, an odd number of them (each lane another bank)
  {
    const u32 per = ((keys + kShortThreads - 1) / kShortThreads) | 1u, k0 = min(keys, tid * per), k1 = min(keys, k0 + per);
    u32 sum = 0;
    for (u32 k = k0; k < k1; ++k) sum += s_start[k];
    u32 run = short_scan(sum, s_warp[0]);
    for (u32 k = k0; k < k1; ++k) {
      const u32 c = s_start[k];
      s_start[k] = run;
      run += c;
    }
    __syncthreads();
    const u32 own = s_share[3] ? 0 : 1u << shift;  // the first bin's keys may be another CTA's to write
    for (u32 k = own + tid; k < keys; k += kShortThreads) out_indptr[key_begin + k] = (i64)(below + s_start[k]);
  }
  // ---- every edge behind those of its key that come before it
  for (u32 j = tid; j < total; j += kShortThreads) {
    const u32 me = s_mine[j], rel = me >> 16, e = me & 0xFFFFu;
    const i64 value = __ldg(other + e);
    u32 pos = below + s_start[rel] + (rel < (1u << shift) ? s_before[rel] : 0u);
    // the key's earlier edges lie between (key, 0) and this one (and so none of them is one of what lies behind the list)
    for (u32 i = 0; i < j; i += 4) {
      const uint4 four = *reinterpret_cast<const uint4*>(s_mine + i);
      pos += (four.x - (rel << 16) < e) + (four.y - (rel << 16) < e) + (four.z - (rel << 16) < e) + (four.w - (rel << 16) < e);
    }
    out_perm[pos] = (i64)e;
    out_other[pos] = value;
  }
}

// ---- COO -> CSC / CSR in one launch ------------------------------------------------------------------------------
// Stable counting sort of E edges by key with the offsets over all keys, as one cooperative kernel with a grid barrier
// between its steps.  The slices that layer-wise sampling converts have 10^4 to 10^6 edges: the radix sort's fifteen
// launches (count, scan, three passes of three, gather, copies) were 60 us of kernels and as much again between them.
//
//   per digit of up to 11 bits (one to three of them):
//     count    CTA c owns the c-th stretch of the current order, warp w the w-th part of that; 16-bit counts per warp and
//              digit in shared memory; the CTA's counts go to matrix[digit][c]
//     scan     a warp per digit (a thread when there are few CTAs: a single one took 10 of its 23 us to walk 1 024 rows a
//              warp at a time) turns its row of the matrix into exclusive prefixes, and notes the digit's total
//     place    every warp walks its part again, 32 items at a time ranked by ballots, and writes each item to
//              digit start + CTA prefix + warp prefix + rank: stable, since everything is numbered in order
//   along the way, the offsets: counts per key (one reduction per edge) during the first scan, totals per CTA of keys
//   during the first place, offsets written during the next step.
// An item is (key << 32 | edge).  The last place step writes the permutation and the other coordinate directly.
constexpr int kConvThreads = 1024;
constexpr int kConvWarps = kConvThreads / 32;
constexpr int kConvMaxBins = 2048;
constexpr int kConvFewCtas = 8;
constexpr i64 kConvMaxEdges = 4ll << 20;  // 28 000 edges per CTA: a warp's count fits 16 bits

struct ConvParams {
  const i64* key;
  const i64* other;
  i64 E, num_keys;
  int digits, digit_bits;
  u64* items[2];   // [E] each
  u32* matrix;     // [bins][CTAs]
  u32* bin_total;  // [bins]
  u32* counts;     // [num_keys]
  u32* key_total;  // [CTAs]
  i64* out_indptr;
  i64* out_other;
  i64* out_perm;
  i64* counters;
  GridSync sync;
};

__global__ void __launch_bounds__(kConvThreads) k_coo2csc(const __grid_constant__ ConvParams p) {
  extern __shared__ __align__(16) unsigned char s_dyn[];
  uint16_t* s_count = reinterpret_cast<uint16_t*>(s_dyn);  // [warps][bins]
  __shared__ u32 s_start[kConvMaxBins];                    // where the CTA's items of a digit go
  __shared__ u32 s_warp[kConvWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, ctas = gridDim.x;
  const int bins = 1 << p.digit_bits;
  const u32 E = (u32)p.E;
  const u32 per_cta = (u32)(((p.E + ctas - 1) / ctas + 32 * kConvWarps - 1) / (32 * kConvWarps) * (32 * kConvWarps));
  const u32 per_warp = per_cta / kConvWarps;
  const u32 begin = min(E, (u32)blockIdx.x * per_cta + (u32)warp * per_warp), end = min(E, begin + per_warp);
  const i64 keys_per_cta = (p.num_keys + ctas - 1) / ctas;
  const i64 key_begin = min(p.num_keys, (i64)blockIdx.x * keys_per_cta), key_end = min(p.num_keys, key_begin + keys_per_cta);
  const unsigned lt = (1u << lane) - 1u;
  uint16_t* my_count = s_count + warp * bins;
  u32 barrier = 0;

  auto load_item = [&](int digit, u32 i) -> u64 {
    if (digit > 0) return __ldcg(p.items[(digit - 1) & 1] + i);
    i64 k = __ldg(p.key + i);
    if ((u64)k >= (u64)p.num_keys) {
      raise_error(p.counters, GSB_ERR_INDEX_RANGE, i);
      k = 0;
    }
    return ((u64)k << 32) | (u64)i;
  };
  // inclusive scan over the CTA of one value per thread, and its total
  auto block_scan = [&](u32 v, u32* total) -> u32 {
    u32 inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    u32 before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kConvWarps; ++w) {
      const u32 t = s_warp[w];
      if (w < warp) before += t;
      all += t;
    }
    *total = all;
    return before + inc;
  };

  // The result of a call that was given up: all edges, in the order of the list, in column 0.
  auto give_up = [&] {
    grid_share(p.E, [&](i64 i) {
      p.out_perm[i] = i;
      p.out_other[i] = __ldg(p.other + i);
    });
    grid_share(p.num_keys, [&](i64 k) { p.out_indptr[k] = k == 0 ? 0 : p.E; });  // the CTA's keys
    if (blockIdx.x == 0) p.out_indptr[p.num_keys] = p.E;
  };

  for (i64 k = key_begin + tid; k < key_end; k += kConvThreads) p.counts[k] = 0;
  for (int digit = 0; digit < p.digits; ++digit) {
    const int shift = 32 + digit * p.digit_bits;
    const u32 mask = (u32)bins - 1;
    // ---- count
    for (int i = tid; i < kConvWarps * bins / 2; i += kConvThreads) reinterpret_cast<u32*>(s_count)[i] = 0;
    __syncthreads();
    for (u32 i0 = begin; i0 < end; i0 += 32) {
      const u32 i = i0 + lane;
      const bool valid = i < end;
      const u32 d = valid ? (u32)(load_item(digit, i) >> shift) & mask : 0;
      const unsigned peers = same_digit(d, p.digit_bits, valid);
      if (valid && (peers & lt) == 0) my_count[d] = (uint16_t)(my_count[d] + __popc(peers));
      __syncwarp();
    }
    __syncthreads();
    for (int b = tid; b < bins; b += kConvThreads) {
      u32 run = 0;
      for (int w0 = 0; w0 < kConvWarps; w0 += 16) {  // counts -> prefixes over the warps
        u32 c[16];
#pragma unroll
        for (int w = 0; w < 16; ++w) c[w] = s_count[(w0 + w) * bins + b];
#pragma unroll
        for (int w = 0; w < 16; ++w) {
          s_count[(w0 + w) * bins + b] = (uint16_t)run;
          run += c[w];
        }
      }
      p.matrix[(size_t)b * ctas + blockIdx.x] = run;
    }
    grid_barrier(p.sync, ++barrier, give_up);
    // ---- scan of the matrix rows; counts per key
    if (ctas <= kConvFewCtas) {  // a row is a few words and there are many rows per warp: a thread per row instead
      for (int b = (int)blockIdx.x * kConvThreads + tid; b < bins; b += ctas * kConvThreads) {
        u32* row = p.matrix + (size_t)b * ctas;
        u32 v[kConvFewCtas], run = 0;
#pragma unroll
        for (int c = 0; c < kConvFewCtas; ++c) v[c] = c < ctas ? __ldcg(row + c) : 0;
#pragma unroll
        for (int c = 0; c < kConvFewCtas; ++c) {
          if (c < ctas) row[c] = run;
          run += v[c];
        }
        p.bin_total[b] = run;
      }
    } else {
      for (int b = (int)blockIdx.x * kConvWarps + warp; b < bins; b += ctas * kConvWarps) {
        u32* row = p.matrix + (size_t)b * ctas;
        u32 carry = 0;
        for (int c0 = 0; c0 < ctas; c0 += 32) {
          const int c = c0 + lane;
          const u32 v = c < ctas ? __ldcg(row + c) : 0;
          u32 inc = v;
  #pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
          }
          if (c < ctas) row[c] = carry + inc - v;
          carry += __shfl_sync(0xffffffffu, inc, 31);
        }
        if (lane == 0) p.bin_total[b] = carry;
      }
    }
    if (digit == 0)
      for (u32 i = begin + lane; i < end; i += 32) {
        const i64 k = __ldg(p.key + i);
        atomicAdd(p.counts + ((u64)k < (u64)p.num_keys ? k : 0), 1u);
      }
    grid_barrier(p.sync, ++barrier, give_up);
    // ---- place
    {
      const int per = bins > kConvThreads ? bins / kConvThreads : 1;  // consecutive digits per thread: 1 or 2
      u32 v[2] = {0, 0}, total;
      for (int j = 0; j < per; ++j)
        if (tid * per + j < bins) v[j] = __ldcg(p.bin_total + tid * per + j);
      u32 run = block_scan(v[0] + v[1], &total) - v[0] - v[1];
      for (int j = 0; j < per; ++j) {
        const int b = tid * per + j;
        if (b < bins) s_start[b] = run + __ldcg(p.matrix + (size_t)b * ctas + blockIdx.x);
        run += v[j];
      }
      __syncthreads();
    }
    const bool last = digit == p.digits - 1;
    for (u32 i0 = begin; i0 < end; i0 += 32) {
      const u32 i = i0 + lane;
      const bool valid = i < end;
      const u64 item = valid ? load_item(digit, i) : 0;
      const u32 d = valid ? (u32)(item >> shift) & mask : 0;
      const unsigned peers = same_digit(d, p.digit_bits, valid);
      u32 base = 0;
      if (valid) base = my_count[d];
      __syncwarp();
      if (valid && (peers & lt) == 0) my_count[d] = (uint16_t)(base + __popc(peers));
      __syncwarp();
      if (valid) {
        const u32 pos = s_start[d] + base + __popc(peers & lt);
        if (last) {
          const u32 e = (u32)item;
          p.out_perm[pos] = (i64)e;
          p.out_other[pos] = __ldg(p.other + e);
        } else {
          p.items[digit & 1][pos] = item;
        }
      }
    }
    // ---- totals of the CTA's keys (their counts are complete since the last barrier)
    if (digit == 0) {
      u32 sum = 0, total;
      for (i64 k = key_begin + tid; k < key_end; k += kConvThreads) sum += __ldcg(p.counts + k);
      block_scan(sum, &total);
      if (tid == 0) p.key_total[blockIdx.x] = total;
    }
    if (!last || digit == 0) grid_barrier(p.sync, ++barrier, give_up);
    if (digit == 0) {  // offsets: the CTA's prefix, then its keys, a thread's share of consecutive ones at a time
      u32 before = 0, total;
      for (int c = tid; c < (int)blockIdx.x; c += kConvThreads) before += __ldcg(p.key_total + c);
      block_scan(before, &total);
      u32 run = total;
      constexpr int kPer = 4;
      for (i64 k0 = key_begin; k0 < key_end; k0 += kConvThreads * kPer) {
        u32 v[kPer], sum = 0, all;
        const i64 mine = k0 + (i64)tid * kPer;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          v[j] = mine + j < key_end ? __ldcg(p.counts + mine + j) : 0;
          sum += v[j];
        }
        u32 at = run + block_scan(sum, &all) - sum;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
          if (mine + j < key_end) p.out_indptr[mine + j] = (i64)at;
          at += v[j];
        }
        run += all;
      }
      if (blockIdx.x == 0 && tid == 0) p.out_indptr[p.num_keys] = p.E;
    }
  }
}

}  // namespace gsb

using namespace gsb;

extern "C" {

int gsb_csc2coo(gsb_ctx* ctx, void* stream_, const int64_t* indptr, int64_t num_cols, int64_t* out_col) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(indptr && num_cols >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (num_cols == 0) return GSB_OK;
  k_csc2coo<<<grid_for(num_cols, kFmtTileCols), kFmtThreads, 0, (cudaStream_t)stream_>>>(indptr, num_cols, out_col);
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 1);
  return GSB_OK;
}

int gsb_coo2csc(gsb_ctx* ctx, void* stream_, const int64_t* key, const int64_t* other, int64_t E, int64_t num_keys,
                int key_sorted, int64_t* out_indptr, int64_t* out_other, int64_t* out_perm) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(out_indptr && E >= 0 && num_keys >= 0, GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(E == 0 || (key && other && out_other), GSB_ERR_INVALID_ARGUMENT);
  GSB_REQUIRE(key_sorted || E == 0 || out_perm, GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  const int grid = min(grid_for(E, kFmtThreads), kNumSMs * 8);
  int bits = 1;
  while (bits < 63 && (1ll << bits) < num_keys) ++bits;
  if (!key_sorted && E > 0 && E <= kShortMaxEdges && num_keys > 0 && num_keys <= kShortMaxKeys) {
    static bool attr_set[64];
    const int dev = ctx_device(ctx);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      GSB_CUDA_OK(cudaFuncSetAttribute(k_coo2csc_short, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)short_smem(short_shape(kShortMaxEdges, kShortMaxKeys))));
      attr_set[dev] = true;
    }
    const ShortShape shape = short_shape(E, num_keys);
    ScopedKernelTimer timer(ctx, KID_FORMAT, stream);
    k_coo2csc_short<<<(int)shape.grid, kShortThreads, short_smem(shape), stream>>>(key, other, (u32)E, num_keys, shape, out_indptr,
                                                                                  out_other, out_perm, ctx_counters(ctx));
    GSB_LAUNCH_OK();
    return GSB_OK;
  }
  // One cooperative launch while a warp's share of the edges fits its 16-bit counts (and keys fit three digits);
  // beyond that the passes are long enough for launches of their own.
  if (!key_sorted && E > 0 && E <= kConvMaxEdges && bits <= 32 && num_keys > 0) {
    ConvParams p{};
    p.digits = (bits + 10) / 11;
    p.digit_bits = max(5, (bits + p.digits - 1) / p.digits);
    const int bins = 1 << p.digit_bits;
    const size_t smem = sizeof(uint16_t) * (size_t)kConvWarps * (size_t)bins;
    static int resident[64];
    static bool attr_set[64];
    const int dev = ctx_device(ctx);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      GSB_CUDA_OK(cudaFuncSetAttribute(k_coo2csc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)(sizeof(uint16_t) * kConvWarps * kConvMaxBins)));
      attr_set[dev] = true;
    }
    const int ctas = min(kNumSMs, ctx_resident_ctas(ctx, (const void*)k_coo2csc, kConvThreads,
                                                    sizeof(uint16_t) * kConvWarps * kConvMaxBins, resident));
    // two items per thread at least: fewer CTAs make the barriers and the matrix of a short list cheaper; the offsets of a
    // long key range want CTAs too
    const i64 want = max((E + 2 * kConvThreads - 1) / (2 * kConvThreads), num_keys / (4 * kConvThreads));
    const int conv_grid = (int)max((i64)1, min((i64)ctas, want));
    if (ctas > 0 && (E + conv_grid - 1) / conv_grid + 32 * kConvWarps <= 65535ll) {
      auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
      const size_t item_bytes = p.digits > 1 ? al(sizeof(u64) * (size_t)E) : 0;
      const size_t matrix_bytes = al(sizeof(u32) * (size_t)bins * (size_t)conv_grid);
      void* ws;
      int st = ctx_reserve_workspace(ctx, stream, item_bytes * (p.digits > 2 ? 2 : 1) + matrix_bytes + al(sizeof(u32) * (size_t)bins) +
                                              al(sizeof(u32) * (size_t)num_keys) + 4096, &ws);
      if (st != GSB_OK) return st;
      char* at = (char*)ws;
      p.items[0] = (u64*)at;
      p.items[1] = (u64*)(at + (p.digits > 2 ? item_bytes : 0));
      at += item_bytes * (p.digits > 2 ? 2 : 1);
      p.matrix = (u32*)at;
      at += matrix_bytes;
      p.bin_total = (u32*)at;
      at += al(sizeof(u32) * (size_t)bins);
      p.key_total = (u32*)at;
      at += 4096;
      p.counts = (u32*)at;
      p.key = key;
      p.other = other;
      p.E = E;
      p.num_keys = num_keys;
      p.out_indptr = out_indptr;
      p.out_other = out_other;
      p.out_perm = out_perm;
      p.counters = ctx_counters(ctx);
      p.sync = ctx_grid_sync(ctx, conv_grid, p.digits == 1 ? 3 : 3 * p.digits - 1);
      ScopedKernelTimer timer(ctx, KID_FORMAT, stream);
      void* args[] = {&p};
      return launch_cooperative(ctx, stream, (const void*)k_coo2csc, conv_grid, kConvThreads, smem, args, p.sync);
    }
  }
  GSB_CUDA_OK(cudaMemsetAsync(out_indptr, 0, sizeof(i64) * (size_t)(num_keys + 1), stream));
  if (E > 0) {
    k_count_keys<<<grid, kFmtThreads, 0, stream>>>(key, E, num_keys, out_indptr, ctx_counters(ctx));
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
  }
  int st = exclusive_scan_i64(ctx, stream, out_indptr, num_keys);
  if (st != GSB_OK) return st;
  if (E == 0) return GSB_OK;
  if (key_sorted) {
    k_conversion_end<<<grid, kFmtThreads, 0, stream>>>(other, nullptr, E, num_keys, out_indptr, out_other, ctx_counters(ctx));
    GSB_LAUNCH_OK();
    ctx_count_launches(ctx, 1);
    return GSB_OK;
  }
  void* ws;
  const size_t sort_bytes = radix_sort_scratch_bytes(E);
  st = ctx_reserve_workspace(ctx, stream, sort_bytes + sizeof(u64) * (size_t)E + 256, &ws);
  if (st != GSB_OK) return st;
  u64* keys = (u64*)((char*)ws + sort_bytes);
  k_make_sort_input<<<grid, kFmtThreads, 0, stream>>>(key, E, keys, out_perm);
  GSB_LAUNCH_OK();
  st = radix_sort_pairs(ctx, stream, keys, out_perm, E, 0, bits, ws);
  if (st != GSB_OK) return st;
  k_conversion_end<<<grid, kFmtThreads, 0, stream>>>(other, out_perm, E, num_keys, out_indptr, out_other, ctx_counters(ctx));
  GSB_LAUNCH_OK();
  ctx_count_launches(ctx, 2);
  return GSB_OK;
}

}  // extern "C"
