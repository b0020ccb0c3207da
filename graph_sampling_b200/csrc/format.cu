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
// The keys of up to 26 624 edges are read from L2 by EVERY CTA (213 KB at most; 6 us for the 25 000 edges of a layer-wise
// minibatch), which needs nothing from the others then: a CTA owns a range of keys, counts the edges with smaller keys (where
// its output starts) and keeps, in order, those of its range; counts per key, their scan (the offsets) and the stable placing, a
// warp per part of the range, happen in shared memory.  A CTA with many edges, whose keys may well be the same, sorts them by two
// digits instead, every warp a part of them.  The cooperative form below, with five grid barriers and 65 536 counters to clear
// and sum up per CTA and digit, takes 42 us for 25 000 edges over a million keys and 17 us for 700 over a thousand, this 16.4 and
// 8.9 (calls in a row); 37 when the keys crowd at one end of their range, as those of a power law do whose ids are sorted by
// degree, and 29 % of the edges are one CTA's.
constexpr int kShortThreads = 1024;
constexpr int kShortWarps = kShortThreads / 32;
constexpr int kKeysAhead = 12;  // keys, and placed edges, of a thread on their way
constexpr int kShortAhead = 8;
// At this many edges the two forms are equal where the keys crowd as those of a power law whose ids are sorted by degree; with keys
// spread evenly this form takes 16.7 us at 32 700 edges, the other 35 to 42.
constexpr i64 kShortMaxEdges = 26624;
constexpr u32 kShortHeavy = 1024;  // edges of a CTA from which every warp places a part of them
constexpr int kShortDigitBits = 7;
constexpr i64 kShortMaxKeys = 8192;  // of a CTA
constexpr size_t short_smem(i64 E, i64 keys) { return 4 * (size_t)keys + 4 * (size_t)((E + 1) & ~1ll); }

__global__ void __launch_bounds__(kShortThreads, 1) k_coo2csc_short(const i64* __restrict__ key, const i64* __restrict__ other,
                                                                   u32 E, i64 num_keys, u32 keys_per_cta,
                                                                   i64* __restrict__ out_indptr, i64* __restrict__ out_other,
                                                                   i64* __restrict__ out_perm,
                                                                   uint16_t* __restrict__ scratch, i64* counters) {
  extern __shared__ __align__(16) u32 s_start[];  // [keys] counts, then where the next edge of the key goes
  uint16_t* s_rel = reinterpret_cast<uint16_t*>(s_start + keys_per_cta);  // [E] key relative to the range, or kOutside
  uint16_t* s_list = s_rel + ((E + 1) & ~1u);                             // [E] the edges of the range, in order
  __shared__ u32 s_warp[2][kShortWarps];
  constexpr u32 kOutside = 0xFFFFu;
  const u32 tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, lt = (1u << lane) - 1u;
  const i64 key_begin = (i64)blockIdx.x * keys_per_cta;
  const u32 keys = (u32)max((i64)0, min((i64)keys_per_cta, num_keys - key_begin));
  const u32 per_warp = (E + kShortThreads - 1) / kShortThreads * 32;
  const u32 begin = min(E, warp * per_warp), end = min(E, begin + per_warp);
  for (u32 k = tid; k < keys; k += kShortThreads) s_start[k] = 0;
  __syncthreads();
  u32 below = 0, inside = 0;  // of the lane's edges
  for (u32 i0 = begin + lane; i0 < end; i0 += 32 * kKeysAhead) {
    i64 k[kKeysAhead];
#pragma unroll
    for (int q = 0; q < kKeysAhead; ++q) k[q] = i0 + 32 * q < end ? __ldg(key + i0 + 32 * q) : num_keys;
#pragma unroll
    for (int q = 0; q < kKeysAhead; ++q) {
      const u32 i = i0 + 32 * q;
      if (i >= end) break;
      if ((u64)k[q] >= (u64)num_keys) {
        if (blockIdx.x == 0) raise_error(counters, GSB_ERR_INDEX_RANGE, i);
        k[q] = 0;
      }
      const i64 rel = k[q] - key_begin;
      const bool in = (u64)rel < (u64)keys;
      s_rel[i] = in ? (uint16_t)rel : (uint16_t)kOutside;
      if (in) atomicAdd(s_start + rel, 1u);
      inside += in;
      below += rel < 0;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    inside += __shfl_xor_sync(0xffffffffu, inside, o);
    below += __shfl_xor_sync(0xffffffffu, below, o);
  }
  if (lane == 0) {
    s_warp[0][warp] = inside;
    s_warp[1][warp] = below;
  }
  __syncthreads();
  u32 at = 0, total = 0;
  below = 0;
#pragma unroll
  for (u32 w = 0; w < kShortWarps; ++w) {
    if (w < warp) at += s_warp[0][w];
    total += s_warp[0][w];
    below += s_warp[1][w];
  }
  if (inside > 0)  // (the whole warp's)
    for (u32 i0 = begin; i0 < end; i0 += 32) {
      const bool in = i0 + lane < end && s_rel[i0 + lane] != kOutside;
      const unsigned bits = __ballot_sync(0xffffffffu, in);
      if (in) s_list[at + __popc(bits & lt)] = (uint16_t)(i0 + lane);
      at += __popc(bits);
    }
  // offsets: a stretch of keys per thread, eight at most
  {
    constexpr u32 kPer = kShortMaxKeys / kShortThreads;
    const u32 per = (keys + kShortThreads - 1) / kShortThreads, first = tid * per;
    u32 v[kPer], sum = 0;
#pragma unroll
    for (u32 j = 0; j < kPer; ++j) {
      v[j] = j < per && first + j < keys ? s_start[first + j] : 0;
      sum += v[j];
    }
    u32 inc = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    __syncthreads();  // s_warp has been read
    if (lane == 31) s_warp[0][warp] = inc;
    __syncthreads();
    u32 run = inc - sum;
#pragma unroll
    for (u32 w = 0; w < kShortWarps; ++w)
      if (w < warp) run += s_warp[0][w];
#pragma unroll
    for (u32 j = 0; j < kPer; ++j) {
      if (j < per && first + j < keys) s_start[first + j] = run;
      run += v[j];
    }
    __syncthreads();
    for (u32 k = tid; k < keys; k += kShortThreads) out_indptr[key_begin + k] = (i64)(below + s_start[k]);
    if (blockIdx.x == 0 && tid == 0) out_indptr[num_keys] = (i64)E;
    __syncthreads();
  }
  // the edges in their new order, placed by the two ways below; the outputs follow from it in one go (a warp that wrote them while
  // placing waited for a random read every 32 edges)
  constexpr u32 kDigits = 1u << kShortDigitBits;
  __shared__ uint16_t s_digit[kShortWarps][kDigits];  // of a warp's part, then where its next edge of the digit goes
  __shared__ u32 s_digit_start[kDigits];
  static_assert(kShortWarps * kDigits >= kShortHeavy, "the order of a light CTA takes the place of the digits");
  uint16_t* order = &s_digit[0][0];
  if (total >= kShortHeavy) {  // a stable counting sort by one or two digits of the key
    const u32 share = (total + kShortThreads - 1) / kShortThreads * 32;
    const u32 lo = min(total, warp * share), hi = min(total, lo + share);
    const int key_bits = keys > 1 ? 32 - __clz(keys - 1) : 0, passes = key_bits > kShortDigitBits ? 2 : 1;
    uint16_t* second = 2 * total <= E ? s_list + total : scratch + below;
    for (int pass = 0; pass < passes; ++pass) {
      const uint16_t* list = pass == 0 ? s_list : second;
      order = pass == 0 ? second : s_list;
      const int bits = pass == 0 ? min(key_bits, kShortDigitBits) : key_bits - kShortDigitBits;
      auto digit_of = [&](u32 e) { return ((u32)s_rel[e] >> (pass * kShortDigitBits)) & (kDigits - 1); };
      for (u32 d = lane; d < kDigits; d += 32) s_digit[warp][d] = 0;
      __syncwarp();
#pragma unroll 4
      for (u32 j0 = lo; j0 < hi; j0 += 32) {
        const bool valid = j0 + lane < hi;
        const u32 d = valid ? digit_of(list[j0 + lane]) : 0;
        const unsigned peers = same_digit(d, bits, valid);
        if (valid && (peers & lt) == 0) s_digit[warp][d] += (uint16_t)__popc(peers);
        __syncwarp();
      }
      __syncthreads();
      if (tid < kDigits) {
        u32 run = 0;
        for (u32 w = 0; w < kShortWarps; ++w) {
          const u32 c = s_digit[w][tid];
          s_digit[w][tid] = (uint16_t)run;
          run += c;
        }
        s_digit_start[tid] = run;
      }
      __syncthreads();
      if (warp == 0) {
        u32 carry = 0;
        for (u32 d0 = 0; d0 < kDigits; d0 += 32) {
          const u32 c = s_digit_start[d0 + lane];
          u32 inc = c;
#pragma unroll
          for (int o = 1; o < 32; o <<= 1) {
            const u32 t = __shfl_up_sync(0xffffffffu, inc, o);
            if (lane >= o) inc += t;
          }
          s_digit_start[d0 + lane] = carry + inc - c;
          carry += __shfl_sync(0xffffffffu, inc, 31);
        }
      }
      __syncthreads();
      for (u32 j0 = lo; j0 < hi; j0 += 32) {
        const bool valid = j0 + lane < hi;
        const u32 e = valid ? list[j0 + lane] : 0, d = valid ? digit_of(e) : 0;
        const unsigned peers = same_digit(d, bits, valid);
        u32 pos = 0;
        if (valid) pos = s_digit[warp][d];
        __syncwarp();
        if (valid && (peers & lt) == 0) s_digit[warp][d] = (uint16_t)(pos + __popc(peers));
        __syncwarp();
        if (valid) order[pos + s_digit_start[d] + __popc(peers & lt)] = (uint16_t)e;
      }
      __syncthreads();  // the other list is complete
    }
  } else {  // a warp takes the edges of its part of the range, in order
    const u32 part = (keys + kShortWarps - 1) / kShortWarps, part_begin = warp * part;
    const u32 part_keys = min(part, keys - min(keys, part_begin));
    for (u32 j0 = 0; j0 < total && part_keys > 0; j0 += 32) {
      const u32 e = j0 + lane < total ? s_list[j0 + lane] : 0;
      const u32 rel = s_rel[e];
      const bool mine = j0 + lane < total && rel - part_begin < part_keys;
      if (!__any_sync(0xffffffffu, mine)) continue;
      const unsigned peers = __match_any_sync(0xffffffffu, mine ? rel : kOutside);
      u32 pos = 0;
      if (mine) pos = s_start[rel];
      __syncwarp();
      if (mine && (peers & lt) == 0) s_start[rel] = pos + __popc(peers);
      __syncwarp();
      if (mine) order[pos + __popc(peers & lt)] = (uint16_t)e;
    }
    __syncthreads();
  }
  for (u32 j0 = tid; j0 < total; j0 += kShortThreads * kShortAhead) {
    u32 e[kShortAhead];
    i64 o[kShortAhead];
#pragma unroll
    for (int q = 0; q < kShortAhead; ++q) e[q] = j0 + q * kShortThreads < total ? order[j0 + q * kShortThreads] : 0;
#pragma unroll
    for (int q = 0; q < kShortAhead; ++q)
      if (j0 + q * kShortThreads < total) o[q] = __ldg(other + e[q]);
#pragma unroll
    for (int q = 0; q < kShortAhead; ++q) {
      const u32 j = j0 + q * kShortThreads;
      if (j >= total) break;
      out_perm[below + j] = (i64)e[q];
      out_other[below + j] = o[q];
    }
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
  if (!key_sorted && E > 0 && E <= kShortMaxEdges && num_keys > 0 && num_keys <= kShortMaxKeys * kNumSMs) {
    static bool attr_set[64];
    const int dev = ctx_device(ctx);
    if (dev >= 0 && dev < 64 && !attr_set[dev]) {
      GSB_CUDA_OK(cudaFuncSetAttribute(k_coo2csc_short, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)short_smem(kShortMaxEdges, kShortMaxKeys)));
      attr_set[dev] = true;
    }
    const u32 keys_per_cta = (u32)((num_keys + kNumSMs - 1) / kNumSMs);
    void* scratch;
    const int st = ctx_reserve_workspace(ctx, stream, sizeof(uint16_t) * (size_t)E, &scratch);
    if (st != GSB_OK) return st;
    ScopedKernelTimer timer(ctx, KID_FORMAT, stream);
    k_coo2csc_short<<<grid_for(num_keys, (int)keys_per_cta), kShortThreads, short_smem(E, keys_per_cta), stream>>>(
        key, other, (u32)E, num_keys, keys_per_cta, out_indptr, out_other, out_perm, (uint16_t*)scratch, ctx_counters(ctx));
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
