// Per-segment reductions over edge data: sum of data^powk per column (CSC / CSR view) or per
// target node (COO), and per-segment normalisation.
//
// One warp per segment with a shuffle reduction (the reference gives each segment to one thread
// that loops over it serially: src/cuda/graph_ops.cu:15-39, 131-158).  powk is applied by repeated
// multiplication, i.e. exact integer powers (the reference's __powf is an approximation and is NaN
// for negative bases).  The COO form accumulates with float atomics into a zero-initialised dense
// vector, like the reference's _SegmentSumCOOKernel (:44-64); its summation order is not fixed.
#include <type_traits>

#include "common.cuh"

namespace gsb {

constexpr int kSegThreads = 256;
constexpr int kSegWarps = kSegThreads / 32;
// Segments longer than this are taken by a whole CTA: with power-law degrees a single hub column would otherwise keep one
// warp busy for hundreds of iterations while the rest of the grid has long finished.
constexpr i64 kLongSegment = 2048;

__device__ __forceinline__ float int_pow(float x, i64 powk) {
  if (powk == 1) return x;
  float r = 1.0f;
  for (i64 i = 0; i < powk; ++i) r *= x;
  return r;
}

constexpr i64 kSegSteps = 8192;  // warps get several segments a step when there are more than this many steps
// edges from which on a warp keeps several loads ahead within one segment
template <bool NORMALIZE>
constexpr int kSegMany = NORMALIZE ? 128 : 192;

// One segment by `width` threads, thread `first` of them: loads kAhead elements before the first is used (with one element per
// iteration a warp waited out a memory round trip per 32 edges), and keeps them in registers when that is the whole segment,
// so that a normalisation reads its data once.  1.2 M edges in 2 048 columns: 45 us with a remainder loop of single loads and 80
// registers a thread (28 % of the warps resident), 12.5 us now.
template <bool NORMALIZE, bool IDS>
struct SegmentReader {
  static constexpr int kAhead = IDS ? 4 : 8;  // more ids would not fit the registers of five CTAs per SM
  const i64* e_ids;
  const float* data;
  i64 powk;
  float v[kAhead];

  __device__ __forceinline__ float value(i64 j) const {
    if (NORMALIZE) return __ldg(data + j);
    return int_pow(data ? __ldg(data + j) : 1.0f, powk);
  }
  __device__ __forceinline__ void load(i64 b, i64 j, i64 len, int width) {
    if (IDS) {
      i64 at[kAhead];
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (j + q * width < len) at[q] = __ldg(e_ids + b + j + q * width);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) v[q] = j + q * width < len ? value(at[q]) : 0.f;
    } else {
#pragma unroll
      for (int q = 0; q < kAhead; ++q) v[q] = j + q * width < len ? value(b + j + q * width) : 0.f;
    }
  }
  __device__ __forceinline__ float sum(i64 b, i64 len, int first, int width) {
    if (len <= width) {  // most of a warp's segments
      v[0] = first < len ? value(IDS ? __ldg(e_ids + b + first) : b + first) : 0.f;
      return v[0];
    }
    float acc = 0.f;
    for (i64 j = first; j < len; j += kAhead * width) {
      load(b, j, len, width);
#pragma unroll
      for (int q = 0; q < kAhead; ++q) acc += v[q];
    }
    return acc;
  }
  __device__ __forceinline__ void divide(i64 b, i64 len, int first, int width, float total, float* __restrict__ out) {
    for (i64 j = first; j < len; j += kAhead * width) {
      if (len > kAhead * width) load(b, j, len, width);  // else they are still in v
#pragma unroll
      for (int q = 0; q < kAhead; ++q)
        if (j + q * width < len) out[IDS ? __ldg(e_ids + b + j + q * width) : b + j + q * width] = v[q] / total;
    }
  }
};

// NORMALIZE: out[j] = data[j] / (sum of its segment); otherwise out[s] = sum of data^powk over segment s.  One launch, three forms:
//   a CTA per segment where they average at least 128 edges (a warp each would leave few warps with everything, and a CTA that
//   meets several hubs does them one after the other);
//   a warp for several segments: up to 16 consecutive ones a step, whose bounds are one load that is asked for a step ahead, two
//   of them side by side, and those with many edges afterwards, one by one with more loads ahead.  Few segments get a warp each;
//   sums of segments that average less than four edges, as in the row view of a slice: 32 a step, lane i reads the bounds of
//   segment s0 + i, sums it itself if it has at most four edges, and the others are summed by the whole warp one after the other.
//   (One warp per segment spent a step, with two dependent loads, on every empty row: 78 us for the 1 M rows of a slice with
//   25 000 edges.)  The short form adds in the order the tree would, (v0 + v2) + (v1 + v3), so a segment's sum does not depend
//   on which form took it.
// Segments too long for a warp are set aside for the whole CTA, when its warps are done with the others.
// What bounds the second form is instruction issue and the warps in flight, and the registers are cut to what that takes (7, 7, 6
// and 4 CTAs per SM; fewer spilled bytes and fewer warps are slower, sums of a million segments 147 us at six).  A million segments
// of 30 edges: sum 129 us with a warp per segment in a kernel of its own, 353 with barriers around every eight segments, 119 now;
// normalised 187, 273, 137.  262 144 of 51: sum 46, 78, 39 us; normalised 63, 74, 64; by edge ids 98, 159, 100.
template <bool NORMALIZE, bool IDS>
__global__ void __launch_bounds__(kSegThreads, !NORMALIZE ? 7 : IDS ? 4 : 6) k_segments(const i64* __restrict__ indptr, i64 num_seg,
                                                             const i64* __restrict__ e_ids, const float* __restrict__ data,
                                                             i64 powk, float* __restrict__ out) {
  __shared__ i64 s_long[kSegThreads];
  __shared__ int s_num_long;  // long segments met by the CTA's warps
  __shared__ float s_part[kSegWarps];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  SegmentReader<NORMALIZE, IDS> reader{e_ids, data, powk};
  auto warp_segment = [&](i64 s, i64 b, i64 e) {
    const i64 len = e - b;
    float acc = reader.sum(b, len, lane, 32);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (NORMALIZE) reader.divide(b, len, lane, 32, acc, out);
    else if (lane == 0) out[s] = acc;
  };
  auto cta_segment = [&](i64 s) {
    const i64 b = __ldg(indptr + s);
    const i64 len = __ldg(indptr + s + 1) - b;
    float acc = reader.sum(b, len, threadIdx.x, kSegThreads);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) s_part[warp] = acc;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int w = 0; w < kSegWarps; ++w) total += s_part[w];
    if (NORMALIZE) reader.divide(b, len, threadIdx.x, kSegThreads, total, out);
    else if (threadIdx.x == 0) out[s] = total;
    __syncthreads();
  };
  const i64 mean = (__ldg(indptr + num_seg) - __ldg(indptr)) / num_seg;
  if (mean >= 128) {
    for (i64 s = blockIdx.x; s < num_seg; s += gridDim.x) cta_segment(s);
    return;
  }
  const bool sparse = !NORMALIZE && mean < 4;
  if (threadIdx.x == 0) s_num_long = 0;
  __syncthreads();
  auto set_aside = [&](i64 s) {
    const int at = atomicAdd(&s_num_long, 1);
    if (at < kSegThreads) s_long[at] = s;
  };
  const i64 first = (i64)blockIdx.x * kSegWarps + warp, warps = (i64)gridDim.x * kSegWarps;
  int per = sparse ? 32 : 1;  // consecutive segments per warp and step: their bounds are one load, asked for a step ahead
  if (!sparse) {
    while (per < 16 && num_seg >= 2ll * per * kSegSteps) per *= 2;
    if (per == 1) {
      for (i64 s = first; s < num_seg; s += warps) {
        const i64 b = __ldg(indptr + s), e = __ldg(indptr + s + 1);
        if (e - b <= kLongSegment) warp_segment(s, b, e);
        else if (lane == 0) set_aside(s);
      }
    }
    auto bounds = [&](i64 s0) { return lane <= per && s0 < num_seg ? __ldg(indptr + min(s0 + lane, num_seg)) : 0; };
    i64 ahead = bounds(first * per);
    for (i64 s0 = first * per; per > 1 && s0 < num_seg; s0 += warps * per) {
      const i64 base = __shfl_sync(0xffffffffu, ahead, 0);
      const int start = (int)min(ahead - base, (i64)1 << 30);  // of the lane's segment, relative to the first one's
      ahead = bounds(s0 + warps * per);
      const int count = (int)min((i64)per, num_seg - s0);
      if (__shfl_sync(0xffffffffu, start, count) == 1 << 30) {  // not in 32 bits
        if (lane < count) set_aside(s0 + lane);
        continue;
      }
      const i64* ids = IDS ? e_ids + base : nullptr;
      const float* from = data && !IDS ? data + base : data;
      using Place = typename std::conditional<IDS, i64, int>::type;
      auto place = [&](int i) -> Place { return IDS ? (Place)__ldg(ids + i) : (Place)i; };
      auto value_at = [&](Place at) {
        const float x = NORMALIZE || data ? __ldg(from + at) : 1.0f;
        return NORMALIZE ? x : int_pow(x, powk);
      };
      unsigned many = 0;  // segments that are worth more loads ahead
      for (int j = 0; j < count; j += 2) {  // two side by side: their loads and their trees overlap
        int b[2], len[2];
        Place at[2];
        float v[2], acc[2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int k = min(j + u, count);
          b[u] = __shfl_sync(0xffffffffu, start, k);
          len[u] = __shfl_sync(0xffffffffu, start, min(k + 1, count)) - b[u];
          if (len[u] > kSegMany<NORMALIZE>) {
            many |= 1u << k;
            len[u] = -1;
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) at[u] = lane < len[u] ? place(b[u] + lane) : 0;
#pragma unroll
        for (int u = 0; u < 2; ++u) acc[u] = v[u] = lane < len[u] ? value_at(at[u]) : 0.f;
#pragma unroll
        for (int u = 0; u < 2; ++u)
          for (int i = 32 + lane; i < len[u]; i += 32) acc[u] += value_at(place(b[u] + i));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
          for (int u = 0; u < 2; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], o);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (NORMALIZE) {
            float* to = IDS ? out : out + base;
            if (lane < len[u]) to[at[u]] = v[u] / acc[u];
            for (int i = 32 + lane; i < len[u]; i += 32) {
              const Place k = place(b[u] + i);
              to[k] = value_at(k) / acc[u];
            }
          } else if (lane == u && len[u] >= 0 && j + u < count) {
            out[s0 + j + u] = acc[u];
          }
        }
      }
      while (many) {
        const int k = __ffs(many) - 1;
        many &= many - 1;
        const int b = __shfl_sync(0xffffffffu, start, k), e = __shfl_sync(0xffffffffu, start, k + 1);
        if (e - b <= kLongSegment) warp_segment(s0 + k, base + b, base + e);
        else if (lane == 0) set_aside(s0 + k);
      }
    }
  } else {
    for (i64 s0 = first * 32; s0 < num_seg; s0 += warps * 32) {
      const i64 s = s0 + lane;
      i64 b = 0, e = 0;
      if (s < num_seg) {
        b = __ldg(indptr + s);
        e = __ldg(indptr + s + 1);
      }
      const i64 len = e - b;
      auto value = [&](i64 j) { return reader.value(IDS ? __ldg(e_ids + j) : j); };
      // the loads of a short segment are issued now and used after the warp-wide part, which hides their latency
      const bool is_short = s < num_seg && len <= 4;
      float v0 = 0.f, v1 = 0.f, v2 = 0.f, v3 = 0.f;
      if (is_short) {
        if (len > 0) v0 = value(b);
        if (len > 1) v1 = value(b + 1);
        if (len > 2) v2 = value(b + 2);
        if (len > 3) v3 = value(b + 3);
      }
      if (len > kLongSegment) set_aside(s);
      unsigned medium = __ballot_sync(0xffffffffu, len > 4 && len <= kLongSegment);
      while (medium) {
        const int src = __ffs(medium) - 1;
        medium &= medium - 1;
        warp_segment(s0 + src, __shfl_sync(0xffffffffu, b, src), __shfl_sync(0xffffffffu, e, src));
      }
      if (is_short) out[s] = (v0 + v2) + (v1 + v3);
    }
  }
  __syncthreads();
  const int num_long = s_num_long;
  if (num_long <= kSegThreads) {
    for (int q = 0; q < num_long; ++q) cta_segment(s_long[q]);
    return;
  }
  for (i64 s0 = first - warp; s0 * per < num_seg; s0 += warps) {  // more than the list holds: the CTA's segments once more
    for (i64 step = s0 * per; step < min(num_seg, (s0 + kSegWarps) * per); step += per) {
      const i64 end = min(num_seg, step + per);
      const bool wide = !sparse && __ldg(indptr + end) - __ldg(indptr + step) >= (i64)1 << 30;
      for (i64 s = step; s < end; ++s)
        if (wide || __ldg(indptr + s + 1) - __ldg(indptr + s) > kLongSegment) cta_segment(s);
    }
  }
}

// FOLD = false: one float atomic per edge (scattered targets).  FOLD = true, for targets that come in runs (a
// column-sorted COO summed per column has 32 equal targets in a row): lanes with the same target add once, in lane
// order — one atomic per distinct target of the warp; a warp without a repeat next door skips the fold.
template <bool FOLD>
__global__ void __launch_bounds__(kSegThreads) k_segment_sum_coo(const i64* __restrict__ target, i64 E,
                                                                 const i64* __restrict__ e_ids,
                                                                 const float* __restrict__ data, i64 powk,
                                                                 float* __restrict__ out) {
  if (!FOLD) {
    for (i64 e = (i64)blockIdx.x * kSegThreads + threadIdx.x; e < E; e += (i64)gridDim.x * kSegThreads) {
      const float x = data ? __ldg(data + (e_ids ? __ldg(e_ids + e) : e)) : 1.0f;
      atomicAdd(out + __ldg(target + e), int_pow(x, powk));
    }
    return;
  }
  const int lane = threadIdx.x & 31;
  for (i64 e0 = (i64)blockIdx.x * kSegThreads + threadIdx.x - lane; e0 < E; e0 += (i64)gridDim.x * kSegThreads) {
    const i64 e = e0 + lane;
    const bool valid = e < E;
    const i64 t = valid ? __ldg(target + e) : -1 - lane;  // distinct dummies: lanes past the end pair with nobody
    const float v = valid ? int_pow(data ? __ldg(data + (e_ids ? __ldg(e_ids + e) : e)) : 1.0f, powk) : 0.0f;
    const int prev_t = __shfl_up_sync(0xffffffffu, (int)t, 1);  // low words: a false match only takes the fold
    if (!__any_sync(0xffffffffu, lane > 0 && prev_t == (int)t)) {
      if (valid) atomicAdd(out + t, v);
      continue;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, t);
    float sum = 0.0f;
    for (int src = 0; src < 32; ++src) {
      const float other = __shfl_sync(0xffffffffu, v, src);
      if ((peers >> src) & 1u) sum += other;
    }
    if (valid && lane == __ffs(peers) - 1) atomicAdd(out + t, sum);
  }
}

// out_data[e] = data[e] / divisor[row[e]] and out_sum[col[e]] += out_data[e] in one pass over the edges
// (gs::impl::fusion::COOEDivUSum, src/cuda/fusion/edge_map_reduce.cu:10-24).
__global__ void __launch_bounds__(kSegThreads) k_edge_div_u_sum(const i64* __restrict__ row,
                                                                const i64* __restrict__ col, i64 E,
                                                                const float* __restrict__ data,
                                                                const float* __restrict__ divisor,
                                                                float* __restrict__ out_data,
                                                                float* __restrict__ out_sum) {
  const int lane = threadIdx.x & 31;
  for (i64 e0 = (i64)blockIdx.x * kSegThreads + threadIdx.x - lane; e0 < E; e0 += (i64)gridDim.x * kSegThreads) {
    const i64 e = e0 + lane;
    const bool valid = e < E;
    float v = 0.0f;
    i64 t = -1 - lane;
    if (valid) {
      v = __fdiv_rn(data ? __ldg(data + e) : 1.0f, __ldg(divisor + __ldg(row + e)));
      out_data[e] = v;
      t = __ldg(col + e);
    }
    // as in k_segment_sum_coo: one atomic per distinct column of the warp when columns repeat next door
    const int prev_t = __shfl_up_sync(0xffffffffu, (int)t, 1);  // low words: a false match only takes the fold
    if (!__any_sync(0xffffffffu, lane > 0 && prev_t == (int)t)) {
      if (valid) atomicAdd(out_sum + t, v);
      continue;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, t);
    float sum = v;
    if (__any_sync(0xffffffffu, valid && __popc(peers) > 1)) {
      sum = 0.0f;
      for (int src = 0; src < 32; ++src) {
        const float other = __shfl_sync(0xffffffffu, v, src);
        if ((peers >> src) & 1u) sum += other;
      }
    }
    if (valid && lane == __ffs(peers) - 1) atomicAdd(out_sum + t, sum);
  }
}

// Grid of k_segments, whose step the device chooses: a CTA per segment, up to 16 per SM.
static inline int segments_grid(i64 num_seg) { return (int)min(num_seg, (i64)kNumSMs * 16); }

}  // namespace gsb

using namespace gsb;

extern "C" {

int gsb_segment_sum_csc(gsb_ctx* ctx, void* stream_, const int64_t* indptr, int64_t num_seg, const int64_t* e_ids,
                        const float* data, int64_t powk, float* out) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(num_seg >= 0 && powk >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (num_seg == 0) return GSB_OK;
  GSB_REQUIRE(indptr && out, GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  {
    ScopedKernelTimer timer(ctx, KID_SEGMENT, stream);
    if (e_ids) k_segments<false, true><<<segments_grid(num_seg), kSegThreads, 0, stream>>>(indptr, num_seg, e_ids, data, powk, out);
    else k_segments<false, false><<<segments_grid(num_seg), kSegThreads, 0, stream>>>(indptr, num_seg, e_ids, data, powk, out);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int gsb_segment_sum_coo(gsb_ctx* ctx, void* stream_, const int64_t* target, int64_t E, const int64_t* e_ids,
                        const float* data, int64_t powk, int targets_in_runs, float* out_zeroed) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(E >= 0 && powk >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (E == 0) return GSB_OK;
  GSB_REQUIRE(target && out_zeroed, GSB_ERR_INVALID_ARGUMENT);
  const int grid = min(grid_for(E, kSegThreads), kNumSMs * 16);
  {
    ScopedKernelTimer timer(ctx, KID_SEGMENT, (cudaStream_t)stream_);
    if (targets_in_runs)
      k_segment_sum_coo<true><<<grid, kSegThreads, 0, (cudaStream_t)stream_>>>(target, E, e_ids, data, powk, out_zeroed);
    else
      k_segment_sum_coo<false><<<grid, kSegThreads, 0, (cudaStream_t)stream_>>>(target, E, e_ids, data, powk, out_zeroed);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int gsb_segment_normalize_csc(gsb_ctx* ctx, void* stream_, const int64_t* indptr, int64_t num_seg,
                              const int64_t* e_ids, const float* data, float* out) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(num_seg >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (num_seg == 0) return GSB_OK;
  GSB_REQUIRE(indptr && data && out, GSB_ERR_INVALID_ARGUMENT);
  cudaStream_t stream = (cudaStream_t)stream_;
  {
    ScopedKernelTimer timer(ctx, KID_SEGMENT, stream);
    if (e_ids) k_segments<true, true><<<segments_grid(num_seg), kSegThreads, 0, stream>>>(indptr, num_seg, e_ids, data, 1, out);
    else k_segments<true, false><<<segments_grid(num_seg), kSegThreads, 0, stream>>>(indptr, num_seg, e_ids, data, 1, out);
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}

int gsb_edge_div_u_sum(gsb_ctx* ctx, void* stream_, const int64_t* coo_row, const int64_t* coo_col, int64_t E,
                       const float* data, const float* divisor, float* out_data, float* out_sum_zeroed) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(E >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (E == 0) return GSB_OK;
  GSB_REQUIRE(coo_row && coo_col && divisor && out_data && out_sum_zeroed, GSB_ERR_INVALID_ARGUMENT);
  ScopedKernelTimer timer(ctx, KID_SEGMENT, (cudaStream_t)stream_);
  k_edge_div_u_sum<<<min(grid_for(E, kSegThreads), kNumSMs * 16), kSegThreads, 0, (cudaStream_t)stream_>>>(
      coo_row, coo_col, E, data, divisor, out_data, out_sum_zeroed);
  GSB_LAUNCH_OK();
  return GSB_OK;
}

}  // extern "C"
