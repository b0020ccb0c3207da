// What the uniform samplers share: the parameters of a call, the count of a column and its draws (slice_sample.cu,
// window_sample.cu).
#pragma once
#include "batch_table.cuh"
#include "common.cuh"
#include "philox.cuh"
#include "scan.cuh"

namespace gsb {

enum CountMode { COUNT_DEGREE = 0, COUNT_WOR = 1, COUNT_WR = 2 };

__device__ __forceinline__ i64 column_count(i64 d, i64 k, int mode) {
  if (mode == COUNT_DEGREE) return d;
  if (mode == COUNT_WOR) return d < k ? d : k;
  return d > 0 ? k : 0;
}

// A seed outside [0, num_cols) counts as an empty column: its offsets are never read, GSB_ERR_INDEX_RANGE is recorded.
__device__ __forceinline__ bool column_in_range(i64 col, i64 num_cols, i64* counters, i64 where) {
  if ((u64)col < (u64)num_cols) return true;
  raise_error(counters, GSB_ERR_INDEX_RANGE, where);
  return false;
}

struct SampleParams {
  const i64* indptr;
  const i64* indices;
  i64 num_cols;
  const i64* seeds;
  i64 S;
  i64 k;
  int replace;
  uint32_t bucket_magic;  // of bucket_count below: see bucket_of_id (here it costs no room: eight bytes more 0.3 us a launch)
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
  TileState ts;
  const i64* S_dev;  // when set, the exact seed count lives on the device and S above is only an upper bound
  // Minibatch form (G > 0): the seeds of minibatch j are seeds[batch_ptr[j] .. batch_ptr[j+1]) and the draws of its
  // column number c are keyed by (batch_ids[j], c) instead of the column's position in the call, so a minibatch
  // receives the same sample whichever call, group or GPU processes it.
  // batch_ptr / G alone (batch_ids null) only tell the kernel which minibatch a column belongs to.
  const i64* batch_ptr;
  const i64* batch_ids;
  i64 G;
  // Per-bucket item counts of the partitioned unique + relabel that follows (thread-per-column kernels only), or null:
  // every seed and every sampled id adds one to the count of its bucket.
  uint32_t* bucket_count;
  const i64* bucket_base;  // [G + 1] first bucket of every minibatch
  Mail mail;               // the edge total, for a caller that waits for it
};

// Random-stream item of the column at position i of the call.
__device__ __forceinline__ u64 sample_item(const SampleParams& p, i64 i, i64 batch) {
  if (!p.batch_ids) return (u64)i;
  return ((u64)__ldg(p.batch_ids + batch) << 32) | (u64)(uint32_t)(i - __ldg(p.batch_ptr + batch));
}

// The picks of the column at position i of the call, minibatch `batch`, with d > 0 edges (positions inside the column): Floyd's
// k-subset in registers, or k draws with replacement, or all edges where there are no more than k.
template <int KMAX>
__device__ __forceinline__ void draw_picks(const SampleParams& p, i64 i, i64 batch, i64 d, uint32_t (&pick)[KMAX]) {
  const int k = (int)p.k;
  if (p.replace || d > k) {
    const u64 item = sample_item(p, i, batch);
    U32x4 blk;
#pragma unroll
    for (int j = 0; j < KMAX; ++j) {
      if (j < k) {
        if ((j & 3) == 0) blk = rand_block(p.seed, item, (u64)(j >> 2), STREAM_UNIFORM);
        const uint32_t word =
            (j & 3) == 0 ? blk.v[0] : (j & 3) == 1 ? blk.v[1] : (j & 3) == 2 ? blk.v[2] : blk.v[3];
        if (p.replace) {
          pick[j] = (uint32_t)bounded_from_word(word, (u64)d);
        } else {
          const uint32_t m = (uint32_t)(d - k + j);
          const uint32_t t = (uint32_t)bounded_from_word(word, (u64)m + 1);
          bool dup = false;
#pragma unroll
          for (int q = 0; q < KMAX; ++q)
            if (q < j) dup |= (pick[q] == t);
          pick[j] = dup ? m : t;
        }
      }
    }
  } else {
#pragma unroll
    for (int j = 0; j < KMAX; ++j) pick[j] = (uint32_t)j;
  }
}

// The launch of the three passes of a call that samples by windows (defined in window_sample.cu), with its scratch.
int window_sample_launch(gsb_ctx* ctx, cudaStream_t stream, const SampleParams& p, i64 num_edges, void* ws);

}  // namespace gsb
