// Walks a stretch of the virtual edge list of a column slice: position q of the list is an edge of the column whose offsets
// off[c] <= q < off[c + 1] it lies between, and sits at position q - off[c] + indptr[seeds[c]] of the operand.
//
// A warp owns a stretch and finds its first column once, by search.  From there it keeps 32 columns in its lanes (offset and
// what to add to get the input position); the offsets and seed ids of the two following windows are on their way, so that a
// new window costs no wait.  32 consecutive positions find their columns without memory: the columns that start among them set
// a bit each, and a lane counts the bits up to its own.  No barrier and no shared memory anywhere.
#pragma once
#include "common.cuh"
#include "scan.cuh"

namespace gsb {

constexpr i64 kNoWalkColumn = (i64)1 << 62;  // a seed outside the operand: its positions are skipped

// Largest c with off[c] <= pos, by a whole warp: 32 pivots per step, so a search over a few hundred thousand columns takes four
// dependent loads instead of eighteen.  Needs off[0] <= pos < off[S].
__device__ __forceinline__ i64 warp_column_search(const i64* __restrict__ off, i64 S, i64 pos) {
  const int lane = threadIdx.x & 31;
  i64 lo = 0, hi = S;
  while (hi - lo > 1) {
    const i64 step = (hi - lo + 31) / 32;
    const i64 idx = lo + (i64)(lane + 1) * step;
    const bool le = idx < hi && __ldg(off + idx) <= pos;  // true for a prefix of the lanes
    const int n = __popc(__ballot_sync(0xffffffffu, le));
    const i64 new_hi = min(hi, lo + (i64)(n + 1) * step);
    lo += (i64)n * step;
    hi = new_hi;
  }
  return lo;
}

struct ColumnWalk {
  const i64* off;
  const i64* seeds;  // null: the columns themselves
  const i64* indptr;
  i64 S, num_cols;
  i64* counters;  // where a bad seed is reported, or null
  i64 begin;      // first position of the stretch
  int len;
  i64 c0;     // the window: columns c0 .. c0 + 31, one per lane
  int start;  // first position of the lane's column, relative to `begin`
  int next;   // of the column after the window
  i64 delta;  // input position minus relative position
  i64 off1, ptr1, off2, col2;  // the two windows that follow
  i64 run_in;   // the column of the last position located: what to add to its positions, its number,
  int run_end;  // and where it ends
  int run_column;

  __device__ __forceinline__ int relative(i64 o) const { return (int)max((i64)0, min(o - begin, (i64)len)); }
  __device__ __forceinline__ void fetch(i64 c, i64& o, i64& col) const {
    o = c <= S ? __ldg(off + c) : (i64)1 << 61;
    col = c < S ? (seeds ? __ldg(seeds + c) : c) : -1;
  }
  __device__ __forceinline__ i64 pointer(i64 col, i64 c) const {
    if ((u64)col < (u64)num_cols) return __ldg(indptr + col);
    if (counters && c < S) raise_error(counters, GSB_ERR_INDEX_RANGE, c);
    return kNoWalkColumn;
  }
  __device__ __forceinline__ void set(i64 o, i64 ptr) {
    start = relative(o);
    delta = ptr == kNoWalkColumn ? kNoWalkColumn : ptr - o + begin;
    next = __shfl_sync(0xffffffffu, relative(off1), 0);
  }
  __device__ __forceinline__ void init(i64 first, int length) {
    const int lane = threadIdx.x & 31;
    begin = first;
    len = length;
    run_end = 0;
    c0 = warp_column_search(off, S, begin);
    i64 o, col, col1;
    fetch(c0 + lane, o, col);
    fetch(c0 + 32 + lane, off1, col1);
    fetch(c0 + 64 + lane, off2, col2);
    const i64 ptr = pointer(col, c0 + lane);
    ptr1 = pointer(col1, c0 + 32 + lane);
    set(o, ptr);
  }
  __device__ __forceinline__ void advance() {
    const int lane = threadIdx.x & 31;
    const i64 o = off1, ptr = ptr1;
    c0 += 32;
    off1 = off2;
    ptr1 = pointer(col2, c0 + 32 + lane);
    fetch(c0 + 64 + lane, off2, col2);
    set(o, ptr);
  }
  // Positions at .. at + 31 of the stretch, a lane each, in ascending calls: the input position (negative: none) and, if
  // wanted, the column.
  template <bool COLUMN>
  __device__ __forceinline__ i64 locate(int at, i64* column) {
    const int lane = threadIdx.x & 31, q = at + lane, end = min(at + 32, len);
    if (end <= run_end) {  // inside a long column
      if (COLUMN) *column = c0 + run_column;
      return q < end && run_in != kNoWalkColumn ? q + run_in : -1;
    }
    i64 in = -1;
    for (;;) {
      const int rel = start - at;
      const unsigned before = __ballot_sync(0xffffffffu, rel <= 0);
      const bool inside = rel > 0 && rel < 32;
      const int starts = __popc(__ballot_sync(0xffffffffu, inside));
      const unsigned heads = __reduce_or_sync(0xffffffffu, inside ? 1u << rel : 0u);
      int c = __popc(before) - 1 + __popc(heads & ((2u << lane) - 1u));
      if (__popc(heads) != starts) {  // empty columns among them share a position: the last one that starts there holds it
        c = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(0xffffffffu, start, c + step) <= q) c += step;
      }
      const i64 d = __shfl_sync(0xffffffffu, delta, max(c, 0));
      if (q >= __shfl_sync(0xffffffffu, start, 0) && q < min(next, end) && d != kNoWalkColumn) {
        in = q + d;
        if (COLUMN) *column = c0 + c;
      }
      if (end <= next) {
        run_column = __shfl_sync(0xffffffffu, max(c, 0), end - 1 - at);
        run_in = __shfl_sync(0xffffffffu, d, end - 1 - at);
        run_end = __shfl_sync(0xffffffffu, start, (run_column + 1) & 31);
        if (run_column == 31) run_end = next;
        return in;
      }
      advance();
    }
  }

  // The other way through the stretch, for columns of some length: pieces of up to 32 positions of ONE column, N of them at a
  // time, so that locating costs a dozen instructions per piece whatever the columns are.  f(at, edge): the lane's position in the
  // N pieces, and the input position (negative: none).  Called by all lanes, behind init(); pieces come in ascending order.
  template <int N, class F>
  __device__ __forceinline__ void for_pieces(F f) {
    static_assert(32 % N == 0, "a warp holds 32 pieces");
    const int lane = threadIdx.x & 31;
    for (;;) {
      int stop = __shfl_down_sync(0xffffffffu, start, 1);
      if (lane == 31) stop = next;
      const int mine = stop > start && delta != kNoWalkColumn ? (stop - start + 31) >> 5 : 0;
      int upto = mine;  // pieces of the window's columns up to the lane's
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
      }
      const int total = __shfl_sync(0xffffffffu, upto, 31);
      for (int base = 0; base < total; base += 32) {
        // piece base + lane: the first column with more pieces up to it than that
        int c = 0;
#pragma unroll
        for (int step = 16; step > 0; step >>= 1)
          if (__shfl_sync(0xffffffffu, upto, c + step - 1) <= base + lane) c += step;
        const int rank = base + lane - (__shfl_sync(0xffffffffu, upto, c) - __shfl_sync(0xffffffffu, mine, c));
        const int first = __shfl_sync(0xffffffffu, start, c) + rank * 32;
        const int end = __shfl_sync(0xffffffffu, stop, c);
        const i64 in = __shfl_sync(0xffffffffu, delta, c) + first;
        const int count = base + lane < total ? min(end - first, 32) : 0;
        for (int piece = 0; piece < min(32, total - base); piece += N) {
          int at[N];
          i64 edge[N];
#pragma unroll
          for (int r = 0; r < N; ++r) {
            at[r] = __shfl_sync(0xffffffffu, first, piece + r) + lane;
            edge[r] = __shfl_sync(0xffffffffu, in, piece + r) + lane;
            if (lane >= __shfl_sync(0xffffffffu, count, piece + r)) edge[r] = -1;
          }
          f(at, edge);
        }
      }
      if (next >= len) return;
      advance();
    }
  }
};

}  // namespace gsb
