// Grid-wide barrier for kernels launched cooperatively (the launch guarantees that the whole grid is resident), so that
// an operator of a few microseconds per pass is one launch instead of one per pass.
//
// The barrier word counts arrivals for ever: a launch is told the count it starts from, and every CTA arrives exactly
// `barriers` times whatever happens, so the word never needs clearing.  The wait is bounded like every other wait of the
// library (GSB_OPT_MAX_POLLS, then GSB_ERR_LOOKBACK_TIMEOUT), and what follows a barrier indexes with what other CTAs wrote
// before it, so nobody may go on from one that was given up.  All CTAs agree on that: giving up is a compare-and-swap of the
// word as it was last seen, incomplete, to the same count with a mark on it.  Whoever sees a complete count therefore sees the
// mark too if there is one, and a count without it means that everybody has arrived.  The mark stays until the error is read
// (ctx_check_device_error), and cooperative kernels launched in between end at their first barrier.
//
// A call that does not wait for its result cannot report the error before its outputs are used, so a kernel that gives up
// leaves results that are wrong but within range: an empty sample or subgraph, a conversion with all edges in column 0.  Every
// CTA of the launch comes to that point and writes its own share of them (grid_share); shares are such that no other CTA writes
// there before the last barrier.
#pragma once
#include "common.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kBarrierCountBits = 56;  // arrivals; the top byte is the mark
constexpr u64 kBarrierGivenUp = 1ull << 63;

struct GridSync {
  u64* word;
  u64 base;
  u32 barriers;
  i64* counters;
  int max_polls;
};

__device__ __forceinline__ u64 ld_acquire_u64(const u64* p) {
  u64 v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// For a CTA that returns early: the arrivals it still owes.
__device__ __forceinline__ void grid_arrive(const GridSync& g, u32 arrivals) {
  if (threadIdx.x == 0) atomicAdd(g.word, (u64)arrivals);
}

// The CTA's share of n things, in one stretch: what thread 0 goes through when a barrier was given up.
template <class F>
__device__ __forceinline__ void grid_share(i64 n, F f) {
  const i64 per = (n + gridDim.x - 1) / gridDim.x, end = min(n, (i64)(blockIdx.x + 1) * per);
  for (i64 i = (i64)blockIdx.x * per; i < end; ++i) f(i);
}

// Barrier number `index` (1, 2, ...) of the launch.  Release / acquire, cumulative over what the CTA did before it.  When this
// barrier or (while the CTA was looking) a later one was given up, the CTA makes the arrivals of its later barriers, thread 0
// runs `give_up`, and the CTA ends here.  It ends by an instruction, and one thread does the work where it waits anyway: with a
// branch to code for all threads, or to the end of the kernel, the compiler keeps more alive across the barrier (36 spilled bytes
// in the weighted sampler, 10 000 columns with replacement 217 -> 259 us).
//
// grid_barrier_arrive and grid_barrier_wait are its halves, for work in between that needs nothing from other CTAs; a CTA waits
// before it arrives at the next barrier.
__device__ __forceinline__ void grid_barrier_arrive(const GridSync& g) {
  __syncthreads();
  if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.word) : "memory");
}

template <class F>
__device__ __forceinline__ void grid_barrier_wait(const GridSync& g, u32 index, F give_up) {
  bool ok = true;
  if (threadIdx.x == 0) {
    const u64 target = g.base + (u64)index * gridDim.x;
    int polls = 0;
    for (;;) {
      const u64 seen = ld_acquire_u64(g.word);
      ok = seen < kBarrierGivenUp;
      if (!ok || (i64)((seen - target) << (64 - kBarrierCountBits)) >= 0) break;
      if (++polls > g.max_polls) {  // fails only when somebody arrived meanwhile: at most as often as there are CTAs
        ok = atomicCAS(g.word, seen, seen | kBarrierGivenUp) != seen;
        if (!ok) break;
      }
      if (polls > 64) __nanosleep(20);
    }
    if (!ok) {
      raise_error(g.counters, GSB_ERR_LOOKBACK_TIMEOUT, blockIdx.x);
      grid_arrive(g, g.barriers - index);
      give_up();
    }
  }
  if (!__syncthreads_and(ok)) asm volatile("exit;");
}

template <class F>
__device__ __forceinline__ void grid_barrier(const GridSync& g, u32 index, F give_up) {
  grid_barrier_arrive(g);
  grid_barrier_wait(g, index, give_up);
}

// CTAs of a kernel that are resident at once on the context's device (0: cooperative launches are not available).  The
// answer is kept in `known`, one entry per device, which the caller provides for each kernel.
int ctx_resident_ctas(gsb_ctx* ctx, const void* kernel, int threads, size_t smem, int (&known)[64]);
// Barrier state for a launch of `grid` CTAs that pass `barriers` barriers, and the launch itself.
GridSync ctx_grid_sync(gsb_ctx* ctx, int grid, int barriers);
int launch_cooperative(gsb_ctx* ctx, cudaStream_t stream, const void* kernel, int grid, int threads, size_t smem,
                       void** args, const GridSync& sync);

}  // namespace gsb
