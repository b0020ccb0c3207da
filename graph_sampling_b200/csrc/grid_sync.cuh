// Grid-wide barrier for kernels launched cooperatively (the launch guarantees that the whole grid is resident), so that
// an operator of a few microseconds per pass is one launch instead of one per pass.
//
// The barrier word counts arrivals for ever: a launch is told the count it starts from, and every CTA arrives exactly
// `barriers` times whatever happens, so the word never needs clearing.  The wait is bounded like every other wait of the
// library (GSB_OPT_MAX_POLLS, then GSB_ERR_LOOKBACK_TIMEOUT).
#pragma once
#include "common.cuh"
#include "scan.cuh"

namespace gsb {

struct GridSync {
  u64* word;
  u64 base;
  i64* counters;
  int max_polls;
};

__device__ __forceinline__ u64 ld_acquire_u64(const u64* p) {
  u64 v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

// Barrier number `index` (1, 2, ...) of the launch.  Release / acquire, cumulative over what the CTA did before it.
__device__ __forceinline__ void grid_barrier(const GridSync& g, u32 index) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(g.word) : "memory");
    const u64 target = g.base + (u64)index * gridDim.x;
    int polls = 0;
    while ((i64)(ld_acquire_u64(g.word) - target) < 0) {
      if (++polls > g.max_polls) {
        raise_error(g.counters, GSB_ERR_LOOKBACK_TIMEOUT, blockIdx.x);
        break;
      }
      if (polls > 64) __nanosleep(20);
    }
  }
  __syncthreads();
}

// For a CTA that returns early: the arrivals it still owes.
__device__ __forceinline__ void grid_arrive(const GridSync& g, u32 arrivals) {
  if (threadIdx.x == 0) atomicAdd(g.word, (u64)arrivals);
}

// CTAs of a kernel that are resident at once on the context's device (0: cooperative launches are not available).  The
// answer is kept in `known`, one entry per device, which the caller provides for each kernel.
int ctx_resident_ctas(gsb_ctx* ctx, const void* kernel, int threads, size_t smem, int (&known)[64]);
// Barrier state for a launch of `grid` CTAs that pass `barriers` barriers, and the launch itself.
GridSync ctx_grid_sync(gsb_ctx* ctx, int grid, int barriers);
int launch_cooperative(gsb_ctx* ctx, cudaStream_t stream, const void* kernel, int grid, int threads, size_t smem,
                       void** args, const GridSync& sync);

}  // namespace gsb
