// Row gather: out[i, :] = src[index[i], :] for rows of `row_len` floats — the feature / edge-data load that
// follows sampling in every training loop (features[frontier]; examples/graphsage/train_minibatch.py), and the
// reference's IndexSelectCPUFromGPU (src/cuda/index_select_uvm.cu:8-45) when `src` is pinned host memory
// that the GPU reads in place.
//
// A group of LPR lanes copies ROWS neighbouring rows of the output at a time (16 bytes per access where rows allow it, else 8
// or 4): all their reads are requested before anything is written, and what it writes is one run of memory.  The copy is
// bound by HBM (or by the host link when src is host memory): 8 bytes of index, row_len * 4 bytes read and row_len * 4 bytes
// written per row; a row in no order that starts on a 16-byte boundary costs up to 64 bytes more.  A million rows of 100
// floats: 184 us with two rows per group, half the grid apart, and half the CTAs; 145 us now, where reading alone takes 93
// and writing alone 65.  Copying the rows through shared memory with bulk copies gave 150 to 158, cutting the output into
// tiles of equal bytes 190.
#include <type_traits>

#include "common.cuh"
#include "scan.cuh"

namespace gsb {

constexpr int kGatherThreads = 256;

template <typename Unit, int LPR, int ROWS>
__global__ void __launch_bounds__(kGatherThreads) k_gather_rows(const Unit* __restrict__ src, i64 num_rows,
                                                                i64 units_per_row, const i64* __restrict__ index,
                                                                i64 n, Unit* __restrict__ out, i64* counters) {
  constexpr int kGroups = kGatherThreads / LPR;
  // a row of one unit per thread: a thread's rows are a CTA apart, so that neighbouring threads have neighbouring rows
  constexpr int kStep = LPR == 1 ? kGroups : 1;
  const int lane = threadIdx.x % LPR, group = threadIdx.x / LPR;
  for (i64 tile = (i64)blockIdx.x * kGroups * ROWS; tile < n; tile += (i64)gridDim.x * kGroups * ROWS) {
    const i64 first = tile + (LPR == 1 ? group : group * ROWS);
    i64 row[ROWS];
#pragma unroll
    for (int q = 0; q < ROWS; ++q) {
      const i64 at = first + q * kStep;
      row[q] = at < n ? __ldg(index + at) : -1;
      if ((u64)row[q] >= (u64)num_rows) {
        if (lane == 0 && at < n) raise_error(counters, GSB_ERR_INDEX_RANGE, at);
        row[q] = -1;
      }
    }
    Unit* to = out + first * units_per_row;
    for (i64 j = lane; j < units_per_row; j += LPR) {
      Unit v[ROWS];
#pragma unroll
      for (int q = 0; q < ROWS; ++q)
        if (row[q] >= 0) v[q] = __ldg(src + row[q] * units_per_row + j);
#pragma unroll
      for (int q = 0; q < ROWS; ++q)
        if (row[q] >= 0) to[q * kStep * units_per_row + j] = v[q];
    }
  }
}

template <typename Unit, int LPR, int ROWS>
static void launch_rows(cudaStream_t stream, const void* src, i64 num_rows, i64 units, const i64* index, i64 n, void* out,
                        i64* counters) {
  constexpr int kRowsPerCta = kGatherThreads / LPR * ROWS;
  const int grid = (int)min((i64)kNumSMs * 32, (n + kRowsPerCta - 1) / kRowsPerCta);
  k_gather_rows<Unit, LPR, ROWS><<<grid, kGatherThreads, 0, stream>>>((const Unit*)src, num_rows, units, index, n, (Unit*)out,
                                                                      counters);
}

// Lanes per row and rows at a time by the units of a row.  A power of two of lanes leaves some of them idle; where half as many
// lanes take the row in no more steps than three quarters of the whole would (5 and 6 units, 9 to 12, 17 to 24, 33 to 48), they
// are the better choice, with two rows: a million rows of 17 floats 63 us against 76, of 33 floats 92 against 108, of 42 floats 93
// against 103, of 160 floats 218 against 251; equal at 24 and 48 floats, and above the three quarters the whole group is ahead (100
// floats 146 against 152).  Rows of several steps are runs of memory by themselves, two at a time are better than four (63 floats
// 156 and 172 us, 300 000 rows of 602 floats 289 and 306, 1 000 rows of 512 floats 5.5 and 8.2) except for 64 units (322 against
// 325) and for odd rows above 4 KB (1 433 floats, 300 000 rows: 925 and 898).
template <typename Unit>
static void launch_gather(cudaStream_t stream, const void* src, i64 num_rows, i64 units, const i64* index, i64 n, void* out,
                          i64* counters) {
  auto go = [&](auto lanes, auto rows) {
    launch_rows<Unit, decltype(lanes)::value, decltype(rows)::value>(stream, src, num_rows, units, index, n, out, counters);
  };
  using std::integral_constant;
  const integral_constant<int, 2> two{};
  const integral_constant<int, 4> four{};
  if (units == 1) go(integral_constant<int, 1>{}, two);
  else if (units == 2) go(two, four);
  else if (units <= 4) go(four, four);
  else if (units <= 6 || (units == 7 && sizeof(Unit) < 16)) go(four, two);
  else if (units <= 8) go(integral_constant<int, 8>{}, four);
  else if (units <= 12) go(integral_constant<int, 8>{}, two);
  else if (units <= 16) go(integral_constant<int, 16>{}, four);
  else if (units <= 24 || (units > 32 && units <= 48)) go(integral_constant<int, 16>{}, two);
  else if (units <= 32 || units == 64) go(integral_constant<int, 32>{}, four);
  else go(integral_constant<int, 32>{}, two);
}

}  // namespace gsb

using namespace gsb;

extern "C" int gsb_gather_rows(gsb_ctx* ctx, void* stream_, const float* src, int64_t num_rows, int64_t row_len,
                               const int64_t* index, int64_t n, float* out) {
  GSB_ENTER(ctx);
  GSB_REQUIRE(num_rows >= 0 && row_len >= 1 && n >= 0, GSB_ERR_INVALID_ARGUMENT);
  if (n == 0) return GSB_OK;
  GSB_REQUIRE(src && index && out, GSB_ERR_INVALID_ARGUMENT);
  // `src` may be device memory or page-locked host memory; the kernel gets the address the DEVICE uses for it.
  // Pageable host memory is refused here instead of faulting in the kernel.
  cudaPointerAttributes attr;
  GSB_CUDA_OK(cudaPointerGetAttributes(&attr, src));
  GSB_REQUIRE(attr.devicePointer != nullptr &&
                  (attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeHost ||
                   attr.type == cudaMemoryTypeManaged),
              GSB_ERR_INVALID_ARGUMENT);
  const void* dsrc = attr.devicePointer;
  cudaStream_t stream = (cudaStream_t)stream_;
  const uintptr_t both = (uintptr_t)dsrc | (uintptr_t)out;
  const int width = row_len % 4 == 0 && both % 16 == 0 ? 4 : row_len % 2 == 0 && both % 8 == 0 ? 2 : 1;  // floats per access
  const i64 units = row_len / width;
  {
    ScopedKernelTimer timer(ctx, KID_OTHER, stream);
    if (width == 4) launch_gather<float4>(stream, dsrc, num_rows, units, index, n, out, ctx_counters(ctx));
    else if (width == 2) launch_gather<float2>(stream, dsrc, num_rows, units, index, n, out, ctx_counters(ctx));
    else launch_gather<float>(stream, dsrc, num_rows, units, index, n, out, ctx_counters(ctx));
  }
  GSB_LAUNCH_OK();
  return GSB_OK;
}
