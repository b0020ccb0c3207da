// Context: scratch arena, look-back tile state, device counters and pinned read-back buffer.
#include <stdio.h>
#include <string.h>

#include <atomic>
#include <chrono>
#include <new>
#include <vector>

#include "common.cuh"
#include "grid_sync.cuh"
#include "scan.cuh"

struct gsb_ctx {
  int device;
  void* workspace;
  size_t workspace_bytes;
  size_t refused_bytes;  // scratch that ctx_try_workspace could not have last time, 0: none
  i64 refused_calls;
  u64* tile_words;
  i64 tile_capacity;
  uint32_t epoch;
  i64* counters;  // device, CNT_NUM entries and the grid-barrier word
  i64* pinned;    // page-locked host memory the device writes: CNT_NUM counters, kMailSlots result words, one ticket
  u64 mail_tag;   // 1 .. 65535, of the last mailbox handed out
  u64 ticket;     // of the last counter fetch
  i64 launches;
  i64 id_bound_refusals;
  char message[512];
  // per-kernel event timing (off by default)
  bool profiling;
  std::vector<cudaEvent_t>* ev_begin;
  std::vector<cudaEvent_t>* ev_end;
  std::vector<int>* ev_kid;
  size_t ev_used;
  double prof_ms[gsb::KID_NUM];
  i64 prof_launches[gsb::KID_NUM];
  i64 options[GSB_OPT_NUM];
  // direct-address tables of the batched unique + relabel (see ctx_direct_tables)
  u64* direct_tables;
  size_t direct_bytes;
  uint32_t direct_epoch;
  // tables of the single-launch unique + relabel (see ctx_epoch_table)
  void* epoch_table[2];
  size_t epoch_bytes[2];
  uint32_t table_epoch[2];
  cudaStream_t stream;   // of the last call that used scratch
  bool stream_known;
  u64 barrier_arrivals;  // the barrier word itself is counters[CNT_NUM]
  cudaEvent_t wait_event;  // created on first use when GSB_OPT_BLOCKING_WAIT is set
};

namespace gsb {

int cuda_fail(gsb_ctx* ctx, cudaError_t e, const char* file, int line) {
  if (ctx) snprintf(ctx->message, sizeof(ctx->message), "%s (%s:%d)", cudaGetErrorString(e), file, line);
  return e == cudaErrorMemoryAllocation ? GSB_ERR_OUT_OF_MEMORY : GSB_ERR_CUDA;
}

// Scratch, look-back words and tables hold one call's work at a time.  A call returns as soon as the size it reports is known,
// while its last kernel may still use them, so the next call must come behind it in stream order.  Where it comes on another
// stream the host waits for the device: not for the stream of the call before, which may have been destroyed since.
static int ctx_on_stream(gsb_ctx* ctx, cudaStream_t stream) {
  if (ctx->stream_known && ctx->stream != stream) GSB_CUDA_OK(cudaDeviceSynchronize());
  ctx->stream = stream;
  ctx->stream_known = true;
  return GSB_OK;
}

int ctx_reserve_workspace(gsb_ctx* ctx, cudaStream_t stream, size_t bytes, void** out) {
  const int st = ctx_on_stream(ctx, stream);
  if (st != GSB_OK) return st;
  if (bytes > ctx->workspace_bytes) {
    // Growing synchronises the device; it only happens the first time a size is seen.
    GSB_CUDA_OK(cudaDeviceSynchronize());
    if (ctx->workspace) GSB_CUDA_OK(cudaFree(ctx->workspace));
    ctx->workspace = nullptr;
    ctx->workspace_bytes = 0;
    size_t want = bytes + bytes / 4;
    want = (want + 255) & ~(size_t)255;
    cudaError_t e = cudaMalloc(&ctx->workspace, want);
    if (e != cudaSuccess) {
      want = (bytes + 255) & ~(size_t)255;
      e = cudaMalloc(&ctx->workspace, want);
    }
    if (e != cudaSuccess) return cuda_fail(ctx, e, __FILE__, __LINE__);
    ctx->workspace_bytes = want;
  }
  *out = ctx->workspace;
  return GSB_OK;
}

// Asking for the free memory takes 0.1 to 0.4 ms: a size that was refused is asked for again by every 64th call that wants it.
constexpr i64 kRefusedCalls = 64;

bool ctx_try_workspace(gsb_ctx* ctx, cudaStream_t stream, size_t bytes, size_t needed, void** out) {
  if (ctx_on_stream(ctx, stream) != GSB_OK) return false;
  if (bytes > ctx->workspace_bytes) {
    bytes = (bytes + 255) & ~(size_t)255;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) return false;
    if (ctx->refused_bytes != 0 && bytes >= ctx->refused_bytes && ++ctx->refused_calls % kRefusedCalls != 0) return false;
    size_t room = 0, total = 0;
    void* grown = nullptr;
    bool fits = cudaMemGetInfo(&room, &total) == cudaSuccess;
    const size_t kept = room + ctx->workspace_bytes;  // what there is for the scratch: growth gives the present one back
    fits = fits && kept >= needed && bytes - needed <= (kept - needed) / 8;
    // the new scratch is there before the old one goes: an attempt that fails leaves everything as it was
    if (!fits || cudaMalloc(&grown, bytes) != cudaSuccess) {
      (void)cudaGetLastError();
      ctx->refused_bytes = bytes;
      return false;
    }
    ctx->refused_bytes = 0;
    if (cudaDeviceSynchronize() != cudaSuccess || (ctx->workspace && cudaFree(ctx->workspace) != cudaSuccess)) {
      (void)cudaFree(grown);
      return false;
    }
    ctx->workspace = grown;
    ctx->workspace_bytes = bytes;
  }
  *out = ctx->workspace;
  return true;
}

int ctx_tile_state(gsb_ctx* ctx, i64 num_tiles, cudaStream_t stream, TileState* out) {
  const int st = ctx_on_stream(ctx, stream);
  if (st != GSB_OK) return st;
  if (num_tiles > ctx->tile_capacity) {
    GSB_CUDA_OK(cudaDeviceSynchronize());
    if (ctx->tile_words) GSB_CUDA_OK(cudaFree(ctx->tile_words));
    ctx->tile_words = nullptr;
    i64 cap = ctx->tile_capacity > 0 ? ctx->tile_capacity : (1 << 16);
    while (cap < num_tiles) cap <<= 1;
    GSB_CUDA_OK(cudaMalloc((void**)&ctx->tile_words, sizeof(u64) * (size_t)cap));
    GSB_CUDA_OK(cudaMemset(ctx->tile_words, 0, sizeof(u64) * (size_t)cap));
    ctx->tile_capacity = cap;
    ctx->epoch = 0;
  }
  ctx->epoch += 1;
  if (ctx->epoch > kEpochMask) {
    // 22-bit epoch wrapped: stale words could alias, clear them (stream-ordered).
    GSB_CUDA_OK(cudaMemsetAsync(ctx->tile_words, 0, sizeof(u64) * (size_t)ctx->tile_capacity, stream));
    ctx->epoch = 1;
  }
  out->words = ctx->tile_words;
  out->epoch = ctx->epoch;
  out->counters = ctx->counters;
  out->max_polls = (int)ctx->options[GSB_OPT_MAX_POLLS];
  return GSB_OK;
}

int ctx_enter(gsb_ctx* ctx) {
  if (!ctx) return GSB_ERR_INVALID_ARGUMENT;
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) return GSB_ERR_CUDA;
  if (dev != ctx->device) {
    snprintf(ctx->message, sizeof(ctx->message),
             "context belongs to CUDA device %d but device %d is current: nothing was launched", ctx->device, dev);
    return GSB_ERR_INVALID_ARGUMENT;
  }
  return GSB_OK;
}

i64 ctx_option(gsb_ctx* ctx, int option) { return ctx->options[option]; }

int ctx_direct_tables(gsb_ctx* ctx, i64 count, i64 num_nodes, cudaStream_t stream, u64** out_table,
                      uint32_t* out_epoch) {
  *out_table = nullptr;
  *out_epoch = 0;
  if (count <= 0 || num_nodes <= 0) return GSB_OK;
  if ((double)count * (double)num_nodes * 8.0 > (double)ctx->options[GSB_OPT_DIRECT_TABLE_BUDGET]) return GSB_OK;
  const int st = ctx_on_stream(ctx, stream);
  if (st != GSB_OK) return st;
  const size_t bytes = (size_t)count * (size_t)num_nodes * sizeof(u64);
  if (bytes > ctx->direct_bytes) {
    // Growing synchronises the device; it only happens the first time a (batches x nodes) size is seen.
    GSB_CUDA_OK(cudaDeviceSynchronize());
    if (ctx->direct_tables) GSB_CUDA_OK(cudaFree(ctx->direct_tables));
    ctx->direct_tables = nullptr;
    ctx->direct_bytes = 0;
    cudaError_t e = cudaMalloc((void**)&ctx->direct_tables, bytes);
    if (e != cudaSuccess) {
      (void)cudaGetLastError();  // not fatal: the caller falls back to the hash tables
      return GSB_OK;
    }
    ctx->direct_bytes = bytes;
    GSB_CUDA_OK(cudaMemsetAsync(ctx->direct_tables, 0xFF, bytes, stream));
    ctx->direct_epoch = 0;
  }
  ctx->direct_epoch += 1;
  if (ctx->direct_epoch >= 0xFFFFFFFEu) {  // the 32-bit epoch is used up: start over from cleared tables
    GSB_CUDA_OK(cudaMemsetAsync(ctx->direct_tables, 0xFF, ctx->direct_bytes, stream));
    ctx->direct_epoch = 1;
  }
  *out_table = ctx->direct_tables;
  *out_epoch = ctx->direct_epoch;
  return GSB_OK;
}

int ctx_epoch_table(gsb_ctx* ctx, int which, size_t bytes, int fill, uint32_t epochs, cudaStream_t stream, void** table,
                    uint32_t* epoch) {
  if (bytes > ctx->epoch_bytes[which]) {
    GSB_CUDA_OK(cudaDeviceSynchronize());
    if (ctx->epoch_table[which]) GSB_CUDA_OK(cudaFree(ctx->epoch_table[which]));
    ctx->epoch_table[which] = nullptr;
    ctx->epoch_bytes[which] = 0;
    size_t cap = 1 << 19;
    while (cap < bytes) cap <<= 1;
    GSB_CUDA_OK(cudaMalloc(&ctx->epoch_table[which], cap));
    ctx->epoch_bytes[which] = cap;
    ctx->table_epoch[which] = epochs - 1;  // filled below
  }
  ctx->table_epoch[which] += 1;
  if (ctx->table_epoch[which] >= epochs) {
    GSB_CUDA_OK(cudaMemsetAsync(ctx->epoch_table[which], fill, ctx->epoch_bytes[which], stream));
    ctx->table_epoch[which] = 1;
  }
  *table = ctx->epoch_table[which];
  *epoch = ctx->table_epoch[which];
  return GSB_OK;
}

int ctx_resident_ctas(gsb_ctx* ctx, const void* kernel, int threads, size_t smem, int (&known)[64]) {
  const int device = ctx->device;
  if (device < 0 || device >= 64) return 0;
  if (known[device] == 0) {
    int coop = 0, sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess)
      (void)cudaGetLastError();
    known[device] = coop && per_sm * sms > 0 ? per_sm * sms : -1;
  }
  return known[device] > 0 ? known[device] : 0;
}

GridSync ctx_grid_sync(gsb_ctx* ctx, int grid, int barriers) {
  const GridSync g{(u64*)(ctx->counters + CNT_NUM), ctx->barrier_arrivals, (u32)barriers, ctx->counters,
                   (int)ctx->options[GSB_OPT_MAX_POLLS]};
  ctx->barrier_arrivals += (u64)grid * (u64)barriers;
  return g;
}

int launch_cooperative(gsb_ctx* ctx, cudaStream_t stream, const void* kernel, int grid, int threads, size_t smem,
                       void** args, const GridSync& sync) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeCooperative;
  attr.val.cooperative = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelExC(&cfg, kernel, args);
  if (e != cudaSuccess) {
    ctx->barrier_arrivals = sync.base;  // nothing ran: the barrier word stands where it stood
    return cuda_fail(ctx, e, __FILE__, __LINE__);
  }
  return GSB_OK;
}

i64* ctx_counters(gsb_ctx* ctx) { return ctx->counters; }
int ctx_device(gsb_ctx* ctx) { return ctx->device; }

// Waits for `stream`.  By default with cudaStreamSynchronize (the calling thread may spin); with
// GSB_OPT_BLOCKING_WAIT through an event created with cudaEventBlockingSync, which puts the thread to sleep — what a
// host that runs several streams from several threads (or several processes per machine) wants.
static int ctx_wait(gsb_ctx* ctx, cudaStream_t stream) {
  if (ctx->options[GSB_OPT_BLOCKING_WAIT] == 0) {
    GSB_CUDA_OK(cudaStreamSynchronize(stream));
    return GSB_OK;
  }
  if (!ctx->wait_event)
    GSB_CUDA_OK(cudaEventCreateWithFlags(&ctx->wait_event, cudaEventBlockingSync | cudaEventDisableTiming));
  GSB_CUDA_OK(cudaEventRecord(ctx->wait_event, stream));
  GSB_CUDA_OK(cudaEventSynchronize(ctx->wait_event));
  return GSB_OK;
}

// Spins until `*word & mask == want`.  The device normally answers within microseconds; from half a millisecond on the
// stream's status is asked now and then, so that a failed launch or a stream that finished without writing the word
// (*answered = false) ends the wait.
static int ctx_spin(gsb_ctx* ctx, cudaStream_t stream, const volatile u64* word, u64 mask, u64 want, bool* answered) {
  *answered = true;
  if (ctx->options[GSB_OPT_BLOCKING_WAIT] != 0) {
    int st = ctx_wait(ctx, stream);
    if (st != GSB_OK) return st;
    *answered = (*word & mask) == want;
    return GSB_OK;
  }
  const auto begin = std::chrono::steady_clock::now();
  auto next_query = std::chrono::microseconds(500);
  for (;;) {
    for (int i = 0; i < 256; ++i) {
      if ((*word & mask) == want) {
        std::atomic_thread_fence(std::memory_order_acquire);
        return GSB_OK;
      }
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
    }
    if (std::chrono::steady_clock::now() - begin < next_query) continue;
    next_query += std::chrono::microseconds(100);
    const cudaError_t e = cudaStreamQuery(stream);
    if (e == cudaErrorNotReady) continue;
    GSB_CUDA_OK(e);
    *answered = (*word & mask) == want;
    return GSB_OK;
  }
}

Mail ctx_mail(gsb_ctx* ctx) {
  if (++ctx->mail_tag > 0xFFFF) {
    // The tags start over, and a slot that few calls post may still hold what one of them left there under a tag that comes
    // again: no word is older than its round of tags.
    volatile u64* slots = (volatile u64*)(ctx->pinned + CNT_NUM);
    for (int q = 0; q < kMailSlots; ++q) slots[q] = 0;
    ctx->mail_tag = 1;
  }
  return Mail{(u64*)(ctx->pinned + CNT_NUM), ctx->mail_tag << 48};
}

int ctx_wait_mail(gsb_ctx* ctx, cudaStream_t stream, const Mail& mail, int n, i64* values, bool* error) {
  *error = false;
  for (int q = 0; q < n; ++q) {
    const volatile u64* word = mail.word + q;
    bool answered;
    int st = ctx_spin(ctx, stream, word, 0xFFFFull << 48, mail.tag, &answered);
    if (st != GSB_OK) return st;
    if (!answered) {  // the stream is done and nothing was posted: only a kernel that gave up does that
      *error = true;
      values[q] = 0;
      continue;
    }
    const u64 w = *word;
    values[q] = (i64)(w & kMailValueMask);
    *error |= ((w >> kMailErrorBit) & 1ull) != 0;
  }
  return GSB_OK;
}

int ctx_mail_result(gsb_ctx* ctx, cudaStream_t stream, const Mail& mail, int n, i64* values) {
  bool error;
  int st = ctx_wait_mail(ctx, stream, mail, n, values, &error);
  if (st != GSB_OK) return st;
  return error ? ctx_check_device_error(ctx, stream) : GSB_OK;
}

// One warp: counters -> page-locked host memory, then the ticket the host spins on.
__global__ void k_publish_counters(const i64* __restrict__ counters, int first, int n, i64* host, u64 ticket) {
  for (int q = threadIdx.x; q < n; q += 32) ((volatile i64*)host)[first + q] = ((const volatile i64*)counters)[first + q];
  __threadfence_system();
  __syncwarp();
  if (threadIdx.x == 0) st_volatile_u64((u64*)host + CNT_NUM + kMailSlots, ticket);
}

int ctx_fetch_counters(gsb_ctx* ctx, cudaStream_t stream, int first, int n, const i64** out) {
  ctx->ticket += 1;
  k_publish_counters<<<1, 32, 0, stream>>>(ctx->counters, first, n, ctx->pinned, ctx->ticket);
  GSB_LAUNCH_OK();
  bool answered;
  int st = ctx_spin(ctx, stream, (const volatile u64*)ctx->pinned + CNT_NUM + kMailSlots, ~0ull, ctx->ticket, &answered);
  if (st != GSB_OK) return st;
  if (!answered) return GSB_ERR_CUDA;
  *out = ctx->pinned + first;
  return GSB_OK;
}

int ctx_check_device_error(gsb_ctx* ctx, cudaStream_t stream) {
  const i64* c;
  int st = ctx_fetch_counters(ctx, stream, CNT_ERROR, 2, &c);
  if (st != GSB_OK) return st;
  if (c[0] != 0) {
    int code = (int)c[0];
    snprintf(ctx->message, sizeof(ctx->message), "device-side error %d (%s), detail %lld", code,
             gsb_status_string(code), (long long)c[1]);
    GSB_CUDA_OK(cudaMemsetAsync(ctx->counters + CNT_ERROR, 0, 2 * sizeof(i64), stream));
    GSB_CUDA_OK(cudaMemsetAsync(ctx->counters + CNT_LOST, 0, sizeof(i64), stream));
    // the mark of a grid barrier that was given up, the top byte of its word (grid_sync.cuh)
    GSB_CUDA_OK(cudaMemsetAsync((char*)(ctx->counters + CNT_NUM) + kBarrierCountBits / 8, 0, 1, stream));
    {
      int st2 = ctx_wait(ctx, stream);
      if (st2 != GSB_OK) return st2;
    }
    return code;
  }
  return GSB_OK;
}

void ctx_count_launches(gsb_ctx* ctx, int n) { ctx->launches += n; }
void ctx_count_id_bound_refusal(gsb_ctx* ctx) { ctx->id_bound_refusals += 1; }

void ctx_prof_begin(gsb_ctx* ctx, int kid, cudaStream_t stream) {
  ctx->launches += 1;
  if (!ctx->profiling) return;
  if (ctx->ev_used == ctx->ev_begin->size()) {
    cudaEvent_t a, b;
    if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) return;
    ctx->ev_begin->push_back(a);
    ctx->ev_end->push_back(b);
    ctx->ev_kid->push_back(kid);
  }
  (*ctx->ev_kid)[ctx->ev_used] = kid;
  cudaEventRecord((*ctx->ev_begin)[ctx->ev_used], stream);
}

void ctx_prof_end(gsb_ctx* ctx, int kid, cudaStream_t stream) {
  (void)kid;
  if (!ctx->profiling || ctx->ev_used >= ctx->ev_begin->size()) return;
  cudaEventRecord((*ctx->ev_end)[ctx->ev_used], stream);
  ctx->ev_used += 1;
}

// Folds the recorded event pairs into the per-kernel totals (waits for the events).
static void prof_collect(gsb_ctx* ctx) {
  for (size_t i = 0; i < ctx->ev_used; ++i) {
    float ms = 0.f;
    if (cudaEventSynchronize((*ctx->ev_end)[i]) == cudaSuccess &&
        cudaEventElapsedTime(&ms, (*ctx->ev_begin)[i], (*ctx->ev_end)[i]) == cudaSuccess) {
      const int k = (*ctx->ev_kid)[i];
      ctx->prof_ms[k] += ms;
      ctx->prof_launches[k] += 1;
    }
  }
  ctx->ev_used = 0;
}

}  // namespace gsb

extern "C" {

int gsb_ctx_create(int device, gsb_ctx** out_ctx) {
  if (!out_ctx) return GSB_ERR_INVALID_ARGUMENT;
  *out_ctx = nullptr;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || device < 0 || device >= count) return e != cudaSuccess ? GSB_ERR_CUDA : GSB_ERR_INVALID_ARGUMENT;
  gsb_ctx* ctx = new (std::nothrow) gsb_ctx();
  if (!ctx) return GSB_ERR_OUT_OF_MEMORY;
  memset(ctx, 0, sizeof(*ctx));
  ctx->device = device;
  ctx->ev_begin = new std::vector<cudaEvent_t>();
  ctx->ev_end = new std::vector<cudaEvent_t>();
  ctx->ev_kid = new std::vector<int>();
  ctx->options[GSB_OPT_MAX_POLLS] = 1 << 22;
  ctx->options[GSB_OPT_TABLE_SLOTS] = 0;
  ctx->options[GSB_OPT_RELABEL_PATH] = 0;
  ctx->options[GSB_OPT_DIRECT_TABLE_BUDGET] = 6ll << 30;
  int prev = 0;
  cudaGetDevice(&prev);
  int st = GSB_OK;
  do {
    if ((e = cudaSetDevice(device)) != cudaSuccess) break;
    if ((e = cudaMalloc((void**)&ctx->counters, sizeof(i64) * (gsb::CNT_NUM + 1))) != cudaSuccess) break;
    if ((e = cudaMemset(ctx->counters, 0, sizeof(i64) * (gsb::CNT_NUM + 1))) != cudaSuccess) break;
    if ((e = cudaMallocHost((void**)&ctx->pinned, sizeof(i64) * (gsb::CNT_NUM + gsb::kMailSlots + 1))) != cudaSuccess) break;
    memset(ctx->pinned, 0, sizeof(i64) * (gsb::CNT_NUM + gsb::kMailSlots + 1));
  } while (0);
  if (e != cudaSuccess) {
    st = gsb::cuda_fail(nullptr, e, __FILE__, __LINE__);
    if (ctx->counters) cudaFree(ctx->counters);
    if (ctx->pinned) cudaFreeHost(ctx->pinned);
    delete ctx->ev_begin;
    delete ctx->ev_end;
    delete ctx->ev_kid;
    delete ctx;
    cudaSetDevice(prev);
    return st;
  }
  cudaSetDevice(prev);
  *out_ctx = ctx;
  return GSB_OK;
}

int gsb_ctx_destroy(gsb_ctx* ctx) {
  if (!ctx) return GSB_OK;
  int prev = 0;
  cudaGetDevice(&prev);
  cudaSetDevice(ctx->device);
  cudaDeviceSynchronize();
  if (ctx->workspace) cudaFree(ctx->workspace);
  if (ctx->tile_words) cudaFree(ctx->tile_words);
  if (ctx->direct_tables) cudaFree(ctx->direct_tables);
  for (void* t : ctx->epoch_table)
    if (t) cudaFree(t);
  if (ctx->wait_event) cudaEventDestroy(ctx->wait_event);
  if (ctx->counters) cudaFree(ctx->counters);
  if (ctx->pinned) cudaFreeHost(ctx->pinned);
  for (size_t i = 0; i < ctx->ev_begin->size(); ++i) {
    cudaEventDestroy((*ctx->ev_begin)[i]);
    cudaEventDestroy((*ctx->ev_end)[i]);
  }
  delete ctx->ev_begin;
  delete ctx->ev_end;
  delete ctx->ev_kid;
  cudaSetDevice(prev);
  delete ctx;
  return GSB_OK;
}

const char* gsb_status_string(int status) {
  switch (status) {
    case GSB_OK: return "ok";
    case GSB_ERR_INVALID_ARGUMENT: return "invalid argument";
    case GSB_ERR_CUDA: return "CUDA runtime error";
    case GSB_ERR_OUT_OF_MEMORY: return "out of device memory";
    case GSB_ERR_CAPACITY: return "output capacity too small";
    case GSB_ERR_LOOKBACK_TIMEOUT: return "bounded device-side wait expired";
    case GSB_ERR_TABLE_FULL: return "hash table full";
    case GSB_ERR_UNSUPPORTED: return "unsupported argument combination";
    case GSB_ERR_INDEX_RANGE: return "index out of range";
    default: return "unknown status";
  }
}

const char* gsb_last_error_message(gsb_ctx* ctx) { return ctx ? ctx->message : ""; }

int gsb_check_device_status(gsb_ctx* ctx, void* stream) {
  GSB_ENTER(ctx);
  return gsb::ctx_check_device_error(ctx, (cudaStream_t)stream);
}

const char* gsb_version(void) { return "gsb200 0.2 sm_100a"; }

int gsb_ctx_set_option(gsb_ctx* ctx, int option, int64_t value) {
  if (!ctx || option < 0 || option >= GSB_OPT_NUM) return GSB_ERR_INVALID_ARGUMENT;
  switch (option) {
    case GSB_OPT_MAX_POLLS:
      if (value < 1 || value > (1ll << 30)) return GSB_ERR_INVALID_ARGUMENT;
      break;
    case GSB_OPT_TABLE_SLOTS:
      if (value < 0) return GSB_ERR_INVALID_ARGUMENT;
      break;
    case GSB_OPT_RELABEL_PATH:
      if (value < 0 || value > 5) return GSB_ERR_INVALID_ARGUMENT;
      break;
    case GSB_OPT_BLOCKING_WAIT:
      if (value < 0 || value > 1) return GSB_ERR_INVALID_ARGUMENT;
      break;
    case GSB_OPT_SAMPLE_PATH:
      if (value < 0 || value > 2) return GSB_ERR_INVALID_ARGUMENT;
      break;
    case GSB_OPT_DIRECT_TABLE_BUDGET:
      if (value < 0) return GSB_ERR_INVALID_ARGUMENT;
      break;
  }
  ctx->options[option] = value;
  return GSB_OK;
}

int gsb_ctx_get_option(gsb_ctx* ctx, int option, int64_t* value_host) {
  if (!ctx || !value_host || option < 0 || option >= GSB_OPT_NUM) return GSB_ERR_INVALID_ARGUMENT;
  *value_host = ctx->options[option];
  return GSB_OK;
}

int64_t gsb_launch_count(gsb_ctx* ctx) { return ctx ? ctx->launches : 0; }

int64_t gsb_id_bound_refusals(gsb_ctx* ctx) { return ctx ? ctx->id_bound_refusals : 0; }

int gsb_read_counts(gsb_ctx* ctx, void* stream, int64_t* nnz_host, int64_t* unique_host) {
  GSB_ENTER(ctx);
  const i64* c;
  int st = gsb::ctx_fetch_counters(ctx, (cudaStream_t)stream, gsb::CNT_NNZ, 2, &c);
  if (st != GSB_OK) return st;
  if (nnz_host) *nnz_host = c[0];
  if (unique_host) *unique_host = c[1];
  return GSB_OK;
}

int gsb_profile_enable(gsb_ctx* ctx, int on) {
  if (!ctx) return GSB_ERR_INVALID_ARGUMENT;
  if (!on && ctx->profiling) gsb::prof_collect(ctx);
  if (on) {
    // Events are created here, not at the first launches that need them: creating an event is a driver call that
    // several processes on one machine contend for, and it would otherwise land inside the caller's timed region.
    constexpr size_t kPool = 4096;
    while (ctx->ev_begin->size() < kPool) {
      cudaEvent_t a, b;
      if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) break;
      ctx->ev_begin->push_back(a);
      ctx->ev_end->push_back(b);
      ctx->ev_kid->push_back(0);
    }
  }
  ctx->profiling = on != 0;
  return GSB_OK;
}

int gsb_profile_reset(gsb_ctx* ctx) {
  if (!ctx) return GSB_ERR_INVALID_ARGUMENT;
  gsb::prof_collect(ctx);
  for (int k = 0; k < gsb::KID_NUM; ++k) {
    ctx->prof_ms[k] = 0.0;
    ctx->prof_launches[k] = 0;
  }
  return GSB_OK;
}

int gsb_profile_num_kernels(void) { return gsb::KID_NUM; }

const char* gsb_profile_kernel_name(int kid) {
  static const char* names[gsb::KID_NUM] = {
      "count_scan",     "slice_fill",   "sample_uniform", "sample_keepdim", "sample_weighted", "table_clear",
      "table_insert",   "first_compact", "relabel",       "random_walk",    "sddmm_dot",       "sddmm_generic",
      "segment",        "row_filter",   "list_sample",    "sort",           "format",          "partition_count",
      "partition_scatter", "bucket_resolve", "first_bits",  "rank_emit",      "other"};
  return (kid >= 0 && kid < gsb::KID_NUM) ? names[kid] : "";
}

int gsb_profile_read(gsb_ctx* ctx, int kid, double* total_ms, int64_t* launches) {
  if (!ctx || kid < 0 || kid >= gsb::KID_NUM) return GSB_ERR_INVALID_ARGUMENT;
  gsb::prof_collect(ctx);
  if (total_ms) *total_ms = ctx->prof_ms[kid];
  if (launches) *launches = ctx->prof_launches[kid];
  return GSB_OK;
}

}  // extern "C"
