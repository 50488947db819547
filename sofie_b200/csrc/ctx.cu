// Context of one emitted Session on one GPU: stream, device arena, persistent allocations (weights),
// pinned staging for host<->device traffic, optional CUDA graph of the infer() kernel sequence.
//
// Replaces what the reference emits as Session data members: one std::vector<float> per weight
// (reference: src/SOFIE_core/src/RModel.cxx:574-595) and the `new char[]` intermediate pool
// (reference: src/SOFIE_core/src/RModel.cxx:597-604).
#include "common.cuh"
#include "contract.cuh"
#include "host_convert.cuh"
#include "host_pool.cuh"

#include <cstdlib>
#include <memory>
#include <utility>
#include <vector>

namespace sofie {

static thread_local char g_last_error[512] = "";
static thread_local int g_last_engine = SOFIE_ENGINE_NONE;
static thread_local int g_default_device = -1; // device of contexts created with device < 0 on this thread (-1: environment)
// Initial kernel-family choice from the environment (SOFIE_CUDA_ENGINE = 0, 1 or 2), for A/B runs.
static int initial_engine()
{
   const char *env = std::getenv("SOFIE_CUDA_ENGINE");
   int v = env ? std::atoi(env) : 0;
   return (v >= 0 && v <= 2) ? v : 0;
}
static int g_forced_engine = initial_engine();

char *last_error_buffer() { return g_last_error; }

int fail(int status, const char *fmt, ...)
{
   va_list ap;
   va_start(ap, fmt);
   vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
   va_end(ap);
   return status;
}

void set_last_engine(int engine) { g_last_engine = engine; }
bool pdl_enabled()
{
   static const bool v = [] { const char *e = getenv("SOFIE_CUDA_PDL"); return !e || atoi(e) != 0; }();
   return v;
}
int forced_engine() { return g_forced_engine; }

// Streams of contexts report into their context's word; every other stream into one word per device,
// allocated on first use with that device current.
static std::mutex g_status_mutex;
static uint32_t *g_status_words[64] = {nullptr};
static std::vector<std::pair<cudaStream_t, uint32_t *>> g_stream_status;

void register_stream_status(cudaStream_t stream, uint32_t *word)
{
   std::lock_guard<std::mutex> lock(g_status_mutex);
   g_stream_status.emplace_back(stream, word);
}

void unregister_stream_status(cudaStream_t stream)
{
   std::lock_guard<std::mutex> lock(g_status_mutex);
   for (size_t i = 0; i < g_stream_status.size(); i++)
      if (g_stream_status[i].first == stream) {
         g_stream_status.erase(g_stream_status.begin() + i);
         return;
      }
}

uint32_t *device_status_word(cudaStream_t stream)
{
   int dev = 0;
   std::lock_guard<std::mutex> lock(g_status_mutex);
   for (auto &e : g_stream_status)
      if (e.first == stream) return e.second;
   if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return nullptr;
   if (!g_status_words[dev]) {
      uint32_t *p = nullptr;
      if (cudaMalloc(&p, 256) != cudaSuccess) return nullptr;
      if (cudaMemset(p, 0, 256) != cudaSuccess) return nullptr;
      g_status_words[dev] = p;
   }
   return g_status_words[dev];
}

} // namespace sofie

// Pageable host memory crosses PCIe through pinned staging slots: while the copy engine drains some slots the CPU fills
// the next, so the host's copy and the DMA overlap instead of alternating. The ring is small enough to stay in the host's
// last-level cache: the filled slot is read by the DMA from there and the host's memory sees the source's bytes alone.
constexpr int kStagingSlots = 8;
constexpr size_t kStagingSlot = size_t(2) << 20;
constexpr size_t kStagingBytes = kStagingSlots * kStagingSlot;
constexpr size_t kLandInPieces = size_t(5) << 19; // a result that lands in one piece below this (sofie_cuda_ctx_result_part)
constexpr int kLandings = 2 * SOFIE_CUDA_MAX_PARTS - 1; // copies of a result: a whole one's pieces and seven parts more
constexpr size_t kPastCaches = size_t(32) << 20; // a result from which on the host's caches hold no useful part of it

struct sofie_cuda_ctx {
   int device = 0;
   cudaStream_t stream = nullptr;
   char *arena = nullptr;
   size_t arena_bytes = 0;
   std::vector<void *> owned;
   char *staging = nullptr; // pinned ring, made on first use
   struct Slot {
      cudaEvent_t event = nullptr;   // the copy that read the slot has completed, when `recorded`
      cudaStream_t stream = nullptr; // the stream that copy was issued on
      bool busy = false, recorded = false;
   } slots[kStagingSlots];
   int next_slot = 0;
   sofie::HostPool *host_pool = nullptr; // borrowed from the process's while a transfer runs
   // one slot being filled by the pool: `bytes` of the slot from `src`
   struct Fill {
      sofie::HostConvert how;
      const char *src = nullptr;
      char *mem = nullptr;
      Slot *slot = nullptr;
      size_t bytes = 0, piece = 0;
   } fills[2];
   int next_fill = 0;
   Fill *ahead = nullptr; // begun by sofie_cuda_ctx_stage_ahead for a copy that is yet to be asked for
   int fail_copy = 0;     // self test: the fail_copy-th staged copy from now on is refused (0: none)
   void *result = nullptr;  // pinned, grown on demand: where results land that were not given a pinned place of their own
   size_t result_bytes = 0;
   // the result of one inference on its way to the host, between result_begin and result_end
   struct Landing {
      bool open = false;
      char *out = nullptr;    // where the caller wants it (nullptr: anywhere)
      char *land = nullptr;   // pinned memory the copies write: out, or `result`
      const char *mapped = nullptr; // the kernels wrote it to host memory themselves
      size_t bytes = 0;
      int parts = 0;  // the caller's
      int pieces = 0; // copies: a part, or (one part only, the whole) a piece of it
      size_t offset[kLandings], count[kLandings];
   } landing;
   cudaStream_t result_stream = nullptr; // results that are copied part by part, under the kernels of later parts
   cudaEvent_t ready_event = nullptr;    // a part's kernels are done
   cudaEvent_t landed_event[kLandings] = {};
   struct Captured {
      cudaGraph_t graph = nullptr;
      cudaGraphExec_t exec = nullptr;
      cudaKernelNodeParams only_kernel = {}; // the graph's one kernel (func set), launched without the graph
   } captured, kept; // kept: set aside by sofie_cuda_ctx_graph_swap
   bool capturing = false;
   // small results written by the last kernel straight into mapped pinned host memory (no device-to-host copy)
   std::vector<std::pair<char *, size_t>> host_outputs;
   // small inputs that the first kernel reads from mapped pinned host memory, each element once
   std::vector<std::pair<char *, size_t>> host_inputs;
   // pipelined input upload: parts of the input are copied on a stream of their own, one event per part
   cudaStream_t copy_stream = nullptr;
   cudaEvent_t part_event[SOFIE_CUDA_MAX_PARTS] = {};
   // status word of this context's kernels (mapped pinned host memory, 256 bytes)
   uint32_t *status = nullptr;
   // per-operator device timers (off unless SOFIE_CUDA_TIMERS is set or sofie_cuda_ctx_timers says so)
   bool timers_on = false;
   std::vector<cudaEvent_t> marks;
   std::vector<char> mark_seen;
};

using namespace sofie;

// The context's status word, read after the stream has been synchronised: a plain host load.
static int report_status(sofie_cuda_ctx *ctx)
{
   volatile uint32_t *w = ctx->status;
   if (w && w[0]) {
      const uint32_t code = w[0], d1 = w[1], d2 = w[2], d3 = w[3];
      w[1] = w[2] = w[3] = 0;
      w[0] = 0;
      return fail(SOFIE_CUDA_ERR_DEVICE, "device status 0x%x (detail 0x%x 0x%x 0x%x)", code, d1, d2, d3);
   }
   return SOFIE_CUDA_OK;
}


namespace {
struct DeviceGuard {
   int prev = -1;
   explicit DeviceGuard(int dev)
   {
      cudaGetDevice(&prev);
      if (prev != dev) cudaSetDevice(dev);
      else prev = -1;
   }
   ~DeviceGuard()
   {
      if (prev >= 0) cudaSetDevice(prev);
   }
};
} // namespace

extern "C" {

const char *sofie_cuda_strerror(int status)
{
   switch (status) {
   case SOFIE_CUDA_OK: return "success";
   case SOFIE_CUDA_ERR_INVALID: return "invalid argument";
   case SOFIE_CUDA_ERR_UNSUPPORTED: return "unsupported configuration";
   case SOFIE_CUDA_ERR_CUDA: return "CUDA error";
   case SOFIE_CUDA_ERR_NOMEM: return "out of device memory or arena range";
   case SOFIE_CUDA_ERR_DEVICE: return "kernel reported a device-side failure";
   default: return "unknown status";
   }
}

const char *sofie_cuda_last_error(void) { return last_error_buffer(); }
int sofie_cuda_abi_version(void) { return SOFIE_CUDA_ABI_VERSION; }
int sofie_cuda_last_engine(void) { return g_last_engine; }

int sofie_cuda_set_engine(int engine)
{
   SOFIE_REQUIRE(engine >= 0 && engine <= 2, "engine must be 0, 1 or 2");
   g_forced_engine = engine;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_set_default_device(int device)
{
   g_default_device = device < 0 ? -1 : device;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_device_count(int *count)
{
   SOFIE_REQUIRE(count != nullptr, "count is NULL");
   *count = 0;
   cudaError_t err = cudaGetDeviceCount(count);
   if (err != cudaSuccess) {
      *count = 0;
      cudaGetLastError();
      return fail(SOFIE_CUDA_ERR_CUDA, "cudaGetDeviceCount: %s", cudaGetErrorString(err));
   }
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_create(sofie_cuda_ctx **out, int device, size_t arena_bytes)
{
   SOFIE_REQUIRE(out != nullptr, "ctx output pointer is NULL");
   *out = nullptr;
   if (device < 0 && g_default_device >= 0) device = g_default_device;
   if (device < 0) {
      const char *env = std::getenv("SOFIE_CUDA_DEVICE");
      device = env ? std::atoi(env) : 0;
   }
   int count = 0;
   int rc = sofie_cuda_device_count(&count);
   if (rc) return rc;
   if (device >= count) return fail(SOFIE_CUDA_ERR_INVALID, "device %d requested, %d visible", device, count);
   DeviceGuard guard(device);
   auto *ctx = new sofie_cuda_ctx();
   ctx->device = device;
   cudaError_t err = cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking);
   if (err == cudaSuccess && arena_bytes) {
      ctx->arena_bytes = (arena_bytes + 255) & ~size_t(255);
      err = cudaMalloc(&ctx->arena, ctx->arena_bytes);
   }
   if (err == cudaSuccess) {
      void *w = nullptr, *d = nullptr;
      err = cudaHostAlloc(&w, 256, cudaHostAllocMapped);
      if (err == cudaSuccess) {
         std::memset(w, 0, 256);
         err = cudaHostGetDevicePointer(&d, w, 0);
         if (err == cudaSuccess && d != w) err = cudaErrorNotSupported; // needs unified addressing
         ctx->status = static_cast<uint32_t *>(w);
      }
   }
   if (err != cudaSuccess) {
      if (ctx->status) cudaFreeHost(ctx->status);
      if (ctx->arena) cudaFree(ctx->arena);
      if (ctx->stream) cudaStreamDestroy(ctx->stream);
      delete ctx;
      cudaGetLastError();
      return fail(err == cudaErrorMemoryAllocation ? SOFIE_CUDA_ERR_NOMEM : SOFIE_CUDA_ERR_CUDA,
                  "context creation on device %d (arena %zu bytes): %s", device, arena_bytes, cudaGetErrorString(err));
   }
   register_stream_status(ctx->stream, ctx->status);
   HostPools::get().user_begins();
   if (const char *t = std::getenv("SOFIE_CUDA_TIMERS")) ctx->timers_on = std::atoi(t) != 0;
   *out = ctx;
   return SOFIE_CUDA_OK;
}

static void settle(sofie_cuda_ctx *ctx);

int sofie_cuda_ctx_destroy(sofie_cuda_ctx *ctx)
{
   if (!ctx) return SOFIE_CUDA_OK;
   DeviceGuard guard(ctx->device);
   // nothing of this context may still be running or copying when its memory goes away
   settle(ctx);
   HostPools::get().user_ends();
   cudaStreamSynchronize(ctx->stream);
   if (ctx->copy_stream) cudaStreamSynchronize(ctx->copy_stream);
   if (ctx->result_stream) cudaStreamSynchronize(ctx->result_stream);
   unregister_stream_status(ctx->stream);
   for (auto *g : {&ctx->captured, &ctx->kept}) {
      if (g->exec) cudaGraphExecDestroy(g->exec);
      if (g->graph) cudaGraphDestroy(g->graph);
   }
   for (void *p : ctx->owned) cudaFree(p);
   if (ctx->arena) cudaFree(ctx->arena);
   for (auto &h : ctx->host_outputs) cudaFreeHost(h.first);
   for (auto &h : ctx->host_inputs) cudaFreeHost(h.first);
   if (ctx->staging) cudaFreeHost(ctx->staging);
   if (ctx->result) cudaFreeHost(ctx->result);
   splitk_scratch_release(ctx->device, ctx->stream);
   if (ctx->copy_stream) cudaStreamDestroy(ctx->copy_stream);
   if (ctx->status) cudaFreeHost(ctx->status);
   if (ctx->result_stream) cudaStreamDestroy(ctx->result_stream);
   for (auto &s : ctx->slots)
      if (s.event) cudaEventDestroy(s.event);
   for (cudaEvent_t e : ctx->landed_event)
      if (e) cudaEventDestroy(e);
   if (ctx->ready_event) cudaEventDestroy(ctx->ready_event);
   for (cudaEvent_t e : ctx->marks)
      if (e) cudaEventDestroy(e);
   for (cudaEvent_t e : ctx->part_event)
      if (e) cudaEventDestroy(e);
   cudaStreamDestroy(ctx->stream);
   delete ctx;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_stream(sofie_cuda_ctx *ctx, void **stream)
{
   SOFIE_REQUIRE(ctx && stream, "NULL argument");
   *stream = ctx->stream;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_device(sofie_cuda_ctx *ctx, int *device)
{
   SOFIE_REQUIRE(ctx && device, "NULL argument");
   *device = ctx->device;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_arena(sofie_cuda_ctx *ctx, size_t offset, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx && dptr, "NULL argument");
   SOFIE_REQUIRE((offset & 255) == 0, "arena offset %zu is not 256-byte aligned", offset);
   if (offset > ctx->arena_bytes || bytes > ctx->arena_bytes - offset)
      return fail(SOFIE_CUDA_ERR_NOMEM, "arena slice [%zu, +%zu) exceeds arena of %zu bytes", offset, bytes,
                  ctx->arena_bytes);
   *dptr = ctx->arena + offset;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_alloc(sofie_cuda_ctx *ctx, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx && dptr, "NULL argument");
   DeviceGuard guard(ctx->device);
   void *p = nullptr;
   cudaError_t err = cudaMalloc(&p, bytes ? bytes : 256);
   if (err != cudaSuccess) {
      cudaGetLastError();
      return fail(SOFIE_CUDA_ERR_NOMEM, "cudaMalloc of %zu bytes: %s", bytes, cudaGetErrorString(err));
   }
   ctx->owned.push_back(p);
   *dptr = p;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_upload(sofie_cuda_ctx *ctx, const void *host, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx && dptr && (host || bytes == 0), "NULL argument");
   int rc = sofie_cuda_ctx_alloc(ctx, bytes, dptr);
   if (rc) return rc;
   DeviceGuard guard(ctx->device);
   if (bytes) {
      SOFIE_CUDA_TRY(cudaMemcpyAsync(*dptr, host, bytes, cudaMemcpyHostToDevice, ctx->stream));
      SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   }
   return SOFIE_CUDA_OK;
}

static int ensure_pool(sofie_cuda_ctx *ctx)
{
   if (!ctx->host_pool) ctx->host_pool = HostPools::get().borrow();
   return ctx->host_pool ? SOFIE_CUDA_OK : fail(SOFIE_CUDA_ERR_NOMEM, "no memory for the helper threads");
}

// No job is left: the helpers are another transfer's.
static void release_pool(sofie_cuda_ctx *ctx)
{
   if (ctx->host_pool) HostPools::get().give_back(ctx->host_pool);
   ctx->host_pool = nullptr;
}

static int ensure_staging(sofie_cuda_ctx *ctx)
{
   int rc = ensure_pool(ctx);
   if (rc || ctx->staging) return rc;
   void *p = nullptr;
   SOFIE_CUDA_TRY(cudaMallocHost(&p, kStagingBytes));
   ctx->staging = static_cast<char *>(p);
   for (auto &s : ctx->slots) SOFIE_CUDA_TRY(cudaEventCreateWithFlags(&s.event, cudaEventDisableTiming));
   return SOFIE_CUDA_OK;
}

// The next slot of the ring, once the copy that last read it is done.
static int take_slot(sofie_cuda_ctx *ctx, sofie_cuda_ctx::Slot **slot, char **mem)
{
   const int i = ctx->next_slot;
   ctx->next_slot = (i + 1) % kStagingSlots;
   sofie_cuda_ctx::Slot &s = ctx->slots[i];
   if (s.busy) {
      if (s.recorded) SOFIE_CUDA_TRY(cudaEventSynchronize(s.event));
      else SOFIE_CUDA_TRY(cudaStreamSynchronize(s.stream));
      s.busy = false;
   }
   *slot = &s;
   *mem = ctx->staging + (size_t)i * kStagingSlot;
   return SOFIE_CUDA_OK;
}

// every copy of this context has completed (its streams were waited for): all slots are free
static void slots_free(sofie_cuda_ctx *ctx)
{
   for (auto &s : ctx->slots) s.busy = false;
}

// Pageable host memory is staged through one pinned buffer in chunks; memory the caller already
// pinned (cudaHostRegister / cudaMallocHost) is copied directly and stays asynchronous.
static bool is_pinned(const void *p)
{
   cudaPointerAttributes attr;
   if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
      cudaGetLastError();
      return false;
   }
   return attr.type == cudaMemoryTypeHost;
}

static void fill_piece(void *arg, size_t i)
{
   const auto &f = *static_cast<const sofie_cuda_ctx::Fill *>(arg);
   const size_t off = i * f.piece, n = f.bytes - off < f.piece ? f.bytes - off : f.piece;
   host_convert(f.how, f.mem + off, f.src + off * f.how.ratio(), n);
}

// Starts filling the ring's next slot with `bytes` (at most a slot) from `src`.
static int begin_fill(sofie_cuda_ctx *ctx, const HostConvert &how, const char *src, size_t bytes, sofie_cuda_ctx::Fill **out)
{
   auto &f = ctx->fills[ctx->next_fill];
   ctx->next_fill ^= 1;
   f.how = how;
   f.src = src;
   f.bytes = bytes;
   int rc = take_slot(ctx, &f.slot, &f.mem);
   if (rc) return rc;
   // 16 to 256 KB of source per piece: several for every thread, each long enough for the prefetchers; a source of less than
   // kAloneBytes is the caller's alone (two threads' hand-over costs as much as it saves)
   const size_t src_bytes = bytes * how.ratio();
   size_t piece = src_bytes / (3 * ctx->host_pool->threads());
   piece = src_bytes < HostPool::kAloneBytes ? src_bytes : (piece < (size_t(16) << 10) ? (size_t(16) << 10) : (piece > HostPool::kPieceBytes ? HostPool::kPieceBytes : piece));
   f.piece = (piece / how.ratio() + 255) & ~size_t(255);
   ctx->host_pool->begin(fill_piece, &f, (bytes + f.piece - 1) / f.piece);
   *out = &f;
   return SOFIE_CUDA_OK;
}

// No job of the pool reads the caller's memory any more.
static void settle(sofie_cuda_ctx *ctx)
{
   if (ctx->host_pool) ctx->host_pool->finish();
   ctx->ahead = nullptr;
   release_pool(ctx);
}

// A small input's way out of pinned memory: read across PCIe by the SMs themselves. The copy engine takes 10 us and more for 256 KB
// (5 us of bytes), this kernel 7, and it costs the host no more than the copy's launch.
constexpr size_t kPullMaxBytes = size_t(512) << 10;
// An input that nothing else is copied beside, in two of them: the second half is put into pinned memory under the first one's way. 0.7 MB (60 images of the fp32 network) 80.8 -> 72.4 us a
// call, 0.8 MB (98 of the residual block) 75 -> 68, 1 MB (4096 rows of the perceptron) 90 -> 80; 1.2 MB no difference, 1.6 MB 95 -> 100; ranges of an input, with results on their
// way out beside them, 284 -> 319 (int8 perceptron, 8192 rows).
constexpr size_t kPullTwiceBytes = size_t(1) << 20;
// Its words are of 16 bytes: a piece behind a fill that was begun ahead, of a length its caller chose, need not start on one and is copied.
constexpr int kPullThreads = 256;
__global__ void __launch_bounds__(kPullThreads) pull_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, uint32_t n16, const uint8_t *__restrict__ src1,
                                                            uint8_t *__restrict__ dst1, uint32_t rest)
{
   const uint32_t i = blockIdx.x * kPullThreads + threadIdx.x;
   if (i < n16) dst[i] = src[i];
   if (i < rest) dst1[i] = src1[i];
}

static int pull(cudaStream_t stream, void *dst, const void *src, size_t bytes)
{
   const uint32_t n16 = (uint32_t)(bytes / 16), rest = (uint32_t)(bytes % 16);
   const uint32_t blocks = (n16 > rest ? n16 : rest) / kPullThreads + 1;
   pull_kernel<<<blocks, kPullThreads, 0, stream>>>(static_cast<const uint4 *>(src), static_cast<uint4 *>(dst), n16, static_cast<const uint8_t *>(src) + 16 * (size_t)n16,
                                                    static_cast<uint8_t *>(dst) + 16 * (size_t)n16, rest);
   SOFIE_LAUNCH_CHECK("pull_kernel");
   return SOFIE_CUDA_OK;
}

static int stage_slots(sofie_cuda_ctx *ctx, const HostConvert &how, void *dst, const void *src_v, size_t bytes, cudaStream_t stream)
{
   int rc = ensure_staging(ctx);
   if (rc || bytes == 0) return rc;
   const char *src = static_cast<const char *>(src_v);
   // slots filled just far enough that the DMA of the first starts early, but not so little that its fixed cost (about 3 us of
   // host time) counts
   const bool small = bytes <= (stream == ctx->stream ? kPullTwiceBytes : kPullMaxBytes) && (reinterpret_cast<uintptr_t>(dst) & 15) == 0;
   size_t step = bytes / 4;
   if (small) step = bytes <= kPullMaxBytes ? bytes : ((bytes / 2 + 4095) & ~size_t(4095));
   else step = step < (size_t(128) << 10) ? (size_t(128) << 10) : (step > kStagingSlot ? kStagingSlot : ((step + 4095) & ~size_t(4095)));
   // an event per slot only where the ring can come round before the stream is waited for anyway
   const bool record = bytes > (size_t(1) << 20);
   sofie_cuda_ctx::Fill *cur = nullptr;
   if (ctx->ahead && ctx->ahead->src == src && ctx->ahead->bytes <= bytes && ctx->ahead->how.kind == how.kind && ctx->ahead->how.scale == how.scale &&
       ctx->ahead->how.zp == how.zp) {
      cur = ctx->ahead;
      ctx->ahead = nullptr;
   } else {
      settle(ctx);
      if ((rc = ensure_pool(ctx)) || (rc = begin_fill(ctx, how, src, bytes < step ? bytes : step, &cur))) return rc;
   }
   for (size_t done = 0; done < bytes;) {
      ctx->host_pool->finish();
      sofie_cuda_ctx::Fill *now = cur;
      const size_t next = done + now->bytes;
      if (next < bytes && (rc = begin_fill(ctx, how, src + next * how.ratio(), bytes - next < step ? bytes - next : step, &cur))) return rc;
      if (ctx->fail_copy > 0 && --ctx->fail_copy == 0) rc = fail(SOFIE_CUDA_ERR_CUDA, "staged copy refused (self test)");
      else if (small && done % 16 == 0) rc = pull(stream, static_cast<char *>(dst) + done, now->mem, now->bytes);
      else SOFIE_CUDA_TRY(cudaMemcpyAsync(static_cast<char *>(dst) + done, now->mem, now->bytes, cudaMemcpyHostToDevice, stream));
      if (rc) return rc;
      now->slot->busy = true;
      now->slot->stream = stream;
      now->slot->recorded = record;
      if (record) SOFIE_CUDA_TRY(cudaEventRecord(now->slot->event, stream));
      done = next;
   }
   return SOFIE_CUDA_OK;
}

// Pageable memory to the device on `stream` (`bytes`: of the destination); returns when the last byte of the source has been
// read, or with an error, after which no helper reads the source either. While the copy of one slot is issued the helpers fill the next.
static int stage_in(sofie_cuda_ctx *ctx, const HostConvert &how, void *dst, const void *src, size_t bytes, cudaStream_t stream)
{
   const int rc = stage_slots(ctx, how, dst, src, bytes, stream);
   settle(ctx);
   return rc;
}

int sofie_cuda_ctx_h2d(sofie_cuda_ctx *ctx, void *dst, const void *src, size_t bytes)
{
   SOFIE_REQUIRE(ctx && dst && src, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "input copies are not part of the captured graph");
   DeviceGuard guard(ctx->device);
   for (auto &h : ctx->host_inputs)
      if (dst == h.first && bytes <= h.second) {
         // host memory: written here, once no kernel of an earlier pass can still be reading it
         const cudaError_t idle = cudaStreamQuery(ctx->stream);
         if (idle == cudaErrorNotReady) SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
         else SOFIE_CUDA_TRY(idle);
         std::memcpy(dst, src, bytes);
         return SOFIE_CUDA_OK;
      }
   if (is_pinned(src)) {
      SOFIE_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
      return SOFIE_CUDA_OK;
   }
   return stage_in(ctx, HostConvert(), dst, src, bytes, ctx->stream);
}

int sofie_cuda_selftest_host_pools(int transfers, int *helpers)
{
   SOFIE_REQUIRE(helpers && transfers >= 1 && transfers <= 64, "bad number of transfers");
   auto &pools = HostPools::get();
   HostPool *lent[64];
   pools.user_begins();
   int rc = SOFIE_CUDA_OK, n = 0;
   for (; n < transfers; n++) {
      if (!(lent[n] = pools.borrow())) {
         rc = fail(SOFIE_CUDA_ERR_NOMEM, "no memory for the helper threads");
         break;
      }
      helpers[n] = (int)lent[n]->threads() - 1;
   }
   while (n > 0) pools.give_back(lent[--n]);
   pools.user_ends();
   return rc;
}

int sofie_cuda_selftest_fail_copy(sofie_cuda_ctx *ctx, int nth)
{
   SOFIE_REQUIRE(ctx && nth >= 0, "NULL context or negative count");
   ctx->fail_copy = nth;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_selftest_host_copy(void *dst, const void *src, size_t bytes, size_t chunk, int threads, int repeats)
{
   SOFIE_REQUIRE((dst && src) || bytes == 0, "NULL buffer");
   SOFIE_REQUIRE(chunk > 0 && threads >= 1 && threads <= 16 && repeats >= 1, "bad chunk size, thread count or repeat count");
   HostPool pool(threads - 1);
   for (int r = 0; r < repeats; r++)
      for (size_t done = 0; done < bytes; done += chunk)
         pool.copy(static_cast<char *>(dst) + done, static_cast<const char *>(src) + done, bytes - done < chunk ? bytes - done : chunk, r % 2 != 0);
   return SOFIE_CUDA_OK;
}

// The copy stream, ready for part `part` of an input.
static int open_part(sofie_cuda_ctx *ctx, int part)
{
   SOFIE_REQUIRE(part >= 0 && part < SOFIE_CUDA_MAX_PARTS, "part index out of range");
   if (!ctx->part_event[part]) SOFIE_CUDA_TRY(cudaEventCreateWithFlags(&ctx->part_event[part], cudaEventDisableTiming));
   if (!ctx->copy_stream) SOFIE_CUDA_TRY(cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
   if (part == 0) {
      // kernels of an earlier pass that was not waited for may still read what this copy overwrites
      if (!ctx->ready_event) SOFIE_CUDA_TRY(cudaEventCreateWithFlags(&ctx->ready_event, cudaEventDisableTiming));
      SOFIE_CUDA_TRY(cudaEventRecord(ctx->ready_event, ctx->stream));
      SOFIE_CUDA_TRY(cudaStreamWaitEvent(ctx->copy_stream, ctx->ready_event, 0));
   }
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_h2d_part(sofie_cuda_ctx *ctx, void *dst, const void *src, size_t bytes, int part)
{
   SOFIE_REQUIRE(ctx && dst && src, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "input copies are not part of the captured graph");
   DeviceGuard guard(ctx->device);
   int rc = open_part(ctx, part);
   if (rc) return rc;
   // pinned memory is copied by the DMA engine alone; from pageable memory the call returns when the part has been staged, so
   // the kernels the caller launches next for this part run while the host stages the following one
   if (is_pinned(src)) {
      SOFIE_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, ctx->copy_stream));
   } else if ((rc = stage_in(ctx, HostConvert(), dst, src, bytes, ctx->copy_stream))) {
      return rc;
   }
   SOFIE_CUDA_TRY(cudaEventRecord(ctx->part_event[part], ctx->copy_stream));
   return SOFIE_CUDA_OK;
}

static int make_convert(HostConvert &how, int kind, float scale, int32_t zp)
{
   SOFIE_REQUIRE(kind >= SOFIE_CUDA_STAGE_COPY && kind <= SOFIE_CUDA_STAGE_E4M3, "unknown kind of staging");
   SOFIE_REQUIRE(kind == SOFIE_CUDA_STAGE_COPY || scale > 0.f, "scale must be positive");
   SOFIE_REQUIRE(zp >= 0 && zp <= 255, "zero point out of range");
   how.kind = kind;
   how.scale = scale;
   how.zp = zp;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_pageable(sofie_cuda_ctx *ctx, const void *src)
{
   return ctx && src && !is_pinned(src);
}

int sofie_cuda_ctx_h2d_quantized(sofie_cuda_ctx *ctx, uint8_t *dst, const float *src, size_t n, int kind, float scale, int32_t zp, int part)
{
   SOFIE_REQUIRE(ctx && dst && src, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "input copies are not part of the captured graph");
   HostConvert how;
   int rc = make_convert(how, kind, scale, zp);
   if (rc) return rc;
   SOFIE_REQUIRE(kind != SOFIE_CUDA_STAGE_COPY, "no quantisation named");
   DeviceGuard guard(ctx->device);
   if (part < 0) return stage_in(ctx, how, dst, src, n, ctx->stream);
   if ((rc = open_part(ctx, part))) return rc;
   if ((rc = stage_in(ctx, how, dst, src, n, ctx->copy_stream))) return rc;
   SOFIE_CUDA_TRY(cudaEventRecord(ctx->part_event[part], ctx->copy_stream));
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_unquantize(sofie_cuda_ctx *ctx, const uint8_t *src, float *dst, size_t n, int kind, float scale, int32_t zp)
{
   SOFIE_REQUIRE(ctx && src && dst, "NULL argument");
   SOFIE_REQUIRE(kind == SOFIE_CUDA_STAGE_U8 || kind == SOFIE_CUDA_STAGE_E4M3, "no quantisation named");
   DeviceGuard guard(ctx->device);
   return kind == SOFIE_CUDA_STAGE_U8 ? sofie_cuda_dequantize_u8(ctx->stream, src, dst, n, scale, zp) : sofie_cuda_dequantize_e4m3_f32(ctx->stream, src, dst, n, scale);
}

int sofie_cuda_ctx_stage_ahead(sofie_cuda_ctx *ctx, const void *src, size_t bytes, int kind, float scale, int32_t zp)
{
   SOFIE_REQUIRE(ctx && src, "NULL argument");
   HostConvert how;
   int rc = make_convert(how, kind, scale, zp);
   if (rc || bytes == 0 || is_pinned(src)) return rc;
   DeviceGuard guard(ctx->device);
   settle(ctx);
   if ((rc = ensure_staging(ctx))) return rc;
   return begin_fill(ctx, how, static_cast<const char *>(src), bytes < kStagingSlot ? bytes : kStagingSlot, &ctx->ahead);
}

int sofie_cuda_ctx_stage_settle(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx != nullptr, "NULL context");
   settle(ctx);
   return SOFIE_CUDA_OK;
}

int sofie_cuda_selftest_host_quantize(uint8_t *dst, const float *src, size_t n, int kind, float scale, int32_t zp)
{
   SOFIE_REQUIRE((dst && src) || n == 0, "NULL buffer");
   HostConvert how;
   int rc = make_convert(how, kind, scale, zp);
   if (rc) return rc;
   SOFIE_REQUIRE(kind != SOFIE_CUDA_STAGE_COPY, "no quantisation named");
   host_convert(how, dst, src, n);
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_wait_part(sofie_cuda_ctx *ctx, int part)
{
   SOFIE_REQUIRE(ctx != nullptr, "NULL context");
   SOFIE_REQUIRE(part >= 0 && part < SOFIE_CUDA_MAX_PARTS && ctx->part_event[part], "no copy was issued for this part");
   SOFIE_REQUIRE(!ctx->capturing, "input copies are not part of the captured graph");
   DeviceGuard guard(ctx->device);
   SOFIE_CUDA_TRY(cudaStreamWaitEvent(ctx->stream, ctx->part_event[part], 0));
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_d2h(sofie_cuda_ctx *ctx, void *dst, const void *src, size_t bytes)
{
   SOFIE_REQUIRE(ctx && dst && src, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "result copies are not part of the captured graph");
   DeviceGuard guard(ctx->device);
   if (is_pinned(dst)) {
      SOFIE_CUDA_TRY(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
      SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
      return SOFIE_CUDA_OK;
   }
   settle(ctx);
   int rc = ensure_staging(ctx);
   if (rc) return rc;
   // every copy that used the slots has to be over before results land in them
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   if (ctx->copy_stream) SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->copy_stream));
   slots_free(ctx);
   // the copies of all slots are queued first, then each is copied out as soon as it has arrived: the host memcpy of
   // one slot overlaps the DMA into the next
   size_t done = 0;
   while (done < bytes) {
      const size_t round = bytes - done < kStagingBytes ? bytes - done : kStagingBytes;
      int n = 0;
      for (size_t off = 0; off < round; off += kStagingSlot, n++) {
         const size_t chunk = round - off < kStagingSlot ? round - off : kStagingSlot;
         SOFIE_CUDA_TRY(cudaMemcpyAsync(ctx->staging + off, static_cast<const char *>(src) + done + off, chunk, cudaMemcpyDeviceToHost, ctx->stream));
         SOFIE_CUDA_TRY(cudaEventRecord(ctx->slots[n].event, ctx->stream));
      }
      for (int i = 0; i < n; i++) {
         const size_t off = (size_t)i * kStagingSlot, chunk = round - off < kStagingSlot ? round - off : kStagingSlot;
         SOFIE_CUDA_TRY(cudaEventSynchronize(ctx->slots[i].event));
         ctx->host_pool->copy(static_cast<char *>(dst) + done + off, ctx->staging + off, chunk);
      }
      done += round;
   }
   release_pool(ctx);
   return SOFIE_CUDA_OK;
}

static int host_mapped(sofie_cuda_ctx *ctx, std::vector<std::pair<char *, size_t>> &list, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx && dptr, "NULL argument");
   SOFIE_REQUIRE(bytes > 0, "empty tensor");
   DeviceGuard guard(ctx->device);
   void *p = nullptr, *d = nullptr;
   SOFIE_CUDA_TRY(cudaHostAlloc(&p, bytes, cudaHostAllocMapped));
   cudaError_t err = cudaHostGetDevicePointer(&d, p, 0);
   if (err != cudaSuccess || d != p) { // without unified addressing the two views differ: not supported here
      cudaFreeHost(p);
      cudaGetLastError();
      return fail(SOFIE_CUDA_ERR_CUDA, "mapped host memory is not addressable by the device at its host address");
   }
   std::memset(p, 0, bytes);
   list.emplace_back(static_cast<char *>(p), bytes);
   *dptr = d;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_host_output(sofie_cuda_ctx *ctx, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx != nullptr, "NULL context");
   return host_mapped(ctx, ctx->host_outputs, bytes, dptr);
}

int sofie_cuda_ctx_host_input(sofie_cuda_ctx *ctx, size_t bytes, void **dptr)
{
   SOFIE_REQUIRE(ctx != nullptr, "NULL context");
   return host_mapped(ctx, ctx->host_inputs, bytes, dptr);
}

static int ensure_result(sofie_cuda_ctx *ctx, size_t bytes)
{
   if (bytes <= ctx->result_bytes) return SOFIE_CUDA_OK;
   if (ctx->result) cudaFreeHost(ctx->result);
   ctx->result = nullptr;
   ctx->result_bytes = 0;
   SOFIE_CUDA_TRY(cudaMallocHost(&ctx->result, bytes));
   ctx->result_bytes = bytes;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_result_begin(sofie_cuda_ctx *ctx, void *out_host, size_t bytes)
{
   SOFIE_REQUIRE(ctx != nullptr, "NULL context");
   SOFIE_REQUIRE(!ctx->capturing, "result copies are not part of the captured graph");
   ctx->landing = {};
   ctx->landing.open = true;
   ctx->landing.out = static_cast<char *>(out_host);
   ctx->landing.bytes = bytes;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_result_part(sofie_cuda_ctx *ctx, const void *src, size_t offset, size_t bytes)
{
   SOFIE_REQUIRE(ctx && src, "NULL argument");
   auto &l = ctx->landing;
   SOFIE_REQUIRE(l.open && offset <= l.bytes && bytes <= l.bytes - offset, "part [%zu, +%zu) of a result of %zu bytes", offset, bytes, l.bytes);
   SOFIE_REQUIRE(l.parts < SOFIE_CUDA_MAX_PARTS, "more than %d parts", SOFIE_CUDA_MAX_PARTS);
   const char *s8 = static_cast<const char *>(src);
   for (auto &h : ctx->host_outputs)
      if (s8 >= h.first && s8 + bytes <= h.first + h.second) {
         l.mapped = s8 - offset; // the kernels write it to host memory themselves
         return SOFIE_CUDA_OK;
      }
   if (bytes == 0) return SOFIE_CUDA_OK;
   DeviceGuard guard(ctx->device);
   if (!l.land) {
      if (l.out && is_pinned(l.out)) {
         l.land = l.out;
      } else {
         int rc = ensure_result(ctx, l.bytes);
         if (rc) return rc;
         l.land = static_cast<char *>(ctx->result);
      }
   }
   cudaStream_t stream = ctx->stream;
   if (bytes != l.bytes) {
      // one part of several: on a stream of its own, so that the copy out runs beside the later parts' kernels and copies in
      if (!ctx->result_stream) SOFIE_CUDA_TRY(cudaStreamCreateWithFlags(&ctx->result_stream, cudaStreamNonBlocking));
      if (!ctx->ready_event) SOFIE_CUDA_TRY(cudaEventCreateWithFlags(&ctx->ready_event, cudaEventDisableTiming));
      SOFIE_CUDA_TRY(cudaEventRecord(ctx->ready_event, ctx->stream));
      SOFIE_CUDA_TRY(cudaStreamWaitEvent(ctx->result_stream, ctx->ready_event, 0));
      stream = ctx->result_stream;
   }
   // A result in one piece that the host carries on into pageable memory lands in several, each carried under the copies of the later ones. 1 MB a piece is not worth its
   // events below 3 MB (72 us either way at 2 MB, 3 MB 111 -> 104); above, 2 MB a piece: 8 / 16 / 31 / 64 MB 254 -> 220, 480 -> 357, 1430 -> 640, 3600 -> 1350 us (a copy over
   // tens of MB that the cores have just read runs at a quarter of the link's rate).
   const bool carried = l.out && l.land != l.out;
   size_t pieces = 1;
   if (carried && bytes == l.bytes && l.pieces == 0 && bytes >= kLandInPieces) {
      pieces = bytes / (size_t(2) << 20);
      pieces = pieces < 2 ? 2 : (pieces > SOFIE_CUDA_MAX_PARTS ? SOFIE_CUDA_MAX_PARTS : pieces);
   }
   const size_t piece = ((bytes + pieces - 1) / pieces + 4095) & ~size_t(4095);
   for (size_t at = 0; at < bytes; at += piece) {
      const size_t n = bytes - at < piece ? bytes - at : piece;
      SOFIE_CUDA_TRY(cudaMemcpyAsync(l.land + offset + at, s8 + at, n, cudaMemcpyDeviceToHost, stream));
      if (carried && (n != l.bytes || l.pieces > 0)) {
         cudaEvent_t &e = ctx->landed_event[l.pieces];
         if (!e) SOFIE_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
         SOFIE_CUDA_TRY(cudaEventRecord(e, stream));
      }
      l.offset[l.pieces] = offset + at;
      l.count[l.pieces++] = n;
   }
   l.parts++;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_result_end(sofie_cuda_ctx *ctx, void **host)
{
   SOFIE_REQUIRE(ctx && host, "NULL argument");
   auto &l = ctx->landing;
   SOFIE_REQUIRE(l.open, "no result was begun");
   settle(ctx);
   DeviceGuard guard(ctx->device);
   const bool carry = l.out && l.land && l.land != l.out; // the caller's memory is pageable: the host carries the bytes over
   if (carry) {
      int rc = ensure_pool(ctx);
      if (rc) return rc;
      if (l.pieces > 1)
         for (int i = 0; i < l.pieces; i++) { // each as soon as it has landed, under the copies of the later ones
            if (i == 0 && l.count[0] == l.bytes) SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream)); // the whole at once, and parts of it again
            else SOFIE_CUDA_TRY(cudaEventSynchronize(ctx->landed_event[i]));
            ctx->host_pool->copy(l.out + l.offset[i], l.land + l.offset[i], l.count[i], l.bytes >= kPastCaches);
         }
   }
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   if (ctx->result_stream) SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->result_stream));
   l.open = false;
   // the stream has waited for every part that was copied in and waited for; a part that was not may still be read out of the ring
   bool copying = false;
   for (auto &slot : ctx->slots) copying = copying || (slot.busy && slot.stream == ctx->copy_stream);
   if (copying) SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->copy_stream));
   slots_free(ctx);
   if (carry && l.pieces == 1) ctx->host_pool->copy(l.out + l.offset[0], l.land + l.offset[0], l.count[0], l.bytes >= kPastCaches);
   release_pool(ctx);
   if (l.mapped && l.out) std::memcpy(l.out, l.mapped, l.bytes);
   *host = l.out ? l.out : (l.mapped ? const_cast<char *>(l.mapped) : l.land);
   return report_status(ctx);
}

int sofie_cuda_ctx_result_abort(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   if (!ctx->landing.open) return SOFIE_CUDA_OK;
   ctx->landing.open = false;
   settle(ctx);
   DeviceGuard guard(ctx->device);
   // inputs on their way out of the caller's memory, and results on their way into it
   cudaError_t err = cudaStreamSynchronize(ctx->stream);
   for (cudaStream_t s : {ctx->copy_stream, ctx->result_stream}) {
      const cudaError_t e = s ? cudaStreamSynchronize(s) : cudaSuccess;
      if (err == cudaSuccess) err = e;
   }
   SOFIE_CUDA_TRY(err);
   slots_free(ctx);
   return SOFIE_CUDA_OK;
}

size_t sofie_cuda_slice_rows(size_t rows, size_t in_bytes, size_t out_bytes, size_t quantum)
{
   static const int forced = [] { const char *e = std::getenv("SOFIE_CUDA_SLICES"); return e ? std::atoi(e) : 0; }();
   if (quantum == 0) quantum = 1;
   const size_t total = rows * (in_bytes > out_bytes ? in_bytes : out_bytes);
   // A slice costs its launches and two copies' fixed cost again (about 10 us each): from 4 MB of traffic on, in slices of about
   // 3 MB (55 us of PCIe). Measured, fp32 CNN on 1003 images (12.3 MB): 416 us in one piece, 357 / 340 / 332 / 358 us in 2 / 3 / 4 / 6
   // slices; int8 MLP on 8192 rows (16.8 MB): 314 / 296 / 277 / 276 us.
   size_t parts = forced > 0 ? (size_t)forced : (total < (size_t(4) << 20) ? 1 : (total < (size_t(6) << 20) ? 2 : total / (size_t(3) << 20)));
   if (parts > 8) parts = 8;
   if (parts <= 1) return rows;
   const size_t per = (rows + parts - 1) / parts;
   return (per + quantum - 1) / quantum * quantum;
}

int sofie_cuda_host_alloc(size_t bytes, void **host)
{
   SOFIE_REQUIRE(host && bytes > 0, "NULL argument or no bytes");
   void *p = nullptr;
   SOFIE_CUDA_TRY(cudaHostAlloc(&p, bytes, cudaHostAllocPortable));
   *host = p;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_host_free(void *host)
{
   if (host) SOFIE_CUDA_TRY(cudaFreeHost(host));
   return SOFIE_CUDA_OK;
}

// Device -> pinned host buffer owned by the context, at full link speed; the caller builds its
// result (the vector Session::infer returns) from the returned pointer in one pass, instead of
// zero-filling a vector first and then staging the copy through it. The pointer stays valid until
// the next fetch on this context.
int sofie_cuda_ctx_fetch(sofie_cuda_ctx *ctx, const void *src, size_t bytes, void **host)
{
   SOFIE_REQUIRE(ctx && src && host, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "result copies are not part of the captured graph");
   DeviceGuard guard(ctx->device);
   for (auto &h : ctx->host_outputs) {
      const char *s8 = static_cast<const char *>(src);
      if (s8 >= h.first && s8 + bytes <= h.first + h.second) {
         // the kernels wrote the result into host memory themselves: wait for them, nothing to copy
         SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
         *host = const_cast<char *>(s8);
         return report_status(ctx);
      }
   }
   int rc = ensure_result(ctx, bytes);
   if (rc) return rc;
   if (bytes) SOFIE_CUDA_TRY(cudaMemcpyAsync(ctx->result, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   *host = ctx->result;
   return report_status(ctx);
}

int sofie_cuda_ctx_sync(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   DeviceGuard guard(ctx->device);
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_check(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(!ctx->capturing, "the stream cannot be synchronised during a graph capture");
   DeviceGuard guard(ctx->device);
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   return report_status(ctx);
}

int sofie_cuda_device_check(int device)
{
   SOFIE_REQUIRE(device >= 0 && device < 64, "device index out of range");
   uint32_t *word = nullptr;
   {
      std::lock_guard<std::mutex> lock(g_status_mutex);
      word = g_status_words[device];
   }
   if (!word) return SOFIE_CUDA_OK; // no kernel with a bounded wait ran outside a context on this device
   DeviceGuard guard(device);
   uint32_t host_word[4] = {0, 0, 0, 0};
   SOFIE_CUDA_TRY(cudaDeviceSynchronize());
   SOFIE_CUDA_TRY(cudaMemcpy(host_word, word, sizeof(host_word), cudaMemcpyDeviceToHost));
   if (host_word[0]) {
      SOFIE_CUDA_TRY(cudaMemset(word, 0, 256));
      return fail(SOFIE_CUDA_ERR_DEVICE, "device status 0x%x (detail 0x%x 0x%x 0x%x)", host_word[0], host_word[1],
                  host_word[2], host_word[3]);
   }
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_timers(sofie_cuda_ctx *ctx, int on)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(!ctx->capturing && !ctx->captured.exec && !ctx->kept.exec, "switch the timers before the first inference is captured");
   ctx->timers_on = on != 0;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_timed(sofie_cuda_ctx *ctx) { return ctx && ctx->timers_on; }

int sofie_cuda_ctx_mark(sofie_cuda_ctx *ctx, int slot)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   if (!ctx->timers_on) return SOFIE_CUDA_OK;
   SOFIE_REQUIRE(slot >= 0 && slot < 4096, "timer slot out of range");
   DeviceGuard guard(ctx->device);
   if ((size_t)slot >= ctx->marks.size()) {
      ctx->marks.resize(slot + 1, nullptr);
      ctx->mark_seen.resize(slot + 1, 0);
   }
   if (!ctx->marks[slot]) SOFIE_CUDA_TRY(cudaEventCreate(&ctx->marks[slot]));
   // inside a capture the record becomes a node of the graph that updates this very event on every replay
   SOFIE_CUDA_TRY(cudaEventRecordWithFlags(ctx->marks[slot], ctx->stream, ctx->capturing ? cudaEventRecordExternal : cudaEventRecordDefault));
   ctx->mark_seen[slot] = 1;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_timers_read(sofie_cuda_ctx *ctx, float *ms, int n, int *count)
{
   SOFIE_REQUIRE(ctx && count, "NULL argument");
   SOFIE_REQUIRE(!ctx->capturing, "the stream cannot be synchronised during a graph capture");
   DeviceGuard guard(ctx->device);
   SOFIE_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
   // intervals between consecutive recorded marks, in slot order
   int prev = -1, k = 0;
   for (int i = 0; i < (int)ctx->marks.size(); i++) {
      if (!ctx->mark_seen[i]) continue;
      if (prev >= 0) {
         if (ms && k < n) SOFIE_CUDA_TRY(cudaEventElapsedTime(&ms[k], ctx->marks[prev], ctx->marks[i]));
         k++;
      }
      prev = i;
   }
   *count = k;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_graph_begin(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(!ctx->capturing, "graph capture already in progress");
   DeviceGuard guard(ctx->device);
   if (ctx->captured.exec) cudaGraphExecDestroy(ctx->captured.exec);
   if (ctx->captured.graph) cudaGraphDestroy(ctx->captured.graph);
   ctx->captured = {};
   SOFIE_CUDA_TRY(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
   ctx->capturing = true;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_graph_end(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(ctx->capturing, "no graph capture in progress");
   DeviceGuard guard(ctx->device);
   ctx->capturing = false;
   auto &g = ctx->captured;
   SOFIE_CUDA_TRY(cudaStreamEndCapture(ctx->stream, &g.graph));
   SOFIE_CUDA_TRY(cudaGraphInstantiate(&g.exec, g.graph, 0));
   // A graph of one kernel saves nothing and its launch costs twice a kernel's (4.5 against 2.2 us of host time): the kernel
   // is launched with the parameters the graph holds (its shared memory was allowed when it was captured, and stays so: allow_smem)
   g.only_kernel = {};
   size_t nodes = 0;
   SOFIE_CUDA_TRY(cudaGraphGetNodes(g.graph, nullptr, &nodes));
   if (nodes == 1) {
      cudaGraphNode_t node;
      cudaGraphNodeType type;
      SOFIE_CUDA_TRY(cudaGraphGetNodes(g.graph, &node, &nodes));
      SOFIE_CUDA_TRY(cudaGraphNodeGetType(node, &type));
      cudaKernelNodeAttrValue cluster = {};
      if (type == cudaGraphNodeTypeKernel && cudaGraphKernelNodeGetAttribute(node, cudaLaunchAttributeClusterDimension, &cluster) == cudaSuccess &&
          cluster.clusterDim.x * cluster.clusterDim.y * cluster.clusterDim.z <= 1) { // a plain launch has no cluster dimensions
         if (cudaGraphKernelNodeGetParams(node, &g.only_kernel) != cudaSuccess) g.only_kernel = {};
      }
      cudaGetLastError();
   }
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_graph_launch(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(ctx->captured.exec != nullptr, "no captured graph");
   DeviceGuard guard(ctx->device);
   const cudaKernelNodeParams &k = ctx->captured.only_kernel;
   if (k.func && k.kernelParams) SOFIE_CUDA_TRY(cudaLaunchKernel(k.func, k.gridDim, k.blockDim, k.kernelParams, k.sharedMemBytes, ctx->stream));
   else SOFIE_CUDA_TRY(cudaGraphLaunch(ctx->captured.exec, ctx->stream));
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_graph_ready(sofie_cuda_ctx *ctx, int *ready)
{
   SOFIE_REQUIRE(ctx && ready, "NULL argument");
   *ready = ctx->captured.exec != nullptr;
   return SOFIE_CUDA_OK;
}

int sofie_cuda_ctx_graph_swap(sofie_cuda_ctx *ctx)
{
   SOFIE_REQUIRE(ctx, "NULL ctx");
   SOFIE_REQUIRE(!ctx->capturing, "graph capture in progress");
   std::swap(ctx->captured, ctx->kept);
   return SOFIE_CUDA_OK;
}

} // extern "C"
