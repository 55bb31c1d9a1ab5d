// Context lifecycle, device memory pool and host<->device copies.
// Stands in for the reference's global backend and residency helpers
// (src/cuda/backend.rs:19-32, src/cuda/runtime.rs:39-124).
#include "fold.h"
#include "nrs_internal.h"

#include <cstring>
#include <mutex>
#include <vector>

static thread_local std::string g_no_ctx_error;

int nrs_fail(nrs_ctx* ctx, int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof(buf), fmt, ap);
  va_end(ap);
  if (ctx) ctx->err = buf; else g_no_ctx_error = buf;
  return code;
}

static void give_back_idle(nrs_ctx* ctx) {   // (cudaFree waits for the kernels in flight)
  NrsPool& pool = ctx->pool;
  for (auto it = pool.free_blocks.upper_bound(NrsPool::kSmall); it != pool.free_blocks.end(); it = pool.free_blocks.erase(it)) {
    cudaFree(it->second);
    pool.bytes_reserved -= it->first;
  }
  if (!ctx->folds.active) nrs_folds_free(ctx);
  for (void* s : pool.take_idle_slabs()) cudaFree(s);
}

int nrs_device_alloc(nrs_ctx* ctx, const char* what, size_t bytes, void** out) {
  *out = nullptr;
  cudaError_t e = ctx->device_malloc(out, bytes);
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    give_back_idle(ctx);
    e = ctx->device_malloc(out, bytes);
  }
  if (e != cudaSuccess && !ctx->folds.waiting.empty()) {   // weight gradients that wait hold what they read
    (void)cudaGetLastError();
    const int st = nrs_folds_relieve(ctx);
    if (st != NRS_OK) return st;
    give_back_idle(ctx);
    e = ctx->device_malloc(out, bytes);
  }
  if (e == cudaSuccess) return NRS_OK;
  (void)cudaGetLastError();
  *out = nullptr;
  return nrs_fail(ctx, NRS_ERR_ALLOC, "%s: cudaMalloc(%zu) failed: %s", what, bytes, cudaGetErrorString(e));
}

// Grow-only blocks of the context's own: small ones out of the pool's slabs.
static void drop_block(nrs_ctx* ctx, void** p, size_t* held) {   // the stream is idle
  if (*p && *held <= NrsPool::kSmall) nrs_free(ctx, *p);
  else if (*p) cudaFree(*p);
  *p = nullptr;
  *held = 0;
}
static int grow_block(nrs_ctx* ctx, const char* what, size_t bytes, void** p, size_t* held) {
  if (bytes <= *held) return NRS_OK;
  if (*p) NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));   // kernels in flight may still read the old block
  drop_block(ctx, p, held);
  const size_t want = (bytes + ((size_t)1 << 20) - 1) >> 20 << 20;
  const int st = want <= NrsPool::kSmall ? nrs_alloc(ctx, want, 0, p) : nrs_device_alloc(ctx, what, want, p);
  if (st == NRS_OK) *held = want;
  return st;
}

int nrs_workspace(nrs_ctx* ctx, size_t bytes, void** out) {
  const int st = grow_block(ctx, "workspace", bytes, &ctx->workspace, &ctx->workspace_bytes);
  *out = ctx->workspace;
  return st;
}

int nrs_ws_slot(nrs_ctx* ctx, int slot, size_t bytes, void** out) {
  if (slot < 0 || slot >= NRS_WS_COUNT) return nrs_fail(ctx, NRS_ERR_ARG, "workspace: bad slot %d", slot);
  const int st = grow_block(ctx, "workspace slot", bytes, &ctx->ws_slot[slot], &ctx->ws_slot_bytes[slot]);
  *out = ctx->ws_slot[slot];
  return st;
}

int nrs_ws_planes(nrs_ctx* ctx, int slot, size_t values, bool split, void** hi, void** lo) {
  const size_t each = (values * (split ? 2 : 4) + 255) / 256 * 256;
  const int st = nrs_ws_slot(ctx, slot, split ? 2 * each : each, hi);
  *lo = st == NRS_OK && split ? (uint8_t*)*hi + each : nullptr;
  return st;
}

void nrs_range_free(nrs_ctx* ctx, NrsRange* r) {
  for (auto& pg : ctx->range_pool.pages)
    if (r >= pg.mem && r < pg.mem + NrsRangePool::kPerPage) { --pg.live; return; }
}
void nrs_range_drop(nrs_ctx* ctx, const void* p) {
  auto it = ctx->ranges.find(p);
  if (it == ctx->ranges.end()) return;
  nrs_range_free(ctx, it->second);
  ctx->ranges.erase(it);
}
int nrs_range_renew(nrs_ctx* ctx, const void* p, NrsRange** out) {
  nrs_range_drop(ctx, p);
  const int st = nrs_range_new(ctx, out);
  if (st == NRS_OK) ctx->ranges[p] = *out;
  return st;
}
int nrs_range_new(nrs_ctx* ctx, NrsRange** out) {
  NrsRangePool& pool = ctx->range_pool;
  *out = nullptr;
  constexpr size_t kBytes = NrsRangePool::kPerPage * sizeof(NrsRange);
  if (pool.captured_left == 0) {   // (ahead of the first capture: the driver may refuse memory during one)
    void* mem = nullptr;
    const int st = nrs_alloc(ctx, NrsRangePool::kCaptured * sizeof(NrsRange), 0, &mem);
    if (st != NRS_OK) return st;
    pool.captured = (NrsRange*)mem;
    pool.captured_left = NrsRangePool::kCaptured;
  }
  cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
  NRS_CUDA(ctx, cudaStreamIsCapturing(ctx->stream, &capturing));
  if (capturing != cudaStreamCaptureStatusNone) {
    *out = pool.captured++;
    --pool.captured_left;
    NRS_CUDA(ctx, cudaMemsetAsync(*out, 0, sizeof(NrsRange), ctx->stream));
    return NRS_OK;
  }
  if (pool.pages.empty() || pool.pages[pool.current].used == NrsRangePool::kPerPage) {
    size_t next = 0;
    while (next < pool.pages.size() && pool.pages[next].live > 0) ++next;
    if (next == pool.pages.size()) {
      void* mem = nullptr;
      const int st = nrs_alloc(ctx, kBytes, 1, &mem);
      if (st != NRS_OK) return st;
      pool.pages.push_back(NrsRangePool::Page{(NrsRange*)mem, 0, 0});
    } else {
      NRS_CUDA(ctx, cudaMemsetAsync(pool.pages[next].mem, 0, kBytes, ctx->stream));
      pool.pages[next].used = 0;
    }
    pool.current = next;
  }
  NrsRangePool::Page& pg = pool.pages[pool.current];
  *out = pg.mem + pg.used++;
  ++pg.live;
  return NRS_OK;
}

// One page-locked block per context: the device error word, and behind it the slot of small read-backs.  Pinning takes
// 1 to 3 ms a call whatever the size, so blocks of closed contexts are kept for the next ones (at most kIdlePinned, by
// any thread; every device may use them).
namespace {
constexpr size_t kBounceBytes = 256 * 1024, kErrBytes = 4096;
constexpr size_t kIdlePinned = 16;
std::mutex g_pinned_lock;
std::vector<void*>& idle_pinned() {
  static auto* v = new std::vector<void*>();   // (not destroyed: contexts may close during static destruction)
  return *v;
}
}  // namespace

static int pinned_block(nrs_ctx* ctx) {
  if (ctx->pinned) return NRS_OK;
  void* p = nullptr;
  {
    std::lock_guard<std::mutex> g(g_pinned_lock);
    if (!idle_pinned().empty()) { p = idle_pinned().back(); idle_pinned().pop_back(); }
  }
  if (!p) NRS_CUDA(ctx, cudaHostAlloc(&p, kErrBytes + kBounceBytes, cudaHostAllocMapped | cudaHostAllocPortable));
  *(int*)p = 0;
  ctx->pinned = p;
  return NRS_OK;
}

void nrs_pinned_release(nrs_ctx* ctx) {   // the context's stream is idle
  if (!ctx->pinned) return;
  std::lock_guard<std::mutex> g(g_pinned_lock);
  if (idle_pinned().size() < kIdlePinned) idle_pinned().push_back(ctx->pinned);
  else cudaFreeHost(ctx->pinned);
  ctx->pinned = nullptr;
  ctx->err_host = nullptr;
  ctx->err_flag = nullptr;
}

// The word lives in mapped host memory: only a kernel that gives up writes it (across the bus, once), and reading it
// after a synchronisation is a plain load instead of a copy and a second synchronisation (some 10 us per read-back).
int nrs_err_flag(nrs_ctx* ctx, int** out) {
  if (!ctx->err_flag) {
    const int st = pinned_block(ctx);
    if (st != NRS_OK) return st;
    void* d = nullptr;
    NRS_CUDA(ctx, cudaHostGetDevicePointer(&d, ctx->pinned, 0));
    ctx->err_host = (volatile int*)ctx->pinned;
    ctx->err_flag = (int*)d;
  }
  *out = ctx->err_flag;
  return NRS_OK;
}

int nrs_fold_ticket(nrs_ctx* ctx, unsigned** out) {
  if (!ctx->fold_ticket) {
    const int st = nrs_alloc(ctx, kNrsFoldTickets * sizeof(unsigned), 1, (void**)&ctx->fold_ticket);
    if (st != NRS_OK) return st;
  }
  *out = ctx->fold_ticket;
  return NRS_OK;
}

int nrs_check_device_error(nrs_ctx* ctx) {
  if (!ctx->err_host) return NRS_OK;
  const int code = *ctx->err_host;
  if (code == 0) return NRS_OK;
  *ctx->err_host = 0;
  if (code == 5)
    return nrs_fail(ctx, NRS_ERR_ARG, "an embedding lookup met a token index outside the vocabulary; that row was read as zeros");
  static const char* what[] = {"", "TMA producer waiting for a free ring slot", "UMMA issuer waiting for a filled ring slot",
                               "epilogue waiting for the accumulator", "draining outstanding TMA loads"};
  return nrs_fail(ctx, NRS_ERR_TIMEOUT, "a tensor-core kernel gave up a bounded wait (%s); its output is invalid",
                  code >= 1 && code <= 4 ? what[code] : "unknown stage");
}

static cudaEvent_t prof_event(nrs_ctx* ctx) {
  if (!ctx->prof_free_events.empty()) {
    cudaEvent_t e = ctx->prof_free_events.back();
    ctx->prof_free_events.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  if (cudaEventCreate(&e) != cudaSuccess) { (void)cudaGetLastError(); return nullptr; }
  return e;
}

NrsProfScope::NrsProfScope(nrs_ctx* c, int kind, double work) : ctx(c) {
  if (!c || !c->profiling) return;
  rec.kind = kind;
  rec.work = work;
  queued = c->folds.queued;
  rec.start = prof_event(c);
  rec.stop = prof_event(c);
  if (!rec.start || !rec.stop) return;
  active = cudaEventRecord(rec.start, c->stream) == cudaSuccess;
}

NrsProfScope::~NrsProfScope() {
  if (!active) return;
  if (queued != ctx->folds.queued) {
    ctx->prof_free_events.push_back(rec.start);
    ctx->prof_free_events.push_back(rec.stop);
    return;
  }
  if (cudaEventRecord(rec.stop, ctx->stream) == cudaSuccess) ctx->prof_records.push_back(rec);
}

// Device -> host: small reads into pageable memory go through a pinned slot of the context's own (one copy, one wait,
// one memcpy: 64 KB 23 -> 15 us); larger ones, and pinned destinations (nrs_host_alloc), are one asynchronous copy.
static int nrs_bounce_d2h(nrs_ctx* ctx, void* dst, const void* src, size_t bytes) {
  if (bytes > kBounceBytes) {
    NRS_CUDA(ctx, cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
    NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return NRS_OK;
  }
  const int st = pinned_block(ctx);
  if (st != NRS_OK) return st;
  void* bounce = (uint8_t*)ctx->pinned + kErrBytes;
  NRS_CUDA(ctx, cudaMemcpyAsync(bounce, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  std::memcpy(dst, bounce, bytes);
  return NRS_OK;
}

extern "C" {

int nrs_selftest_smem_attr_bookkeeping(void) {
  NrsSmemAttr a;
  int bad = 0;
  bad += nrs_smem_attr_update(a, 0, 40 * 1024) ? 1 : 0;      // fits the default: never requested
  bad += nrs_smem_attr_update(a, 0, 100 * 1024) ? 0 : 1;     // first request on device 0
  bad += nrs_smem_attr_update(a, 0, 100 * 1024) ? 1 : 0;     // already set there
  bad += nrs_smem_attr_update(a, 0, 90 * 1024) ? 1 : 0;      // smaller than what is set
  bad += nrs_smem_attr_update(a, 1, 100 * 1024) ? 0 : 1;     // another device starts from nothing
  bad += nrs_smem_attr_update(a, 0, 200 * 1024) ? 0 : 1;     // growth
  bad += nrs_smem_attr_update(a, 1, 100 * 1024) ? 1 : 0;
  bad += nrs_smem_attr_update(a, kNrsMaxDevices, 100 * 1024) ? 0 : 1;   // untracked ordinals always request
  bad += nrs_smem_attr_update(a, kNrsMaxDevices, 100 * 1024) ? 0 : 1;
  return bad;
}

int nrs_selftest_pool_bookkeeping(void) {
  int bad = 0;
  NrsPool p;
  const size_t kb = 1024;
  uint8_t* base = (uint8_t*)(uintptr_t)((size_t)1 << 40);   // addresses only
  auto at = [&](int slab, size_t off) { return (void*)(base + (size_t)slab * 2 * NrsPool::kSlab + off); };
  for (int i = 0; i < 3; ++i) p.slabs.push_back(at(i, 0));
  p.bytes_reserved = 3 * NrsPool::kSlab + 64 * kb * kb;
  p.slab_used = 4 * kb;
  p.free_blocks.emplace(kb, at(0, 0));
  p.live[at(1, 0)] = kb;                                    // the middle slab is in use
  p.live[at(1, NrsPool::kSlab - kb)] = kb;
  p.free_blocks.emplace(kb, at(1, kb));
  p.free_blocks.emplace(2 * kb, at(2, 0));
  p.free_blocks.emplace(64 * kb * kb, at(7, 0));            // a block of its own
  bad += p.take_idle_slabs() == std::vector<void*>{at(0, 0), at(2, 0)} ? 0 : 1;
  bad += p.slabs == std::vector<void*>{at(1, 0)} && p.slab_used == NrsPool::kSlab ? 0 : 1;
  bad += p.free_blocks.size() == 2 && p.free_blocks.begin()->second == at(1, kb) ? 0 : 1;
  bad += p.bytes_reserved == NrsPool::kSlab + 64 * kb * kb ? 0 : 1;
  bad += p.take_idle_slabs().empty() ? 0 : 1;
  p.live.clear();
  bad += p.take_idle_slabs().size() == 1 && p.slabs.empty() && p.free_blocks.size() == 1 ? 0 : 1;
  return bad;
}

// A driver that is out of memory, played by an allocator that refuses until something has been given back.
int nrs_selftest_memory_pressure(nrs_ctx* ctx) {
  NRS_REQUIRE_CTX(ctx);
  static thread_local int refuse;
  static thread_local int calls;
  const auto real = ctx->device_malloc;
  ctx->device_malloc = [](void** p, size_t n) { ++calls; return refuse-- > 0 ? cudaErrorMemoryAllocation : cudaMalloc(p, n); };
  int bad = 0;
  void* p[40] = {};
  for (int i = 0; i < 40; ++i) bad += nrs_alloc(ctx, (size_t)900 << 10, 0, &p[i]) == NRS_OK ? 0 : 1;   // three slabs
  for (void* q : p) bad += nrs_free(ctx, q) == NRS_OK ? 0 : 1;
  const size_t slabs = ctx->pool.slabs.size();
  refuse = 1;
  bad += nrs_alloc(ctx, (size_t)40 << 20, 0, &p[0]) == NRS_OK && ctx->pool.slabs.size() + 2 <= slabs ? 0 : 1;
  bad += nrs_free(ctx, p[0]) == NRS_OK ? 0 : 1;
  refuse = 1 << 20;                                          // nothing to be had: an error, and the context goes on
  calls = 0;
  bad += nrs_alloc(ctx, (size_t)50 << 20, 0, &p[0]) == NRS_ERR_ALLOC && p[0] == nullptr && calls == 2 ? 0 : 1;
  // fold scratch: a full block while folds are queued means that they run and the block starts over
  refuse = 0;
  float *a = nullptr, *b = nullptr, *dst = nullptr;
  bad += nrs_alloc(ctx, 40960, 1, (void**)&dst) == NRS_OK ? 0 : 1;
  nrs_folds_begin(ctx);
  bad += nrs_fold_partial(ctx, -1, (size_t)40 << 20, &a) == NRS_OK ? 0 : 1;
  bad += nrs_memset_zero(ctx, a, 4096) == NRS_OK && nrs_fold_columns(ctx, a, dst, 4, 256, 256, 0) == NRS_OK ? 0 : 1;
  refuse = 1 << 20;
  bad += nrs_fold_partial(ctx, -1, (size_t)40 << 20, &b) == NRS_OK && b == a && ctx->folds.jobs.empty() ? 0 : 1;
  refuse = 0;
  // weight gradients that wait hold what they read: they run, and it goes back, before an allocation fails, and ahead of the
  // next one where too much is held
  const int mode = ctx->math_mode;
  ctx->math_mode = NRS_MATH_3XTF32;
  const int n = 8, c = 32, hw = 16;
  const size_t image = sizeof(float) * n * c * hw * hw, weight = sizeof(float) * c * c * 9;
  float *x = nullptr, *dy = nullptr, *dw = nullptr;
  bad += nrs_alloc(ctx, image, 1, (void**)&x) == NRS_OK && nrs_alloc(ctx, image, 1, (void**)&dy) == NRS_OK && nrs_alloc(ctx, weight, 0, (void**)&dw) == NRS_OK ? 0 : 1;
  bad += nrs_planes_cache(ctx, x, n, c, hw, hw) == NRS_OK && nrs_planes_cache(ctx, dy, n, c, hw, hw) == NRS_OK ? 0 : 1;
  const NrsFolds& f = ctx->folds;
  for (int limit = 0; limit < 2; ++limit) {
    bad += cudaMemsetAsync(dw, 0xff, weight, ctx->stream) == cudaSuccess ? 0 : 1;
    bad += nrs_conv2d_bwd(ctx, x, dw /*no data gradient reads it*/, dy, nullptr, dw, nullptr, n, c, hw, hw, c, 3, 3, 1, 1, 0) == NRS_OK && f.waiting.size() == 1 ? 0 : 1;
    void *held = nullptr, *more = nullptr;
    bad += nrs_alloc(ctx, (size_t)60 << 20, 0, &held) == NRS_OK ? 0 : 1;
    nrs_free_after_wgrads(ctx, held);
    bad += f.kept.size() == 1 && f.kept_bytes == (size_t)60 << 20 ? 0 : 1;
    if (limit) {
      ctx->folds.kept_bytes = kNrsKeptBytes + 1;
      bad += nrs_conv2d_bwd(ctx, x, dw, dy, nullptr, dst, nullptr, n, c, hw, hw, c, 3, 3, 1, 1, 0) == NRS_OK && f.waiting.size() == 1 ? 0 : 1;
    } else {
      refuse = 2;   // what the context keeps idle is not enough
      bad += nrs_alloc(ctx, (size_t)70 << 20, 0, &more) == NRS_OK && f.waiting.empty() ? 0 : 1;
      refuse = 0;
      bad += nrs_free(ctx, more) == NRS_OK ? 0 : 1;
    }
    bad += f.kept.empty() && f.kept_bytes == 0 ? 0 : 1;
    float got[2] = {1.0f, 1.0f};
    bad += nrs_d2h(ctx, got, dw, sizeof(got)) == NRS_OK && got[0] == 0.0f && got[1] == 0.0f ? 0 : 1;
  }
  bad += nrs_folds_flush(ctx) == NRS_OK && f.waiting.empty() ? 0 : 1;
  // memory of a job that is being made stays its own while others run for the sake of memory
  bad += nrs_fold_partial(ctx, -1, 1024, &a) == NRS_OK && nrs_folds_relieve(ctx) == NRS_OK && nrs_fold_partial(ctx, -1, 1024, &b) == NRS_OK && a != b ? 0 : 1;
  bad += nrs_planes_drop(ctx, x) == NRS_OK && nrs_planes_drop(ctx, dy) == NRS_OK ? 0 : 1;
  ctx->math_mode = mode;
  nrs_folds_end(ctx);
  ctx->device_malloc = real;
  for (void* q : {(void*)x, (void*)dy, (void*)dw}) bad += nrs_free(ctx, q) == NRS_OK ? 0 : 1;
  bad += nrs_free(ctx, dst) == NRS_OK && nrs_sync(ctx) == NRS_OK ? 0 : 1;
  return bad;
}

int nrs_profile_enable(nrs_ctx* ctx, int on) {
  NRS_REQUIRE_CTX(ctx);
  ctx->profiling = on != 0;
  return NRS_OK;
}

int nrs_profile_reset(nrs_ctx* ctx) {
  NRS_REQUIRE_CTX(ctx);
  NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  for (auto& r : ctx->prof_records) {
    ctx->prof_free_events.push_back(r.start);
    ctx->prof_free_events.push_back(r.stop);
  }
  ctx->prof_records.clear();
  return NRS_OK;
}

int nrs_profile_get(nrs_ctx* ctx, int kind, double* ms_out, double* work_out, uint64_t* calls_out) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, kind >= 0 && kind < NRS_PROF_KINDS, NRS_ERR_ARG, "nrs_profile_get: unknown kind %d", kind);
  NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  double ms = 0.0, work = 0.0;
  uint64_t calls = 0;
  for (auto& r : ctx->prof_records) {
    if (r.kind != kind) continue;
    float t = 0.0f;
    NRS_CUDA(ctx, cudaEventElapsedTime(&t, r.start, r.stop));
    ms += t;
    work += r.work;
    ++calls;
  }
  if (ms_out) *ms_out = ms;
  if (work_out) *work_out = work;
  if (calls_out) *calls_out = calls;
  return NRS_OK;
}

int nrs_init(int device, nrs_ctx** out) {
  if (!out) return nrs_fail(nullptr, NRS_ERR_ARG, "nrs_init: null out pointer");
  *out = nullptr;
  int count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) {
    (void)cudaGetLastError();
    return nrs_fail(nullptr, NRS_ERR_CUDA,
                    "nrs_init: no usable CUDA device (%s); this library has no CPU fallback",
                    e != cudaSuccess ? cudaGetErrorString(e) : "device count is 0");
  }
  if (device < 0 || device >= count)
    return nrs_fail(nullptr, NRS_ERR_ARG, "nrs_init: device %d out of range [0,%d)", device, count);
  e = cudaSetDevice(device);
  if (e != cudaSuccess)
    return nrs_fail(nullptr, NRS_ERR_CUDA, "nrs_init: cudaSetDevice(%d): %s", device, cudaGetErrorString(e));
  cudaDeviceProp prop;
  e = cudaGetDeviceProperties(&prop, device);
  if (e != cudaSuccess)
    return nrs_fail(nullptr, NRS_ERR_CUDA, "nrs_init: cudaGetDeviceProperties: %s", cudaGetErrorString(e));
  if (prop.major != 10)
    return nrs_fail(nullptr, NRS_ERR_CUDA,
                    "nrs_init: device %d is sm_%d%d; this library is built for sm_100a only",
                    device, prop.major, prop.minor);
  nrs_ctx* ctx = new nrs_ctx();
  ctx->device = device;
  ctx->sm_count = prop.multiProcessorCount;
  e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking);
  if (e != cudaSuccess) {
    delete ctx;
    return nrs_fail(nullptr, NRS_ERR_CUDA, "nrs_init: cudaStreamCreate: %s", cudaGetErrorString(e));
  }
  ctx->stream = ctx->own_stream;
  *out = ctx;
  return NRS_OK;
}

int nrs_destroy(nrs_ctx* ctx) {
  if (!ctx) return NRS_OK;
  cudaSetDevice(ctx->device);
  cudaStreamSynchronize(ctx->stream);
  drop_block(ctx, &ctx->workspace, &ctx->workspace_bytes);
  for (int i = 0; i < NRS_WS_COUNT; ++i) drop_block(ctx, &ctx->ws_slot[i], &ctx->ws_slot_bytes[i]);
  nrs_folds_free(ctx);
  nrs_weight_set_clear(ctx);
  for (auto& kv : ctx->pool.free_blocks) if (kv.first > NrsPool::kSmall) cudaFree(kv.second);
  for (auto& kv : ctx->pool.live) if (kv.second > NrsPool::kSmall) cudaFree(kv.first);
  for (void* s : ctx->pool.slabs) cudaFree(s);
  nrs_pinned_release(ctx);
  for (auto& r : ctx->prof_records) { cudaEventDestroy(r.start); cudaEventDestroy(r.stop); }
  for (auto& e : ctx->prof_free_events) cudaEventDestroy(e);
  if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
  delete ctx;
  return NRS_OK;
}

const char* nrs_last_error(const nrs_ctx* ctx) {
  return ctx ? ctx->err.c_str() : g_no_ctx_error.c_str();
}

int nrs_set_stream(nrs_ctx* ctx, void* cuda_stream) {
  NRS_REQUIRE_CTX(ctx);
  ctx->stream = cuda_stream ? (cudaStream_t)cuda_stream : ctx->own_stream;
  return NRS_OK;
}

void* nrs_get_stream(nrs_ctx* ctx) { return ctx ? (void*)ctx->stream : nullptr; }

int nrs_set_math_mode(nrs_ctx* ctx, int mode) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, mode == NRS_MATH_3XTF32 || mode == NRS_MATH_TF32 || mode == NRS_MATH_FP32,
              NRS_ERR_ARG, "nrs_set_math_mode: unknown mode %d", mode);
  ctx->math_mode = mode;
  return NRS_OK;
}

int nrs_get_math_mode(const nrs_ctx* ctx) { return ctx ? ctx->math_mode : -1; }

uint64_t nrs_launch_count(const nrs_ctx* ctx) { return ctx ? ctx->launches : 0; }

int nrs_alloc(nrs_ctx* ctx, size_t bytes, int zero, void** dptr) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, dptr != nullptr, NRS_ERR_ARG, "nrs_alloc: null out pointer");
  *dptr = nullptr;
  const size_t want = NrsPool::round_up(bytes ? bytes : 1);
  void* p = nullptr;
  auto it = ctx->pool.free_blocks.find(want);
  if (it != ctx->pool.free_blocks.end()) {
    p = it->second;
    ctx->pool.free_blocks.erase(it);
  } else {
    NrsPool& pool = ctx->pool;
    const bool small = want <= NrsPool::kSmall;
    if (small && pool.slab_used + want <= NrsPool::kSlab) {
      p = (uint8_t*)pool.slabs.back() + pool.slab_used;
      pool.slab_used += want;
    } else {
      const size_t ask = small ? NrsPool::kSlab : want;
      const int st = nrs_device_alloc(ctx, "nrs_alloc", ask, &p);
      if (st != NRS_OK) return st;
      pool.bytes_reserved += ask;
      if (small) {
        pool.slabs.push_back(p);
        pool.slab_used = want;
      }
    }
  }
  ctx->pool.live[p] = want;
  if (zero) NRS_CUDA(ctx, cudaMemsetAsync(p, 0, bytes, ctx->stream));
  *dptr = p;
  return NRS_OK;
}

int nrs_free(nrs_ctx* ctx, void* dptr) {
  NRS_REQUIRE_CTX(ctx);
  if (!dptr) return NRS_OK;
  auto it = ctx->pool.live.find(dptr);
  NRS_REQUIRE(ctx, it != ctx->pool.live.end(), NRS_ERR_ARG, "nrs_free: %p was not allocated by nrs_alloc", dptr);
  nrs_range_drop(ctx, dptr);
  ctx->pool.free_blocks.emplace(it->second, dptr);
  ctx->pool.live.erase(it);
  return NRS_OK;
}

int nrs_memset_zero(nrs_ctx* ctx, void* dptr, size_t bytes) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, dptr || bytes == 0, NRS_ERR_ARG, "nrs_memset_zero: null pointer");
  if (bytes) NRS_CUDA(ctx, cudaMemsetAsync(dptr, 0, bytes, ctx->stream));
  return NRS_OK;
}

int nrs_h2d(nrs_ctx* ctx, void* dst_dev, const void* src_host, size_t bytes) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, (dst_dev && src_host) || bytes == 0, NRS_ERR_ARG, "nrs_h2d: null pointer");
  if (bytes) NRS_CUDA(ctx, cudaMemcpyAsync(dst_dev, src_host, bytes, cudaMemcpyHostToDevice, ctx->stream));
  return NRS_OK;
}

int nrs_d2h(nrs_ctx* ctx, void* dst_host, const void* src_dev, size_t bytes) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, (dst_host && src_dev) || bytes == 0, NRS_ERR_ARG, "nrs_d2h: null pointer");
  if (bytes) {
    const int st = nrs_bounce_d2h(ctx, dst_host, src_dev, bytes);
    if (st != NRS_OK) return st;
  } else {
    NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  }
  return nrs_check_device_error(ctx);
}

int nrs_host_alloc(size_t bytes, void** out) {
  if (!out) return nrs_fail(nullptr, NRS_ERR_ARG, "nrs_host_alloc: null out pointer");
  *out = nullptr;
  if (cudaHostAlloc(out, bytes ? bytes : 1, cudaHostAllocPortable) != cudaSuccess) {
    (void)cudaGetLastError();
    *out = nullptr;
    return nrs_fail(nullptr, NRS_ERR_ALLOC, "nrs_host_alloc: no pinned memory for %zu bytes", bytes);
  }
  return NRS_OK;
}

int nrs_host_free(void* ptr) {
  if (ptr && cudaFreeHost(ptr) != cudaSuccess) {
    (void)cudaGetLastError();
    return nrs_fail(nullptr, NRS_ERR_ARG, "nrs_host_free: not a pinned block of nrs_host_alloc");
  }
  return NRS_OK;
}

int nrs_d2d(nrs_ctx* ctx, void* dst_dev, const void* src_dev, size_t bytes) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, (dst_dev && src_dev) || bytes == 0, NRS_ERR_ARG, "nrs_d2d: null pointer");
  if (bytes) NRS_CUDA(ctx, cudaMemcpyAsync(dst_dev, src_dev, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
  return NRS_OK;
}

int nrs_sync(nrs_ctx* ctx) {
  NRS_REQUIRE_CTX(ctx);
  NRS_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
  return nrs_check_device_error(ctx);
}

}  // extern "C"
