// Internal declarations shared by the translation units of libnrs_b200.so.
#pragma once

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <iterator>
#include <map>
#include <memory>
#include <string>
#include <unordered_map>
#include <utility>
#include <vector>

#include "nrs.h"

// Size-bucketed device memory pool.  Blocks are handed back to a free list
// keyed by their rounded size instead of being cudaFree'd, so a training loop
// whose shapes repeat stops calling cudaMalloc after its first step.  All work
// runs on one stream, so reuse right after release is ordered correctly.
struct NrsPool {
  std::multimap<size_t, void*> free_blocks;   // rounded size -> block
  std::map<void*, size_t> live;               // block -> rounded size
  size_t bytes_reserved = 0;
  // Blocks up to kSmall bytes, the context's own workspaces of that size among them, are cut from slabs: cudaMalloc takes
  // 0.3 ms for anything from 2 MB to 256 MB, and a small model's first step asks for dozens of sizes (the first step of
  // the digit classifier in a new context: 14 calls of cudaMalloc without, 3 with).
  static constexpr size_t kSmall = (size_t)2 << 20, kSlab = (size_t)32 << 20;
  std::vector<void*> slabs;
  size_t slab_used = kSlab;                   // of the last one
  static size_t round_up(size_t bytes) {
    const size_t g = bytes <= (1u << 20) ? 512 : (size_t)1 << 16;
    return (bytes + g - 1) / g * g;
  }
  // Takes the slabs none of whose blocks is in use out of the pool, for the caller to give back.
  std::vector<void*> take_idle_slabs() {
    std::vector<void*> out;
    for (size_t i = 0; i < slabs.size();) {
      uint8_t *lo = (uint8_t*)slabs[i], *hi = lo + kSlab;
      const auto used = live.lower_bound(lo);
      if (used != live.end() && (uint8_t*)used->first < hi) { ++i; continue; }
      for (auto it = free_blocks.begin(); it != free_blocks.end() && it->first <= kSmall;)
        it = (uint8_t*)it->second >= lo && (uint8_t*)it->second < hi ? free_blocks.erase(it) : std::next(it);
      if (i + 1 == slabs.size()) slab_used = kSlab;   // the one that was being cut
      slabs.erase(slabs.begin() + i);
      bytes_reserved -= kSlab;
      out.push_back(lo);
    }
    return out;
  }
};

// What is known on the device about the magnitudes of a tensor whose values exist as f16 pairs (pair.cuh): `bound`, which
// no finite value exceeds and which the pairs' exponent comes from, and `top`, the largest finite magnitude that was
// written (where its writer only has a bound: that), which bounds of results are made of.
struct NrsRange {
  float bound, top;
  float pad[6];   // a sector each
};
// Ranges are cut from pages that are zeroed as a whole, on the context's stream, once all ranges of a page are back.  While
// the stream is being captured they come from memory apart: a graph may be replayed at any time, so its ranges are cleared
// one by one, by the graph itself, and nobody else ever gets them.
struct NrsRangePool {
  static constexpr int kPerPage = 256, kCaptured = 1024;
  struct Page { NrsRange* mem; int used, live; };
  std::vector<Page> pages;
  size_t current = 0;
  NrsRange* captured = nullptr;
  int captured_left = 0;
};

struct NrsProfRecord {
  int kind;
  double work;
  cudaEvent_t start, stop;
};

// The address of value `at` of a plane.
inline float* nrs_plane_at(const float* plane, size_t at, bool split) { return (float*)((uint8_t*)plane + at * (split ? 2 : 4)); }
// Operand planes: TF32 mode: the values rounded to TF32, in f32 storage (hi).  3xTF32: f16 pairs (pair.cuh), hi and lo in
// f16 storage each; the tensor's NrsRange is found by the address of hi (nrs_range_of).  The pointers are typed float* in
// both cases.
// NHWC planes of an NCHW activation, staged ahead of time by a caller that knows
// the tensor will feed several tensor-core convolutions (forward and weight gradient,
// or data and weight gradient).  lo is null unless `split` (3xTF32).
struct NrsPlanes {
  float* hi;
  float* lo;
  int split;
  // Set for the planes of a 2-D tensor [rows][cols] (cols a multiple of 32) staged for a GEMM; zero for
  // image planes, whose NHWC order is not the tensor's own row-major order.
  int rows = 0, cols = 0;
};

// Patch planes of an image tensor [n][ci][h][w]: for every output pixel of a convolution the ci*kh*kw input values
// under it, [n*oh*ow][nrs_plane_ld(ci*kh*kw)].
struct NrsPatchPlanes {
  float* hi;
  float* lo;
  int kh, kw, stride, pad;
};
// Layers that run on patches: with fewer than 8 input channels a 32-channel K-block per tap would be mostly padding
// (a factor of 4 and more), while all taps together fill a few blocks (up to 128 values, at most 1 KB per pixel).
// (Images of a few hundred pixels in all take the direct kernels of conv_smallc.cu where those apply: fewer launches.)
constexpr long kNrsPatchMinPixels = 1024;
inline bool nrs_conv_uses_patches(int ci, int kh, int kw) { return ci < 8 && kh * kw > 1 && ci * kh * kw <= 128; }

// Floats between two pixels of a tensor's NHWC planes: its channels rounded up to whole 32-byte sectors (TMA wants
// 16-byte strides; with 112-byte rows, 27 values padded to 28, a convolution over them ran 41 us instead of 28).
constexpr inline int nrs_plane_ld(int channels) { return (channels + 7) & ~7; }

// Extra work a convolution kernel can fold into the epilogue that writes `out` (keyed by the
// output pointer in nrs_ctx::out_extras).  A kernel that honours the request erases the entry;
// an entry still present after the call means the caller has to do the work itself.
struct NrsOutExtras {
  const float* relu_mask_src;   // NCHW tensor of out's shape: out = relu_mask_src > 0 ? out : 0 (or null)
  float* hi;                    // NHWC operand planes of the (masked) result, or null
  float* lo;                    // (3xTF32)
  NrsRange* measure = nullptr;  // 3xTF32, no planes: largest magnitude of the result goes here
  bool planes_suffice = false;  // the result itself need not be written where its planes and channel sums are
};

// Request for per-tile channel sums of a convolution kernel's (masked) output, keyed by the output
// pointer in nrs_ctx::colsum_requests: the bias gradient of the layer below is then a fold of
// [rows][channels] partial sums instead of a pass over the whole gradient.  A kernel that honours
// it sets `rows` (> 0); the caller removes the entry either way.
struct NrsColsumRequest {
  float* partial;   // [cap_rows][channels]
  int cap_rows;
  int rows;         // out: rows written, 0 = not honoured
};

// Weight operand planes staged ahead of the contractions by a caller that knows its weights (the
// trainer): see weight_set.cu.  Forms: convolution forward [co][tap*ci + ci] and data gradient
// [ci][tap*co + co]; Linear W[in,out] transposed to [out][in] (B operand of x@W) and as stored
// [in][out] (B operand of dz@W^T), rows padded to a multiple of 32 floats.
enum NrsWeightForm { NRS_WF_CONV_FWD = 0, NRS_WF_CONV_DGRAD = 1, NRS_WF_LINEAR_T = 2, NRS_WF_LINEAR_ROWS = 3 };
struct NrsWeightDesc {
  const float* w;
  int form;
  int rows, K;        // linear forms: the DESTINATION's row count and reduction length
  int co, ci, taps;   // convolution forms
  int group = 0;      // not 0: consecutive weights of one group share a range (they meet in one product)
};
struct NrsWeightPlanes {
  float* hi;
  float* lo;          // null unless 3xTF32
  const NrsRange* range;
  int rows, K, co, ci, taps;
};
struct NrsWeightSet {
  void* storage = nullptr;
  void* jobs_dev = nullptr;
  int n_jobs = 0;
  unsigned blocks = 0;
  bool split = false;
  bool fresh = false;   // staged since the weights last changed (the owner clears it when it updates them)
  const void* owner = nullptr;   // whoever built the set (a trainer); a different owner rebuilds it
  int mode = -1;                 // math mode it was built for
  std::map<std::pair<const void*, int>, NrsWeightPlanes> planes;
  // per job, in launch order: the weight it reads and its first block (the last entry of job_first is `blocks`)
  std::vector<const float*> job_src;
  std::vector<unsigned> job_first;
  std::vector<unsigned> job_scan;   // the same of the launch that measures ranges (3xTF32)
  std::vector<int> job_group;       // first job of its group
  NrsRange* ranges = nullptr;
  int refreshed_jobs = 0;   // jobs restaged range by range since the last full refresh / reset (refresh_range)
};

// Cross-rank sum of a few per-channel statistics (batch normalisation under data parallelism): set by
// whoever owns a communicator (the trainer); null = statistics are per process.  Sums `count` floats at
// `dev` over all ranks in place, in order on the context's stream; every rank must make the same calls.
struct NrsStatSync {
  int (*all_reduce_sum)(void* user, float* dev, size_t count) = nullptr;
  void* user = nullptr;
};

// One fold (fold.cu).  Kinds: column sums; the partial tiles of the general and of the row-streaming weight gradient.
enum { NRS_FOLD_COLUMNS = 0, NRS_FOLD_WGRAD = 1, NRS_FOLD_WGRAD_ROWS = 2 };
struct NrsFoldJob {
  const float* src;
  float* dst;
  float* scratch;          // columns with several row splits: [splits][cols]
  float* dst2;             // columns: those from cols1 on go here (null: all to dst)
  unsigned* tickets;
  unsigned first_block;
  int kind, accumulate, splits, lanes;
  union { int rows; int co; };
  union { int cols; int ci; };
  union { int stride; int taps; };
  // weight gradients: the partial tiles' layout (see the kernels)
  int taps_per_group, n_groups, col_blocks, cblocks, group_cols;
  int chunk, n_chunks, jtypes, a_blocks, pack;
  int cols1;
  int vec;                 // 1x1: outputs written 16 bytes at a time
  int out_cols;            // general kernel, 1x1: the columns are several [co][out_cols] matrices side by side (0: one)
  size_t split_stride;     // floats between two splits
};
struct NrsFolds {
  bool active = false;
  std::vector<NrsFoldJob> jobs;
  unsigned tickets_used = 1;
  std::vector<std::pair<void*, size_t>> chunks;   // memory for partial sums that wait
  size_t chunk = 0, used = 0;
  bool open = false;       // some of it has been handed out for a job that is not submitted yet
  int holding = 0;         // queued jobs with partial sums in it (others read memory of their own)
  uint64_t launched_at = ~0ull;   // nrs_ctx::launches right after the last launch of folds
  // Weight gradients that wait for the pass's end (wgrad_queue.h): where they write, their kernels' own queues, and memory
  // they read whose owner has let go of it.
  std::vector<std::pair<const float*, size_t>> waiting;
  uint64_t queued = 0;     // how many have ever waited
  std::shared_ptr<void> waiting_rows, waiting_tiles;
  std::vector<void*> kept;
  size_t kept_bytes = 0;
  bool relieving = false;  // the waiting gradients run for the sake of memory, maybe while a job is being made
};

struct nrs_ctx {
  int device = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  int math_mode = NRS_MATH_3XTF32;
  bool internal_graph = false;   // nodes made now belong to a native trainer: nobody else reads them (see nrs::Node::internal)
  int sm_count = 148;
  uint64_t launches = 0;
  std::string err;
  NrsPool pool;
  // Grow-only scratch for split-K partial sums and operand staging.
  void* workspace = nullptr;
  size_t workspace_bytes = 0;
  // Named grow-only scratch blocks (operand staging for the tensor-core kernels).
  void* ws_slot[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  size_t ws_slot_bytes[5] = {0, 0, 0, 0, 0};
  // Device word the tensor-core kernels set when a bounded wait runs out; read at sync points.
  int* err_flag = nullptr;
  volatile int* err_host = nullptr;  // the same word as the host sees it (mapped memory)
  void* pinned = nullptr;            // page-locked: the error word, and a slot for small read-backs; made on first use
  unsigned* fold_ticket = nullptr;   // arrival counter of kernels whose last block folds the blocks' partial sums
  // Bounds of tensors for the duration of a call that stages them (an operator that had them measured in another launch).
  std::map<const void*, const NrsRange*> known_tops;
  // Planes registered for a source tensor (keyed by its device pointer); the conv kernels
  // use them instead of staging again.  Whoever registers keeps both alive and unregisters.
  std::map<const void*, NrsPlanes> plane_hints;
  std::map<const void*, NrsPlanes> owned_planes;   // nrs_planes_cache: planes the context itself allocated
  std::unordered_map<const void*, NrsRange*> ranges;   // of f16 pair planes, by the address of hi
  NrsRangePool range_pool;
  char scratch_range[2];   // addresses that own the ranges of measurements inside a call
  std::map<const void*, NrsOutExtras> out_extras;
  std::map<const void*, NrsColsumRequest> colsum_requests;
  // Patch planes (see conv_patch.cu) of a tensor with few channels, keyed by its device pointer: the host graph
  // makes them once per step for the layer's forward pass and weight gradient.
  std::map<const void*, NrsPatchPlanes> patch_hints;
  NrsWeightSet weight_set;
  // Set by a caller that has just issued a kernel whose output the NEXT tensor-core weight-gradient launch
  // does not read (see NRS_PDL_PROLOGUE): that launch may overlap it.  Consumed by the launch.
  bool independent_next = false;
  NrsStatSync stat_sync;
  NrsFolds folds;
  // Counter-based generator state of the dropout masks (dropout.cu): seed, and the next unused counter block.
  uint64_t rng_seed = 0, rng_offset = 0;
  // A process that works on samples [shard_begin, shard_begin + shard_local) of a batch of shard_global
  // (data parallelism; set by the trainer for the duration of a step, 0 = off): per-sample random draws
  // (dropout masks, augmentation) then take the counters those samples have in the GLOBAL batch's stream
  // and the stream advances by the global batch's amount, so N processes draw what one process would.
  int shard_begin = 0, shard_local = 0, shard_global = 0;
  // cudaMalloc, or what a self-test puts in its place.
  cudaError_t (*device_malloc)(void** p, size_t bytes) = [](void** p, size_t bytes) { return cudaMalloc(p, bytes); };
  // Optional per-family device timing (nrs_profile_*).
  bool profiling = false;
  std::vector<NrsProfRecord> prof_records;
  std::vector<cudaEvent_t> prof_free_events;
};

// Marks, for the duration of a scope, that the kernel launched last wrote nothing the next tensor-core
// weight-gradient launch reads (nrs_ctx::independent_next).  Not where folds went out in between (asking for the place
// of a shared weight's gradient may run the queue): that launch reads memory which the weight gradient's partial sums
// are written to next.
struct NrsIndependentNext {
  nrs_ctx* c;
  NrsIndependentNext(nrs_ctx* ctx, bool on) : c(ctx) { c->independent_next = on && c->launches != c->folds.launched_at; }
  ~NrsIndependentNext() { c->independent_next = false; }
  NrsIndependentNext(const NrsIndependentNext&) = delete;
  NrsIndependentNext& operator=(const NrsIndependentNext&) = delete;
};

// Brackets the launches issued during its lifetime with two events when
// profiling is on; free otherwise.  A product that was queued meanwhile is not counted here but where
// it is launched.
struct NrsProfScope {
  nrs_ctx* ctx;
  bool active = false;
  uint64_t queued = 0;
  NrsProfRecord rec{};
  NrsProfScope(nrs_ctx* c, int kind, double work);
  ~NrsProfScope();
};

int nrs_fail(nrs_ctx* ctx, int code, const char* fmt, ...);
// Device memory from the driver.  Where there is none left, what the context keeps without using it (large blocks and
// whole slabs of its pool, idle fold scratch) goes back first.  NRS_ERR_ALLOC names `what`.
int nrs_device_alloc(nrs_ctx* ctx, const char* what, size_t bytes, void** out);
int nrs_workspace(nrs_ctx* ctx, size_t bytes, void** out);
// (the weight-gradient kernels keep their split partials in a slot of their own: they may run while the
// data gradient's K-split is still being folded out of NRS_WS_PARTIAL)
enum { NRS_WS_A = 0, NRS_WS_B = 1, NRS_WS_PARTIAL = 2, NRS_WS_WGRAD_PARTIAL = 3, NRS_WS_FOLD = 4, NRS_WS_COUNT = 5 };
int nrs_ws_slot(nrs_ctx* ctx, int slot, size_t bytes, void** out);
// Room for operand planes of `values` values in one slot (with `split` both of a pair in one block); *lo is null without.
int nrs_ws_planes(nrs_ctx* ctx, int slot, size_t values, bool split, void** hi, void** lo);
// A new range, all zero, for what is written to `p` next; it belongs to the address until that is renewed, dropped or
// freed (nrs_free).
int nrs_range_renew(nrs_ctx* ctx, const void* p, NrsRange** out);
// The same without an address: the caller gives it back.
int nrs_range_new(nrs_ctx* ctx, NrsRange** out);
void nrs_range_free(nrs_ctx* ctx, NrsRange* r);
void nrs_range_drop(nrs_ctx* ctx, const void* p);
inline NrsRange* nrs_range_of(const nrs_ctx* ctx, const void* p) {
  auto it = ctx->ranges.find(p);
  return it == ctx->ranges.end() ? nullptr : it->second;
}
// Largest finite magnitude of `count` values at `src` into r->top and r->bound (tc_stage.cu).
int nrs_absmax(nrs_ctx* ctx, const float* src, size_t count, NrsRange* r);
// The same of two tensors in one launch.
int nrs_absmax2(nrs_ctx* ctx, const float* a, size_t na, NrsRange* ra, const float* b, size_t nb, NrsRange* rb);
// dst = the values of n consecutive f16 pairs.
int nrs_pair_unpack(nrs_ctx* ctx, const float* hi, const float* lo, float* dst, size_t n);
int nrs_err_flag(nrs_ctx* ctx, int** out);
void nrs_pinned_release(nrs_ctx* ctx);
// Zero-initialised device counters (kNrsFoldTickets of them) for "the last block to arrive folds the partials"
// reductions; the folding block resets its counter, so consecutive launches on the context's stream can share
// them.  Slot 0 serves kernels with one counter, slots 1.. kernels with a counter per column block.
constexpr int kNrsFoldTickets = 4096;
int nrs_fold_ticket(nrs_ctx* ctx, unsigned** out);
// LayerNorm with the operand planes of its result written by the kernel (norm_softmax.cu).
extern "C" int nrs_layernorm_fwd_planes(nrs_ctx* ctx, const float* a, const float* b, const float* gamma, const float* beta,
                                        float* y, float* xhat, float* istd, int rows, int f, float eps, float* y_hi, float* y_lo,
                                        int* emitted, NrsRange* istd_range);
extern "C" int nrs_layernorm_bwd_planes(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma,
                                        float* da, float* db, float* dgamma, float* dbeta, int rows, int f, int accumulate_da,
                                        int accumulate_db, int accumulate_params, float* d_hi, float* d_lo, int* emitted,
                                        const NrsRange* range_g, const NrsRange* range_istd,
                                        float* sums /*[nrs_layernorm_sum_rows][f] partial column sums of the gradient, or null*/,
                                        int* sums_rows /*how many rows of it were written; 0: none*/);
static inline int nrs_layernorm_sum_rows(const nrs_ctx* ctx) { return 4 * ctx->sm_count; }
// Operand planes of a batch of [rows][K] matrices (tc_stage.cu); see tc_mainloop.cuh for the layouts.  3xTF32: the range
// of `hi` is renewed and measured, in the same launch for small tensors, unless the caller knows a bound of the source's
// values (NrsRange::top).
int nrs_tc_stage(nrs_ctx* ctx, const float* src, float* hi, float* lo, int rows, int K, int ldk, int batch,
                 size_t src_bstride, size_t dst_bstride, bool src_k_by_rows, const NrsRange* known = nullptr,
                 const float* also = nullptr /*rows as stored, f16 pairs, one matrix: a tensor to measure in the same launch*/,
                 size_t also_count = 0, NrsRange* also_range = nullptr);
// The same of `count` matrices that lie anywhere, with one range for all of them; four to a launch, measured and staged.
int nrs_tc_stage_each(nrs_ctx* ctx, const float* const* src, int count, float* hi, float* lo, int rows, int K, int ldk, size_t dst_bstride,
                      bool src_k_by_rows);
// NHWC planes of an NCHW tensor [n][c][hw], pixel stride nrs_plane_ld(c) floats (zeros between c and there).
// chan_partial (hw > 1): [nrs_batchnorm_tiles(n, hw)][c] channel sums of the pixels of each tile.
int nrs_tc_stage_image(nrs_ctx* ctx, const float* src, float* hi, float* lo, int n, int c, int hw, float* chan_partial = nullptr,
                       const NrsRange* known = nullptr);
// Counter window of a per-sample draw of `count` elements (count = samples * per-sample) in blocks of four:
// first block to use and by how many blocks the stream advances.  Falls back to the plain stream (this
// process's own draws) when no shard is set, the call is not per-sample, or the shard does not start on a
// block boundary.
inline void nrs_rng_window(const nrs_ctx* ctx, size_t count, uint64_t* first_block, uint64_t* advance) {
  *first_block = ctx->rng_offset;
  *advance = (count + 3) / 4;
  if (ctx->shard_global <= 0 || ctx->shard_local <= 0 || count % (size_t)ctx->shard_local != 0) return;
  const size_t per = count / (size_t)ctx->shard_local, before = (size_t)ctx->shard_begin * per;
  if (before % 4 != 0) return;
  *first_block = ctx->rng_offset + before / 4;
  *advance = ((size_t)ctx->shard_global * per + 3) / 4;
}

inline const NrsPlanes* nrs_planes_find(nrs_ctx* ctx, const void* src, bool split) {
  auto it = ctx->plane_hints.find(src);
  if (it == ctx->plane_hints.end() || (it->second.split != 0) != split) return nullptr;
  return &it->second;
}
// Reads and clears the device error word (the stream must be idle); NRS_ERR_TIMEOUT if a kernel gave up a wait.
int nrs_check_device_error(nrs_ctx* ctx);

// Batch normalisation for the graph (batchnorm.cu): saves the means instead of xhat, and takes x back for the backward
// pass.  hi / lo (optional, 4-D tensors with c a multiple of 8): NHWC planes of y, or of dx, which is then overwritten
// and leaves chan_partial[nrs_batchnorm_tiles(n, hw)][c], its channel sums.
int nrs_batchnorm_fwd_saving_mean(nrs_ctx* ctx, const float* x, const float* gamma, const float* beta, float* running_mean, float* running_var,
                                  float* y, float* mean, float* istd, int n, int c, int hw, float eps, float momentum, int training, int act,
                                  float* hi, float* lo, const NrsRange* range_x = nullptr);
int nrs_batchnorm_bwd_from_x(nrs_ctx* ctx, const float* g, const float* x, const float* mean, const float* istd, const float* gamma,
                             const float* beta, float* dx, float* dgamma, float* dbeta, int n, int c, int hw, int training, int accumulate_dx,
                             int accumulate_params, int act, float* hi, float* lo, float* chan_partial);
int nrs_batchnorm_tiles(int n, int hw);

// Batched weight staging (weight_set.cu).  build: allocates planes for the described weights in the
// context's current math mode (nothing in FP32 mode) and replaces any earlier set; refresh: one launch
// that stages them all from the weights' current values; find: the planes of (w, form) when the set is
// fresh and was built for the current mode, else null.
int nrs_weight_set_build(nrs_ctx* ctx, const NrsWeightDesc* descs, int count);
int nrs_weight_set_refresh(nrs_ctx* ctx);
// Restages only the weights stored in [lo, hi) (a bucket of parameters that has just been updated), on the
// context's current stream; counts the jobs done in refreshed_jobs.  The caller decides when the set as a
// whole is fresh again.
int nrs_weight_set_refresh_range(nrs_ctx* ctx, const float* lo, const float* hi);
void nrs_weight_set_clear(nrs_ctx* ctx);
inline const NrsWeightPlanes* nrs_weight_planes_find(nrs_ctx* ctx, const void* w, int form) {
  const NrsWeightSet& ws = ctx->weight_set;
  if (!ws.fresh || ws.n_jobs == 0 || ws.split != (ctx->math_mode == NRS_MATH_3XTF32) || ctx->math_mode == NRS_MATH_FP32) return nullptr;
  auto it = ws.planes.find(std::make_pair(w, form));
  return it == ws.planes.end() ? nullptr : &it->second;
}

#define NRS_REQUIRE_CTX(ctx) \
  do { if (!(ctx)) return nrs_fail(nullptr, NRS_ERR_ARG, "%s: null context", __func__); } while (0)
#define NRS_REQUIRE(ctx, cond, code, ...) \
  do { if (!(cond)) return nrs_fail((ctx), (code), __VA_ARGS__); } while (0)
#define NRS_CUDA(ctx, call)                                                              \
  do {                                                                                   \
    cudaError_t e__ = (call);                                                            \
    if (e__ != cudaSuccess)                                                              \
      return nrs_fail((ctx), NRS_ERR_CUDA, "%s: %s failed: %s", __func__, #call,         \
                      cudaGetErrorString(e__));                                          \
  } while (0)
// After a kernel launch: count it and surface launch-configuration errors.
#define NRS_LAUNCHED(ctx)                                                                \
  do {                                                                                   \
    (ctx)->launches++;                                                                   \
    cudaError_t e__ = cudaGetLastError();                                                \
    if (e__ != cudaSuccess)                                                              \
      return nrs_fail((ctx), NRS_ERR_CUDA, "%s: kernel launch failed: %s", __func__,     \
                      cudaGetErrorString(e__));                                          \
  } while (0)

// cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a (kernel, device) pair, and one process may hold
// contexts on several devices.  Each launcher keeps one NrsSmemAttr per kernel instantiation: the largest
// value already set on every device ordinal.
constexpr int kNrsMaxDevices = 64;
struct NrsSmemAttr {
  size_t bytes[kNrsMaxDevices] = {};
};
// True when `bytes` of dynamic shared memory on `device` still has to be requested (values that fit the
// 48 KB default never do); records the request.
inline bool nrs_smem_attr_update(NrsSmemAttr& a, int device, size_t bytes) {
  if (bytes <= 48 * 1024) return false;
  if (device < 0 || device >= kNrsMaxDevices) return true;   // not tracked: always set
  if (bytes <= a.bytes[device]) return false;
  a.bytes[device] = bytes;
  return true;
}
#define NRS_ENSURE_SMEM(ctx, attr, kernel, bytes)                                                          \
  do {                                                                                                     \
    if (nrs_smem_attr_update((attr), (ctx)->device, (size_t)(bytes)))                                      \
      NRS_CUDA((ctx), cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(bytes))); \
  } while (0)

// Programmatic dependent launch.  A kernel launched through nrs_pdl_launch may be scheduled while
// the kernel before it in the stream is still running (as SMs free up in its last wave), so that its
// launch latency and prologue overlap with that kernel's tail; it must execute NRS_PDL_WAIT() before
// its first global-memory access — the wait returns once the preceding kernel has completed and its
// writes are visible.  NRS_PDL_TRIGGER() lets the NEXT kernel start the same way; every CTA of a grid
// has to issue it (or exit) before that happens, so only a grid's last wave is ever shared.
#define NRS_PDL_WAIT() asm volatile("griddepcontrol.wait;" ::: "memory")
#define NRS_PDL_TRIGGER() asm volatile("griddepcontrol.launch_dependents;" ::: "memory")
// Order: every kernel WAITS first and only then triggers.  That keeps one property a few kernels rely on:
// when kernel N+1 has been launched, every CTA of kernel N has passed its wait, so kernel N-1 and all
// before it have completed.  A kernel that does not depend on its immediate predecessor (a weight
// gradient issued right after the data gradient of the same layer: both read the same inputs) may then
// skip the wait at its start, begin on the SMs its predecessor's last wave leaves idle, and wait just
// before it exits instead, so that kernels after it still see everything before them complete.  Such a
// kernel triggers at once: its successor's own wait returns only when this kernel has completed, late wait
// included, so the successor still sees everything before it.  Two such kernels are never adjacent: the
// callers mark a launch independent only right after issuing the data gradient it may overlap.
#define NRS_PDL_PROLOGUE() \
  do { NRS_PDL_WAIT(); NRS_PDL_TRIGGER(); } while (0)

template <class... P, class... A>
inline cudaError_t nrs_pdl_launch_cluster(unsigned cluster, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                          A&&... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
template <class... P, class... A>
inline cudaError_t nrs_pdl_launch(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
  return nrs_pdl_launch_cluster(1, kernel, grid, block, smem, stream, static_cast<A&&>(args)...);
}
// kernel<<<grid, block, smem, stream>>>(args...) as a programmatic dependent launch.  The kernel
// expression goes in parentheses when its template arguments contain commas.
#define NRS_PDL_LAUNCH(kernel, grid, block, smem, stream, ...) \
  (void)nrs_pdl_launch(kernel, dim3(grid), dim3(block), (size_t)(smem), stream, __VA_ARGS__)

// How many threads share one output of a weight gradient's split reduce (each summing every lanes-th split) for a
// given number of splits.
static inline int reduce_lanes(int splits) { return splits >= 32 ? 8 : splits >= 16 ? 4 : splits >= 8 ? 2 : 1; }

static inline unsigned nrs_blocks(size_t work, unsigned per_block) {
  return (unsigned)((work + per_block - 1) / per_block);
}

// Tensor-core contraction entry points (tc_gemm.cu / tc_conv.cu).  Each returns
// NRS_ERR_UNSUPPORTED (without setting an error text) when the shape is outside
// what the tcgen05 kernels cover, and the caller then runs the FFMA kernels.
// What else the epilogue of a tensor-core GEMM may write or take part in (all optional).
struct NrsGemmExtras {
  float* pre = nullptr;        // [batch][m][n]: the value before the activation (what GELU's derivative needs)
  // The result times the derivative of the activation that produced the operand it is the gradient of: `dact` is
  // NRS_ACT_RELU (dact_src = that activation's output) or NRS_ACT_GELU (dact_src = its pre-activation), [m][n].  c keeps
  // the value without the factor; planes and column sums are of the value with it.
  int dact = NRS_ACT_NONE;
  const float* dact_src = nullptr;
  float* hi = nullptr;         // operand planes [m][n] for the GEMM that reads the result next (n a multiple of 8)
  float* lo = nullptr;
  NrsRange* range = nullptr;   // 3xTF32: of the planes (out; belongs to hi); without planes: where the largest magnitude of c goes
  float* colsum = nullptr;     // [colsum_cap][n] partial column sums
  int colsum_cap = 0;
  int colsum_rows = 0;         // out: rows of it written (0: none, the caller sums the columns itself)
  bool skip_c = false;         // c is not written (its planes are all that is read)
  bool skip_c_unsplit = false; // ... only where the result leaves in one pass (a K-split's second pass writes c and makes no column sums)
  bool honoured = false;       // out: the tensor-core kernel ran and did all of the above (but colsum: see colsum_rows)
};
int nrs_tc_gemm(nrs_ctx* ctx, int trans_a, int trans_b, int batch, int m, int n, int k,
                const float* a, const float* b, float* c, const float* bias, int act, float beta, NrsGemmExtras* extras = nullptr);
// x times several weights of one shape in one product (tc_gemm.cu); NRS_ERR_UNSUPPORTED (no error text) outside its range.
int nrs_tc_gemm_weights(nrs_ctx* ctx, int reduce, int count, int m, int n, int k, const float* x, const float* const* w, float* c,
                        float beta, NrsGemmExtras* extras);
// nrs_gemm with extras; NRS_ERR_UNSUPPORTED (no error text) when the product would not run on the tensor cores.
int nrs_gemm_extras(nrs_ctx* ctx, int trans_a, int trans_b, int m, int n, int k, const float* a, const float* b, float* c,
                    const float* bias, int act, float beta, NrsGemmExtras* extras);
int nrs_tc_conv_fwd(nrs_ctx* ctx, const float* x, const float* w, const float* b, float* y, int n, int ci, int h,
                    int wd, int co, int kh, int kw, int stride, int pad, int act);
int nrs_tc_conv_dgrad(nrs_ctx* ctx, const float* w, const float* dy, float* dx, int n, int ci, int h, int wd, int co,
                      int kh, int kw, int stride, int pad, int accumulate);
// out_cols (1x1 only): the ci columns are matrices of out_cols columns side by side, written one behind the other.
int nrs_tc_conv_wgrad(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co,
                      int kh, int kw, int stride, int pad, int accumulate, int out_cols = 0);
bool nrs_gemm_on_tensor_cores(const nrs_ctx* ctx, int m, int n, int k);
// Whether nrs_gemm's A^T B [m,n] runs on row planes of A and B (never on the f32 tensors): then a caller may hand it
// planes without the tensor behind them.
inline bool nrs_gemm_tn_reads_planes(int m, int n) { return m >= 32 && n >= 32 && ((long)m * n <= (4L << 20) || (m % 32 == 0 && n % 32 == 0)); }
// C[m,n] (+)= A^T B, A stored [k][m], B stored [k][n], on the weight-gradient kernel (no transposes).
int nrs_tc_gemm_tn(nrs_ctx* ctx, int m, int n, int k, const float* a, const float* b, float* c, int accumulate);
// Row-streaming variant for 3x3 / stride 1 / pad 1 (tc_wgrad_rows.cu); tried first.
int nrs_tc_conv_wgrad_rows(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co,
                           int kh, int kw, int stride, int pad, int accumulate);
// Fused attention core on the tensor cores (attention_tc.cu); NRS_ERR_UNSUPPORTED (no error text) outside its range.
int nrs_tc_attention_fwd(nrs_ctx* ctx, const float* q, const float* k, const float* v, float* out, float* probs, int batch,
                         int seq, int heads, int d_head, int causal);
int nrs_tc_attention_bwd(nrs_ctx* ctx, const float* q, const float* k, const float* v, const float* probs, const float* dout,
                         float* dq, float* dk, float* dv, int batch, int seq, int heads, int d_head, int acc_q, int acc_k,
                         int acc_v);
// Tensor-core convolution through patch planes (conv_patch.cu); NRS_ERR_UNSUPPORTED (no error text) for layers that
// do not use patches.
int nrs_patch_planes(nrs_ctx* ctx, const float* x, float* hi, float* lo, int n, int ci, int h, int wd, int kh, int kw, int stride, int pad);
int nrs_patch_conv_fwd(nrs_ctx* ctx, const float* x, const float* w, const float* b, float* y, int n, int ci, int h, int wd, int co,
                       int kh, int kw, int stride, int pad, int act);
int nrs_patch_conv_wgrad(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co, int kh, int kw,
                         int stride, int pad, int accumulate);
// Direct FFMA kernels for 3x3 stride-1 layers over 1 or 3 input channels (conv_smallc.cu).
int nrs_smallc_conv_fwd(nrs_ctx* ctx, const float* x, const float* w, const float* b, float* y, int n, int ci, int h,
                        int wd, int co, int kh, int kw, int stride, int pad, int act);
int nrs_smallc_conv_wgrad(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co,
                          int kh, int kw, int stride, int pad, int accumulate);
