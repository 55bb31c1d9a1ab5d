// Folds: the second stages of the split reductions that end a layer's backward pass (column sums of bias and LayerNorm
// parameter gradients, K-split partial tiles of weight gradients), each a few microseconds of mostly latency.
//
// Nothing in a backward pass reads these gradients, so inside nrs::backward_graph they are collected and run as ONE
// launch at its end (nrs_folds_begin / nrs_folds_flush); outside of it each runs as a batch of one.  The job table
// travels as a kernel parameter.  Every sum has a fixed order, whatever the batch.  Measured on the CIFAR CNN at batch
// 100: 15 launches, 104 us, become one of 38 us; on the language model (32 x 128 tokens) 21 launches, 125 us, one of 40.
#include "fold.h"
#include "wgrad_queue.h"

#include <algorithm>

#include "igemm_problems.cuh"

namespace {

constexpr int kMaxJobs = 32;
// Rows of a column fold that one block takes at least: 16 per warp, two rounds of loads.  (1024 rows to a block are
// thirteen rounds of loads, one behind the other.)
constexpr int kColumnRows = 128;
// The divisions that place a weight gradient's outputs, as multiplications (with 32-bit divisions the pass was bound by
// instructions: 740 per warp, most of them there).
struct FoldDiv {
  NrsFastDiv run, run4, taps, cblks, group, chunk;
};
template <int CAP>
struct FoldBatch {
  int n;
  unsigned first_block[CAP];   // of each job, side by side: the search over them is one or two lines of constant memory
  NrsFoldJob job[CAP];
  FoldDiv div[CAP];
};
static_assert(sizeof(FoldBatch<kMaxJobs>) <= 8000, "the job table is a kernel parameter");

__device__ __forceinline__ void put(float* dst, float v, int accumulate) { *dst = accumulate ? *dst + v : v; }

__device__ __forceinline__ float* column_dst(const NrsFoldJob& j, int c) { return j.dst2 && c >= j.cols1 ? j.dst2 + (c - j.cols1) : j.dst + c; }

// dst[c] (+)= sum over rows of src[r*stride + c].  A block takes 32 columns of a row split: its eight warps every eighth
// row, eight rows in flight per thread, combined in warp order; with several splits the last block of a column group to
// arrive adds the splits in the same way: warp w splits w, w + 8, ...
__device__ void fold_columns(const NrsFoldJob& j, unsigned blk, float* sm) {
  __shared__ bool last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int groups = (j.cols + 31) / 32, grp = (int)(blk % groups), split = (int)(blk / groups);
  const int c = grp * 32 + lane;
  const int per = (j.rows + j.splits - 1) / j.splits, r0 = split * per, r1 = min(j.rows, r0 + per);
  float t = 0.0f;
  if (c < j.cols) {
    const size_t step = (size_t)8 * j.stride;
    const float* s = j.src + (size_t)(r0 + warp) * j.stride + c;
    for (int r = r0 + warp; r < r1; r += 64, s += 8 * step) {   // eight loads under way, the last round's too
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = r + 8 * u < r1 ? s[u * step] : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (r + 8 * u < r1) t += v[u];
    }
  }
  sm[warp * 32 + lane] = t;
  __syncthreads();
  if (warp == 0 && c < j.cols) {
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += sm[w * 32 + lane];
    if (j.splits == 1) put(column_dst(j, c), sum, j.accumulate);
    else j.scratch[(size_t)split * j.cols + c] = sum;
  }
  if (j.splits == 1) return;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicAdd(&j.tickets[grp], 1u) == (unsigned)j.splits - 1;
  __syncthreads();
  if (!last) return;
  __threadfence();
  t = 0.0f;
  if (c < j.cols)
    for (int z = warp; z < j.splits; z += 64) {
      float v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) v[u] = z + 8 * u < j.splits ? __ldcg(j.scratch + (size_t)(z + 8 * u) * j.cols + c) : 0.0f;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (z + 8 * u < j.splits) t += v[u];
    }
  sm[warp * 32 + lane] = t;
  __syncthreads();
  if (warp == 0 && c < j.cols) {
    float sum = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) sum += sm[w * 32 + lane];
    put(column_dst(j, c), sum, j.accumulate);
  }
  if (threadIdx.x == 0) j.tickets[grp] = 0;
}

// dw (+)= sum over splits of partial tiles.  A block is (256 / lanes) outputs (quads of four input channels) x `lanes`
// split lanes: lane y sums splits y, y + lanes, ... and the lanes are combined in lane order through shared memory: a
// fixed order of additions without one serial chain of loads per output.  Outputs are counted (co, 32-channel block,
// tap, quad), so that reads of the partials are 128-byte runs along ci and the 8 * taps outputs of a block of channels
// are one run of dw: with several taps the sums go back through shared memory and leave in dw's order (written from
// their quads, 4 bytes every 4 * taps, they took twice as long as the reads).
__device__ void fold_tiles(const NrsFoldJob& j, const FoldDiv& dv, unsigned blk, float4* sums) {
  const int per_block = 256 / j.lanes;
  const int lane = threadIdx.x / per_block, slot = threadIdx.x - lane * per_block;
  const uint32_t cblks = (uint32_t)(j.ci + 31) / 32, run = 8u * j.taps;
  const uint32_t total = (uint32_t)j.co * cblks * run;   // (below 2^31: nrs_fold_submit)
  const uint32_t idx = blk * per_block + slot;
  uint32_t r, u, co_u, cb;
  dv.run.divmod(idx, r, u);
  dv.cblks.divmod(r, co_u, cb);
  const int tap = (int)(u >> 3), co = (int)co_u, c = (int)(cb * 32 + (u & 7) * 4);
  const bool live = idx < total && c < j.ci;
  size_t off;
  if (j.kind == NRS_FOLD_WGRAD) {                 // [m block][group][column block][128][group_cols]
    const int mb = co >> 7, row = co & 127;
    const int grp = (int)dv.group.div((uint32_t)tap), t = tap - grp * j.taps_per_group;
    const int cbk = j.col_blocks > 1 ? c >> (31 - __clz(j.group_cols)) : 0;   // (column blocks are a power of two wide)
    const size_t col = j.col_blocks > 1 ? (size_t)(c - cbk * j.group_cols) : (size_t)t * j.cblocks * 32 + c;
    off = ((((size_t)mb * j.n_groups + grp) * j.col_blocks + cbk) * 128 + row) * j.group_cols + col;
  } else {                                        // rows kernel: a (horizontal j, vertical i) pair per tap
    const int i = (int)((unsigned)tap / 3u), jt = tap - 3 * i;
    int mb = co >> 7, row = co & 127, jk = jt;
    if (j.pack) {   // tap 1 -> kind 0 rows [0,h); tap 0 -> kind 0 rows [h,2h); tap 2 -> kind 1 rows [0,h)
      mb = 0;
      jk = jt == 2 ? 1 : 0;
      row = co + (jt == 0 ? 32 * j.a_blocks : 0);
    }
    const int cc = (int)dv.chunk.div((uint32_t)c);
    const int cta = (mb * j.jtypes + jk) * j.n_chunks + cc;
    const size_t cols = (size_t)3 * j.chunk;
    off = ((size_t)cta * 128 + row) * cols + (size_t)i * j.chunk + (c - cc * j.chunk);
  }
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (live) {
    const float* src = j.src + off;
    for (int z = lane; z < j.splits; z += 8 * j.lanes) {   // eight loads under way, the last round's too
      float4 v[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (z + u * j.lanes < j.splits) v[u] = *reinterpret_cast<const float4*>(src + (size_t)(z + u * j.lanes) * j.split_stride);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (z + u * j.lanes < j.splits) { s.x += v[u].x; s.y += v[u].y; s.z += v[u].z; s.w += v[u].w; }
    }
  }
  if (j.lanes > 1) {
    sums[threadIdx.x] = s;
    __syncthreads();
    if (lane == 0)
      for (int l = 1; l < j.lanes; ++l) {
        const float4 v = sums[l * per_block + slot];
        s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
      }
  }
  if (j.taps == 1) {
    // [co][ci]; with out_cols (several matrices side by side) columns c of matrix c / out_cols, each [co][out_cols]
    if (lane != 0 || !live) return;
    if (j.vec) {
      const int mat = j.out_cols ? c / j.out_cols : 0, ld = j.out_cols ? j.out_cols : j.ci;
      float4* dst = reinterpret_cast<float4*>(j.dst + (size_t)mat * j.co * ld + (size_t)co * ld + (c - mat * ld));
      if (j.accumulate) {
        const float4 o = *dst;
        s = make_float4(o.x + s.x, o.y + s.y, o.z + s.z, o.w + s.w);
      }
      *dst = s;
      return;
    }
    const float e[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (c + k >= j.ci) continue;
      const int mat = j.out_cols ? (c + k) / j.out_cols : 0, ld = j.out_cols ? j.out_cols : j.ci;
      put(j.dst + (size_t)mat * j.co * ld + (size_t)co * ld + (c + k - mat * ld), e[k], j.accumulate);
    }
    return;
  }
  __syncthreads();   // (the lanes' sums have been read)
  if (lane == 0) sums[slot] = s;
  __syncthreads();
  const float* f = reinterpret_cast<const float*>(sums);
  const uint32_t first = blk * per_block, end = min(first + per_block, total);
  if (first >= total) return;
  const uint32_t r0 = dv.run.div(first), r1 = dv.run.div(end - 1) + 1;
  for (uint32_t q = threadIdx.x; q < (r1 - r0) * 4 * run; q += 256) {   // output values of the runs this block has a share in
    uint32_t rr, pos, ch, t, o, ob;
    dv.run4.divmod(q, rr, pos);
    dv.taps.divmod(pos, ch, t);
    const uint32_t id = (r0 + rr) * run + t * 8 + (ch >> 2) - first;
    dv.cblks.divmod(r0 + rr, o, ob);
    const uint32_t cc = ob * 32 + ch;
    if (id < end - first && cc < (uint32_t)j.ci)   // (unsigned: below `first` counts as beyond)
      put(j.dst + ((size_t)o * j.ci + cc) * j.taps + t, f[id * 4 + (ch & 3)], j.accumulate);
  }
}

// CAP: room in the job table.  A fold outside of a backward pass comes alone, and 7 KB of empty table cost it 0.7 us
// (LayerNorm's parameter gradients of [819][256]: 7.5 us with the full table, 6.7 with room for one).
template <int CAP>
__global__ void __launch_bounds__(256) fold_kernel(const __grid_constant__ FoldBatch<CAP> b) {
  NRS_PDL_PROLOGUE();
  __shared__ float4 sm[256];
  int i = CAP - 1;
  if (CAP > 1) {
    i = b.n - 1;
    while (i > 0 && b.first_block[i] > blockIdx.x) --i;
  }
  const NrsFoldJob& j = b.job[i];
  const unsigned blk = blockIdx.x - j.first_block;
  if (j.kind == NRS_FOLD_COLUMNS) fold_columns(j, blk, reinterpret_cast<float*>(sm));
  else fold_tiles(j, b.div[i], blk, sm);
}

unsigned job_blocks(const NrsFoldJob& j) {
  if (j.kind == NRS_FOLD_COLUMNS) return (unsigned)((j.cols + 31) / 32) * (unsigned)j.splits;
  const size_t total = (size_t)j.co * ((j.ci + 31) / 32) * 8 * j.taps;
  return (unsigned)((total + 256 / j.lanes - 1) / (256 / j.lanes));
}

template <int CAP>
int run_table(nrs_ctx* ctx, NrsFoldJob* jobs, int n) {
  FoldBatch<CAP> b{};
  unsigned blocks = 0;
  unsigned ticket = 1;   // slot 0 serves kernels with one counter
  unsigned* tickets = nullptr;   // made when a job asks for some
  for (int i = 0; i < n; ++i) {
    NrsFoldJob& j = jobs[i];
    if (j.kind == NRS_FOLD_COLUMNS && j.splits > 1) {
      const int st = tickets ? NRS_OK : nrs_fold_ticket(ctx, &tickets);
      if (st != NRS_OK) return st;
      j.tickets = tickets + ticket;
      ticket += (unsigned)((j.cols + 31) / 32);
    }
    j.first_block = blocks;
    blocks += job_blocks(j);
    if (j.kind != NRS_FOLD_COLUMNS) {
      const bool general = j.kind == NRS_FOLD_WGRAD;
      b.div[b.n] = FoldDiv{NrsFastDiv(8 * j.taps), NrsFastDiv(32 * j.taps), NrsFastDiv(j.taps), NrsFastDiv((j.ci + 31) / 32),
                           NrsFastDiv(general ? j.taps_per_group : 1), NrsFastDiv(general ? 1 : j.chunk)};
    }
    b.first_block[b.n] = j.first_block;
    b.job[b.n++] = j;
  }
  if (blocks == 0) return NRS_OK;
  NRS_PDL_LAUNCH(fold_kernel<CAP>, blocks, 256, 0, ctx->stream, b);
  NRS_LAUNCHED(ctx);
  ctx->folds.launched_at = ctx->launches;
  return NRS_OK;
}
int run(nrs_ctx* ctx, NrsFoldJob* jobs, int n) { return n == 1 ? run_table<1>(ctx, jobs, n) : run_table<kMaxJobs>(ctx, jobs, n); }

// Launches what is queued.  Its partial sums stay where they are: place() says when their memory starts over.
int run_queue(nrs_ctx* ctx) {
  NrsFolds& f = ctx->folds;
  if (f.jobs.empty()) return NRS_OK;
  const int st = run(ctx, f.jobs.data(), (int)f.jobs.size());
  ctx->independent_next = false;   // whoever writes into that memory next waits for this launch
  f.jobs.clear();
  f.tickets_used = 1;
  f.holding = 0;
  return st;
}

// Memory for partial sums out of the blocks there are, or null.  The blocks start over only when nothing in them is
// still to be read: no job with sums there is queued, and none is being made (its memory is handed out before the kernel that fills it
// is launched and the job is submitted, and what comes in between may run the queue, or other jobs for the sake of memory).
float* place(NrsFolds& f, size_t bytes) {
  if (f.holding == 0 && !f.open && !f.relieving) f.chunk = f.used = 0;
  for (; f.chunk < f.chunks.size(); ++f.chunk, f.used = 0)
    if (f.used + bytes <= f.chunks[f.chunk].second) {
      float* p = (float*)((uint8_t*)f.chunks[f.chunk].first + f.used);
      f.used += bytes;
      f.open = true;
      return p;
    }
  return nullptr;
}

}  // namespace

void nrs_folds_begin(nrs_ctx* ctx) { ctx->folds.active = true; }

static void drop_kept(nrs_ctx* ctx) {
  for (void* p : ctx->folds.kept) nrs_free(ctx, p);
  ctx->folds.kept.clear();
  ctx->folds.kept_bytes = 0;
}

int nrs_folds_flush(nrs_ctx* ctx) {
  NrsFolds& f = ctx->folds;
  int st = NRS_OK;
  if (!f.waiting.empty()) {
    f.waiting.clear();
    st = nrs_wgrad_rows_run(ctx);
    if (st == NRS_OK) st = nrs_wgrad_tiles_run(ctx);
  }
  if (st == NRS_OK) st = run_queue(ctx);
  drop_kept(ctx);
  return st;
}

int nrs_folds_relieve(nrs_ctx* ctx) {
  NrsFolds& f = ctx->folds;
  const bool open = f.open, relieving = f.relieving;
  f.relieving = true;
  const int st = nrs_folds_flush(ctx);
  f.relieving = relieving;
  f.open = open;                  // whose job is being made still has its memory
  ctx->independent_next = false;  // the kernel launched last is not the one its caller had in mind
  return st;
}

void nrs_free_after_wgrads(nrs_ctx* ctx, void* p) {
  NrsFolds& f = ctx->folds;
  if (f.waiting.empty()) {
    nrs_free(ctx, p);
  } else if (p) {
    f.kept.push_back(p);
    const auto it = ctx->pool.live.find(p);
    f.kept_bytes += it == ctx->pool.live.end() ? 0 : it->second;
  }
}

void nrs_folds_end(nrs_ctx* ctx) {
  ctx->folds.active = ctx->folds.open = false;
  ctx->folds.jobs.clear();
  ctx->folds.tickets_used = 1;
  ctx->folds.holding = 0;
  ctx->folds.waiting.clear();
  ctx->folds.waiting_rows.reset();
  ctx->folds.waiting_tiles.reset();
  drop_kept(ctx);
}

void nrs_folds_free(nrs_ctx* ctx) {
  for (auto& c : ctx->folds.chunks)
    if (c.second <= NrsPool::kSmall) nrs_free(ctx, c.first);
    else cudaFree(c.first);
  ctx->folds.chunks.clear();
  ctx->folds.chunk = ctx->folds.used = 0;
}

// Whether a job writes any of the `len` floats at `p`.  (One job may write several tensors: a column pair has two
// outputs, the weight gradients of Q, K and V lie one behind the other.)
static bool writes(const NrsFoldJob& j, const float* p, size_t len) {
  auto meets = [p, len](const float* at, size_t n) { return at < p + len && p < at + n; };
  if (j.kind != NRS_FOLD_COLUMNS) return meets(j.dst, (size_t)j.co * j.ci * j.taps);
  if (!j.dst2) return meets(j.dst, (size_t)j.cols);
  return meets(j.dst, (size_t)j.cols1) || meets(j.dst2, (size_t)(j.cols - j.cols1));
}

int nrs_folds_settle(nrs_ctx* ctx, const float* dst, size_t len) {
  for (const auto& w : ctx->folds.waiting)
    if (w.first < dst + len && dst < w.first + w.second) return nrs_folds_flush(ctx);
  for (const NrsFoldJob& j : ctx->folds.jobs)
    if (writes(j, dst, len)) return nrs_folds_flush(ctx);
  return NRS_OK;
}

// Partial sums of a job that may wait live in blocks of their own (not pool blocks, which are handed out again as soon
// as the host releases them, and not a shared slot, which the next layer overwrites).  The first is small and comes out of
// a slab (a small model needs no more); then 64 MB at a time; at 512 MB what is queued runs and the blocks start over, or,
// while a job is being made, there is one block more.
int nrs_fold_partial(nrs_ctx* ctx, int ws_slot, size_t bytes, float** out) {
  NrsFolds& f = ctx->folds;
  void* p = nullptr;
  if (!f.active) {
    const int st = ws_slot >= 0 ? nrs_ws_slot(ctx, ws_slot, bytes, &p) : nrs_workspace(ctx, bytes, &p);
    *out = (float*)p;
    return st;
  }
  constexpr size_t kChunk = (size_t)64 << 20, kLimit = (size_t)512 << 20;
  bytes = (bytes + 255) / 256 * 256;
  if ((*out = place(f, bytes))) return NRS_OK;
  size_t total = 0;
  for (auto& c : f.chunks) total += c.second;
  if (total + bytes > kLimit && !f.open && !f.jobs.empty()) {
    const int st = run_queue(ctx);
    if (st != NRS_OK) return st;
    if ((*out = place(f, bytes))) return NRS_OK;
  }
  const size_t want = f.chunks.empty() && bytes <= NrsPool::kSmall ? NrsPool::kSmall : std::max(kChunk, bytes);
  auto more = [&] { return want <= NrsPool::kSmall ? nrs_alloc(ctx, want, 0, &p) : nrs_device_alloc(ctx, "fold scratch", want, &p); };
  int st = more();
  if (st != NRS_OK && !f.open && !f.jobs.empty()) {   // what is queued runs, and its memory is to be had again
    st = run_queue(ctx);
    if (st != NRS_OK) return st;
    if ((*out = place(f, bytes))) return NRS_OK;
    st = more();
  }
  if (st != NRS_OK) return st;
  f.chunks.push_back({p, want});
  *out = place(f, bytes);
  return NRS_OK;
}

int nrs_fold_submit(nrs_ctx* ctx, NrsFoldJob job) {
  NrsFolds& f = ctx->folds;
  if (job.kind != NRS_FOLD_COLUMNS) {
    NRS_REQUIRE(ctx, (size_t)job.co * ((job.ci + 31) / 32) * 8 * job.taps < 0x7fffffffu, NRS_ERR_SHAPE, "weight gradient: too large");
    const int ld = job.out_cols ? job.out_cols : job.ci;
    job.vec = job.taps == 1 && ld % 4 == 0 && (reinterpret_cast<uintptr_t>(job.dst) & 15) == 0;
  }
  if (!f.active) return run(ctx, &job, 1);
  const unsigned need = job.kind == NRS_FOLD_COLUMNS && job.splits > 1 ? (unsigned)((job.cols + 31) / 32) : 0;
  if (f.jobs.size() >= (size_t)kMaxJobs || f.tickets_used + need > kNrsFoldTickets) {
    const int st = run_queue(ctx);
    if (st != NRS_OK) return st;
  }
  // a second share of the same gradient: the first one goes ahead of it
  const bool pair = job.kind == NRS_FOLD_COLUMNS && job.dst2;
  int st = nrs_folds_settle(ctx, job.dst, job.kind != NRS_FOLD_COLUMNS ? (size_t)job.co * job.ci * job.taps : (size_t)(pair ? job.cols1 : job.cols));
  if (st == NRS_OK && pair) st = nrs_folds_settle(ctx, job.dst2, (size_t)(job.cols - job.cols1));
  if (st != NRS_OK) return st;
  f.tickets_used += need;
  f.jobs.push_back(job);
  bool held = f.open;   // (one launch may leave the sums of several jobs: `open` speaks for the first of them to be submitted)
  for (const auto& c : f.chunks) {
    const uintptr_t lo = (uintptr_t)c.first, src = (uintptr_t)job.src, scratch = (uintptr_t)job.scratch;
    held = held || (src >= lo && src < lo + c.second) || (scratch >= lo && scratch < lo + c.second);
  }
  f.holding += held ? 1 : 0;
  f.open = false;
  return NRS_OK;
}

static int fold_columns_to(nrs_ctx* ctx, const float* src, float* dst, float* dst2, int cols1, int rows, int cols, int stride, int accumulate) {
  if (cols <= 0) return NRS_OK;
  NrsFoldJob j{};
  j.dst2 = dst2;
  j.cols1 = cols1;
  j.kind = NRS_FOLD_COLUMNS;
  j.src = src;
  j.dst = dst;
  j.rows = rows; j.cols = cols; j.stride = stride;
  j.accumulate = accumulate;
  const int groups = (cols + 31) / 32;
  j.splits = 1;
  if (rows >= 2 * kColumnRows && groups + 1 <= kNrsFoldTickets) {
    j.splits = std::min(rows / kColumnRows, (2 * ctx->sm_count + groups - 1) / groups);
    if (j.splits < 1) j.splits = 1;
  }
  if (j.splits > 1) {
    float* p = nullptr;
    const int st = nrs_fold_partial(ctx, NRS_WS_FOLD, (size_t)j.splits * cols * sizeof(float), &p);
    if (st != NRS_OK) return st;
    j.scratch = p;
  }
  return nrs_fold_submit(ctx, j);
}

int nrs_fold_columns(nrs_ctx* ctx, const float* src, float* dst, int rows, int cols, int stride, int accumulate) {
  return fold_columns_to(ctx, src, dst, nullptr, cols, rows, cols, stride, accumulate);
}
int nrs_fold_column_pair(nrs_ctx* ctx, const float* src, float* dst, float* dst2, int rows, int cols, int stride, int accumulate) {
  return fold_columns_to(ctx, src, dst, dst2, cols, rows, 2 * cols, stride, accumulate);
}

// Host bookkeeping of the queue, without a device: how many checks failed (0 = all hold).
extern "C" int nrs_selftest_fold_bookkeeping(void) {
  int bad = 0;
  static float mem[4096];   // addresses only
  NrsFoldJob qkv{};         // three [8][8] weight gradients one behind the other
  qkv.kind = NRS_FOLD_WGRAD;
  qkv.dst = mem + 1024; qkv.co = 8; qkv.ci = 24; qkv.taps = 1; qkv.out_cols = 8;
  for (int m = 0; m < 3; ++m) bad += writes(qkv, mem + 1024 + m * 64, 64) ? 0 : 1;
  bad += writes(qkv, mem + 1024 - 64, 64) ? 1 : 0;
  bad += writes(qkv, mem + 1024 + 192, 64) ? 1 : 0;
  bad += writes(qkv, mem, 4096) ? 0 : 1;               // a gradient that holds all of it
  NrsFoldJob conv{};                                    // [4][2][3][3]
  conv.kind = NRS_FOLD_WGRAD_ROWS;
  conv.dst = mem; conv.co = 4; conv.ci = 2; conv.taps = 9;
  bad += writes(conv, mem + 71, 1) ? 0 : 1;
  bad += writes(conv, mem + 72, 1) ? 1 : 0;
  NrsFoldJob pair{};
  pair.kind = NRS_FOLD_COLUMNS;
  pair.dst = mem; pair.dst2 = mem + 512; pair.cols = 20; pair.cols1 = 10;
  bad += writes(pair, mem + 9, 4) ? 0 : 1;
  bad += writes(pair, mem + 10, 502) ? 1 : 0;
  bad += writes(pair, mem + 521, 1) ? 0 : 1;
  bad += writes(pair, mem + 522, 1) ? 1 : 0;
  pair.dst2 = nullptr;                                  // all twenty columns in one place
  bad += writes(pair, mem + 19, 1) ? 0 : 1;
  bad += writes(pair, mem + 512, 10) ? 1 : 0;

  // memory handed out stays its job's own until that job has been launched, whatever is launched before it
  nrs_ctx c;
  NrsFolds& f = c.folds;
  f.active = true;
  f.chunks = {{mem, 8192}, {mem + 2048, 8192}};
  float* p[6] = {};
  for (int i = 0; i < 2; ++i) bad += nrs_fold_partial(&c, -1, 1000, &p[i]) == NRS_OK ? 0 : 1;   // two blocks of one job
  bad += p[0] == mem && p[1] == mem + 256 ? 0 : 1;
  bad += nrs_fold_submit(&c, pair) == NRS_OK && f.jobs.size() == 1 ? 0 : 1;
  bad += nrs_fold_partial(&c, -1, 4096, &p[2]) == NRS_OK && p[2] == mem + 512 ? 0 : 1;
  f.jobs.clear();            // the queue is launched while the second job is being made
  f.holding = 0;
  bad += nrs_fold_partial(&c, -1, 4096, &p[3]) == NRS_OK && p[3] == mem + 2048 ? 0 : 1;
  bad += nrs_fold_submit(&c, pair) == NRS_OK ? 0 : 1;
  bad += nrs_fold_partial(&c, -1, 4096, &p[4]) == NRS_OK && p[4] == mem + 3072 ? 0 : 1;
  bad += nrs_fold_submit(&c, qkv) == NRS_OK && f.jobs.size() == 2 ? 0 : 1;
  f.jobs.clear();
  f.holding = 0;
  bad += nrs_fold_submit(&c, pair) == NRS_OK && f.holding == 0 ? 0 : 1;   // sums in memory of its own: nobody's concern
  bad += nrs_fold_partial(&c, -1, 16, &p[5]) == NRS_OK && p[5] == mem ? 0 : 1;   // nothing waits: from the start again

  // two jobs' sums from one launch, and the queue is launched when the first of them has been submitted
  f.jobs.clear();
  f.holding = 0;
  f.open = false;
  NrsFoldJob sums = pair;
  for (int i = 0; i < 2; ++i) bad += nrs_fold_partial(&c, -1, 4096, &p[i]) == NRS_OK ? 0 : 1;
  sums.src = p[0];
  bad += nrs_fold_submit(&c, sums) == NRS_OK ? 0 : 1;
  f.jobs.clear();
  f.holding = 0;
  sums.src = p[1];
  bad += nrs_fold_submit(&c, sums) == NRS_OK && f.holding == 1 ? 0 : 1;
  bad += nrs_fold_partial(&c, -1, 16, &p[2]) == NRS_OK && p[2] != p[0] && p[2] != p[1] ? 0 : 1;
  f.jobs.clear();
  f.holding = 0;
  f.open = false;

  // a weight gradient never starts under a launch of folds
  c.launches = 7;
  { NrsIndependentNext on(&c, true); bad += c.independent_next ? 0 : 1; }
  f.launched_at = 7;
  { NrsIndependentNext on(&c, true); bad += c.independent_next ? 1 : 0; }
  c.launches = 8;            // the data gradient, issued after the folds
  { NrsIndependentNext on(&c, true); bad += c.independent_next ? 0 : 1; }
  { NrsIndependentNext off(&c, false); bad += c.independent_next ? 1 : 0; }
  return bad;
}
