// Cross-entropy on raw logits with dense one-hot (f32) targets.
// Reference: ce_forward / ce_backward (src/cuda/loss/cross_entropy.rs:18-57),
// host side :74-128; CPU semantics src/nn/loss.rs:50-107.  The reference runs
// one thread per row and sums the per-row losses on the host after a blocking
// device-to-host copy; here a warp owns a row (shuffle reductions, the row is
// re-read from L1), forward and backward share one pass, and the batch mean is
// reduced on the device in a fixed order.
#include "nrs_internal.h"
#include "row_pipe.cuh"

namespace {

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Batch mean without a second launch: wsum[0..n) (shared memory, one sum per warp or team) -> block, in order ->
// block_partial[block]; the block that arrives last folds the partials in block order (lane l takes l, l+32, ..., then
// a butterfly), so the order of the additions is fixed whichever block that is.
__device__ __forceinline__ void fold_batch_loss(const float* wsum, int n, float* block_partial, unsigned* ticket, float* loss_dev,
                                                float inv_div) {
  __shared__ bool last;
  __syncthreads();
  if (threadIdx.x == 0) {
    float s = 0.0f;
    for (int w = 0; w < n; ++w) s += wsum[w];
    block_partial[blockIdx.x] = s;
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x >= 32) return;
  __threadfence();
  float s = 0.0f;
  for (unsigned i = threadIdx.x; i < gridDim.x; i += 32) s += __ldcg(block_partial + i);
  s = warp_sum(s);
  if (threadIdx.x == 0) {
    loss_dev[0] = s * inv_div;
    *ticket = 0;
  }
}

// Large batches and odd widths (row_pipe.cuh): logits in the first buffer, the one-hot row (when there is one) in the
// second; the gradient replaces the logits.
struct CeOp {
  const int32_t* labels;
  float *row_loss, *block_partial, *loss_dev;
  unsigned* ticket;
  float inv_div;
  int has_target;
  template <int NPL> struct State { float loss; };
  template <class C, class S> __device__ __forceinline__ void start(const C&, S& s) const { s.loss = 0.0f; }
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void row(const rowpipe::Team& tm, const C& c, S& s, float* buf0, float* buf1, int r) const {
    float x[NPL], t[NPL], mx = -INFINITY;
    c.load(buf0, x, -INFINITY);
    if (has_target) {
      c.load(buf1, t);
    } else {
      const int label = labels[r];
#pragma unroll
      for (int i = 0; i < NPL; ++i) t[i] = c.first(i / VEC) + i % VEC == label ? 1.0f : 0.0f;
    }
    float v[3] = {0.0f, 0.0f, 0.0f};   // sum exp(x - max), sum t*x, sum t
#pragma unroll
    for (int i = 0; i < NPL; ++i)
      if (c.live(i / VEC)) {
        mx = fmaxf(mx, x[i]);
        v[1] += t[i] * x[i];
        v[2] += t[i];
      }
    mx = tm.max(mx);
#pragma unroll
    for (int i = 0; i < NPL; ++i)
      if (c.live(i / VEC)) { x[i] = expf(x[i] - mx); v[0] += x[i]; }
    tm.sum(v);
    const float lse = logf(v[0]) + mx, inv_se = 1.0f / v[0];
#pragma unroll
    for (int i = 0; i < NPL; ++i) x[i] = (x[i] * inv_se - t[i]) * inv_div;
    c.store(buf0, x);
    const float rl = lse * v[2] - v[1];
    if (row_loss && tm.warp == 0 && tm.lane == 0) row_loss[r] = rl;
    s.loss += rl;
  }
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void finish(const rowpipe::Team& tm, const C&, S& s, float* smem, int team, int teams) const {
    if (!loss_dev) return;
    if (tm.warp == 0 && tm.lane == 0) smem[team] = s.loss;
    fold_batch_loss(smem, teams, block_partial, ticket, loss_dev, inv_div);
  }
  static size_t finish_bytes(int teams, int) { return (size_t)teams * sizeof(float); }
};

// One warp per row.  row_loss (optional) gets -sum_c t*(x - lse); grad (optional)
// gets (softmax - t) * inv_div.  Scalar path (any width / alignment).
// FOLD: the kernel also folds the batch mean, which saves a launch; without, row_loss is left to ce_mean_kernel.  The
// fold costs the loops registers (48 against 40) and every block a fence and an atomic, so it is for small calls and a few
// others (see run_ce): [64][10] 6.0 us with two launches, 4.0 with one; [16760][1001] with labels 64 and 85.
template <bool FOLD>
__global__ void __launch_bounds__(256)
ce_rows_kernel(const float* __restrict__ logits, const float* __restrict__ target, const int32_t* __restrict__ labels,
               float* __restrict__ row_loss, float* __restrict__ grad, int batch, int classes, float inv_div, float* block_partial,
               unsigned* ticket, float* loss_dev) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  float warp_loss = 0.0f;   // this warp's rows, in the order it takes them
  for (int b = blockIdx.x * warps_per_block + (threadIdx.x >> 5); b < batch; b += gridDim.x * warps_per_block) {
    const float* row = logits + (size_t)b * classes;
    const float* trow = target ? target + (size_t)b * classes : nullptr;
    const int label = labels ? labels[b] : -1;
    float mx = -INFINITY;
    for (int c = lane; c < classes; c += 32) mx = fmaxf(mx, row[c]);
    mx = warp_max(mx);
    float se = 0.0f;
    for (int c = lane; c < classes; c += 32) se += expf(row[c] - mx);
    se = warp_sum(se);
    const float lse = logf(se) + mx;
    float loss = 0.0f;
    for (int c = lane; c < classes; c += 32) {
      const float xv = row[c], tv = trow ? trow[c] : (c == label ? 1.0f : 0.0f);
      loss += -tv * (xv - lse);
      if (grad) grad[(size_t)b * classes + c] = (expf(xv - mx) / se - tv) * inv_div;
    }
    if (FOLD || row_loss) {
      loss = warp_sum(loss);
      if (row_loss && lane == 0) row_loss[b] = loss;
      if (FOLD) warp_loss += loss;
    }
  }
  if (FOLD) {
    __shared__ float wsum[32];
    if (lane == 0) wsum[threadIdx.x >> 5] = warp_loss;
    fold_batch_loss(wsum, warps_per_block, block_partial, ticket, loss_dev, inv_div);
  }
}

// loss_dev[0] = (sum_b row_loss[b]) * inv_div, one block, fixed summation tree.
__global__ void __launch_bounds__(1024)
ce_mean_kernel(const float* __restrict__ row_loss, float* __restrict__ loss_dev, int batch, float inv_div) {
  NRS_PDL_PROLOGUE();
  __shared__ float sm[32];
  float s = 0.0f;
  int i = threadIdx.x;
  const int step = blockDim.x;
  for (; i + 7 * step < batch; i += 8 * step) {   // eight loads in flight; the additions keep the order of i
    float v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = row_loss[i + u * step];
#pragma unroll
    for (int u = 0; u < 8; ++u) s += v[u];
  }
  for (; i < batch; i += step) s += row_loss[i];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float t = threadIdx.x < (blockDim.x >> 5) ? sm[threadIdx.x] : 0.0f;
    t = warp_sum(t);
    if (threadIdx.x == 0) loss_dev[0] = t * inv_div;
  }
}

// The same with the row held in registers: logits (and the one-hot row) are read once with 128-bit
// loads (lane l takes float4s l, l+32, ...: 512 contiguous bytes per load instruction), every
// exponential is evaluated once, the gradient is written once.  Rows of up to 1024 classes whose
// width is a multiple of four.  With `labels` (int32 class per row) the dense one-hot tensor is not read.
// Registers hold two rows only, which is what bounds the rows in flight per SM (three blocks per SM): the
// target row, and the logits row that is overwritten by its exponentials once sum(t*x) and sum(t) have been
// taken (the row loss is lse*sum(t) - sum(t*x)).
template <int VPL>
__global__ void __launch_bounds__(256, 3)
ce_rows_vec_kernel(const float* __restrict__ logits, const float* __restrict__ target, const int32_t* __restrict__ labels,
                   float* __restrict__ row_loss, float* __restrict__ grad, int batch, int classes, float inv_div,
                   float* block_partial, unsigned* ticket, float* loss_dev) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31;
  const int warps_per_block = blockDim.x >> 5;
  const int c4 = classes >> 2;
  float warp_loss = 0.0f;   // this warp's rows, in the order it takes them
  for (int b = blockIdx.x * warps_per_block + (threadIdx.x >> 5); b < batch; b += gridDim.x * warps_per_block) {
    const size_t base = (size_t)b * classes;
    float4 x[VPL], t[VPL];
    float mx = -INFINITY;
    const int label = labels ? labels[b] : -1;
    // the row this warp takes next is pulled into L2 while this one is worked on: a warp is a serial chain
    // (loads, two reductions, stores), and this takes the DRAM round trip out of the next link
    {
      const int nb = b + gridDim.x * warps_per_block;
      if (nb < batch) {
        const char* nx = reinterpret_cast<const char*>(logits + (size_t)nb * classes);
        for (int off = lane * 128; off < classes * 4; off += 32 * 128) {
          asm volatile("prefetch.global.L2 [%0];" ::"l"(nx + off));
          if (target) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(target + (size_t)nb * classes) + off));
        }
      }
    }
    // every load of the row (logits and one-hot row) is in flight before the first reduction waits
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < c4) {
        x[k] = __ldcs(reinterpret_cast<const float4*>(logits + base) + c);
        if (target) {
          t[k] = __ldcs(reinterpret_cast<const float4*>(target + base) + c);
        } else {
          const int d = label - 4 * c;     // position of the label inside this float4, if any
          t[k] = make_float4(d == 0 ? 1.0f : 0.0f, d == 1 ? 1.0f : 0.0f, d == 2 ? 1.0f : 0.0f, d == 3 ? 1.0f : 0.0f);
        }
      }
    }
    float stx = 0.0f, st = 0.0f;   // sum(t*x), sum(t) of this lane's elements
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (lane + 32 * k < c4) {
        mx = fmaxf(mx, fmaxf(fmaxf(x[k].x, x[k].y), fmaxf(x[k].z, x[k].w)));
        stx += (t[k].x * x[k].x + t[k].y * x[k].y) + (t[k].z * x[k].z + t[k].w * x[k].w);
        st += (t[k].x + t[k].y) + (t[k].z + t[k].w);
      }
    mx = warp_max(mx);
    float se = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (lane + 32 * k < c4) {
        x[k] = make_float4(expf(x[k].x - mx), expf(x[k].y - mx), expf(x[k].z - mx), expf(x[k].w - mx));
        se += (x[k].x + x[k].y) + (x[k].z + x[k].w);
      }
    se = warp_sum(se);          // three independent butterflies: their shuffles interleave
    stx = warp_sum(stx);
    st = warp_sum(st);
    const float lse = logf(se) + mx;
    const float inv_se = 1.0f / se;
    if (grad) {
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int c = lane + 32 * k;
        if (c < c4)
          __stcs(reinterpret_cast<float4*>(grad + base) + c,
                 make_float4((x[k].x * inv_se - t[k].x) * inv_div, (x[k].y * inv_se - t[k].y) * inv_div,
                             (x[k].z * inv_se - t[k].z) * inv_div, (x[k].w * inv_se - t[k].w) * inv_div));
      }
    }
    const float rl = lse * st - stx;
    if (row_loss && lane == 0) row_loss[b] = rl;
    warp_loss += rl;
  }
  if (!loss_dev) return;
  __shared__ float wsum[32];
  if (lane == 0) wsum[threadIdx.x >> 5] = warp_loss;
  fold_batch_loss(wsum, warps_per_block, block_partial, ticket, loss_dev, inv_div);
}

int run_ce(nrs_ctx* ctx, const char* who, const float* logits, const float* target, const int32_t* labels, float* loss_dev,
           float* row_loss, float* grad, int batch, int classes, int divisor) {
  NRS_REQUIRE(ctx, batch >= 0 && classes > 0, NRS_ERR_SHAPE, "%s: bad shape [%d,%d]", who, batch, classes);
  NRS_REQUIRE(ctx, divisor > 0, NRS_ERR_ARG, "%s: divisor must be positive", who);
  if (batch == 0) {
    if (loss_dev) NRS_CUDA(ctx, cudaMemsetAsync(loss_dev, 0, sizeof(float), ctx->stream));
    return NRS_OK;
  }
  NRS_REQUIRE(ctx, logits && (target || labels), NRS_ERR_ARG, "%s: null tensor", who);
  const float inv_div = 1.0f / (float)divisor;
  // Where the row pipeline is the better kernel: from 8 M elements up (us here -> there, tensors that are not in L2).
  // Float4 rows: with a one-hot target [16384][1000] 52 -> 48, 1024 columns 52 -> 45, 512 46 -> 43 (but 64 M elements 146,
  // 155); not 256 (50, 61) or 384 (46, 52); with labels nowhere (1000: 40, 50; 256: 46, 71).  Scalar loops, with a one-hot
  // target: 16 M elements of 250 columns 107 -> 53, 385 95 -> 85, 1001 129 -> 107, 3000 136 -> 61, not 1281 (120, 162; 2.5
  // live warps) or 700 (44, 52 in [20000][700]); with labels, one tensor less to bring in, only with more columns at work:
  // 250 73 -> 61, 1002 64 -> 50, 4096 97 -> 51, not 385 (54, 60), 1001 (64, 70), 1281 (59, 73) or 2999 (75, 90).  Rows of 257
  // to 512 columns with a one-hot target wait for 12 M elements: 8 M of 385 that lie in L2 take 39 and 48.
  const bool vec = classes % 4 == 0 && classes <= 1024 &&
                   ((reinterpret_cast<uintptr_t>(logits) | reinterpret_cast<uintptr_t>(target) | reinterpret_cast<uintptr_t>(grad)) & 15) == 0;
  const double fill = rowpipe::fill(classes), live = rowpipe::live_warps(classes, target ? 2 : 1);
  const bool wide = classes <= 512 || classes >= 960;
  const size_t elems = (size_t)batch * classes;
  const bool pipe = elems >= (size_t)1 << 23 && fill >= 0.75 &&
                    (vec      ? target && (classes >= 960 || (classes >= 448 && classes <= 512 && elems < (size_t)1 << 25))
                     : target ? wide && live >= (classes > 512 || elems >= (size_t)12 << 20 ? 3.5 : 4.5)
                              : wide && live >= 9.5 && (fill >= 0.85 || classes > 1500));
  if (pipe && rowpipe::applies(batch, classes, {logits, target, grad})) {
    rowpipe::Params p{};
    p.in[0] = logits; p.in[1] = target;
    p.n_in = p.n_buf = target ? 2 : 1;
    p.out[0] = grad;
    p.rows = batch; p.f = classes;
    CeOp op{labels, row_loss, nullptr, loss_dev, nullptr, inv_div, target != nullptr};
    if (loss_dev) {
      void* ws = nullptr;
      int st = nrs_workspace(ctx, (size_t)ctx->sm_count * sizeof(float), &ws);
      if (st == NRS_OK) st = nrs_fold_ticket(ctx, &op.ticket);
      if (st != NRS_OK) return st;
      op.block_partial = (float*)ws;
    }
    const int st = rowpipe::launch(ctx, p, op);
    if (st != NRS_ERR_UNSUPPORTED) return st;
  }
  int blocks = (batch + 7) / 8;
  if (blocks > ctx->sm_count * 8) blocks = ctx->sm_count * 8;
  // wide rows: one resident wave (three blocks of 80 registers per SM) of warps that walk several rows each,
  // prefetching the next
  if (classes > 512 && blocks > ctx->sm_count * 3) blocks = ctx->sm_count * 3;
  // The vector kernels fold the batch mean themselves (per-block partial sums, last block folds), the scalar one where
  // a launch weighs more, or where the mean's own launch has very many rows to add.  us with two launches and with one:
  // 64 x 10 6.0, 4.0; 2048 x 33 6.0, 4.6; 8192 x 33 6.4, 8.5; 512 x 127 5.9, 6.3, with labels (a tensor less to read) 5.9,
  // 5.0; 512 x 255 7.0, 7.5; with labels 133455 x 33 63, 58 and 9532 x 33 8.6, 9.0; with a one-hot target 508400 x 33 241,
  // 232 and 133455 x 33 67, 67; beyond 1800 columns always (1024 x 4096 86, 82, with labels 33, 30; 2990 x 1401 39, 41).
  const bool small = batch <= 4096 && classes <= (target ? 64 : 128) && (size_t)batch * classes <= (size_t)1 << (target ? 17 : 18);
  const bool many = batch >= 1 << (target ? 18 : 16) && classes <= 256;
  const bool fold = vec || small || many || classes >= 1800;
  float* rl = row_loss;
  float* partial = nullptr;
  unsigned* ticket = nullptr;
  if (loss_dev) {
    void* ws = nullptr;
    int st = nrs_workspace(ctx, (size_t)(fold ? blocks : rl ? 0 : batch) * sizeof(float) + 16, &ws);
    if (st == NRS_OK && fold) st = nrs_fold_ticket(ctx, &ticket);
    if (st != NRS_OK) return st;
    if (fold) partial = (float*)ws;
    else if (!rl) rl = (float*)ws;
  }
  if (vec && classes <= 128) {
    NRS_PDL_LAUNCH(ce_rows_vec_kernel<1>, blocks, 256, 0, ctx->stream, logits, target, labels, row_loss, grad, batch, classes, inv_div,
                   partial, ticket, loss_dev);
  } else if (vec && classes <= 512) {
    NRS_PDL_LAUNCH(ce_rows_vec_kernel<4>, blocks, 256, 0, ctx->stream, logits, target, labels, row_loss, grad, batch, classes, inv_div,
                   partial, ticket, loss_dev);
  } else if (vec) {
    NRS_PDL_LAUNCH(ce_rows_vec_kernel<8>, blocks, 256, 0, ctx->stream, logits, target, labels, row_loss, grad, batch, classes, inv_div,
                   partial, ticket, loss_dev);
  } else {
    if (loss_dev && fold)
      NRS_PDL_LAUNCH(ce_rows_kernel<true>, blocks, 256, 0, ctx->stream, logits, target, labels, rl, grad, batch, classes, inv_div, partial,
                     ticket, loss_dev);
    else
      NRS_PDL_LAUNCH(ce_rows_kernel<false>, blocks, 256, 0, ctx->stream, logits, target, labels, rl, grad, batch, classes, inv_div,
                     (float*)nullptr, (unsigned*)nullptr, (float*)nullptr);
  }
  NRS_LAUNCHED(ctx);
  if (loss_dev && !fold) {
    NRS_PDL_LAUNCH(ce_mean_kernel, 1, 1024, 0, ctx->stream, rl, loss_dev, batch, inv_div);
    NRS_LAUNCHED(ctx);
  }
  return NRS_OK;
}

}  // namespace

extern "C" {

int nrs_ce_fwd(nrs_ctx* ctx, const float* logits, const float* target, float* loss_dev, float* row_loss,
               int batch, int classes, int divisor) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, loss_dev || row_loss, NRS_ERR_ARG, "nrs_ce_fwd: no output requested");
  return run_ce(ctx, "nrs_ce_fwd", logits, target, nullptr, loss_dev, row_loss, nullptr, batch, classes, divisor);
}

int nrs_ce_bwd(nrs_ctx* ctx, const float* logits, const float* target, float* grad, int batch, int classes,
               int divisor) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, grad || batch == 0, NRS_ERR_ARG, "nrs_ce_bwd: null grad");
  return run_ce(ctx, "nrs_ce_bwd", logits, target, nullptr, nullptr, nullptr, grad, batch, classes, divisor);
}

int nrs_ce_fwd_bwd(nrs_ctx* ctx, const float* logits, const float* target, float* loss_dev, float* grad,
                   int batch, int classes, int divisor) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, loss_dev && (grad || batch == 0), NRS_ERR_ARG, "nrs_ce_fwd_bwd: null output");
  return run_ce(ctx, "nrs_ce_fwd_bwd", logits, target, nullptr, loss_dev, nullptr, grad, batch, classes, divisor);
}

int nrs_ce_fwd_bwd_indexed(nrs_ctx* ctx, const float* logits, const int32_t* labels, float* loss_dev, float* grad,
                           int batch, int classes, int divisor) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, loss_dev && (grad || batch == 0), NRS_ERR_ARG, "nrs_ce_fwd_bwd_indexed: null output");
  NRS_REQUIRE(ctx, labels || batch == 0, NRS_ERR_ARG, "nrs_ce_fwd_bwd_indexed: null labels");
  return run_ce(ctx, "nrs_ce_fwd_bwd_indexed", logits, nullptr, labels, loss_dev, nullptr, grad, batch, classes, divisor);
}

}  // extern "C"
