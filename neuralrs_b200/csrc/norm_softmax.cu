// LayerNorm and row softmax, forward and backward.
//
// One warp owns a row and keeps it in registers: rows whose width is a multiple of four (up to
// 1024 floats) are read ONCE with 128-bit loads — lane l takes the float4s l, l+32, l+64, ... so every
// load instruction of the warp covers 512 contiguous bytes — reduced with shuffles, and written once.
// Other widths run scalar loops with the same arithmetic.  The LayerNorm backward pass produces the
// input gradient (optionally into two destinations: the fused residual add) and the parameter
// gradients from one read of g and xhat: every warp keeps column partials of dgamma / dbeta in
// registers over the rows it visits, the block folds its warps in warp order through shared memory,
// and the blocks are folded in block order (fold.cu) — fixed order, no atomics, bit-reproducible.
// Large tensors and odd widths run on the row pipeline where that is the better one (row_pipe.cuh).
// (The reference runs one thread per row and three kernels.)
// Reference: ln_forward / ln_reduce / ln_dx (src/cuda/nn/normalization.rs:14-78),
// softmax_forward / softmax_backward (src/cuda/graph/softmax.rs:12-35); CPU
// semantics src/nn/normalization.rs:38-103, src/autograd/graph/softmax.rs:23-60.
#include "fold.h"
#include "nrs_internal.h"
#include "pair.cuh"
#include "row_pipe.cuh"
#include "tc_common.cuh"

namespace {

// ------------------------------------------------------------------ large tensors and odd widths (row_pipe.cuh)
struct NoState {};

// x = a (+ b); xhat replaces a, y = gamma*xhat + beta goes to the second buffer.
struct LnFwdOp {
  const float *gamma, *beta;
  float* istd_out;
  float eps;
  int has_b;
  template <int NPL> struct State { float gamma[NPL], beta[NPL]; };   // the lane's columns, for all rows it meets
  template <class C, class S> __device__ __forceinline__ void start(const C& c, S& s) const {
    c.load(gamma, s.gamma);
    c.load(beta, s.beta);
  }
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void row(const rowpipe::Team& tm, const C& c, S& s, float* buf0, float* buf1, int r) const {
    float v[NPL], t[1] = {0.0f};
    c.load(buf0, v);
    if (has_b) {
      float w[NPL];
      c.load(buf1, w);
#pragma unroll
      for (int i = 0; i < NPL; ++i) v[i] += w[i];
    }
#pragma unroll
    for (int i = 0; i < NPL; ++i) t[0] += v[i];
    tm.sum(t);
    const float mean = t[0] / (float)c.f;
    t[0] = 0.0f;
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      v[i] -= mean;
      if (c.live(i / VEC)) t[0] += v[i] * v[i];
    }
    tm.sum(t);
    const float istd = 1.0f / sqrtf(t[0] / (float)c.f + eps);
    if (istd_out && tm.warp == 0 && tm.lane == 0) istd_out[r] = istd;
#pragma unroll
    for (int i = 0; i < NPL; ++i) v[i] *= istd;
    c.store(buf0, v);
#pragma unroll
    for (int i = 0; i < NPL; ++i) v[i] = s.gamma[i] * v[i] + s.beta[i];
    c.store(buf1, v);
  }
  template <int NPL, int VEC, class C, class S>
  __device__ void finish(const rowpipe::Team&, const C&, S&, float*, int, int) const {}
  static size_t finish_bytes(int, int) { return 0; }
};

// g in the first buffer, xhat in the second; the input gradient replaces g.  With `partial` every lane also keeps the
// column sums of g*xhat and g over all rows it meets; they are folded team by team into partial[block][2][f].
struct LnBwdOp {
  const float *istd, *gamma;
  float* partial;
  int want_dx;
  template <int NPL> struct State { float pg[NPL], pb[NPL], gamma[NPL]; };
  template <class C, class S> __device__ __forceinline__ void start(const C& c, S& s) const {
    c.load(gamma, s.gamma);
#pragma unroll
    for (int i = 0; i < (int)(sizeof(s.pg) / sizeof(float)); ++i) s.pg[i] = s.pb[i] = 0.0f;
  }
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void row(const rowpipe::Team& tm, const C& c, S& s, float* buf0, float* buf1, int r) const {
    const float is = want_dx ? __ldg(istd + r) : 0.0f;   // on its way while the row is reduced
    float g[NPL], xh[NPL];
    c.load(buf0, g);
    c.load(buf1, xh);
    if (partial) {
#pragma unroll
      for (int i = 0; i < NPL; ++i) { s.pg[i] += g[i] * xh[i]; s.pb[i] += g[i]; }
    }
    if (!want_dx) return;
    float t[2] = {0.0f, 0.0f};
#pragma unroll
    for (int i = 0; i < NPL; ++i) {
      g[i] *= s.gamma[i];
      t[0] += g[i];
      t[1] += g[i] * xh[i];
    }
    tm.sum(t);
    const float s1 = t[0] / (float)c.f, s2 = t[1] / (float)c.f;
#pragma unroll
    for (int i = 0; i < NPL; ++i) g[i] = is * (g[i] - s1 - xh[i] * s2);
    c.store(buf0, g);
  }
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void finish(const rowpipe::Team&, const C& c, S& s, float* smem, int team, int teams) const {
    if (!partial) return;
    float* mine = smem + (size_t)team * 2 * c.f;
#pragma unroll
    for (int k = 0; k < NPL; ++k) {
      const int col = c.first(k / VEC) + k % VEC;
      if (col < c.f) { mine[col] = s.pg[k]; mine[c.f + col] = s.pb[k]; }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * c.f; i += blockDim.x) {
      float t = 0.0f;
      for (int w = 0; w < teams; ++w) t += smem[(size_t)w * 2 * c.f + i];
      partial[(size_t)blockIdx.x * 2 * c.f + i] = t;
    }
  }
  static size_t finish_bytes(int teams, int f) { return (size_t)teams * 2 * f * sizeof(float); }
};

struct SoftmaxFwdOp {
  template <int NPL> using State = NoState;
  template <class C, class S> __device__ void start(const C&, S&) const {}
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void row(const rowpipe::Team& tm, const C& c, S&, float* buf0, float*, int) const {
    float v[NPL], mx = -INFINITY, t[1] = {0.0f};
    c.load(buf0, v, -INFINITY);
#pragma unroll
    for (int i = 0; i < NPL; ++i) mx = fmaxf(mx, v[i]);
    mx = tm.max(mx);
#pragma unroll
    for (int i = 0; i < NPL; ++i)
      if (c.live(i / VEC)) { v[i] = expf(v[i] - mx); t[0] += v[i]; }
    tm.sum(t);
#pragma unroll
    for (int i = 0; i < NPL; ++i) v[i] = v[i] / t[0];
    c.store(buf0, v);
  }
  template <int NPL, int VEC, class C, class S>
  __device__ void finish(const rowpipe::Team&, const C&, S&, float*, int, int) const {}
  static size_t finish_bytes(int, int) { return 0; }
};

// y in the first buffer, g in the second; the gradient replaces y.
struct SoftmaxBwdOp {
  template <int NPL> using State = NoState;
  template <class C, class S> __device__ void start(const C&, S&) const {}
  template <int NPL, int VEC, class C, class S>
  __device__ __forceinline__ void row(const rowpipe::Team& tm, const C& c, S&, float* buf0, float* buf1, int) const {
    float y[NPL], g[NPL], t[1] = {0.0f};
    c.load(buf0, y);
    c.load(buf1, g);
#pragma unroll
    for (int i = 0; i < NPL; ++i) t[0] += y[i] * g[i];
    tm.sum(t);
#pragma unroll
    for (int i = 0; i < NPL; ++i) y[i] *= g[i] - t[0];
    c.store(buf0, y);
  }
  template <int NPL, int VEC, class C, class S>
  __device__ void finish(const rowpipe::Team&, const C&, S&, float*, int, int) const {}
  static size_t finish_bytes(int, int) { return 0; }
};

// The TF32 operand planes of a value that the next tensor-core GEMM will read (rows x f, the tensor's own
// layout): written by the producing kernel so that no separate staging pass reads the tensor again.
__device__ __forceinline__ void put_planes(float* hi, float* lo, size_t at, float4 v, float scale, uint32_t& top) {
  if (lo) {
    top = pr::seen4(top, v);
    pr::put4(hi, lo, at, v, scale);
  } else {
    *reinterpret_cast<float4*>(hi + at) = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
  }
}
// f16 pairs: the scale of a result of `bound`, which one thread of the grid leaves as its range.
__device__ __forceinline__ float open_pairs(NrsRange* range, float bound) {
  bound = fminf(bound * 1.001f, 3.0e38f);
  if (blockIdx.x == 0 && threadIdx.x == 0) range->bound = bound;
  return pr::scale_of(bound);
}

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float wmax(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

constexpr int kMaxVpl = 8;                 // float4s per lane: rows of up to 32 * 4 * 8 = 1024 floats
constexpr int kRowThreads = 256;

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
// streaming variants for tensors that are read or written exactly once
__device__ __forceinline__ float4 ld4_stream(const float* p) { return __ldcs(reinterpret_cast<const float4*>(p)); }
__device__ __forceinline__ void st4_stream(float* p, float4 v) { __stcs(reinterpret_cast<float4*>(p), v); }

// ------------------------------------------------------------------ LayerNorm forward
// x = a (+ b when given: the residual add folded in); y = gamma * xhat + beta.
// EMIT: also write the operand planes of y (a separate instantiation, so that the plain kernel keeps its registers).
template <int VPL, bool EMIT>
__global__ void __launch_bounds__(kRowThreads)
ln_fwd_vec_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ gamma,
                  const float* __restrict__ beta, float* __restrict__ y, float* __restrict__ xhat,
                  float* __restrict__ istd_out, int rows, int f, float eps, float* __restrict__ y_hi,
                  float* __restrict__ y_lo, NrsRange* __restrict__ range, NrsRange* __restrict__ istd_range) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int f4 = f >> 2;
  const float inv_f = 1.0f / (float)f;
  [[maybe_unused]] float scale = 1.0f;
  [[maybe_unused]] uint32_t top = 0, top_istd = 0;
  if (EMIT && y_lo) {   // |xhat| <= sqrt(f)
    uint32_t mg = 0, mb = 0;
    for (int c = lane; c < f4; c += 32) {
      mg = pr::seen4(mg, ld4(gamma + 4 * c));
      mb = pr::seen4(mb, ld4(beta + 4 * c));
    }
    mg = __reduce_max_sync(0xffffffffu, mg);
    mb = __reduce_max_sync(0xffffffffu, mb);
    scale = open_pairs(range, sqrtf((float)f) * __uint_as_float(mg) + __uint_as_float(mb));
  }
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const size_t base = (size_t)r * f;
    float4 v[VPL];
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      v[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (c < f4) {
        v[k] = ld4_stream(a + base + 4 * c);
        if (b) {
          const float4 w = ld4_stream(b + base + 4 * c);
          v[k].x += w.x; v[k].y += w.y; v[k].z += w.z; v[k].w += w.w;
        }
        s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
      }
    }
    const float mean = wsum(s) * inv_f;
    float vs = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (lane + 32 * k < f4) {
        const float dx = v[k].x - mean, dy = v[k].y - mean, dz = v[k].z - mean, dw = v[k].w - mean;
        vs += (dx * dx + dy * dy) + (dz * dz + dw * dw);
      }
    const float istd = 1.0f / sqrtf(wsum(vs) * inv_f + eps);
    if (lane == 0 && istd_out) istd_out[r] = istd;
    if (EMIT) top_istd = pr::seen(top_istd, istd);
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < f4) {
        const float4 gm = ld4(gamma + 4 * c), bt = ld4(beta + 4 * c);
        float4 xn;
        xn.x = (v[k].x - mean) * istd; xn.y = (v[k].y - mean) * istd;
        xn.z = (v[k].z - mean) * istd; xn.w = (v[k].w - mean) * istd;
        if (xhat) st4_stream(xhat + base + 4 * c, xn);
        const float4 out = make_float4(gm.x * xn.x + bt.x, gm.y * xn.y + bt.y, gm.z * xn.z + bt.z, gm.w * xn.w + bt.w);
        st4_stream(y + base + 4 * c, out);
        if (EMIT) put_planes(y_hi, y_lo, base + 4 * c, out, scale, top);
      }
    }
  }
  if (EMIT && y_lo) {
    pr::report_block(range, top);
    if (istd_range) {
      __syncthreads();
      pr::report_block(istd_range, top_istd);
    }
  }
}

__global__ void __launch_bounds__(kRowThreads)
ln_fwd_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ gamma,
              const float* __restrict__ beta, float* __restrict__ y, float* __restrict__ xhat,
              float* __restrict__ istd_out, int rows, int f, float eps) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const float* ra = a + (size_t)r * f;
    const float* rb = b ? b + (size_t)r * f : nullptr;
    float s = 0.0f;
    for (int i = lane; i < f; i += 32) s += rb ? ra[i] + rb[i] : ra[i];
    const float mean = wsum(s) / (float)f;
    float vs = 0.0f;
    for (int i = lane; i < f; i += 32) { const float d = (rb ? ra[i] + rb[i] : ra[i]) - mean; vs += d * d; }
    const float var = wsum(vs) / (float)f;
    const float istd = 1.0f / sqrtf(var + eps);
    if (lane == 0 && istd_out) istd_out[r] = istd;
    for (int i = lane; i < f; i += 32) {
      const float xn = ((rb ? ra[i] + rb[i] : ra[i]) - mean) * istd;
      if (xhat) xhat[(size_t)r * f + i] = xn;
      y[(size_t)r * f + i] = gamma[i] * xn + beta[i];
    }
  }
}

// ------------------------------------------------------------------ LayerNorm backward
// dx (+)= istd * (g*gamma - mean(g*gamma) - xhat * mean(g*gamma*xhat)), optionally also into dx2 (the
// second addend of a fused residual add receives the same gradient); per-block column partials of
// dgamma = sum_r g*xhat and dbeta = sum_r g into partial[block][2][f] when `partial` is given, and with it (EMIT) those of
// the gradient itself, without what it is added to, into sums[block][f]: the bias gradient of a linear layer that made the
// addend.  (A launch of its own for those, two per language model step: 6.5 us each at 4096 x 256.)
template <int VPL, bool EMIT>
__global__ void __launch_bounds__(kRowThreads)
ln_bwd_vec_kernel(const float* __restrict__ g, const float* __restrict__ xhat, const float* __restrict__ istd,
                  const float* __restrict__ gamma, float* dx, float* dx2, float* __restrict__ partial, int rows, int f,
                  int acc1, int acc2, float* __restrict__ d_hi, float* __restrict__ d_lo, float* __restrict__ sums,
                  const NrsRange* __restrict__ range_g, const NrsRange* __restrict__ range_istd, NrsRange* __restrict__ range) {
  NRS_PDL_PROLOGUE();
  extern __shared__ float ln_smem[];          // [warps][2][f] when partial != nullptr
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5, wpb = blockDim.x >> 5;
  const int f4 = f >> 2;
  const float inv_f = 1.0f / (float)f;
  float4 gm[VPL], pg[VPL], pb[VPL];
  [[maybe_unused]] float4 pd[EMIT ? VPL : 1];
#pragma unroll
  for (int k = 0; k < VPL; ++k) {
    const int c = lane + 32 * k;
    gm[k] = c < f4 ? ld4(gamma + 4 * c) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    pg[k] = pb[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (EMIT) pd[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  }
  [[maybe_unused]] float scale = 1.0f;
  [[maybe_unused]] uint32_t top = 0;
  if (EMIT && d_lo) {   // both means are at most the largest |g * gamma| (times |xhat| <= sqrt(f))
    uint32_t mg = 0;
#pragma unroll
    for (int k = 0; k < VPL; ++k) mg = pr::seen4(mg, gm[k]);
    mg = __reduce_max_sync(0xffffffffu, mg);
    scale = open_pairs(range, (2.0f + sqrtf((float)f)) * __uint_as_float(mg) * range_g->top * range_istd->top);
  }
  for (int r = blockIdx.x * wpb + wrp; r < rows; r += gridDim.x * wpb) {
    const size_t base = (size_t)r * f;
    float4 gv[VPL], xh[VPL];
    float s1 = 0.0f, s2 = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      gv[k] = xh[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (c < f4) {
        gv[k] = ld4_stream(g + base + 4 * c);
        xh[k] = ld4_stream(xhat + base + 4 * c);
        if (partial) {
          pg[k].x += gv[k].x * xh[k].x; pg[k].y += gv[k].y * xh[k].y; pg[k].z += gv[k].z * xh[k].z; pg[k].w += gv[k].w * xh[k].w;
          pb[k].x += gv[k].x; pb[k].y += gv[k].y; pb[k].z += gv[k].z; pb[k].w += gv[k].w;
        }
        gv[k].x *= gm[k].x; gv[k].y *= gm[k].y; gv[k].z *= gm[k].z; gv[k].w *= gm[k].w;    // dxhat
        s1 += (gv[k].x + gv[k].y) + (gv[k].z + gv[k].w);
        s2 += (gv[k].x * xh[k].x + gv[k].y * xh[k].y) + (gv[k].z * xh[k].z + gv[k].w * xh[k].w);
      }
    }
    if (dx) {
      s1 = wsum(s1) * inv_f;
      s2 = wsum(s2) * inv_f;
      const float is = istd[r];
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int c = lane + 32 * k;
        if (c < f4) {
          float4 o;
          o.x = is * (gv[k].x - s1 - xh[k].x * s2); o.y = is * (gv[k].y - s1 - xh[k].y * s2);
          o.z = is * (gv[k].z - s1 - xh[k].z * s2); o.w = is * (gv[k].w - s1 - xh[k].w * s2);
          if (EMIT) {   // planes and sums of the gradient itself (before any accumulation)
            put_planes(d_hi, d_lo, base + 4 * c, o, scale, top);
            pd[k].x += o.x; pd[k].y += o.y; pd[k].z += o.z; pd[k].w += o.w;
          }
          float4 w = o;
          if (acc1) { const float4 old = ld4(dx + base + 4 * c); w.x += old.x; w.y += old.y; w.z += old.z; w.w += old.w; }
          st4(dx + base + 4 * c, w);
          if (dx2) {
            if (acc2) { const float4 old = ld4(dx2 + base + 4 * c); o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w; }
            st4(dx2 + base + 4 * c, o);
          }
        }
      }
    }
  }
  if (EMIT && d_lo) pr::report_block(range, top);
  if (partial) {
    float* mine = ln_smem + (size_t)wrp * 2 * f;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < f4) { st4(mine + 4 * c, pg[k]); st4(mine + f + 4 * c, pb[k]); }
    }
    __syncthreads();
    float* out = partial + (size_t)blockIdx.x * 2 * f;
    for (int i = threadIdx.x; i < 2 * f; i += blockDim.x) {
      float t = 0.0f;
      for (int w = 0; w < wpb; ++w) t += ln_smem[(size_t)w * 2 * f + i];     // warp order
      out[i] = t;
    }
    if (EMIT && sums) {
      __syncthreads();
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int c = lane + 32 * k;
        if (c < f4) st4(mine + 4 * c, pd[k]);
      }
      __syncthreads();
      for (int i = threadIdx.x; i < f; i += blockDim.x) {
        float t = 0.0f;
        for (int w = 0; w < wpb; ++w) t += ln_smem[(size_t)w * 2 * f + i];
        sums[(size_t)blockIdx.x * f + i] = t;
      }
    }
  }
}

__global__ void __launch_bounds__(kRowThreads)
ln_dx_kernel(const float* __restrict__ g, const float* __restrict__ xhat, const float* __restrict__ istd,
             const float* __restrict__ gamma, float* dx, float* dx2, int rows, int f, int acc1, int acc2) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const float nf = (float)f;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const size_t st = (size_t)r * f;
    float s1 = 0.0f, s2 = 0.0f;
    for (int i = lane; i < f; i += 32) {
      const float dxh = g[st + i] * gamma[i];
      s1 += dxh;
      s2 += dxh * xhat[st + i];
    }
    s1 = wsum(s1);
    s2 = wsum(s2);
    const float is = istd[r];
    for (int i = lane; i < f; i += 32) {
      const float dxh = g[st + i] * gamma[i];
      const float v = is * (dxh - s1 / nf - xhat[st + i] * s2 / nf);
      dx[st + i] = acc1 ? dx[st + i] + v : v;
      if (dx2) dx2[st + i] = acc2 ? dx2[st + i] + v : v;
    }
  }
}

// Scalar path of the parameter gradients: dgamma[c] = sum_r g*xhat, dbeta[c] = sum_r g over a row split;
// 32 columns per block.
__global__ void __launch_bounds__(256)
ln_param_kernel(const float* __restrict__ g, const float* __restrict__ xhat, float* __restrict__ partial,
                int rows, int f, int splits) {
  NRS_PDL_PROLOGUE();
  __shared__ float sg[8][33], sb[8][33];
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + lane, split = blockIdx.y;
  const int rows_per = (rows + splits - 1) / splits;
  const int r0 = split * rows_per, r1 = min(rows, r0 + rows_per);
  float dg = 0.0f, db = 0.0f;
  if (c < f)
    for (int r = r0 + wrp; r < r1; r += 8) {
      const float gv = g[(size_t)r * f + c];
      dg += gv * xhat[(size_t)r * f + c];
      db += gv;
    }
  sg[wrp][lane] = dg;
  sb[wrp][lane] = db;
  __syncthreads();
  if (wrp == 0 && c < f) {
    float tg = 0.0f, tb = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) { tg += sg[i][lane]; tb += sb[i][lane]; }
    partial[((size_t)split * 2 + 0) * f + c] = tg;
    partial[((size_t)split * 2 + 1) * f + c] = tb;
  }
}
// ------------------------------------------------------------------ softmax
template <int VPL>
__global__ void __launch_bounds__(kRowThreads)
softmax_fwd_vec_kernel(const float* __restrict__ x, float* __restrict__ y, int rows, int width) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int w4 = width >> 2;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const size_t base = (size_t)r * width;
    float4 v[VPL];
    float mx = -INFINITY;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < w4) {
        v[k] = ld4_stream(x + base + 4 * c);
        mx = fmaxf(mx, fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w)));
      }
    }
    mx = wmax(mx);
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k)
      if (lane + 32 * k < w4) {
        v[k].x = expf(v[k].x - mx); v[k].y = expf(v[k].y - mx); v[k].z = expf(v[k].z - mx); v[k].w = expf(v[k].w - mx);
        s += (v[k].x + v[k].y) + (v[k].z + v[k].w);
      }
    s = wsum(s);
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < w4) st4_stream(y + base + 4 * c, make_float4(v[k].x / s, v[k].y / s, v[k].z / s, v[k].w / s));
    }
  }
}

__global__ void __launch_bounds__(kRowThreads)
softmax_fwd_kernel(const float* __restrict__ x, float* __restrict__ y, int rows, int width) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const float* row = x + (size_t)r * width;
    float mx = -INFINITY;
    for (int i = lane; i < width; i += 32) mx = fmaxf(mx, row[i]);
    mx = wmax(mx);
    float s = 0.0f;
    for (int i = lane; i < width; i += 32) s += expf(row[i] - mx);
    s = wsum(s);
    for (int i = lane; i < width; i += 32) y[(size_t)r * width + i] = expf(row[i] - mx) / s;
  }
}

template <int VPL>
__global__ void __launch_bounds__(kRowThreads)
softmax_bwd_vec_kernel(const float* __restrict__ y, const float* __restrict__ g, float* dx, int rows, int width,
                       int accumulate) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  const int w4 = width >> 2;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const size_t base = (size_t)r * width;
    float4 yv[VPL], gv[VPL];
    float dot = 0.0f;
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < w4) {
        yv[k] = ld4_stream(y + base + 4 * c);
        gv[k] = ld4_stream(g + base + 4 * c);
        dot += (yv[k].x * gv[k].x + yv[k].y * gv[k].y) + (yv[k].z * gv[k].z + yv[k].w * gv[k].w);
      }
    }
    dot = wsum(dot);
#pragma unroll
    for (int k = 0; k < VPL; ++k) {
      const int c = lane + 32 * k;
      if (c < w4) {
        float4 o = make_float4(yv[k].x * (gv[k].x - dot), yv[k].y * (gv[k].y - dot), yv[k].z * (gv[k].z - dot),
                               yv[k].w * (gv[k].w - dot));
        if (accumulate) { const float4 old = ld4(dx + base + 4 * c); o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w; }
        st4(dx + base + 4 * c, o);
      }
    }
  }
}

__global__ void __launch_bounds__(kRowThreads)
softmax_bwd_kernel(const float* __restrict__ y, const float* __restrict__ g, float* dx, int rows, int width,
                   int accumulate) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
  for (int r = blockIdx.x * wpb + (threadIdx.x >> 5); r < rows; r += gridDim.x * wpb) {
    const size_t st = (size_t)r * width;
    float dot = 0.0f;
    for (int i = lane; i < width; i += 32) dot += y[st + i] * g[st + i];
    dot = wsum(dot);
    for (int i = lane; i < width; i += 32) {
      const float v = y[st + i] * (g[st + i] - dot);
      dx[st + i] = accumulate ? dx[st + i] + v : v;
    }
  }
}

int row_grid(const nrs_ctx* ctx, int rows, int warps_per_block = 8) {
  int blocks = (rows + warps_per_block - 1) / warps_per_block;
  if (blocks > ctx->sm_count * 8) blocks = ctx->sm_count * 8;
  return blocks < 1 ? 1 : blocks;
}

// float4s per lane for a row of `width` floats, or 0 when the vector path does not apply.
int vec_vpl(int width, std::initializer_list<const void*> ptrs) {
  if (width % 4 != 0 || width > 32 * 4 * kMaxVpl) return 0;
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15) return 0;
  const int f4 = width / 4;
  return f4 <= 32 ? 1 : f4 <= 64 ? 2 : f4 <= 128 ? 4 : 8;
}

#define NRS_DISPATCH_VPL(vpl, CALL) \
  do {                              \
    switch (vpl) {                  \
      case 1: { constexpr int V = 1; CALL; } break; \
      case 2: { constexpr int V = 2; CALL; } break; \
      case 4: { constexpr int V = 4; CALL; } break; \
      default: { constexpr int V = 8; CALL; } break; \
    }                               \
  } while (0)

int layernorm_fwd(nrs_ctx* ctx, const char* who, const float* a, const float* b, const float* gamma, const float* beta,
                  float* y, float* xhat, float* istd, int rows, int f, float eps, float* y_hi = nullptr, float* y_lo = nullptr,
                  int* emitted = nullptr, NrsRange* istd_range = nullptr) {
  if (emitted) *emitted = 0;
  NRS_REQUIRE(ctx, rows >= 0 && f > 0, NRS_ERR_SHAPE, "%s: bad shape [%d,%d]", who, rows, f);
  if (rows == 0) return NRS_OK;
  NRS_REQUIRE(ctx, a && gamma && beta && y, NRS_ERR_ARG, "%s: null tensor", who);
  const int vpl = vec_vpl(f, {a, b, gamma, beta, y, xhat, y_hi, y_lo});
  // Where the row pipeline is the better kernel (us here -> there, tensors that are not in L2).  Float4 rows without a
  // residual: 16 M elements of 384 columns 40 -> 39, 448 43 -> 36, 512 40 -> 38, 896 42 -> 39, 1000 42 -> 36; not 256 (39,
  // 51) or 768 (40, 45; a quarter of the lanes idle).  With a residual (two inputs, two outputs) 8 M of 448 28 -> 26, 896 29
  // -> 26; not 256 (25, 30), and not far beyond L2 (40 M of 1000 114, 124), although up to there the register kernel's
  // stores, which pass the cache by, cost the operator that reads y next 4 us of 16 M elements.  Scalar loops: 1502 columns
  // 62 -> 51, 3000 76 -> 43, not 1401 (83, 112; 2.7 live warps); with a residual 1001 100 -> 82, 3000 128 -> 49, not 1281
  // (98, 130).  Tensors that still lie in L2 suit the other kernels (8 M elements: 384 columns 19, 22; 2050 27, 33): lines
  // that are close wait for 12 M.
  const size_t elems = (size_t)rows * f;
  const double fill = rowpipe::fill(f), live = rowpipe::live_warps(f, 2);
  const bool beyond_l2 = elems >= (size_t)12 << 20, full_warp = f >= 448 && f <= 512;
  bool pipe;
  if (vpl && b) pipe = f >= 832 ? elems < (size_t)24 << 20 : full_warp && !beyond_l2;
  else if (vpl) pipe = full_warp || f >= 928 || (beyond_l2 && (f >= 832 || (f >= 384 && f <= 512)));
  else pipe = fill >= 0.75 && (b ? f >= 960 && live >= 3.8 : f >= 1400 && live >= 5.0 && (beyond_l2 || fill >= 0.85));
  pipe = pipe && elems >= 6000000;
  if (!(y_hi && vpl) && pipe && rowpipe::applies(rows, f, {a, b, gamma, beta, y, xhat})) {
    rowpipe::Params p{};
    p.in[0] = a; p.in[1] = b; p.n_in = b ? 2 : 1; p.n_buf = 2;
    p.out[0] = xhat; p.out_buf[0] = 0;
    p.out[1] = y; p.out_buf[1] = 1;
    p.rows = rows; p.f = f;
    const int st = rowpipe::launch(ctx, p, LnFwdOp{gamma, beta, istd, eps, b != nullptr});
    if (st != NRS_ERR_UNSUPPORTED) return st;
  }
  if (vpl) {
    NrsRange* range = nullptr;
    if (y_hi && y_lo) {
      const int st = nrs_range_renew(ctx, y_hi, &range);
      if (st != NRS_OK) return st;
    }
    if (y_hi)
      NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH((ln_fwd_vec_kernel<V, true>), row_grid(ctx, rows), kRowThreads, 0, ctx->stream, a, b, gamma,
                                           beta, y, xhat, istd, rows, f, eps, y_hi, y_lo, range, istd_range));
    else
      NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH((ln_fwd_vec_kernel<V, false>), row_grid(ctx, rows), kRowThreads, 0, ctx->stream, a, b, gamma,
                                           beta, y, xhat, istd, rows, f, eps, y_hi, y_lo, range, istd_range));
    if (emitted && y_hi) *emitted = 1;
  } else {
    NRS_PDL_LAUNCH(ln_fwd_kernel, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, a, b, gamma, beta, y, xhat, istd, rows, f, eps);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

// partial[part][2][f] -> dgamma, dbeta.
int fold_params(nrs_ctx* ctx, const float* partial, float* dgamma, float* dbeta, int f, int parts, int accumulate) {
  return nrs_fold_column_pair(ctx, partial, dgamma, dbeta, parts, f, 2 * f, accumulate);
}

int layernorm_bwd(nrs_ctx* ctx, const char* who, const float* g, const float* xhat, const float* istd, const float* gamma,
                  float* dx, float* dx2, float* dgamma, float* dbeta, int rows, int f, int acc1, int acc2, int accumulate_params,
                  float* d_hi = nullptr, float* d_lo = nullptr, int* emitted = nullptr, const NrsRange* range_g = nullptr,
                  const NrsRange* range_istd = nullptr, float* sums = nullptr, int* sums_rows = nullptr) {
  if (emitted) *emitted = 0;
  if (sums_rows) *sums_rows = 0;
  NRS_REQUIRE(ctx, rows >= 0 && f > 0, NRS_ERR_SHAPE, "%s: bad shape [%d,%d]", who, rows, f);
  NRS_REQUIRE(ctx, (dgamma == nullptr) == (dbeta == nullptr), NRS_ERR_ARG, "%s: dgamma and dbeta must be given together", who);
  NRS_REQUIRE(ctx, dx || !dx2, NRS_ERR_ARG, "%s: a second input gradient without the first", who);
  if (rows == 0) {
    if (dgamma && !accumulate_params) {
      NRS_CUDA(ctx, cudaMemsetAsync(dgamma, 0, sizeof(float) * f, ctx->stream));
      NRS_CUDA(ctx, cudaMemsetAsync(dbeta, 0, sizeof(float) * f, ctx->stream));
    }
    return NRS_OK;
  }
  NRS_REQUIRE(ctx, g && xhat && istd && gamma, NRS_ERR_ARG, "%s: null tensor", who);
  if (!dx && !dgamma) return NRS_OK;
  const int vpl = vec_vpl(f, {g, xhat, gamma, dx, dx2, d_hi, d_lo});
  // Where the row pipeline is the better kernel (us here -> there, tensors that are not in L2).  Float4 rows: beyond 256
  // columns, from 4 M elements up (8 M below 280 columns).  dx and parameters of 16 M elements: 260 columns 71 -> 68, 320
  // 69 -> 58, 512 59 -> 42, 768 98 -> 46, 1000 104 -> 41; but 64 columns 76, 87, 128 48, 67, 256 44, 56 (dx alone 38, 52;
  // parameters alone 30, 36).
  // Scalar loops, which read g and xhat twice.  dx and parameters: from 256 K elements (17 columns 9.8 -> 9.2, 1001 14 ->
  // 12; 128 K of 385: 8.8, 11.0), with 60 to 256 columns (128 K of 127 9.5 -> 8.1) or 1024 and more (128 K of 1401 15.5 ->
  // 11.6) always.  Parameters alone, one read of each: from 12 M (16 M of 1001 columns 64 -> 32), where rows are neither
  // very short nor very long from 8 M (1001: 34 -> 20; 17 62 -> 57, 6000 29 -> 24), up to 256 columns from 4 M (250: 21 ->
  // 14); 1 M of 1001 8.5, 10.9.  dx alone: any width of 961 columns and more (4 M of 1028 20 -> 15), narrower ones with
  // few lanes idle (4 M of 450 16 -> 15) or beyond L2 (16 M of 33 164 -> 134, 301 61 -> 51) or for few rows (512 K of 705
  // 7.2 -> 5.2); not 16 M of 777 (58, 70; 3.1 live warps) or 1281 (64, 83; 2.5).  Tensors that still lie in L2 suit the
  // loops, which is why lines that are close wait for more elements: dx and parameters of 4 M of 1281 22, 31, parameters of
  // 8 M of 17 27, 56, dx of 4 M of 385 14, 18.
  const size_t elems = (size_t)rows * f, m = (size_t)1 << 20;
  const double fill = rowpipe::fill(f), live = rowpipe::live_warps(f, 2);
  const bool beyond_l2 = elems >= 12 * m, large = elems >= 8 * m, small = elems < 3 * m, few = elems < 3 * m / 2;
  bool pipe;
  if (vpl) pipe = f > 256 && elems >= (f < 280 ? 8 : 4) * m;
  else if (dx && dgamma) pipe = (f >= 1024 || elems >= m / 4 || (f >= 60 && f <= 256)) && (live >= 3.0 || f <= 256 || large || small);
  else if (dgamma) pipe = beyond_l2 || (large && f >= 24 && f <= 3000 && (live >= 3.0 || f <= 256)) ||
                          (elems >= 4 * m && f >= 100 && f <= 256);
  else if (f > 960) pipe = live >= 3.0 || small;
  else pipe = (fill >= 0.85 && (live >= 3.9 || small || beyond_l2)) || (live >= 7.0 && f > 512 && (fill >= 0.75 || small)) ||
              (beyond_l2 && (f <= 512 || live >= 4.3)) || (large && f <= 40) || (few && f > 256 && fill >= 0.55 && elems >= m / 4);
  if (!(d_hi && vpl) && pipe && rowpipe::applies(rows, f, {g, xhat, gamma, dx, dx2})) {
    rowpipe::Params p{};
    p.in[0] = g; p.in[1] = xhat; p.n_in = p.n_buf = 2;
    p.out[0] = dx; p.out_add[0] = acc1;
    p.out[1] = dx2; p.out_add[1] = acc2;
    p.rows = rows; p.f = f;
    float* partial = nullptr;
    if (dgamma) {
      const int st = nrs_fold_partial(ctx, -1, (size_t)ctx->sm_count * 2 * f * sizeof(float), &partial);
      if (st != NRS_OK) return st;
    }
    int blocks = 0;
    const int st = rowpipe::launch(ctx, p, LnBwdOp{istd, gamma, partial, dx != nullptr}, &blocks);
    if (st != NRS_ERR_UNSUPPORTED) {
      if (st != NRS_OK || !dgamma) return st;
      return fold_params(ctx, partial, dgamma, dbeta, f, blocks, accumulate_params);
    }
  }
  if (vpl) {
    // one pass over g and xhat for everything; the block size keeps the per-warp column partials within 32 KB
    if (!(dx && d_hi && dgamma)) sums = nullptr;
    int warps = 8;
    while (dgamma && warps > 1 && (size_t)warps * 2 * f * sizeof(float) > 32 * 1024) warps >>= 1;
    int blocks = row_grid(ctx, rows, warps);
    if (dgamma && blocks > 4 * ctx->sm_count) blocks = 4 * ctx->sm_count;   // one resident wave of longer-lived blocks: fewer partial rows to fold
    float* partial = nullptr;
    if (dgamma) {
      const int st = nrs_fold_partial(ctx, -1, (size_t)blocks * 2 * f * sizeof(float), &partial);
      if (st != NRS_OK) return st;
    }
    const size_t smem = dgamma ? (size_t)warps * 2 * f * sizeof(float) : 0;
    NrsRange* range = nullptr;
    if (dx && d_hi && d_lo) {
      int st = nrs_range_renew(ctx, d_hi, &range);
      NrsRange *mg = nullptr, *mi = nullptr;
      if (!range_g && st == NRS_OK) st = nrs_range_renew(ctx, &ctx->scratch_range[0], &mg);
      if (!range_istd && st == NRS_OK) st = nrs_range_renew(ctx, &ctx->scratch_range[1], &mi);
      if (st == NRS_OK && mg) st = nrs_absmax(ctx, g, elems, mg);
      if (st == NRS_OK && mi) st = nrs_absmax(ctx, istd, (size_t)rows, mi);
      if (st != NRS_OK) return st;
      if (mg) range_g = mg;
      if (mi) range_istd = mi;
    }
    if (dx && d_hi)
      NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH((ln_bwd_vec_kernel<V, true>), blocks, warps * 32, smem, ctx->stream, g, xhat, istd, gamma, dx,
                                           dx2, partial, rows, f, acc1, acc2, d_hi, d_lo, sums, range_g, range_istd, range));
    else
      NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH((ln_bwd_vec_kernel<V, false>), blocks, warps * 32, smem, ctx->stream, g, xhat, istd, gamma, dx,
                                           dx2, partial, rows, f, acc1, acc2, (float*)nullptr, (float*)nullptr, (float*)nullptr, (const NrsRange*)nullptr,
                                           (const NrsRange*)nullptr, (NrsRange*)nullptr));
    if (emitted && dx && d_hi) *emitted = 1;
    if (sums) *sums_rows = blocks;
    NRS_LAUNCHED(ctx);
    return dgamma ? fold_params(ctx, partial, dgamma, dbeta, f, blocks, accumulate_params) : NRS_OK;
  }
  if (dx) {
    NRS_PDL_LAUNCH(ln_dx_kernel, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, g, xhat, istd, gamma, dx, dx2, rows, f, acc1, acc2);
    NRS_LAUNCHED(ctx);
  }
  if (dgamma) {
    const int col_blocks = (f + 31) / 32;
    int splits = (2 * ctx->sm_count + col_blocks - 1) / col_blocks;
    if (splits > rows / 32) splits = rows / 32;
    if (splits < 1) splits = 1;
    if (splits > 65535) splits = 65535;
    float* ws = nullptr;
    const int st = nrs_fold_partial(ctx, -1, (size_t)splits * 2 * f * sizeof(float), &ws);
    if (st != NRS_OK) return st;
    NRS_PDL_LAUNCH(ln_param_kernel, dim3(col_blocks, splits), 256, 0, ctx->stream, g, xhat, ws, rows, f, splits);
    NRS_LAUNCHED(ctx);
    return fold_params(ctx, ws, dgamma, dbeta, f, splits, accumulate_params);
  }
  return NRS_OK;
}

}  // namespace

extern "C" {

int nrs_layernorm_fwd(nrs_ctx* ctx, const float* x, const float* gamma, const float* beta, float* y,
                      float* xhat, float* istd, int rows, int f, float eps) {
  NRS_REQUIRE_CTX(ctx);
  return layernorm_fwd(ctx, "nrs_layernorm_fwd", x, nullptr, gamma, beta, y, xhat, istd, rows, f, eps);
}

int nrs_layernorm_residual_fwd(nrs_ctx* ctx, const float* a, const float* b, const float* gamma, const float* beta, float* y,
                               float* xhat, float* istd, int rows, int f, float eps) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, b != nullptr || rows == 0, NRS_ERR_ARG, "nrs_layernorm_residual_fwd: null second addend");
  return layernorm_fwd(ctx, "nrs_layernorm_residual_fwd", a, b, gamma, beta, y, xhat, istd, rows, f, eps);
}

int nrs_layernorm_bwd(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma,
                      float* dx, float* dgamma, float* dbeta, int rows, int f, int accumulate_dx,
                      int accumulate_params) {
  NRS_REQUIRE_CTX(ctx);
  return layernorm_bwd(ctx, "nrs_layernorm_bwd", g, xhat, istd, gamma, dx, nullptr, dgamma, dbeta, rows, f, accumulate_dx, 0,
                       accumulate_params);
}

int nrs_layernorm_residual_bwd(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma,
                               float* da, float* db, float* dgamma, float* dbeta, int rows, int f, int accumulate_da,
                               int accumulate_db, int accumulate_params) {
  NRS_REQUIRE_CTX(ctx);
  // the gradient of a + b is the same for both addends; either may be absent
  float* first = da ? da : db;
  float* second = da ? db : nullptr;
  const int acc_first = da ? accumulate_da : accumulate_db;
  return layernorm_bwd(ctx, "nrs_layernorm_residual_bwd", g, xhat, istd, gamma, first, second, dgamma, dbeta, rows, f, acc_first,
                       accumulate_db, accumulate_params);
}

// The same two operators with the operand planes of their result written by the kernel itself (y forward; the
// input gradient backward): *emitted = 1 when the planes were written (vector path), 0 when the caller has
// to stage them itself.  Internal: the graph's fused transformer block calls them.
int nrs_layernorm_fwd_planes(nrs_ctx* ctx, const float* a, const float* b, const float* gamma, const float* beta, float* y,
                             float* xhat, float* istd, int rows, int f, float eps, float* y_hi, float* y_lo, int* emitted,
                             NrsRange* istd_range) {
  NRS_REQUIRE_CTX(ctx);
  return layernorm_fwd(ctx, "nrs_layernorm_fwd_planes", a, b, gamma, beta, y, xhat, istd, rows, f, eps, y_hi, y_lo, emitted, istd_range);
}

int nrs_layernorm_bwd_planes(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma, float* da,
                             float* db, float* dgamma, float* dbeta, int rows, int f, int accumulate_da, int accumulate_db,
                             int accumulate_params, float* d_hi, float* d_lo, int* emitted, const NrsRange* range_g,
                             const NrsRange* range_istd, float* sums, int* sums_rows) {
  NRS_REQUIRE_CTX(ctx);
  float* first = da ? da : db;
  float* second = da ? db : nullptr;
  const int acc_first = da ? accumulate_da : accumulate_db;
  return layernorm_bwd(ctx, "nrs_layernorm_bwd_planes", g, xhat, istd, gamma, first, second, dgamma, dbeta, rows, f, acc_first,
                       accumulate_db, accumulate_params, d_hi, d_lo, emitted, range_g, range_istd, sums, sums_rows);
}

int nrs_softmax_fwd(nrs_ctx* ctx, const float* x, float* y, int rows, int width) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, rows >= 0 && width > 0, NRS_ERR_SHAPE, "nrs_softmax_fwd: bad shape [%d,%d]", rows, width);
  if (rows == 0) return NRS_OK;
  NRS_REQUIRE(ctx, x && y, NRS_ERR_ARG, "nrs_softmax_fwd: null tensor");
  const int vpl = vec_vpl(width, {x, y});
  // (widths the vector kernel takes stay there at every size: bound by its exponentials and divisions, not by HBM, it
  // does better with a full SM of warps: [16384][1000] 23 us against 54)
  // Against the scalar loops, with hardly a lane idle and enough columns at work (us there -> here): 8 M elements of 1502
  // columns 34 -> 26, 3000 39 -> 35; 16 M of 4096 91 -> 46.  Not 1401 (34, 48), 2050 (30, 48; a fifth of the lanes idle)
  // or 2001 (30, 40; 7.8 live warps), and up to 3400 columns not beyond 24 M elements (40 M of 2000: 118, 128).
  const size_t elems = (size_t)rows * width;
  const double live = rowpipe::live_warps(width, 1);
  const bool pipe = !vpl && width >= 1400 && elems >= 6000000 && rowpipe::fill(width) >= 0.95 &&
                    ((width >= 3400 && live >= 13.0) || (elems <= (size_t)24 << 20 && live >= 9.5));
  if (pipe && rowpipe::applies(rows, width, {x, y})) {
    rowpipe::Params p{};
    p.in[0] = x; p.n_in = p.n_buf = 1;
    p.out[0] = y;
    p.rows = rows; p.f = width;
    const int st = rowpipe::launch(ctx, p, SoftmaxFwdOp{});
    if (st != NRS_ERR_UNSUPPORTED) return st;
  }
  if (vpl) {
    NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH(softmax_fwd_vec_kernel<V>, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, x, y, rows, width));
  } else {
    NRS_PDL_LAUNCH(softmax_fwd_kernel, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, x, y, rows, width);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_softmax_bwd(nrs_ctx* ctx, const float* y, const float* g, float* dx, int rows, int width, int accumulate) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, rows >= 0 && width > 0, NRS_ERR_SHAPE, "nrs_softmax_bwd: bad shape [%d,%d]", rows, width);
  if (rows == 0) return NRS_OK;
  NRS_REQUIRE(ctx, y && g && dx, NRS_ERR_ARG, "nrs_softmax_bwd: null tensor");
  const int vpl = vec_vpl(width, {y, g, dx});
  // Only against the scalar loops ([16384][1001] 61 us, 37 here; 1 M elements of 50 columns, most lanes idle, 6.2, 8.2):
  // the register kernel takes 32 us for [16384][1000], and is the better one at every float4 width.
  if (!vpl && rowpipe::fill(width) >= 0.75 && rowpipe::applies(rows, width, {y, g, dx})) {
    rowpipe::Params p{};
    p.in[0] = y; p.in[1] = g; p.n_in = p.n_buf = 2;
    p.out[0] = dx; p.out_add[0] = accumulate;
    p.rows = rows; p.f = width;
    const int st = rowpipe::launch(ctx, p, SoftmaxBwdOp{});
    if (st != NRS_ERR_UNSUPPORTED) return st;
  }
  if (vpl) {
    NRS_DISPATCH_VPL(vpl, NRS_PDL_LAUNCH(softmax_bwd_vec_kernel<V>, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, y, g, dx, rows,
                                         width, accumulate));
  } else {
    NRS_PDL_LAUNCH(softmax_bwd_kernel, row_grid(ctx, rows), kRowThreads, 0, ctx->stream, y, g, dx, rows, width, accumulate);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

}  // extern "C"
