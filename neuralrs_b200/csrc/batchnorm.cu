// Batch normalisation over [n, c, hw] (hw == 1 is the [batch, features] layer), forward and backward.
// Reference: bn2d_stats / bn2d_normalize / bn2d_reduce / bn2d_dx (src/cuda/nn/batchnorm2d.rs:22-128) and their
// 2-D twins bn_stats / bn_normalize / bn_reduce / bn_dx (src/cuda/nn/batchnorm.rs:20-108); CPU semantics
// src/nn/batchnorm2d.rs:28-164, src/nn/batchnorm.rs:28-150.
//
// The reference walks a channel with one thread (two serial passes for the statistics).  Here every
// per-channel reduction is a pair of sums spread over (channel, sample-split) blocks and folded in a fixed
// order, so results are bit-reproducible and the pass runs at HBM speed:
//   forward   S = sum(x - K), Q = sum((x - K)^2) with the pivot K = the channel's first element, which keeps
//             Q/N - (S/N)^2 free of the cancellation a raw sum of squares has when |mean| >> std;
//   backward  S = sum(g) = dbeta, Q = sum(g * xhat) = dgamma.
// x is read twice in the forward pass (statistics, normalise) and g / xhat twice in the backward pass.  The graph keeps
// no xhat: it saves the means, and the backward kernels take x and recompute (x - mean) * istd, the forward pass's very
// expression (4 B per element less written).  Where a tensor-core convolution reads the output, or made the input, the
// normalise and dx kernels also write the NHWC planes that it wants, and the dx kernel the per-tile channel sums that
// the convolution's bias gradient folds.  Measured (256 images of 64 x 32 x 32, TF32): staging and channel sums as
// passes of their own took 27 and 26 us a tensor.
#include "image_tile.cuh"
#include "nrs_internal.h"

namespace {

constexpr int kThreads = 256;

__host__ __device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

__device__ __forceinline__ float wsum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The two values an element contributes.  FWD: a = x, b unused, k = pivot.  BWD: a = g, b = xhat.
template <bool FWD>
__device__ __forceinline__ void contribute(float a, float b, float k, float& s, float& q) {
  if (FWD) {
    const float d = a - k;
    s += d;
    q += d * d;
  } else {
    s += a;
    q += a * b;
  }
}

// 3xTF32, where the planes of the result are written: their exponent comes from a bound of it, which is made of what the
// reduction ahead of it meets in its own reading of the tensors (a bound from the count, |xhat| <= sqrt(count), is far
// looser, and does not hold where the variance is lost in the rounding of its sums: a channel that is constant but for its
// first value).  extremes[split][ch] = forward (largest |x - k|, 0), backward (largest |g|, largest |xhat|); of finite values.
struct BnBound {
  NrsRange* out;         // null: no planes, or the bound is not made here
  const NrsRange* x;     // evaluation, forward: the input's
  const float *gamma, *beta, *istd;
  int training;
};
// By any thread, once a channel.  (A channel whose statistics are not finite has no finite results to bound.)
__device__ __forceinline__ void take_bound(NrsRange* out, float b) {
  atomicMax(reinterpret_cast<unsigned*>(&out->bound), __float_as_uint(fminf(b * 1.001f, 3.0e38f)));
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) < __int_as_float(0x7f800000); }
__device__ __forceinline__ void bound_output(const BnBound& b, int ch, float far /*of x from k*/, float k, float mean, float istd) {
  if (!b.out || !finite(mean) || !finite(istd)) return;
  const float xhat = istd * (b.training ? far + fabsf(k - mean) : b.x->top + fabsf(mean));
  take_bound(b.out, fabsf(b.gamma[ch]) * xhat + fabsf(b.beta[ch]));
}
__device__ __forceinline__ void bound_dx(const BnBound& b, int ch, float g, float xhat, float s, float q, float count) {
  const float ga = fabsf(b.gamma[ch]), istd = b.istd[ch];
  const float means = b.training ? ga * fabsf(s) / count + xhat * (ga * fabsf(q) / count) : 0.0f;
  if (!b.out || !finite(istd) || !finite(s) || !finite(q)) return;
  take_bound(b.out, istd * (ga * g + means));
}

// What the folded sums of a channel become; done by the last block of the channel to arrive (an integer ticket; the
// splits are added in order whichever block that is), or by a kernel of its own where there are more channels than
// tickets, columns instead of planes, or sums to be shared across processes first.
struct BnFinish {
  unsigned* tickets;   // null: not here
  // forward: mean, biased variance, running statistics (running = momentum * running + (1 - momentum) * batch value,
  // batchnorm2d.rs:52-53), 1/sqrt(var + eps)
  float *mean, *istd, *running_mean, *running_var;
  float count, eps, momentum;
  // backward: sums[ch] = (dbeta, dgamma) of this call feeds the dx kernel, and the parameter gradients receive them (+)=
  float2* sums;
  float *dgamma, *dbeta;
  int accumulate;
  BnBound bound;
};
__device__ __forceinline__ void finish_stats(int ch, float s, float q, float k, float count, float eps, float momentum, float* mean,
                                             float* istd, float* running_mean, float* running_var, const BnBound& bound, float far) {
  const float d = s / count;
  const float m = k + d;
  const float v = fmaxf(q / count - d * d, 0.0f);
  running_mean[ch] = momentum * running_mean[ch] + (1.0f - momentum) * m;
  running_var[ch] = momentum * running_var[ch] + (1.0f - momentum) * v;
  mean[ch] = m;
  const float is = 1.0f / sqrtf(v + eps);
  istd[ch] = is;
  bound_output(bound, ch, far, k, m, is);
}
__device__ __forceinline__ void finish_grads(int ch, float s, float q, float2* sums, float* dgamma, float* dbeta, int accumulate) {
  sums[ch] = make_float2(s, q);
  if (dgamma) dgamma[ch] = accumulate ? dgamma[ch] + q : q;
  if (dbeta) dbeta[ch] = accumulate ? dbeta[ch] + s : s;
}

// Planes layout (hw >= 2): one block per (channel, sample split), 128-bit loads when the plane allows.
// partial[split][ch] = (S, Q).  MEASURE: extremes too (see BnBound).
// RELU (backward only): the layer's output went through a ReLU fused into the normalise pass; the incoming
// gradient is masked where that output was not positive, the output being recomputed from xhat with the very
// expression of the forward pass (fmaf(gamma, xhat, beta)), so the mask is the forward one bit for bit.
template <bool FWD, bool RELU, bool MEASURE>
__global__ void __launch_bounds__(kThreads)
bn_pair_planes_kernel(const float* __restrict__ a, const float* __restrict__ b, float2* __restrict__ partial, float2* __restrict__ extremes,
                      int n, int c, int hw, int splits, const float* __restrict__ gamma, const float* __restrict__ beta,
                      const float* __restrict__ pivot, const float* __restrict__ mean, const float* __restrict__ istd, const BnFinish fin, const NrsFastDiv div_per, const int vec /*planes of whole float4s*/) {
  NRS_PDL_PROLOGUE();
  __shared__ float2 sm[kThreads / 32];
  [[maybe_unused]] __shared__ uint2 sm_top[kThreads / 32];
  [[maybe_unused]] uint32_t top_a = 0, top_b = 0;
  const int ch = blockIdx.x, split = blockIdx.y;
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  const int n_per = (n + splits - 1) / splits;
  const int n0 = split * n_per, n1 = min(n, n0 + n_per);
  const float k = FWD ? (pivot ? pivot[ch] : a[(size_t)ch * hw]) : 0.0f;
  const float ga = RELU ? gamma[ch] : 0.0f, be = RELU ? beta[ch] : 0.0f;
  const float mu = mean ? mean[ch] : 0.0f, is = mean ? istd[ch] : 1.0f;   // b is x; without them xhat itself
  // The block's threads walk the split's (image, element) pairs as one flat index, so that planes shorter
  // than a warp's reach (8x8, 4x4 feature maps) still keep every lane loading.
  float s = 0.0f, q = 0.0f, s1 = 0.0f, q1 = 0.0f;
  const int per = vec ? hw / 4 : hw;                       // items per plane
  const int items = max(n1 - n0, 0) * per;               // n * hw < 2^31 is checked on the host
  if (vec) {
    constexpr int kDeep = 4;   // float4s of each tensor under way per thread, in the last round too
    for (int j = threadIdx.x; j < items; j += kDeep * kThreads) {
      float4 fa[kDeep], fb[kDeep];
#pragma unroll
      for (int u = 0; u < kDeep; ++u) {
        const int at = j + u * kThreads;
        const int di = (int)div_per.div((uint32_t)at), i = at - di * per;
        const size_t base = ((size_t)(n0 + di) * c + ch) * hw;
        if (at < items) {
          fa[u] = reinterpret_cast<const float4*>(a + base)[i];
          if (!FWD) fb[u] = reinterpret_cast<const float4*>(b + base)[i];
        }
      }
#pragma unroll
      for (int u = 0; u < kDeep; ++u) {
        if (j + u * kThreads >= items) break;
        float4 va = fa[u], vb = make_float4(0.f, 0.f, 0.f, 0.f);
        if (!FWD) vb = make_float4((fb[u].x - mu) * is, (fb[u].y - mu) * is, (fb[u].z - mu) * is, (fb[u].w - mu) * is);
        if (RELU) {
          va.x = fmaf(ga, vb.x, be) > 0.0f ? va.x : 0.0f;
          va.y = fmaf(ga, vb.y, be) > 0.0f ? va.y : 0.0f;
          va.z = fmaf(ga, vb.z, be) > 0.0f ? va.z : 0.0f;
          va.w = fmaf(ga, vb.w, be) > 0.0f ? va.w : 0.0f;
        }
        contribute<FWD>(va.x, vb.x, k, s, q);
        contribute<FWD>(va.y, vb.y, k, s1, q1);
        contribute<FWD>(va.z, vb.z, k, s, q);
        contribute<FWD>(va.w, vb.w, k, s1, q1);
        if (MEASURE) {
          top_a = pr::seen4(top_a, FWD ? make_float4(va.x - k, va.y - k, va.z - k, va.w - k) : va);
          if (!FWD) top_b = pr::seen4(top_b, vb);
        }
      }
    }
  } else {
#pragma unroll 2
    for (int j = threadIdx.x; j < items; j += kThreads) {
      const int di = (int)div_per.div((uint32_t)j), i = j - di * per;
      const size_t base = ((size_t)(n0 + di) * c + ch) * hw;
      const float vb = FWD ? 0.0f : (b[base + i] - mu) * is;
      float va = a[base + i];
      if (RELU) va = fmaf(ga, vb, be) > 0.0f ? va : 0.0f;
      contribute<FWD>(va, vb, k, s, q);
      if (MEASURE) {
        top_a = pr::seen(top_a, FWD ? va - k : va);
        if (!FWD) top_b = pr::seen(top_b, vb);
      }
    }
  }
  s += s1;
  q += q1;
  s = wsum(s);
  q = wsum(q);
  if (lane == 0) sm[wrp] = make_float2(s, q);
  if (MEASURE) {
    top_a = __reduce_max_sync(0xffffffffu, top_a);
    top_b = __reduce_max_sync(0xffffffffu, top_b);
    if (lane == 0) sm_top[wrp] = make_uint2(top_a, top_b);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float2 t = sm[0];
#pragma unroll
    for (int i = 1; i < kThreads / 32; ++i) { t.x += sm[i].x; t.y += sm[i].y; }
    partial[(size_t)split * c + ch] = t;
    if (MEASURE) {
      for (int i = 1; i < kThreads / 32; ++i) { top_a = max(top_a, sm_top[i].x); top_b = max(top_b, sm_top[i].y); }
      extremes[(size_t)split * c + ch] = make_float2(__uint_as_float(top_a), __uint_as_float(top_b));
    }
    if (!fin.tickets) return;
    __threadfence();
    if (atomicAdd(&fin.tickets[ch], 1u) != (unsigned)splits - 1) return;
    __threadfence();
    fin.tickets[ch] = 0;
    float ts = 0.0f, tq = 0.0f;
#pragma unroll 4
    for (int z = 0; z < splits; ++z) {
      const float2 v = __ldcg(partial + (size_t)z * c + ch);
      ts += v.x;
      tq += v.y;
    }
    [[maybe_unused]] float2 ext = make_float2(0.0f, 0.0f);
    if (MEASURE) {
#pragma unroll 4
      for (int z = 0; z < splits; ++z) {
        const float2 v = __ldcg(extremes + (size_t)z * c + ch);
        ext = make_float2(fmaxf(ext.x, v.x), fmaxf(ext.y, v.y));
      }
    }
    if (FWD) {
      finish_stats(ch, ts, tq, k, fin.count, fin.eps, fin.momentum, fin.mean, fin.istd, fin.running_mean, fin.running_var, fin.bound, ext.x);
    } else {
      finish_grads(ch, ts, tq, fin.sums, fin.dgamma, fin.dbeta, fin.accumulate);
      if (MEASURE && fin.bound.out) bound_dx(fin.bound, ch, ext.x, ext.y, ts, tq, fin.count);
    }
  }
}
__device__ __forceinline__ float2 fold_extremes(const float2* __restrict__ extremes, int ch, int c, int splits) {
  float2 e = make_float2(0.0f, 0.0f);
  for (int z = 0; extremes && z < splits; ++z) {
    const float2 v = extremes[(size_t)z * c + ch];
    e = make_float2(fmaxf(e.x, v.x), fmaxf(e.y, v.y));
  }
  return e;
}

// Columns layout (hw == 1): a block owns 32 features and a slice of the rows; its 8 warps stride the rows
// reading 128-byte row segments.
template <bool FWD, bool RELU>
__global__ void __launch_bounds__(kThreads)
bn_pair_cols_kernel(const float* __restrict__ a, const float* __restrict__ b, float2* __restrict__ partial,
                    float2* __restrict__ extremes /*or null*/, int rows, int cols, int splits, const float* __restrict__ gamma, const float* __restrict__ beta,
                    const float* __restrict__ pivot, const float* __restrict__ mean, const float* __restrict__ istd) {
  NRS_PDL_PROLOGUE();
  __shared__ float2 sm[kThreads / 32][33];
  __shared__ uint2 sm_top[kThreads / 32][33];
  uint32_t top_a = 0, top_b = 0;
  const int lane = threadIdx.x & 31, wrp = threadIdx.x >> 5;
  const int col = blockIdx.x * 32 + lane, split = blockIdx.y;
  const int rows_per = (rows + splits - 1) / splits;
  const int r0 = split * rows_per, r1 = min(rows, r0 + rows_per);
  float s = 0.0f, q = 0.0f;
  if (col < cols) {
    const float k = FWD ? (pivot ? pivot[col] : a[col]) : 0.0f;
    const float ga = RELU ? gamma[col] : 0.0f, be = RELU ? beta[col] : 0.0f;
    const float mu = mean ? mean[col] : 0.0f, is = mean ? istd[col] : 1.0f;
    for (int r = r0 + wrp; r < r1; r += kThreads / 32) {
      const size_t i = (size_t)r * cols + col;
      const float vb = FWD ? 0.0f : (b[i] - mu) * is;
      float va = a[i];
      if (RELU) va = fmaf(ga, vb, be) > 0.0f ? va : 0.0f;
      contribute<FWD>(va, vb, k, s, q);
      if (extremes) {
        top_a = pr::seen(top_a, FWD ? va - k : va);
        if (!FWD) top_b = pr::seen(top_b, vb);
      }
    }
  }
  sm[wrp][lane] = make_float2(s, q);
  sm_top[wrp][lane] = make_uint2(top_a, top_b);
  __syncthreads();
  if (wrp == 0 && col < cols) {
    float2 t = sm[0][lane];
#pragma unroll
    for (int i = 1; i < kThreads / 32; ++i) { t.x += sm[i][lane].x; t.y += sm[i][lane].y; }
    partial[(size_t)split * cols + col] = t;
    if (extremes) {
      for (int i = 1; i < kThreads / 32; ++i) { top_a = max(top_a, sm_top[i][lane].x); top_b = max(top_b, sm_top[i][lane].y); }
      extremes[(size_t)split * cols + col] = make_float2(__uint_as_float(top_a), __uint_as_float(top_b));
    }
  }
}

// One thread per channel folds the splits in order and finishes the statistics: mean, biased variance,
// running statistics (running = momentum * running + (1 - momentum) * batch value, batchnorm2d.rs:52-53),
// 1/sqrt(var + eps).  In evaluation mode the running statistics are used as they are (batchnorm2d.rs:57-60).
// `pivot` / `count_dev` (both or neither): the sums were taken around pivot[ch] (the running mean, read here
// before it is updated) over *count_dev elements — statistics summed over several processes.
__global__ void bn_stats_finish_kernel(const float2* __restrict__ partial, const float* __restrict__ x, float* mean,
                                       float* istd, float* running_mean, float* running_var, int c, int hw,
                                       int splits, float count, float eps, float momentum, int training,
                                       const float* __restrict__ pivot, const float* __restrict__ count_dev,
                                       const float2* __restrict__ extremes, int extreme_splits, const BnBound bound) {
  NRS_PDL_PROLOGUE();
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= c) return;
  if (!training) {
    const float m = running_mean[ch], is = 1.0f / sqrtf(running_var[ch] + eps);
    mean[ch] = m;
    istd[ch] = is;
    bound_output(bound, ch, 0.0f, 0.0f, m, is);
    return;
  }
  float s = 0.0f, q = 0.0f;
  for (int z = 0; z < splits; ++z) {
    const float2 t = partial[(size_t)z * c + ch];
    s += t.x;
    q += t.y;
  }
  const float k = pivot ? pivot[ch] : x[(size_t)ch * hw];
  if (count_dev) count = *count_dev;
  finish_stats(ch, s, q, k, count, eps, momentum, mean, istd, running_mean, running_var, bound, fold_extremes(extremes, ch, c, extreme_splits).x);
}

// Folds the backward sums; sums[ch] = (dbeta, dgamma) of this call feeds the dx kernel, and the parameter
// gradients receive them (+)=.
__global__ void bn_grad_finish_kernel(const float2* __restrict__ partial, float2* __restrict__ sums, float* dgamma,
                                      float* dbeta, int c, int splits, int accumulate, const float2* __restrict__ extremes,
                                      float count, const BnBound bound) {
  NRS_PDL_PROLOGUE();
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= c) return;
  float s = 0.0f, q = 0.0f;
  for (int z = 0; z < splits; ++z) {
    const float2 t = partial[(size_t)z * c + ch];
    s += t.x;
    q += t.y;
  }
  finish_grads(ch, s, q, sums, dgamma, dbeta, accumulate);
  if (!bound.out) return;
  const float2 e = fold_extremes(extremes, ch, c, splits);
  bound_dx(bound, ch, e.x, e.y, s, q, count);
}

// y = gamma * xhat + beta, xhat = (x - mean) * istd (bn2d_normalize, batchnorm2d.rs:62-75).
template <bool VEC, bool RELU>
__global__ void __launch_bounds__(kThreads)
bn_normalize_kernel(const float* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ istd,
                    const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ y,
                    float* __restrict__ xhat, size_t total, int c, int hw) {
  NRS_PDL_PROLOGUE();
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC) {   // hw % 4 == 0: the four elements of a vector share their channel
    for (size_t i = tid; i < total / 4; i += stride) {
      const int ch = (int)((i * 4 / hw) % c);
      const float m = mean[ch], is = istd[ch], ga = gamma[ch], be = beta[ch];
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      const float4 h = make_float4((v.x - m) * is, (v.y - m) * is, (v.z - m) * is, (v.w - m) * is);
      if (xhat) reinterpret_cast<float4*>(xhat)[i] = h;
      float4 o = make_float4(fmaf(ga, h.x, be), fmaf(ga, h.y, be), fmaf(ga, h.z, be), fmaf(ga, h.w, be));
      if (RELU) o = make_float4(fmaxf(o.x, 0.0f), fmaxf(o.y, 0.0f), fmaxf(o.z, 0.0f), fmaxf(o.w, 0.0f));
      reinterpret_cast<float4*>(y)[i] = o;
    }
  } else {
    for (size_t i = tid; i < total; i += stride) {
      const int ch = (int)((i / hw) % c);
      const float h = (x[i] - mean[ch]) * istd[ch];
      if (xhat) xhat[i] = h;
      const float o = fmaf(gamma[ch], h, beta[ch]);
      y[i] = RELU ? fmaxf(o, 0.0f) : o;
    }
  }
}

// bn2d_dx (batchnorm2d.rs:96-117): training dx = istd * (g*gamma - gamma*dbeta/N - xhat*gamma*dgamma/N);
// evaluation dx = g * gamma * istd.
template <bool VEC, bool RELU>
__global__ void __launch_bounds__(kThreads)
bn_dx_kernel(const float* __restrict__ g, const float* __restrict__ xhat, const float* __restrict__ istd,
             const float* __restrict__ gamma, const float* __restrict__ beta, const float2* __restrict__ sums, float* dx,
             size_t total, int c, int hw, float count, int training, int accumulate, const float* __restrict__ count_dev,
             const float* __restrict__ mean /* null: xhat is xhat; else it is x */) {
  NRS_PDL_PROLOGUE();
  if (count_dev) count = *count_dev;   // elements per channel over all processes
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (VEC) {
    for (size_t i = tid; i < total / 4; i += stride) {
      const int ch = (int)((i * 4 / hw) % c);
      const float ga = gamma[ch], is = istd[ch];
      float4 vg = reinterpret_cast<const float4*>(g)[i];
      float4 vh = make_float4(0.f, 0.f, 0.f, 0.f);
      if (training || RELU) vh = reinterpret_cast<const float4*>(xhat)[i];
      if (mean) {
        const float mu = mean[ch];
        vh = make_float4((vh.x - mu) * is, (vh.y - mu) * is, (vh.z - mu) * is, (vh.w - mu) * is);
      }
      if (RELU) {
        const float be = beta[ch];
        vg.x = fmaf(ga, vh.x, be) > 0.0f ? vg.x : 0.0f;
        vg.y = fmaf(ga, vh.y, be) > 0.0f ? vg.y : 0.0f;
        vg.z = fmaf(ga, vh.z, be) > 0.0f ? vg.z : 0.0f;
        vg.w = fmaf(ga, vh.w, be) > 0.0f ? vg.w : 0.0f;
      }
      float4 r;
      if (training) {
        const float2 sm = sums[ch];
        const float m1 = ga * sm.x / count, m2 = ga * sm.y / count;
        r = make_float4(is * (vg.x * ga - m1 - vh.x * m2), is * (vg.y * ga - m1 - vh.y * m2),
                        is * (vg.z * ga - m1 - vh.z * m2), is * (vg.w * ga - m1 - vh.w * m2));
      } else {
        r = make_float4(vg.x * ga * is, vg.y * ga * is, vg.z * ga * is, vg.w * ga * is);
      }
      float4* dst = reinterpret_cast<float4*>(dx) + i;
      if (accumulate) {
        const float4 o = *dst;
        r = make_float4(o.x + r.x, o.y + r.y, o.z + r.z, o.w + r.w);
      }
      *dst = r;
    }
  } else {
    for (size_t i = tid; i < total; i += stride) {
      const int ch = (int)((i / hw) % c);
      const float ga = gamma[ch], is = istd[ch];
      float gi = g[i], h = training || RELU ? xhat[i] : 0.0f;
      if (mean) h = (h - mean[ch]) * is;
      if (RELU) gi = fmaf(ga, h, beta[ch]) > 0.0f ? gi : 0.0f;
      float r;
      if (training) {
        const float2 sm = sums[ch];
        r = is * (gi * ga - ga * sm.x / count - h * (ga * sm.y / count));
      } else {
        r = gi * ga * is;
      }
      dx[i] = accumulate ? dx[i] + r : r;
    }
  }
}

// The bound of dx where the sums are those of several processes (elsewhere it is made where the sums are finished).
__global__ void bn_dx_bound_kernel(const float2* __restrict__ sums, const float2* __restrict__ extremes, int splits,
                                   const float* __restrict__ count_dev, int c, const BnBound bound) {
  NRS_PDL_PROLOGUE();
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch >= c) return;
  const float2 e = fold_extremes(extremes, ch, c, splits), t = sums[ch];
  bound_dx(bound, ch, e.x, e.y, t.x, t.y, *count_dev);
}

// The normalise pass with the NHWC planes of y (no xhat).
template <bool SPLIT, bool RELU>
__global__ void __launch_bounds__(kThreads)
bn_normalize_planes_kernel(const float* __restrict__ x, const float* __restrict__ mean, const float* __restrict__ istd,
                           const float* __restrict__ gamma, const float* __restrict__ beta, float* __restrict__ y,
                           float* __restrict__ hi, float* __restrict__ lo, const img::Grid g, NrsRange* __restrict__ range) {
  NRS_PDL_PROLOGUE();
  __shared__ img::Tile tile;
  const float scale = SPLIT ? pr::scale_of(range->bound) : 1.0f;
  uint32_t top = 0;
  const uint32_t p0 = blockIdx.x * img::kTilePx;
  const int c0 = blockIdx.y * img::kTileCh, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const img::Pixels px(g, p0);
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int c = c0 + warp + 8 * (i >> 2);
    v[i] = (c < g.c && px.live[i & 3]) ? x[px.base + (px.at[i & 3] + (uint32_t)c * g.hw)] : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int cl = warp + 8 * k, c = c0 + cl;
    const bool ok = c < g.c;
    const float m = ok ? mean[c] : 0.0f, is = ok ? istd[c] : 0.0f, ga = ok ? gamma[c] : 0.0f, be = ok ? beta[c] : 0.0f;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float h = (v[4 * k + s] - m) * is;
      float o = fmaf(ga, h, be);
      if (RELU) o = fmaxf(o, 0.0f);
      if (ok && px.live[s]) {
        y[px.base + (px.at[s] + (uint32_t)c * g.hw)] = o;
        if (SPLIT) top = pr::seen(top, o);
      }
      tile[cl][s * 32 + lane] = o;
    }
  }
  __syncthreads();
  img::tile_to_planes<SPLIT>(tile, g, p0, c0, hi, lo, scale);
  if (SPLIT) pr::report_block(range, top);
}

// dx (overwritten; null: planes only) with its NHWC planes, and chan_partial[tile of 128 pixels][c], its sums over the tile.
template <bool SPLIT, bool RELU>
__global__ void __launch_bounds__(kThreads, 3)
bn_dx_planes_kernel(const float* __restrict__ gr, const float* __restrict__ x, const float* __restrict__ mean,
                    const float* __restrict__ istd, const float* __restrict__ gamma, const float* __restrict__ beta,
                    const float2* __restrict__ sums, float* __restrict__ dx, float* __restrict__ hi, float* __restrict__ lo,
                    float* __restrict__ chan_partial, const img::Grid g, float count, int training, const float* __restrict__ count_dev,
                    NrsRange* __restrict__ range) {
  NRS_PDL_PROLOGUE();
  __shared__ img::Tile tile;
  const float scale = SPLIT ? pr::scale_of(range->bound) : 1.0f;
  uint32_t top = 0;
  if (count_dev) count = *count_dev;
  const uint32_t p0 = blockIdx.x * img::kTilePx;
  const int c0 = blockIdx.y * img::kTileCh, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const img::Pixels px(g, p0);
  float vg[16], vx[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int c = c0 + warp + 8 * (i >> 2);
    const bool ok = c < g.c && px.live[i & 3];
    const size_t at = px.base + (px.at[i & 3] + (uint32_t)c * g.hw);
    vg[i] = ok ? gr[at] : 0.0f;
    vx[i] = ok ? x[at] : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int cl = warp + 8 * k, c = c0 + cl;
    const bool ok = c < g.c;
    const float m = ok ? mean[c] : 0.0f, is = ok ? istd[c] : 0.0f, ga = ok ? gamma[c] : 0.0f, be = ok && RELU ? beta[c] : 0.0f;
    const float2 sm = ok && training ? sums[c] : make_float2(0.0f, 0.0f);
    const float m1 = ga * sm.x / count, m2 = ga * sm.y / count;
    float total = 0.0f;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const float h = (vx[4 * k + s] - m) * is;
      float gi = vg[4 * k + s];
      if (RELU) gi = fmaf(ga, h, be) > 0.0f ? gi : 0.0f;
      const bool live = ok && px.live[s];
      const float r = !live ? 0.0f : training ? is * (gi * ga - m1 - h * m2) : gi * ga * is;
      if (live && dx) dx[px.base + (px.at[s] + (uint32_t)c * g.hw)] = r;
      tile[cl][s * 32 + lane] = r;
      if (SPLIT) top = pr::seen(top, r);
      total += r;
    }
    total = wsum(total);
    if (lane == 0 && ok) chan_partial[(size_t)blockIdx.x * g.c + c] = total;
  }
  __syncthreads();
  img::tile_to_planes<SPLIT>(tile, g, p0, c0, hi, lo, scale);
  if (SPLIT) pr::report_block(range, top);
}

// Statistics shared by several processes: the splits of this process folded in order into out[ch], the
// element count behind them (one slot), ready for one cross-rank sum of 2c + 1 floats.
__global__ void bn_fold_for_sync_kernel(const float2* __restrict__ partial, float2* __restrict__ out, float* count_slot,
                                        int c, int splits, float local_count) {
  NRS_PDL_PROLOGUE();
  const int ch = blockIdx.x * blockDim.x + threadIdx.x;
  if (ch == 0) *count_slot = local_count;
  if (ch >= c) return;
  float s = 0.0f, q = 0.0f;
  for (int z = 0; z < splits; ++z) {
    const float2 t = partial[(size_t)z * c + ch];
    s += t.x;
    q += t.y;
  }
  out[ch] = make_float2(s, q);
}
__global__ void bn_set_count_kernel(float* count_slot, float local_count) {
  NRS_PDL_PROLOGUE();
  if (blockIdx.x == 0 && threadIdx.x == 0) *count_slot = local_count;
}

// How many sample splits the per-channel reductions use: enough blocks to fill the device a few times over,
// no fewer than 8 images (planes) or 64 rows (columns) per block.
int plan_splits(const nrs_ctx* ctx, int n, int c, int hw) {
  const int blocks_c = hw == 1 ? (c + 31) / 32 : c;
  const int min_per = hw == 1 ? 64 : 8;
  int splits = (4 * ctx->sm_count + blocks_c - 1) / blocks_c;
  if (splits > n / min_per) splits = n / min_per;
  if (splits < 1) splits = 1;
  if (splits > 65535) splits = 65535;
  return splits;
}

template <bool FWD, bool RELU>
int launch_pair(nrs_ctx* ctx, const float* a, const float* b, float2* partial, float2* extremes, int n, int c, int hw, int splits,
                const float* gamma, const float* beta, const float* pivot = nullptr, const float* mean = nullptr,
                const float* istd = nullptr, const BnFinish& fin = BnFinish{}) {
  if (hw == 1) {
    NRS_PDL_LAUNCH((bn_pair_cols_kernel<FWD, RELU>), dim3((c + 31) / 32, splits), kThreads, 0, ctx->stream, a, b, partial, extremes,
                   n, c, splits, gamma, beta, pivot, mean, istd);
  } else {
    const bool vec = (hw & 3) == 0 && aligned16(a) && (FWD || aligned16(b));
#define NRS_BN_PAIR(M)                                                                                                         \
  NRS_PDL_LAUNCH((bn_pair_planes_kernel<FWD, RELU, M>), dim3(c, splits), kThreads, 0, ctx->stream, a, b, partial, extremes, n, c, hw, \
                 splits, gamma, beta, pivot, mean, istd, fin, NrsFastDiv(vec ? hw / 4 : hw), vec ? 1 : 0)
    if (extremes) NRS_BN_PAIR(true); else NRS_BN_PAIR(false);
#undef NRS_BN_PAIR
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}
// Tickets for a planes-layout reduction that finishes its channels itself; null when it cannot.
int finish_tickets(nrs_ctx* ctx, int c, int hw, unsigned** out) {
  *out = nullptr;
  if (hw == 1 || c + 1 > kNrsFoldTickets) return NRS_OK;
  const int st = nrs_fold_ticket(ctx, out);
  if (st == NRS_OK) *out += 1;   // slot 0 belongs to the single-counter users
  return st;
}

unsigned ew_blocks(const nrs_ctx* ctx, size_t work_items) {
  const size_t want = (work_items + kThreads - 1) / kThreads;
  const size_t cap = (size_t)ctx->sm_count * 16;
  return (unsigned)(want < 1 ? 1 : (want > cap ? cap : want));
}

bool check_dims(int n, int c, int hw) {
  return n >= 1 && c >= 1 && hw >= 1 && (size_t)n * c * hw <= (size_t)1 << 40 && (size_t)c * hw <= 0x7fffffffu &&
         (size_t)n * hw <= 0x7fffffffu;
}

}  // namespace

namespace {

int bn_forward(nrs_ctx* ctx, const char* who, const float* x, const float* gamma, const float* beta, float* running_mean,
               float* running_var, float* y, float* xhat, float* istd, int n, int c, int hw, float eps, float momentum,
               int training, bool relu, float* mean_out = nullptr, float* hi = nullptr, float* lo = nullptr,
               const NrsRange* known_x = nullptr) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, check_dims(n, c, hw), NRS_ERR_SHAPE, "%s: bad shape [%d,%d,%d]", who, n, c, hw);
  NRS_REQUIRE(ctx, x && gamma && beta && running_mean && running_var && y && istd, NRS_ERR_ARG, "%s: null tensor", who);
  NrsProfScope prof(ctx, NRS_PROF_BATCHNORM, 12.0 * (double)n * c * hw);   // x in; y, xhat out
  const int splits = training ? plan_splits(ctx, n, c, hw) : 1;
  // statistics over every process's shard: sums around a pivot all ranks share (the running mean), folded,
  // summed across ranks together with the element count, then finished as usual
  const bool shared = training && ctx->stat_sync.all_reduce_sum != nullptr;
  void* ws = nullptr;
  const bool pairs = hi && lo;
  const int st = nrs_workspace(ctx, ((size_t)splits * c * (pairs ? 4 : 2) + c + (size_t)c * 2 + 4) * sizeof(float), &ws);
  if (st != NRS_OK) return st;
  float2* partial = (float2*)ws;
  float2* extremes = pairs ? partial + (size_t)splits * c : nullptr;
  float* mean_ws = (float*)(partial + (size_t)splits * c * (pairs ? 2 : 1));
  float* mean = mean_out ? mean_out : mean_ws;
  float2* summed = (float2*)(mean_ws + c + (c & 1));   // 8-byte aligned; [c] pairs + the count
  float* count_slot = (float*)(summed + c);
  BnFinish fin{};
  NrsRange* range = nullptr;
  if (pairs) {
    int rs = nrs_range_renew(ctx, hi, &range);
    if (rs == NRS_OK && !training && !known_x) {
      NrsRange* measured = nullptr;
      rs = nrs_range_renew(ctx, &ctx->scratch_range[0], &measured);
      if (rs == NRS_OK) rs = nrs_absmax(ctx, x, (size_t)n * c * hw, measured);
      known_x = measured;
    }
    if (rs != NRS_OK) return rs;
  }
  const BnBound bound{range, known_x, gamma, beta, nullptr, training};
  fin.bound = bound;
  if (training) {
    if (!shared) {
      const int ft = finish_tickets(ctx, c, hw, &fin.tickets);
      if (ft != NRS_OK) return ft;
      fin.mean = mean; fin.istd = istd; fin.running_mean = running_mean; fin.running_var = running_var;
      fin.count = (float)((double)n * hw); fin.eps = eps; fin.momentum = momentum;
    }
    const int sp = launch_pair<true, false>(ctx, x, nullptr, partial, extremes, n, c, hw, splits, nullptr, nullptr,
                                            shared ? running_mean : nullptr, nullptr, nullptr, fin);
    if (sp != NRS_OK) return sp;
  }
  if (shared) {
    NRS_PDL_LAUNCH(bn_fold_for_sync_kernel, nrs_blocks(c, 128), 128, 0, ctx->stream, (const float2*)partial, summed, count_slot, c,
                   splits, (float)((double)n * hw));
    NRS_LAUNCHED(ctx);
    const int sr = ctx->stat_sync.all_reduce_sum(ctx->stat_sync.user, (float*)summed, (size_t)c * 2 + 1);
    if (sr != NRS_OK) return sr;
    NRS_PDL_LAUNCH(bn_stats_finish_kernel, nrs_blocks(c, 128), 128, 0, ctx->stream, (const float2*)summed, x, mean, istd,
                   running_mean, running_var, c, hw, 1, 0.0f, eps, momentum, training, (const float*)running_mean,
                   (const float*)count_slot, (const float2*)extremes, splits, bound);   // (this process's own extremes: its planes)
    NRS_LAUNCHED(ctx);
  } else if (!fin.tickets) {
    NRS_PDL_LAUNCH(bn_stats_finish_kernel, nrs_blocks(c, 128), 128, 0, ctx->stream, (const float2*)partial, x, mean, istd,
                   running_mean, running_var, c, hw, splits, (float)((double)n * hw), eps, momentum, training,
                   (const float*)nullptr, (const float*)nullptr, (const float2*)extremes, splits, bound);
    NRS_LAUNCHED(ctx);
  }
  if (hi) {
    const img::Grid grid(n, c, hw);
#define NRS_BN_NORM(S, R)                                                                                               \
  NRS_PDL_LAUNCH((bn_normalize_planes_kernel<S, R>), grid.blocks(), kThreads, 0, ctx->stream, x, (const float*)mean, (const float*)istd, \
                 gamma, beta, y, hi, lo, grid, range)
    if (lo) { if (relu) NRS_BN_NORM(true, true); else NRS_BN_NORM(true, false); }
    else { if (relu) NRS_BN_NORM(false, true); else NRS_BN_NORM(false, false); }
#undef NRS_BN_NORM
    NRS_LAUNCHED(ctx);
    return NRS_OK;
  }
  const size_t total = (size_t)n * c * hw;
  const bool vec = (hw & 3) == 0 && ((uintptr_t)x & 15) == 0 && ((uintptr_t)y & 15) == 0 && ((uintptr_t)xhat & 15) == 0;
  const unsigned blocks = ew_blocks(ctx, vec ? total / 4 : total);
#define NRS_BN_NORM(V, R)                                                                                          \
  NRS_PDL_LAUNCH((bn_normalize_kernel<V, R>), blocks, kThreads, 0, ctx->stream, x, (const float*)mean, (const float*)istd, \
                 gamma, beta, y, xhat, total, c, hw)
  if (vec) { if (relu) NRS_BN_NORM(true, true); else NRS_BN_NORM(true, false); }
  else { if (relu) NRS_BN_NORM(false, true); else NRS_BN_NORM(false, false); }
#undef NRS_BN_NORM
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int bn_backward(nrs_ctx* ctx, const char* who, const float* g, const float* xhat, const float* istd, const float* gamma,
                const float* beta, float* dx, float* dgamma, float* dbeta, int n, int c, int hw, int training,
                int accumulate_dx, int accumulate_params, bool relu, const float* mean = nullptr /* xhat is x then */,
                float* hi = nullptr, float* lo = nullptr, float* chan_partial = nullptr) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, check_dims(n, c, hw), NRS_ERR_SHAPE, "%s: bad shape [%d,%d,%d]", who, n, c, hw);
  NRS_REQUIRE(ctx, (dgamma == nullptr) == (dbeta == nullptr), NRS_ERR_ARG, "%s: dgamma and dbeta must be given together", who);
  NRS_REQUIRE(ctx, g && xhat && istd && gamma && (!relu || beta), NRS_ERR_ARG, "%s: null tensor", who);
  if (!dx && !hi && !dgamma) return NRS_OK;
  NrsProfScope prof(ctx, NRS_PROF_BATCHNORM, 12.0 * (double)n * c * hw);   // g, xhat in; dx out
  const bool pairs = hi && lo;
  const bool need_sums = dgamma || training || pairs;   // (pairs: the same reading bounds dx)
  const int splits = need_sums ? plan_splits(ctx, n, c, hw) : 1;
  void* ws = nullptr;
  const int st = nrs_workspace(ctx, ((size_t)splits * c * (pairs ? 4 : 2) + (size_t)c * 2 + 4) * sizeof(float), &ws);
  if (st != NRS_OK) return st;
  float2* partial = (float2*)ws;
  float2* extremes = pairs ? partial + (size_t)splits * c : nullptr;
  float2* sums = partial + (size_t)splits * c * (pairs ? 2 : 1);
  float* count_slot = (float*)(sums + c);
  // with shared statistics dx needs the sums over every process's shard; the parameter gradients keep this
  // process's own sums (they are summed across ranks with all other gradients)
  const bool shared = training && (dx || hi) && ctx->stat_sync.all_reduce_sum != nullptr;
  const float count = (float)((double)n * hw);
  NrsRange* range = nullptr;
  if (pairs) {
    const int rs = nrs_range_renew(ctx, hi, &range);
    if (rs != NRS_OK) return rs;
  }
  const BnBound bound{range, nullptr, gamma, nullptr, istd, training};
  if (need_sums) {
    BnFinish fin{};
    if (!shared) fin.bound = bound;   // (else once the sums are those of all processes)
    fin.count = count;
    const int ft = finish_tickets(ctx, c, hw, &fin.tickets);
    if (ft != NRS_OK) return ft;
    fin.sums = sums; fin.dgamma = dgamma; fin.dbeta = dbeta; fin.accumulate = accumulate_params;
    const int sp = relu ? launch_pair<false, true>(ctx, g, xhat, partial, extremes, n, c, hw, splits, gamma, beta, nullptr, mean, istd, fin)
                        : launch_pair<false, false>(ctx, g, xhat, partial, extremes, n, c, hw, splits, nullptr, nullptr, nullptr, mean, istd, fin);
    if (sp != NRS_OK) return sp;
    if (!fin.tickets) {
      NRS_PDL_LAUNCH(bn_grad_finish_kernel, nrs_blocks(c, 128), 128, 0, ctx->stream, (const float2*)partial, sums, dgamma, dbeta,
                     c, splits, accumulate_params, (const float2*)extremes, count, fin.bound);
      NRS_LAUNCHED(ctx);
    }
  }
  if (!dx && !hi) return NRS_OK;
  if (shared) {
    NRS_PDL_LAUNCH(bn_set_count_kernel, 1, 32, 0, ctx->stream, count_slot, (float)((double)n * hw));
    NRS_LAUNCHED(ctx);
    const int sr = ctx->stat_sync.all_reduce_sum(ctx->stat_sync.user, (float*)sums, (size_t)c * 2 + 1);
    if (sr != NRS_OK) return sr;
    if (pairs) {
      NRS_PDL_LAUNCH(bn_dx_bound_kernel, nrs_blocks(c, 128), 128, 0, ctx->stream, (const float2*)sums, (const float2*)extremes, splits,
                     (const float*)count_slot, c, bound);
      NRS_LAUNCHED(ctx);
    }
  }
  if (hi) {
    const img::Grid grid(n, c, hw);
#define NRS_BN_DX(S, R)                                                                                                  \
  NRS_PDL_LAUNCH((bn_dx_planes_kernel<S, R>), grid.blocks(), kThreads, 0, ctx->stream, g, xhat, mean, istd, gamma, beta,  \
                 (const float2*)sums, dx, hi, lo, chan_partial, grid, count, training, shared ? (const float*)count_slot : (const float*)nullptr, range)
    if (lo) { if (relu) NRS_BN_DX(true, true); else NRS_BN_DX(true, false); }
    else { if (relu) NRS_BN_DX(false, true); else NRS_BN_DX(false, false); }
#undef NRS_BN_DX
    NRS_LAUNCHED(ctx);
    return NRS_OK;
  }
  const size_t total = (size_t)n * c * hw;
  const bool vec = (hw & 3) == 0 && ((uintptr_t)g & 15) == 0 && ((uintptr_t)xhat & 15) == 0 && ((uintptr_t)dx & 15) == 0;
  const unsigned blocks = ew_blocks(ctx, vec ? total / 4 : total);
#define NRS_BN_DX(V, R)                                                                                              \
  NRS_PDL_LAUNCH((bn_dx_kernel<V, R>), blocks, kThreads, 0, ctx->stream, g, xhat, istd, gamma, beta, (const float2*)sums, dx, \
                 total, c, hw, count, training, accumulate_dx, shared ? (const float*)count_slot : (const float*)nullptr, mean)
  if (vec) { if (relu) NRS_BN_DX(true, true); else NRS_BN_DX(true, false); }
  else { if (relu) NRS_BN_DX(false, true); else NRS_BN_DX(false, false); }
#undef NRS_BN_DX
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

bool act_ok(int act) { return act == NRS_ACT_NONE || act == NRS_ACT_RELU; }

}  // namespace

int nrs_batchnorm_fwd(nrs_ctx* ctx, const float* x, const float* gamma, const float* beta, float* running_mean,
                      float* running_var, float* y, float* xhat, float* istd, int n, int c, int hw, float eps,
                      float momentum, int training) {
  return bn_forward(ctx, "nrs_batchnorm_fwd", x, gamma, beta, running_mean, running_var, y, xhat, istd, n, c, hw, eps,
                    momentum, training, false);
}

int nrs_batchnorm_bwd(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma, float* dx,
                      float* dgamma, float* dbeta, int n, int c, int hw, int training, int accumulate_dx,
                      int accumulate_params) {
  return bn_backward(ctx, "nrs_batchnorm_bwd", g, xhat, istd, gamma, nullptr, dx, dgamma, dbeta, n, c, hw, training,
                     accumulate_dx, accumulate_params, false);
}

int nrs_batchnorm_act_fwd(nrs_ctx* ctx, const float* x, const float* gamma, const float* beta, float* running_mean,
                          float* running_var, float* y, float* xhat, float* istd, int n, int c, int hw, float eps,
                          float momentum, int training, int act) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, act_ok(act), NRS_ERR_ARG, "nrs_batchnorm_act_fwd: activation %d is not NONE or RELU", act);
  NRS_REQUIRE(ctx, act == NRS_ACT_NONE || xhat, NRS_ERR_ARG, "nrs_batchnorm_act_fwd: a fused ReLU needs xhat saved");
  return bn_forward(ctx, "nrs_batchnorm_act_fwd", x, gamma, beta, running_mean, running_var, y, xhat, istd, n, c, hw, eps,
                    momentum, training, act == NRS_ACT_RELU);
}

int nrs_batchnorm_act_bwd(nrs_ctx* ctx, const float* g, const float* xhat, const float* istd, const float* gamma,
                          const float* beta, float* dx, float* dgamma, float* dbeta, int n, int c, int hw, int training,
                          int accumulate_dx, int accumulate_params, int act) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, act_ok(act), NRS_ERR_ARG, "nrs_batchnorm_act_bwd: activation %d is not NONE or RELU", act);
  return bn_backward(ctx, "nrs_batchnorm_act_bwd", g, xhat, istd, gamma, beta, dx, dgamma, dbeta, n, c, hw, training,
                     accumulate_dx, accumulate_params, act == NRS_ACT_RELU);
}

int nrs_batchnorm_fwd_saving_mean(nrs_ctx* ctx, const float* x, const float* gamma, const float* beta, float* running_mean, float* running_var,
                                  float* y, float* mean, float* istd, int n, int c, int hw, float eps, float momentum, int training, int act,
                                  float* hi, float* lo, const NrsRange* range_x) {
  return bn_forward(ctx, "batchnorm", x, gamma, beta, running_mean, running_var, y, nullptr, istd, n, c, hw, eps, momentum, training,
                    act == NRS_ACT_RELU, mean, hi, lo, range_x);
}

int nrs_batchnorm_bwd_from_x(nrs_ctx* ctx, const float* g, const float* x, const float* mean, const float* istd, const float* gamma,
                             const float* beta, float* dx, float* dgamma, float* dbeta, int n, int c, int hw, int training, int accumulate_dx,
                             int accumulate_params, int act, float* hi, float* lo, float* chan_partial) {
  return bn_backward(ctx, "batchnorm backward", g, x, istd, gamma, beta, dx, dgamma, dbeta, n, c, hw, training, accumulate_dx, accumulate_params,
                     act == NRS_ACT_RELU, mean, hi, lo, chan_partial);
}

int nrs_batchnorm_tiles(int n, int hw) { return (int)(((size_t)n * hw + img::kTilePx - 1) / img::kTilePx); }
