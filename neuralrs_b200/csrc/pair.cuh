// Operands of the 3xTF32 mode: an f32 value as a pair of f16 values,
//
//   x = (hi + lo / 2048) / 2^e,     hi = f16(x * 2^e),  lo = f16((x * 2^e - hi) * 2048),
//
// with one exponent e per tensor, taken from a bound of its largest magnitude (NrsRange::bound): bound * 2^e lies in
// [2^14, 2^15).  Both roundings are to nearest, so the pair carries x to 2^-23 of itself (a TF32 value and its residual as
// the tensor core reads it, truncated: 2^-22) down to 2^-29 of the bound, and to 2^-51 of the bound below that.  A product
// is hi.hi + (hi.lo + lo.hi) / 2048, on kind::f16 at twice the rate of kind::tf32 and with half the bytes per value; the
// two parts are summed in accumulators of their own, and the epilogue brings them together and takes the exponents out.
// Infinities and NaNs make hi the same and lo NaN, as a TF32 value and its residual did.
#pragma once

#include <cuda_fp16.h>

#include "nrs_internal.h"

namespace pr {

constexpr float kLoScale = 2048.0f, kLoUnscale = 1.0f / 2048.0f;

// The exponent for a tensor bounded by `bound` (finite, not negative).
__device__ __forceinline__ int scale_exp(float bound) { return min(126, 141 - (int)(__float_as_uint(bound) >> 23)); }
__device__ __forceinline__ float pow2(int e) { return __uint_as_float((uint32_t)(e + 127) << 23); }   // -126 <= e <= 127
__device__ __forceinline__ float scale_of(float bound) { return pow2(scale_exp(bound)); }
// The factor that takes two operands' exponents out of their product, in two halves (by itself it may leave f32's range).
struct Unscale {
  float a, a_lo, b;
  bool halves;   // nearly never: one factor does
  __device__ __forceinline__ Unscale(float bound_a, float bound_b) {
    const int e = -(scale_exp(bound_a) + scale_exp(bound_b));
    halves = e < -115 || e > 127;
    const int first = halves ? e / 2 : e;
    a = pow2(first);
    a_lo = a * kLoUnscale;
    b = pow2(e - first);
  }
  __device__ __forceinline__ float operator()(float hh, float cross) const {
    const float v = fmaf(cross, a_lo, hh * a);
    return halves ? v * b : v;
  }
  template <int N>
  __device__ __forceinline__ void apply(uint32_t (&hh)[N], const uint32_t (&cross)[N]) const {
#pragma unroll
    for (int j = 0; j < N; ++j) hh[j] = __float_as_uint(fmaf(__uint_as_float(cross[j]), a_lo, __uint_as_float(hh[j]) * a));
    if (!halves) return;
#pragma unroll
    for (int j = 0; j < N; ++j) hh[j] = __float_as_uint(__uint_as_float(hh[j]) * b);
  }
};

__device__ __forceinline__ void split(float v, float scale, __half* hi, __half* lo) {
  const float x = v * scale;
  *hi = __float2half_rn(x);
  *lo = __float2half_rn((x - __half2float(*hi)) * kLoScale);
}
__device__ __forceinline__ void split2(float x, float y, __half2* hi, __half2* lo) {   // already scaled
  *hi = __floats2half2_rn(x, y);
  const float2 f = __half22float2(*hi);
  *lo = __floats2half2_rn((x - f.x) * kLoScale, (y - f.y) * kLoScale);
}
__device__ __forceinline__ uint32_t bits(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
__device__ __forceinline__ void split4(float4 v, float scale, uint2* hi, uint2* lo) {
  __half2 h0, h1, l0, l1;
  split2(v.x * scale, v.y * scale, &h0, &l0);
  split2(v.z * scale, v.w * scale, &h1, &l1);
  *hi = make_uint2(bits(h0), bits(h1));
  *lo = make_uint2(bits(l0), bits(l1));
}
__device__ __forceinline__ void put(void* hi, void* lo, size_t at, float v, float scale) {
  split(v, scale, reinterpret_cast<__half*>(hi) + at, reinterpret_cast<__half*>(lo) + at);
}
// Four values to an index that is a multiple of 4.
__device__ __forceinline__ void put4(void* hi, void* lo, size_t at, float4 v, float scale) {
  uint2 h, l;
  split4(v, scale, &h, &l);
  *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(hi) + at) = h;
  *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(lo) + at) = l;
}
__device__ __forceinline__ float4 get4(const void* hi, const void* lo, size_t at, float unscale) {
  const uint2 h = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(hi) + at);
  const uint2 l = *reinterpret_cast<const uint2*>(reinterpret_cast<const __half*>(lo) + at);
  auto two = [](uint32_t u) { return __half22float2(*reinterpret_cast<const __half2*>(&u)); };
  const float2 h0 = two(h.x), h1 = two(h.y), l0 = two(l.x), l1 = two(l.y);
  return make_float4(fmaf(l0.x, kLoUnscale, h0.x) * unscale, fmaf(l0.y, kLoUnscale, h0.y) * unscale, fmaf(l1.x, kLoUnscale, h1.x) * unscale,
                     fmaf(l1.y, kLoUnscale, h1.y) * unscale);
}

// Largest finite magnitude seen, as the bits of a float (which order like the magnitudes).
__device__ __forceinline__ uint32_t seen(uint32_t top, float v) {
  const uint32_t u = __float_as_uint(v) & 0x7fffffffu;
  return u < 0x7f800000u && u > top ? u : top;
}
template <int N>
__device__ __forceinline__ uint32_t seen_all(uint32_t top, const float (&v)[N]) {   // infinities and NaNs looked for once
  uint32_t m = 0;
#pragma unroll
  for (int j = 0; j < N; ++j) m = max(m, __float_as_uint(v[j]) & 0x7fffffffu);
  if (m < 0x7f800000u) return max(top, m);
#pragma unroll
  for (int j = 0; j < N; ++j) top = seen(top, v[j]);
  return top;
}
__device__ __forceinline__ uint32_t seen4(uint32_t top, float4 v) {
  const float a[4] = {v.x, v.y, v.z, v.w};
  return seen_all(top, a);
}
// A whole warp's, into the tensor's range.
__device__ __forceinline__ void report(NrsRange* r, uint32_t top) {
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) atomicMax(reinterpret_cast<unsigned*>(&r->top), top);   // (no result: nothing waits for it)
}
// What one block finds in n values (all of its threads ask; at most kScanAlone values, else absmax_kernel measures them).
constexpr int kScanAlone = 32768;
__device__ __forceinline__ uint32_t scan(const float* __restrict__ src, int n) {
  __shared__ uint32_t found[32];
  uint32_t top = 0;
  const int head = min(n, (int)(((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15) / 4)), quads = (n - head) / 4;
  const float4* body = reinterpret_cast<const float4*>(src + head);
  for (int i = threadIdx.x; i < quads; i += 8 * blockDim.x) {   // eight loads under way: latency is all there is here
    float v[32];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int at = i + u * (int)blockDim.x;
      const float4 q = at < quads ? body[at] : make_float4(0.f, 0.f, 0.f, 0.f);
      v[4 * u] = q.x; v[4 * u + 1] = q.y; v[4 * u + 2] = q.z; v[4 * u + 3] = q.w;
    }
    top = seen_all(top, v);
  }
  if ((int)threadIdx.x < head) top = seen(top, src[threadIdx.x]);
  const int rest = head + 4 * quads + (int)threadIdx.x;
  if (rest < n) top = seen(top, src[rest]);   // at most 3
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) found[threadIdx.x >> 5] = top;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  top = __reduce_max_sync(0xffffffffu, lane < (int)(blockDim.x >> 5) ? found[lane] : 0u);
  __syncthreads();
  return top;
}
// The scale of planes whose values are bounded by *top, or (scan_n > 0) are the scan_n values at `src`; one thread of the
// grid leaves the bound as their range.
__device__ __forceinline__ float open_range(const float* top, const float* src, int scan_n, NrsRange* range) {
  const float bound = scan_n > 0 ? __uint_as_float(scan(src, scan_n)) : *reinterpret_cast<const volatile float*>(top);
  if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) {
    range->bound = bound;
    if (top != &range->top) range->top = bound;
  }
  return scale_of(bound);
}
// The same for a whole block (all of its threads ask).
__device__ __forceinline__ void report_block(NrsRange* r, uint32_t top) {
  __shared__ uint32_t all;
  if (threadIdx.x == 0) all = 0;
  __syncthreads();
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) atomicMax(&all, top);
  __syncthreads();
  if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned*>(&r->top), all);
}
// Bound of a sum of `k` products of values up to a and b, plus a value up to c: with room for the sum's own rounding,
// and finite.
__device__ __forceinline__ float product_bound(float k, float a, float b, float c) { return fminf((k * a * b + c) * 1.001f, 3.0e38f); }

}  // namespace pr
