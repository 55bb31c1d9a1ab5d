// Operand staging for the tensor-core kernels: one memory-bound pass that brings an
// operand into the K-major form with 16-byte aligned rows that TMA wants and, for 3xTF32,
// makes f16 pairs of it (pair.cuh).  Without the split the single plane is still rounded to nearest
// TF32: the tensor core truncates its inputs, and truncation's systematic bias
// compounds through a deep network where rounding's does not.  Transposed sources ([K][rows], e.g. NCHW images seen as
// [C][H*W]) go through 32x32 shared-memory tiles so both sides stay coalesced.
#include "image_tile.cuh"
#include "tc_mainloop.cuh"

namespace {

// Largest finite magnitude of n values into r->top.  A read of the tensor, from HBM where it exceeds L2.
struct Measured { const float* src; size_t n; NrsRange* r; };
constexpr int kSources = 4;   // tensors of one launch
struct MeasuredSet { Measured m[kSources]; };
__global__ void __launch_bounds__(256)
absmax_kernel(const __grid_constant__ MeasuredSet set) {
  NRS_PDL_PROLOGUE();
  __shared__ uint32_t part[8];
  const Measured& m = set.m[blockIdx.y];
  const float* __restrict__ src = m.src;
  const size_t n = m.n;
  const size_t head = min(n, (size_t)(((16 - (reinterpret_cast<uintptr_t>(src) & 15)) & 15) / 4)), quads = (n - head) / 4;
  const float4* body = reinterpret_cast<const float4*>(src + head);
  const size_t step = (size_t)gridDim.x * blockDim.x, first = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t top = 0;
  size_t i = first;
  for (; i + 3 * step < quads; i += 4 * step) {
    float4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = body[i + u * step];
#pragma unroll
    for (int u = 0; u < 4; ++u) top = pr::seen4(top, v[u]);
  }
  for (; i < quads; i += step) top = pr::seen4(top, body[i]);
  if (first < head) top = pr::seen(top, src[first]);
  if (head + 4 * quads + first < n) top = pr::seen(top, src[head + 4 * quads + first]);   // (at most 3, in the first block)
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = top;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  pr::report(m.r, threadIdx.x < 8 ? part[threadIdx.x] : 0u);
}

__global__ void __launch_bounds__(256)
pair_unpack_kernel(const float* __restrict__ hi, const float* __restrict__ lo, const NrsRange* __restrict__ range, float* __restrict__ dst, size_t n) {
  NRS_PDL_PROLOGUE();
  const float unscale = pr::pow2(-pr::scale_exp(range->bound));
  const size_t step = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step)
    dst[i] = fmaf(__half2float(reinterpret_cast<const __half*>(lo)[i]), pr::kLoUnscale, __half2float(reinterpret_cast<const __half*>(hi)[i])) * unscale;
}

// Where the bound of a tensor's planes comes from: *top, or a scan of the `scan_n` values at src by every block.
struct Bound {
  const float* top;
  const float* src;
  int scan_n;
  NrsRange* range;
};
template <bool SPLIT>
__device__ __forceinline__ float open_range(const Bound& b) { return SPLIT ? pr::open_range(b.top, b.src, b.scan_n, b.range) : 1.0f; }

// `also`: a tensor whose largest magnitude the grid's last blocks measure meanwhile (the weight that the staged rows are to
// be multiplied with: a launch of its own costs a small model's step 3 us).
struct Also {
  const float* src;
  size_t count;
  NrsRange* range;
  unsigned blocks;
};
__device__ __forceinline__ void measure_also(const Also& a, unsigned first) {
  uint32_t top = 0;
  const size_t step = (size_t)a.blocks * blockDim.x, tid = (size_t)(blockIdx.x - first) * blockDim.x + threadIdx.x;
  const size_t quads = (reinterpret_cast<uintptr_t>(a.src) & 15) == 0 ? a.count / 4 : 0;
  const float4* body = reinterpret_cast<const float4*>(a.src);
  for (size_t i = tid; i < quads; i += 4 * step) {
    float v[16];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const float4 q = i + u * step < quads ? body[i + u * step] : make_float4(0.f, 0.f, 0.f, 0.f);
      v[4 * u] = q.x; v[4 * u + 1] = q.y; v[4 * u + 2] = q.z; v[4 * u + 3] = q.w;
    }
    top = pr::seen_all(top, v);
  }
  for (size_t i = 4 * quads + tid; i < a.count; i += step) top = pr::seen(top, a.src[i]);
  pr::report_block(a.range, top);
}

// Where the matrices of a batch lie: at equal distances, or (weights that meet in one product) each by itself.
struct Sources {
  const float* first;
  size_t stride;
  const float* each[kSources];   // null: by the stride
  Sources(const float* src, size_t bstride) : first(src), stride(bstride), each{} {}
  __device__ __forceinline__ const float* at(int b) const { return each[0] ? each[b] : first + b * stride; }
};

template <bool SPLIT>
__global__ void __launch_bounds__(256)
stage_rows_kernel(const __grid_constant__ Sources sources, float* __restrict__ hi, float* __restrict__ lo, int rows, int K,
                  int ldk, size_t dst_bstride, const NrsFastDiv div_q, const Bound bound, const Also also) {
  NRS_PDL_PROLOGUE();
  const unsigned blocks = gridDim.x - also.blocks;
  if (SPLIT && blockIdx.x >= blocks) {
    measure_also(also, blocks);
    return;
  }
  const float scale = open_range<SPLIT>(bound);
  const int b = blockIdx.y;
  const float* __restrict__ src = sources.at(b);
  const size_t dst = b * dst_bstride;
  const int q = ldk / 4;
  const size_t total4 = (size_t)rows * q;
  const size_t stride = (size_t)blocks * blockDim.x;
  const bool vec = (K & 3) == 0 && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < total4; i += stride) {
    const size_t r = total4 < ((size_t)1 << 31) ? div_q.div((uint32_t)i) : i / q;   // (a 64-bit division is some 80 instructions)
    const int k = (int)(i - r * q) * 4;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
      if (k < K) v = *reinterpret_cast<const float4*>(src + r * K + k);
    } else {
      if (k + 0 < K) v.x = src[r * K + k + 0];
      if (k + 1 < K) v.y = src[r * K + k + 1];
      if (k + 2 < K) v.z = src[r * K + k + 2];
      if (k + 3 < K) v.w = src[r * K + k + 3];
    }
    if (SPLIT) pr::put4(hi, lo, dst + r * ldk + k, v, scale);
    else *reinterpret_cast<float4*>(hi + dst + r * ldk + k) = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
  }
}

template <bool SPLIT>
__global__ void __launch_bounds__(256)
stage_transpose_kernel(const __grid_constant__ Sources sources, float* __restrict__ hi, float* __restrict__ lo, int rows, int K,
                       int ldk, size_t dst_bstride, const Bound bound) {
  NRS_PDL_PROLOGUE();
  __shared__ float tile[32][33];
  const float scale = open_range<SPLIT>(bound);
  const int b = blockIdx.z;
  const float* __restrict__ src = sources.at(b);
  const size_t dst = b * dst_bstride;
  const int r0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = ty; i < 32; i += 8) {
    const int k = k0 + i, r = r0 + tx;
    tile[i][tx] = (k < K && r < rows) ? src[(size_t)k * rows + r] : 0.0f;
  }
  __syncthreads();
  if (SPLIT) {   // two values a thread (ldk is even): 64 bytes of a row per half warp
    for (int i = threadIdx.x >> 4; i < 32; i += 16) {
      const int r = r0 + i, c = 2 * (threadIdx.x & 15), k = k0 + c;
      if (r >= rows || k >= ldk) continue;
      __half2 h, l;
      pr::split2(tile[c][i] * scale, tile[c + 1][i] * scale, &h, &l);
      *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(hi) + dst + (size_t)r * ldk + k) = h;
      *reinterpret_cast<__half2*>(reinterpret_cast<__half*>(lo) + dst + (size_t)r * ldk + k) = l;
    }
    return;
  }
  for (int i = ty; i < 32; i += 8) {
    const int r = r0 + i, k = k0 + tx;
    if (r < rows && k < ldk) hi[dst + (size_t)r * ldk + k] = tc::tf32_rn(tile[tx][i]);
  }
}

// NCHW [n][c][hw] -> NHWC planes [n][hw][ld].  HBM-bound: 4 B read and 4 or 8 B written per element.  SUMS: also
// chan_partial[tile][c], the channel sums over the tile's pixels (a bias gradient's first stage without a pass of its own:
// 29 us for 256 images of 128 x 32 x 32).
template <bool SPLIT, bool SUMS>
__global__ void __launch_bounds__(256)
stage_image_kernel(const float* __restrict__ src, float* __restrict__ hi, float* __restrict__ lo, float* __restrict__ chan_partial, const img::Grid g,
                   const Bound bound) {
  __shared__ img::Tile tile;
  const uint32_t p0 = blockIdx.x * img::kTilePx;
  const int c0 = blockIdx.y * img::kTileCh, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const img::Pixels px(g, p0);
  NRS_PDL_PROLOGUE();
  float v[16];
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int c = c0 + warp + 8 * (i >> 2);
    v[i] = (c < g.c && px.live[i & 3]) ? src[px.base + (px.at[i & 3] + (uint32_t)c * g.hw)] : 0.0f;
  }
  const float scale = open_range<SPLIT>(bound);   // (its loads behind those)
#pragma unroll
  for (int i = 0; i < 16; ++i) tile[warp + 8 * (i >> 2)][(i & 3) * 32 + lane] = v[i];
  if (SUMS) {
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      float t = (v[4 * k] + v[4 * k + 1]) + (v[4 * k + 2] + v[4 * k + 3]);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) t += __shfl_xor_sync(0xffffffffu, t, d);
      const int c = c0 + warp + 8 * k;
      if (lane == 0 && c < g.c) chan_partial[(size_t)blockIdx.x * g.c + c] = t;
    }
  }
  __syncthreads();
  img::tile_to_planes<SPLIT>(tile, g, p0, c0, hi, lo, scale);
}

// A weight that every block scans itself is staged by blocks of kWideStage threads: five loads a thread instead of eighteen
// for 64 x 32 x 3 x 3.
constexpr int kWideStage = 1024, kWideScan = 4096;
template <bool SPLIT>
__global__ void __launch_bounds__(kWideStage)
stage_conv_weight_kernel(const float* __restrict__ w, float* __restrict__ hi, float* __restrict__ lo, int co_n, int ci_n,
                         int kh, int kw, int for_dgrad, const Bound bound) {
  const int taps = kh * kw, rows = for_dgrad ? ci_n : co_n, inner = for_dgrad ? co_n : ci_n, ld = (inner + 31) / 32 * 32;
  const size_t total = (size_t)rows * ld * taps;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  // idx enumerates the OUTPUT [row][t*ld + k] so writes are coalesced.
  size_t above;   // row * taps + t
  int row, t;
  if (total < (size_t)1 << 31) {
    above = (uint32_t)idx / (uint32_t)ld;
    row = (int)((uint32_t)above / (uint32_t)taps);
  } else {
    above = idx / ld;
    row = (int)(above / taps);
  }
  const int k = (int)(idx - above * ld);
  t = (int)(above - (size_t)row * taps);
  const int co = for_dgrad ? k : row, ci = for_dgrad ? row : k;
  NRS_PDL_PROLOGUE();
  const float v = idx < total && k < inner ? w[((size_t)co * ci_n + ci) * taps + t] : 0.0f;
  const float scale = open_range<SPLIT>(bound);   // (its loads behind that one)
  if (idx >= total) return;
  if (SPLIT) pr::put(hi, lo, idx, v, scale);
  else hi[idx] = tc::tf32_rn(v);
}

// Gradient staging fused with the masks that precede a convolution's backward pass.
//   MODE 0  v = (y > 0) ? dy : 0                          (ReLU folded into the conv: y is its output)
//   MODE 1  v = (argmax[o] == idx && y[o] > 0) ? g[o] : 0  (k x k / stride k max-pool on top of that;
//           y is the POOLED output here: the window's maximum is > 0 exactly where the winner
//           passed the ReLU, so the full-resolution activation is not read at all)
// One pass reads the NCHW sources through 32 channel x 32 pixel tiles and writes the
// masked gradient in NCHW (optional) and as NHWC operand planes (optional).
template <bool SPLIT, int MODE>
__global__ void __launch_bounds__(256)
stage_masked_kernel(const float* __restrict__ g, const float* __restrict__ y, const int32_t* __restrict__ argmax,
                    float* __restrict__ nchw_out, float* __restrict__ hi, float* __restrict__ lo, int c_n, int h,
                    int w, int k, int oh, int ow, const Bound bound) {
  NRS_PDL_PROLOGUE();
  const float scale = open_range<SPLIT>(bound);
  __shared__ float tile[32][33];
  const int img = blockIdx.z, hw = h * w;
  const int p0 = blockIdx.x * 32, c0 = blockIdx.y * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int i = ty; i < 32; i += 8) {
    const int c = c0 + i, px = p0 + tx;
    float v = 0.0f;
    if (c < c_n && px < hw) {
      const size_t idx = ((size_t)img * c_n + c) * hw + px;
      if (MODE == 0) {
        v = y[idx] > 0.0f ? g[idx] : 0.0f;
      } else {
        const int yy = px / w, xx = px - yy * w;
        const int oy = yy / k, ox = xx / k;
        if (oy < oh && ox < ow) {
          const size_t o = (((size_t)img * c_n + c) * oh + oy) * ow + ox;
          if ((size_t)argmax[o] == idx && y[o] > 0.0f) v = g[o];
        }
      }
      if (nchw_out) nchw_out[idx] = v;
    }
    tile[i][tx] = v;
  }
  if (!hi) return;
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int px = p0 + i, c = c0 + tx;
    if (px < hw && c < c_n) {
      const float v = tile[tx][i];
      const size_t o = ((size_t)img * hw + px) * c_n + c;
      if (SPLIT) pr::put(hi, lo, o, v, scale);
      else hi[o] = tc::tf32_rn(v);
    }
  }
}


// The tile of the two 2x2 / stride-2 pooling kernels below: 32 channels x 32 consecutive pooled positions, counted across
// the even-sized images.  A thread reads its four channels' values together, all loads under way before the first is used,
// and writes four channels of a pixel at once.
struct PoolGrid {
  int c, h, w;
  uint32_t positions;   // pooled, in the batch
  NrsFastDiv div_ohw, div_ow;
  PoolGrid(int n, int c_, int h_, int w_)
      : c(c_), h(h_), w(w_), positions((uint32_t)n * (uint32_t)(h_ / 2) * (uint32_t)(w_ / 2)), div_ohw((h_ / 2) * (w_ / 2)), div_ow(w_ / 2) {}
  static bool fits(int n, int c_, int h_, int w_) { return (double)n * (h_ / 2) * (w_ / 2) < 2147483648.0 && (double)c_ * h_ * w_ < 2147483648.0; }
  dim3 blocks() const { return dim3((positions + 31) / 32, (unsigned)((c + 31) / 32)); }
};
struct PoolPlace {
  bool live;
  uint32_t img, po, corner;   // image, pooled position and top left pixel inside its plane
  __device__ __forceinline__ PoolPlace(const PoolGrid& g, uint32_t pos) {
    uint32_t oy, ox;
    live = pos < g.positions;
    g.div_ohw.divmod(live ? pos : 0u, img, po);
    g.div_ow.divmod(po, oy, ox);
    corner = 2 * oy * (uint32_t)g.w + 2 * ox;
  }
};

// The backward pass of 2x2 / stride-2 pooling and the ReLU ahead of it, organised around the POOLED elements (a quarter of
// the output): g, the pooled output and argmax are read once, coalesced; the 2x2 windows leave as float2 row segments
// (NCHW) and, through a shared-memory tile, as NHWC planes, four channels a store.  Bound by memory where the tensor is
// large: 12 B read per pooled element and 16 to 32 written.  Small tensors are bound by instructions and latency: with
// 64-bit divisions per thread, loads one behind the other and two channels a store, the two launches of a step of the small
// CNN (batch 64, 3xTF32) took 14.7 us, now 9.0; the three of the CIFAR CNN at batch 100 28.6, now 25.
template <bool SPLIT>
__global__ void __launch_bounds__(256)
pool2_bwd_planes_kernel(const float* __restrict__ g, const float* __restrict__ pooled, const int32_t* __restrict__ argmax,
                        float* __restrict__ nchw_out, float* __restrict__ hi, float* __restrict__ lo,
                        float* __restrict__ chan_partial /*[gridDim.x][c] per-block channel sums, or null*/, const PoolGrid pg, const Bound bound) {
  __shared__ float tile[32][129];    // [channel][q*32 + position], q = 2*dy + dx inside the window
  __shared__ long long pix_base[32]; // linear index of each position's top-left pixel, -1 beyond the end
  const uint32_t gp0 = blockIdx.x * 32u;
  const int c0 = blockIdx.y * 32, w = pg.w, hw = pg.h * w, ohw = hw >> 2;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const PoolPlace at(pg, gp0 + tx);
  if (ty == 0) pix_base[tx] = at.live ? (long long)at.img * hw + at.corner : -1;
  NRS_PDL_PROLOGUE();
  const size_t chan0 = (size_t)at.img * pg.c + c0 + ty;
  float gv[4], pv[4];
  int32_t am[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const bool ok = at.live && c0 + ty + 8 * i < pg.c;
    const size_t o = (chan0 + 8 * i) * ohw + at.po;
    gv[i] = ok ? g[o] : 0.0f;
    pv[i] = ok ? pooled[o] : 0.0f;
    am[i] = ok ? argmax[o] : 0;
  }
  const float scale = open_range<SPLIT>(bound);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int cl = ty + 8 * i;
    const bool ok = at.live && c0 + cl < pg.c;
    const size_t plane = (chan0 + 8 * i) * hw + at.corner;
    const float v = pv[i] > 0.0f ? gv[i] : 0.0f;
    const int d = (int)((size_t)am[i] - plane);   // the winner from the window's corner: 0, 1, w, w + 1
    const int q = d >= w ? d - w + 2 : d;
    const float v0 = ok && q == 0 ? v : 0.0f, v1 = ok && q == 1 ? v : 0.0f, v2 = ok && q == 2 ? v : 0.0f, v3 = ok && q == 3 ? v : 0.0f;
    if (nchw_out && ok) {
      float* dst = nchw_out + plane;
      *reinterpret_cast<float2*>(dst) = make_float2(v0, v1);
      *reinterpret_cast<float2*>(dst + w) = make_float2(v2, v3);
    }
    float* t = &tile[cl][tx];
    t[0] = v0; t[32] = v1; t[64] = v2; t[96] = v3;
    if (chan_partial) {   // the window's four outputs sum to v: fixed-order butterfly over the 32 positions
      float sum = v;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, s);
      if (tx == 0 && c0 + cl < pg.c) chan_partial[(size_t)blockIdx.x * pg.c + c0 + cl] = sum;
    }
  }
  if (!hi) return;
  __syncthreads();
  const int cq = (threadIdx.x & 7) * 4, pl = threadIdx.x >> 3;   // (the channels of a tensor with planes are a multiple of 8)
  const long long base = pix_base[pl];
  if (c0 + cq >= pg.c || base < 0) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int k = q * 32 + pl;
    const float4 f = make_float4(tile[cq][k], tile[cq + 1][k], tile[cq + 2][k], tile[cq + 3][k]);
    const size_t o = ((size_t)base + (size_t)(q >> 1) * w + (q & 1)) * pg.c + c0 + cq;
    if (SPLIT) pr::put4(hi, lo, o, f, scale);
    else *reinterpret_cast<float4*>(hi + o) = make_float4(tc::tf32_rn(f.x), tc::tf32_rn(f.y), tc::tf32_rn(f.z), tc::tf32_rn(f.w));
  }
}

// 2x2 / stride-2 max-pool forward that also writes the pooled output's NHWC planes (the next convolution's operand), in
// the same tiles; the first maximum in row-major window order wins and argmax is the flat input index, as in
// maxpool2x2_fwd_kernel.
template <bool SPLIT>
__global__ void __launch_bounds__(256)
pool2_fwd_planes_kernel(const float* __restrict__ x, float* __restrict__ y, int32_t* __restrict__ argmax,
                        float* __restrict__ hi, float* __restrict__ lo, const PoolGrid pg, const Bound bound) {
  __shared__ float tile[32][33];
  const uint32_t gp0 = blockIdx.x * 32u;
  const int c0 = blockIdx.y * 32, w = pg.w, hw = pg.h * w, ohw = hw >> 2;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const PoolPlace at(pg, gp0 + tx);
  NRS_PDL_PROLOGUE();
  const size_t chan0 = (size_t)at.img * pg.c + c0 + ty;
  float2 r0[4], r1[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float* s = x + (chan0 + 8 * i) * hw + at.corner;
    const bool ok = at.live && c0 + ty + 8 * i < pg.c;
    r0[i] = ok ? *reinterpret_cast<const float2*>(s) : make_float2(0.0f, 0.0f);
    r1[i] = ok ? *reinterpret_cast<const float2*>(s + w) : make_float2(0.0f, 0.0f);
  }
  const float scale = open_range<SPLIT>(bound);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const size_t first = (chan0 + 8 * i) * hw + at.corner;
    float best = r0[i].x;
    size_t bi = first;
    if (r0[i].y > best) { best = r0[i].y; bi = first + 1; }
    if (r1[i].x > best) { best = r1[i].x; bi = first + w; }
    if (r1[i].y > best) { best = r1[i].y; bi = first + w + 1; }
    if (at.live && c0 + ty + 8 * i < pg.c) {
      const size_t o = (chan0 + 8 * i) * ohw + at.po;
      y[o] = best;
      if (argmax) argmax[o] = (int32_t)bi;
    }
    tile[ty + 8 * i][tx] = best;
  }
  __syncthreads();
  const int cq = (threadIdx.x & 7) * 4, pl = threadIdx.x >> 3;
  if (c0 + cq >= pg.c || gp0 + pl >= pg.positions) return;
  const float4 f = make_float4(tile[cq][pl], tile[cq + 1][pl], tile[cq + 2][pl], tile[cq + 3][pl]);
  const size_t o = (size_t)(gp0 + pl) * pg.c + c0 + cq;
  if (SPLIT) pr::put4(hi, lo, o, f, scale);
  else *reinterpret_cast<float4*>(hi + o) = make_float4(tc::tf32_rn(f.x), tc::tf32_rn(f.y), tc::tf32_rn(f.z), tc::tf32_rn(f.w));
}

}  // namespace

static unsigned absmax_blocks(const nrs_ctx* ctx, size_t count) {
  const size_t blocks = (count / 4 + 255) / 256 + 1, cap = (size_t)ctx->sm_count * 8;
  return (unsigned)(blocks < cap ? blocks : cap);
}
int nrs_absmax(nrs_ctx* ctx, const float* src, size_t count, NrsRange* r) {
  if (count == 0) return NRS_OK;
  MeasuredSet set{};
  set.m[0] = Measured{src, count, r};
  NRS_PDL_LAUNCH(absmax_kernel, absmax_blocks(ctx, count), 256, 0, ctx->stream, set);
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}
int nrs_absmax2(nrs_ctx* ctx, const float* a, size_t na, NrsRange* ra, const float* b, size_t nb, NrsRange* rb) {
  MeasuredSet set{};
  set.m[0] = Measured{a, na, ra};
  set.m[1] = Measured{b, nb, rb};
  NRS_PDL_LAUNCH(absmax_kernel, dim3(absmax_blocks(ctx, na > nb ? na : nb), 2), 256, 0, ctx->stream, set);
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}
int nrs_pair_unpack(nrs_ctx* ctx, const float* hi, const float* lo, float* dst, size_t n) {
  const NrsRange* range = nrs_range_of(ctx, hi);
  NRS_REQUIRE(ctx, range != nullptr, NRS_ERR_ARG, "f16 pairs without a range");
  if (n == 0) return NRS_OK;
  NRS_PDL_LAUNCH(pair_unpack_kernel, absmax_blocks(ctx, n), 256, 0, ctx->stream, hi, lo, range, dst, n);
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

// A fresh range for `hi` (or the caller's, measured), and where its bound comes from: the source's own where `known` has
// it, a scan by the staging kernel's blocks for small sources, else a launch that measures.
static int open_planes(nrs_ctx* ctx, const float* hi, const float* src, size_t count, const NrsRange* known, Bound* b) {
  *b = Bound{nullptr, src, 0, nullptr};
  if (!known && !ctx->known_tops.empty()) {
    auto it = ctx->known_tops.find(src);
    if (it != ctx->known_tops.end()) known = it->second;
  }
  int st = nrs_range_renew(ctx, hi, &b->range);
  if (st != NRS_OK) return st;
  b->top = known ? &known->top : &b->range->top;
  if (known) return NRS_OK;
  if (count > (size_t)pr::kScanAlone) return nrs_absmax(ctx, src, count, b->range);
  b->top = nullptr;
  b->scan_n = (int)count;
  return NRS_OK;
}

int nrs_tc_pool2_fwd_planes(nrs_ctx* ctx, const float* x, float* y, int32_t* argmax, float* hi, float* lo, int n, int c,
                            int h, int w, const NrsRange* x_range) {
  if (n <= 0 || c <= 0) return NRS_OK;
  if (h % 2 != 0 || w % 2 != 0 || !hi || (reinterpret_cast<uintptr_t>(x) & 7) != 0) return NRS_ERR_UNSUPPORTED;
  if (h == 0 || w == 0 || !PoolGrid::fits(n, c, h, w) || (c + 31) / 32 > 65535) return NRS_ERR_UNSUPPORTED;
  const PoolGrid pg(n, c, h, w);
  const dim3 grid = pg.blocks();
  Bound bound{};
  if (lo) {
    const int st = open_planes(ctx, hi, x, (size_t)n * c * h * w, x_range, &bound);
    if (st != NRS_OK) return st;
    NRS_PDL_LAUNCH((pool2_fwd_planes_kernel<true>), grid, 256, 0, ctx->stream, x, y, argmax, hi, lo, pg, bound);
  } else {
    NRS_PDL_LAUNCH((pool2_fwd_planes_kernel<false>), grid, 256, 0, ctx->stream, x, y, argmax, hi, nullptr, pg, bound);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_tc_stage_masked(nrs_ctx* ctx, int mode, const float* g, const float* y, const int32_t* argmax, int n, int c,
                        int h, int w, int k, float* nchw_out, float* hi, float* lo, float* chan_partial,
                        int* chan_partial_rows, const NrsRange* g_range) {
  if (chan_partial_rows) *chan_partial_rows = 0;
  if (n <= 0 || c <= 0) return NRS_OK;
  const int oh = mode == 1 ? h / k : h, ow = mode == 1 ? w / k : w;
  dim3 grid((unsigned)((h * w + 31) / 32), (unsigned)((c + 31) / 32), (unsigned)n);
  if (grid.y > 65535 || grid.z > 65535) return NRS_ERR_UNSUPPORTED;
  const bool split = lo != nullptr;
  Bound bound{};
  if (split) {
    const int st = open_planes(ctx, hi, g, (size_t)n * c * oh * ow, g_range, &bound);
    if (st != NRS_OK) return st;
  }
  if (mode == 1 && k == 2 && h % 2 == 0 && w % 2 == 0 && h > 0 && w > 0 && PoolGrid::fits(n, c, h, w)) {
    const PoolGrid pg(n, c, h, w);
    const dim3 pgrid = pg.blocks();
    if (split) NRS_PDL_LAUNCH((pool2_bwd_planes_kernel<true>), pgrid, 256, 0, ctx->stream, g, y, argmax, nchw_out, hi, lo, chan_partial, pg, bound);
    else NRS_PDL_LAUNCH((pool2_bwd_planes_kernel<false>), pgrid, 256, 0, ctx->stream, g, y, argmax, nchw_out, hi, lo, chan_partial, pg, bound);
    NRS_LAUNCHED(ctx);
    if (chan_partial && chan_partial_rows) *chan_partial_rows = (int)pgrid.x;
    return NRS_OK;
  }
#define NRS_MASKED(S, M) NRS_PDL_LAUNCH((stage_masked_kernel<S, M>), grid, 256, 0, ctx->stream, g, y, argmax, nchw_out, hi, lo, c, h, w, k, oh, ow, bound)
  if (mode == 0) { if (split) NRS_MASKED(true, 0); else NRS_MASKED(false, 0); }
  else { if (split) NRS_MASKED(true, 1); else NRS_MASKED(false, 1); }
#undef NRS_MASKED
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

static int stage(nrs_ctx* ctx, const Sources& src, float* hi, float* lo, int rows, int K, int ldk, int batch, size_t dst_bstride, bool src_k_by_rows,
                 const Bound& bound, const float* also, size_t also_count, NrsRange* also_range) {
  if (!src_k_by_rows) {
    size_t blocks = ((size_t)rows * (ldk / 4) + 255) / 256;
    const size_t cap = (size_t)ctx->sm_count * 16;
    if (blocks > cap) blocks = cap;
    if (batch > 65535) return NRS_ERR_UNSUPPORTED;
    Also more{};
    if (also && lo && batch == 1) more = Also{also, also_count, also_range, absmax_blocks(ctx, also_count)};
    dim3 grid((unsigned)blocks + more.blocks, (unsigned)batch);
    if (lo) NRS_PDL_LAUNCH((stage_rows_kernel<true>), grid, 256, 0, ctx->stream, src, hi, lo, rows, K, ldk, dst_bstride, NrsFastDiv(ldk / 4), bound, more);
    else NRS_PDL_LAUNCH((stage_rows_kernel<false>), grid, 256, 0, ctx->stream, src, hi, nullptr, rows, K, ldk, dst_bstride, NrsFastDiv(ldk / 4), bound, more);
  } else {
    dim3 grid((unsigned)((rows + 31) / 32), (unsigned)((ldk + 31) / 32), (unsigned)batch);
    if (grid.y > 65535 || grid.z > 65535) return NRS_ERR_UNSUPPORTED;
    if (lo) NRS_PDL_LAUNCH((stage_transpose_kernel<true>), grid, 256, 0, ctx->stream, src, hi, lo, rows, K, ldk, dst_bstride, bound);
    else NRS_PDL_LAUNCH((stage_transpose_kernel<false>), grid, 256, 0, ctx->stream, src, hi, nullptr, rows, K, ldk, dst_bstride, bound);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_tc_stage(nrs_ctx* ctx, const float* src, float* hi, float* lo, int rows, int K, int ldk, int batch,
                 size_t src_bstride, size_t dst_bstride, bool src_k_by_rows, const NrsRange* known,
                 const float* also, size_t also_count, NrsRange* also_range) {
  if (rows <= 0 || K <= 0 || batch <= 0) return NRS_OK;
  Bound bound{};
  if (lo) {
    const int st = open_planes(ctx, hi, src, batch == 1 ? (size_t)rows * K : src_bstride * (batch - 1) + (size_t)rows * K, known, &bound);
    if (st != NRS_OK) return st;
  }
  return stage(ctx, Sources(src, src_bstride), hi, lo, rows, K, ldk, batch, dst_bstride, src_k_by_rows, bound, also, also_count, also_range);
}

int nrs_tc_stage_each(nrs_ctx* ctx, const float* const* src, int count, float* hi, float* lo, int rows, int K, int ldk, size_t dst_bstride,
                      bool src_k_by_rows) {
  if (rows <= 0 || K <= 0 || count <= 0) return NRS_OK;
  NrsRange* range = nullptr;
  if (lo) {
    const int st = nrs_range_renew(ctx, hi, &range);
    if (st != NRS_OK) return st;
    for (int i = 0; i < count; i += kSources) {
      MeasuredSet set{};
      const int n = std::min(count - i, kSources);
      for (int k = 0; k < n; ++k) set.m[k] = Measured{src[i + k], (size_t)rows * K, range};
      NRS_PDL_LAUNCH(absmax_kernel, dim3(absmax_blocks(ctx, (size_t)rows * K), n), 256, 0, ctx->stream, set);
      NRS_LAUNCHED(ctx);
    }
  }
  const Bound bound{range ? &range->top : nullptr, nullptr, 0, range};
  for (int i = 0; i < count; i += kSources) {
    Sources s(nullptr, 0);
    const int n = std::min(count - i, kSources);
    for (int k = 0; k < n; ++k) s.each[k] = src[i + k];
    const int st = stage(ctx, s, nrs_plane_at(hi, i * dst_bstride, lo != nullptr), lo ? nrs_plane_at(lo, i * dst_bstride, true) : nullptr, rows, K, ldk, n,
                         dst_bstride, src_k_by_rows, bound, nullptr, 0, nullptr);
    if (st != NRS_OK) return st;
  }
  return NRS_OK;
}

int nrs_tc_stage_image(nrs_ctx* ctx, const float* src, float* hi, float* lo, int n, int c, int hw, float* chan_partial,
                       const NrsRange* known) {
  if (n <= 0 || c <= 0 || hw <= 0) return NRS_OK;
  const int ld = nrs_plane_ld(c);
  if (hw == 1) return nrs_tc_stage(ctx, src, hi, lo, n, c, ld, 1, 0, 0, false, known);   // already pixel-major: split only
  if ((size_t)n * hw > 0x7fffffffu) return NRS_ERR_UNSUPPORTED;
  const img::Grid g(n, c, hw);
  Bound bound{};
  if (lo) {
    const int st = open_planes(ctx, hi, src, (size_t)n * c * hw, known, &bound);
    if (st != NRS_OK) return st;
  }
#define NRS_STAGE(S, C) NRS_PDL_LAUNCH((stage_image_kernel<S, C>), g.blocks(), 256, 0, ctx->stream, src, hi, lo, chan_partial, g, bound)
  if (lo) { if (chan_partial) NRS_STAGE(true, true); else NRS_STAGE(true, false); }
  else { if (chan_partial) NRS_STAGE(false, true); else NRS_STAGE(false, false); }
#undef NRS_STAGE
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_tc_stage_conv_weight(nrs_ctx* ctx, const float* w, float* hi, float* lo, int co, int ci, int kh, int kw,
                             int for_dgrad) {
  const size_t total = (size_t)(for_dgrad ? ci : co) * (((for_dgrad ? co : ci) + 31) / 32 * 32) * kh * kw;
  if (total == 0) return NRS_OK;
  Bound bound{};
  if (lo) {
    const int st = open_planes(ctx, hi, w, (size_t)co * ci * kh * kw, nullptr, &bound);
    if (st != NRS_OK) return st;
    const int threads = bound.scan_n > kWideScan ? kWideStage : 256;
    NRS_PDL_LAUNCH((stage_conv_weight_kernel<true>), nrs_blocks(total, threads), threads, 0, ctx->stream, w, hi, lo, co, ci, kh, kw, for_dgrad, bound);
  } else {
    NRS_PDL_LAUNCH((stage_conv_weight_kernel<false>), nrs_blocks(total, 256), 256, 0, ctx->stream, w, hi, nullptr, co, ci, kh, kw, for_dgrad, bound);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}
