// Convolutions over few input channels on the tensor cores, through patch planes.
//
// With K = c_in*kh*kw of a few dozen (an image layer: 9 or 27) the contraction is too short for one
// 32-channel K-block per filter tap.  The input is written out once as [output pixels][K] operand planes
// (the K values under each output pixel, in the order of a weight's row), which makes the layer a 1x1
// convolution over K channels: its forward pass and its weight gradient then run on the general
// tensor-core kernels, whose B operand is the weight as it is stored ([co][K]) and whose result is the
// weight gradient as it is stored.  HBM-bound: 4*K or 8*K bytes per output pixel, written once per step.
// The data gradient reads no patches (tc_conv.cu).
//
// Reference counterparts: conv2d_im2col + matmul_nn + col2out and im2col + matmul_nt_splitk
// (src/cuda/nn/conv.rs:244-320).
#include "fold.h"
#include "igemm_problems.cuh"
#include "nrs_internal.h"
#include "pair.cuh"
#include "tc_common.cuh"

namespace {

constexpr int kMaxPatch = 128;

// A thread owns four consecutive values of one pixel's patch: 128-bit stores, consecutive threads
// consecutive addresses; the four gathers hit L1 (neighbouring pixels share their input rows).
template <bool SPLIT>
__global__ void __launch_bounds__(256)
patch_planes_kernel(const float* __restrict__ x, float* __restrict__ hi, float* __restrict__ lo, const NrsConvGeom g, int kh,
                    int kw, const NrsFastDiv div_quads, uint32_t total /*pixels * (row length / 4)*/, int scan_n, NrsRange* range) {
  __shared__ int off[kMaxPatch];        // offset of patch value k from the patch's origin
  __shared__ short2 tap[kMaxPatch];     // its (row, column) inside the window
  const int K = g.ci * kh * kw;
  for (int k = threadIdx.x; k < K; k += blockDim.x) {
    const int c = k / (kh * kw), t = k - c * kh * kw, i = t / kw, j = t - i * kw;
    off[k] = (c * g.h + i) * g.w + j;
    tap[k] = make_short2((short)i, (short)j);
  }
  __syncthreads();
  NRS_PDL_PROLOGUE();   // (the tables are made ahead of the wait)
  const float scale = SPLIT ? pr::open_range(scan_n > 0 ? nullptr : &range->top, x, scan_n, range) : 1.0f;
  const int ld = nrs_plane_ld(K);
  const uint32_t stride = gridDim.x * blockDim.x;
  for (uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x; idx < total; idx += stride) {
    uint32_t p32, kq, img, pix, oy, ox;
    div_quads.divmod(idx, p32, kq);
    const size_t p = p32;
    const int k0 = (int)kq * 4;
    g.div_ohow.divmod(p32, img, pix);
    g.div_ow.divmod(pix, oy, ox);
    const int iy0 = (int)oy * g.stride - g.pad, ix0 = (int)ox * g.stride - g.pad;
    const float* src = x + (size_t)img * g.ci * g.h * g.w + (long)iy0 * g.w + ix0;
    float v[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = 0.0f;
      if (k0 + e < K) {
        const short2 t = tap[k0 + e];
        if ((unsigned)(iy0 + t.x) < (unsigned)g.h && (unsigned)(ix0 + t.y) < (unsigned)g.w) v[e] = src[off[k0 + e]];
      }
    }
    if (SPLIT) pr::put4(hi, lo, p * ld + k0, make_float4(v[0], v[1], v[2], v[3]), scale);
    else *reinterpret_cast<float4*>(hi + p * ld + k0) = make_float4(tc::tf32_rn(v[0]), tc::tf32_rn(v[1]), tc::tf32_rn(v[2]), tc::tf32_rn(v[3]));
  }
}

// The patch planes of x for a layer: the caller's registered ones, or fresh ones in pool blocks given back at the
// end of the scope.
struct Patches {
  nrs_ctx* ctx;
  float *hi = nullptr, *lo = nullptr;
  bool owned = false;
  explicit Patches(nrs_ctx* c) : ctx(c) {}
  int get(const float* x, int n, int ci, int h, int wd, int kh, int kw, int stride, int pad) {
    const bool split = ctx->math_mode == NRS_MATH_3XTF32;
    auto it = ctx->patch_hints.find(x);
    if (it != ctx->patch_hints.end()) {
      const NrsPatchPlanes& q = it->second;
      if ((q.lo != nullptr) == split && q.kh == kh && q.kw == kw && q.stride == stride && q.pad == pad) {
        hi = q.hi;
        lo = q.lo;
        return NRS_OK;
      }
    }
    const NrsConvGeom g(n, ci, h, wd, 1, kh, kw, stride, pad);
    const size_t bytes = (size_t)n * g.oh * g.ow * nrs_plane_ld(ci * kh * kw) * (split ? 2 : 4);
    void *phi = nullptr, *plo = nullptr;
    int st = nrs_alloc(ctx, bytes, 0, &phi);
    if (st != NRS_OK) return st;
    owned = true;
    hi = (float*)phi;
    if (split) {
      st = nrs_alloc(ctx, bytes, 0, &plo);
      if (st != NRS_OK) return st;
      lo = (float*)plo;
    }
    return nrs_patch_planes(ctx, x, hi, lo, n, ci, h, wd, kh, kw, stride, pad);
  }
  ~Patches() {
    if (!owned) return;
    nrs_free_after_wgrads(ctx, hi);
    if (lo) nrs_free_after_wgrads(ctx, lo);
  }
};

}  // namespace

int nrs_patch_planes(nrs_ctx* ctx, const float* x, float* hi, float* lo, int n, int ci, int h, int wd, int kh, int kw, int stride,
                     int pad) {
  if (!nrs_conv_uses_patches(ci, kh, kw)) return NRS_ERR_UNSUPPORTED;
  const NrsConvGeom g(n, ci, h, wd, 1, kh, kw, stride, pad);
  const int quads = nrs_plane_ld(ci * kh * kw) / 4;
  const size_t total = (size_t)n * g.oh * g.ow * quads;
  if (total >= (1ull << 31) - (1u << 20)) return NRS_ERR_UNSUPPORTED;
  size_t blocks = (total + 255) / 256;
  const size_t cap = (size_t)ctx->sm_count * 16;
  if (blocks > cap) blocks = cap;
  NrsRange* range = nullptr;
  int scan_n = 0;
  if (lo) {
    int st = nrs_range_renew(ctx, hi, &range);
    const size_t count = (size_t)n * ci * h * wd;
    if (count <= (size_t)pr::kScanAlone) scan_n = (int)count;
    else if (st == NRS_OK) st = nrs_absmax(ctx, x, count, range);
    if (st != NRS_OK) return st;
  }
  if (lo) NRS_PDL_LAUNCH((patch_planes_kernel<true>), (unsigned)blocks, 256, 0, ctx->stream, x, hi, lo, g, kh, kw, NrsFastDiv(quads), (uint32_t)total, scan_n, range);
  else NRS_PDL_LAUNCH((patch_planes_kernel<false>), (unsigned)blocks, 256, 0, ctx->stream, x, hi, nullptr, g, kh, kw, NrsFastDiv(quads), (uint32_t)total, scan_n, range);
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_patch_conv_fwd(nrs_ctx* ctx, const float* x, const float* w, const float* b, float* y, int n, int ci, int h, int wd, int co,
                       int kh, int kw, int stride, int pad, int act) {
  if (!nrs_conv_uses_patches(ci, kh, kw) || !tc::tensor_map_encoder()) return NRS_ERR_UNSUPPORTED;
  const NrsConvGeom g(n, ci, h, wd, co, kh, kw, stride, pad);
  Patches p(ctx);
  int st = p.get(x, n, ci, h, wd, kh, kw, stride, pad);
  if (st != NRS_OK) return st;
  ctx->plane_hints[p.hi] = NrsPlanes{p.hi, p.lo, p.lo ? 1 : 0};
  st = nrs_tc_conv_fwd(ctx, p.hi, w, b, y, n, ci * kh * kw, g.oh, g.ow, co, 1, 1, 1, 0, act);
  ctx->plane_hints.erase(p.hi);
  return st;
}

int nrs_patch_conv_wgrad(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co, int kh, int kw,
                         int stride, int pad, int accumulate) {
  if (!nrs_conv_uses_patches(ci, kh, kw) || !tc::tensor_map_encoder()) return NRS_ERR_UNSUPPORTED;
  const NrsConvGeom g(n, ci, h, wd, co, kh, kw, stride, pad);
  Patches p(ctx);
  int st = p.get(x, n, ci, h, wd, kh, kw, stride, pad);
  if (st != NRS_OK) return st;
  if (p.owned) ctx->independent_next = false;   // the patches were written by the kernel just launched
  ctx->plane_hints[p.hi] = NrsPlanes{p.hi, p.lo, p.lo ? 1 : 0};
  st = nrs_tc_conv_wgrad(ctx, p.hi, dy, dw, n, ci * kh * kw, g.oh, g.ow, co, 1, 1, 1, 0, accumulate);
  ctx->plane_hints.erase(p.hi);
  return st;
}
