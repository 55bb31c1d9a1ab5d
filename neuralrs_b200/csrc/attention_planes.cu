// Multi-head attention over TF32 operand planes: any sequence length up to 4096 and any head size that is a
// multiple of 8, where the one-CTA-per-head kernels (attention_tc.cu: 128 keys, 32 columns) end.
//
//   forward   S = Q K^T                 P = softmax(scale S, causal)      O = P V
//   backward  dP = dO V^T               dS = P o (dP - rowsum(dP o P)) scale
//             dV = P^T dO               dQ = dS K                         dK = dS^T Q
//
// Six products on the persistent tensor-core kernel (tc_mainloop.cuh) and two row kernels.  Nothing is transposed,
// permuted or masked in a pass of its own: the head slices of Q, K, V and of their gradients are addressed in place by
// 4-D tensor maps (columns, rows, head, sample) over the projections' planes, every operand is taken in the order it
// lies in memory (K-major, or MN-major where the reduction index is the slow one), a causal product neither computes
// the tiles above the diagonal nor walks the K-slices that are zero, and P, dS, O and the three gradients leave
// their kernels as the planes the next product reads.  HBM-bound by the [batch*heads][seq][seq] matrices: 4 B written
// and read per element for S and dP, 8 B for P and dS, half of it when causal.
//
// Measured on the 512-wide model (6 sequences of 500, 8 heads of 64, causal, 3xTF32), one layer forward + backward:
// 204 us (products 163, row kernels 41); with the permutations, transposes, scale, mask and softmax kernels that it
// replaces there, and Q, K, V as three products each way, a step of two layers took 0.92 ms more.  At 32 sequences of
// 128, 8 heads of 32: 96 us, where the one-CTA-per-head kernels take 107 and need K, V and the gradients unsplit.
//
// Replaces, per head, slice_cols x3 -> transpose -> bmm -> scale -> softmax -> bmm -> concat_cols of
// src/cuda/nn/multihead.rs:57-85 and src/cuda/nn/attention.rs:23-32.
#include "attention_planes.h"
#include "tc_mainloop.cuh"

namespace {

// A matrix per (sample, head): element (r, c) of head h of sample b at b*bs + h*hs + r*ld + c.
struct HeadMat {
  const float *hi, *lo;
  int cols, rows;      // extent of one head's matrix
  size_t ld, hs, bs;   // floats
};

// C[b][h] = scale * op(A) op(B).  AMN / BMN: that operand is stored with the reduction index slow.
template <bool AMN, bool BMN>
struct HeadPolicy {
  float* c;            // f32 result, or null
  float *hi, *lo;      // planes of the result, or null; same addressing
  size_t ldc, hs, bs;
  int M, N, heads;
  bool vec;            // rows start on 16 bytes
  // Causal products: kTiles: result tiles above the diagonal do not exist.  kUpTo: K-slices beyond the tile's last row
  // are zero.  kFrom: K-slices before the tile's first row are zero.
  enum { kDense = tc::kRaster, kTiles = tc::kTriangle, kUpTo = tc::kLastFirst, kFrom = tc::kFirstFirst };
  int causal;
  static constexpr bool kCanEmit = false, kMaySplit = false;
  static constexpr bool kAMnMajor = AMN, kBMnMajor = BMN;
  static constexpr int kEpiWarps = 16;
  int order() const { return causal; }   // the same numbers

  __device__ __forceinline__ bool clip(int tile_m, int tile_n, int bn, int* kb_begin, int* kb_end) const {
    if (causal == kUpTo) *kb_end = min(*kb_end, (tile_m * tc::BM + tc::BM) / tc::BK);
    if (causal == kFrom) *kb_begin = tile_m * tc::BM / tc::BK;
    return *kb_begin < *kb_end;
  }
  __device__ __forceinline__ uint32_t a_slice_bytes() const { return tc::BM * tc::BK * 4; }
  struct Cursor { int k, row, h, b; };
  __device__ __forceinline__ Cursor cursor(int tile_m, int batch, int kb) const {
    const int b = batch / heads;
    return Cursor{kb * tc::BK, tile_m * tc::BM, batch - b * heads, b};
  }
  __device__ __forceinline__ void advance(Cursor& c) const { c.k += tc::BK; }
  template <bool PAIR>
  __device__ __forceinline__ void load_a(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c) const {
    if (AMN) {
#pragma unroll
      for (int i = 0; i < tc::BM / 32; ++i) tc::tma_load_4d_to<PAIR>((uint8_t*)dst + i * 4096, tm, bar, c.row + 32 * i, c.k, c.h, c.b);
    } else {
      tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.k, c.row, c.h, c.b);
    }
  }
  template <int BN, bool PAIR>
  __device__ __forceinline__ void load_b(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c, int n0) const {
    if (BMN) {
#pragma unroll
      for (int i = 0; i < BN / 32; ++i) tc::tma_load_4d_to<PAIR>((uint8_t*)dst + i * 4096, tm, bar, n0 + 32 * i, c.k, c.h, c.b);
    } else {
      tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.k, n0, c.h, c.b);
    }
  }
  __device__ __forceinline__ int row(int, int, int) const { return 0; }
  __device__ __forceinline__ void store(int, int, int, int, float) const {}   // no K-split
  __device__ __forceinline__ void epilogue(int tile_m, int batch, int r0, int n, float4 (&v)[4]) const {
    const int b = batch / heads, m0 = tile_m * tc::BM + r0, nn = N - n;
    const size_t at0 = (size_t)b * bs + (size_t)(batch - b * heads) * hs + (size_t)m0 * ldc + n;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (m0 + 8 * i >= M) continue;
      const size_t at = at0 + (size_t)(8 * i) * ldc;
      if (c) tc::store_guarded(c + at, v[i], nn, vec);
      if (hi) {
        const float4 h = make_float4(tc::tf32_rn(v[i].x), tc::tf32_rn(v[i].y), tc::tf32_rn(v[i].z), tc::tf32_rn(v[i].w));
        tc::store_guarded(hi + at, h, nn, vec);
        if (lo) tc::store_guarded(lo + at, make_float4(v[i].x - h.x, v[i].y - h.y, v[i].z - h.z, v[i].w - h.w), nn, vec);
      }
    }
  }
};

// mn: box {32 columns, 32 rows}; else {32 columns, `rows` rows}.
bool head_map(CUtensorMap* t, const float* p, const HeadMat& m, int heads, int batch, bool mn, int rows) {
  const uint64_t dim[4] = {(uint64_t)m.cols, (uint64_t)m.rows, (uint64_t)heads, (uint64_t)batch};
  const uint64_t str[3] = {m.ld * 4, m.hs * 4, m.bs * 4};
  const uint32_t box[4] = {32, (uint32_t)(mn ? tc::BK : rows), 1, 1};
  return tc::encode_tmap_f32(t, p, 4, dim, str, box, mn);
}

template <int BN, int NPLANES, bool AMN, bool BMN>
int run(nrs_ctx* ctx, const HeadMat& A, const HeadMat& B, const HeadPolicy<AMN, BMN>& pol, int batch, int k) {
  CUtensorMap a_hi, a_lo, b_hi, b_lo;
  bool ok = head_map(&a_hi, A.hi, A, pol.heads, batch, AMN, tc::BM) && head_map(&b_hi, B.hi, B, pol.heads, batch, BMN, BN);
  if (NPLANES == 2) ok = ok && head_map(&a_lo, A.lo, A, pol.heads, batch, AMN, tc::BM) && head_map(&b_lo, B.lo, B, pol.heads, batch, BMN, BN);
  else { a_lo = a_hi; b_lo = b_hi; }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed");
  return tc::launch<BN, NPLANES, false, HeadPolicy<AMN, BMN>>(ctx, a_hi, a_lo, b_hi, b_lo, pol, (pol.M + tc::BM - 1) / tc::BM, pol.N,
                                                       batch * pol.heads, (k + tc::BK - 1) / tc::BK);
}

struct Out {
  float *c, *hi, *lo;
  size_t ld, hs, bs;
};

template <bool AMN, bool BMN>
int product(nrs_ctx* ctx, const HeadMat& A, const HeadMat& B, const Out& o, int batch, int heads, int m, int n, int k, int causal) {
  auto ok16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  HeadPolicy<AMN, BMN> pol{o.c, o.hi, o.lo, o.ld, o.hs, o.bs, m, n, heads, false, causal};
  pol.vec = o.ld % 4 == 0 && o.hs % 4 == 0 && o.bs % 4 == 0 && ok16(o.c) && ok16(o.hi) && ok16(o.lo);
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  NrsProfScope prof(ctx, NRS_PROF_GEMM, 2.0 * batch * heads * m * n * k * (causal ? 0.5 : 1.0));
  if (n > 64) return split ? run<128, 2, AMN, BMN>(ctx, A, B, pol, batch, k) : run<128, 1, AMN, BMN>(ctx, A, B, pol, batch, k);
  if (n > 32) return split ? run<64, 2, AMN, BMN>(ctx, A, B, pol, batch, k) : run<64, 1, AMN, BMN>(ctx, A, B, pol, batch, k);
  return split ? run<32, 2, AMN, BMN>(ctx, A, B, pol, batch, k) : run<32, 1, AMN, BMN>(ctx, A, B, pol, batch, k);
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
__device__ __forceinline__ void put_planes(float* hi, float* lo, size_t at, float4 v) {
  const float4 h = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
  *reinterpret_cast<float4*>(hi + at) = h;
  if (lo) *reinterpret_cast<float4*>(lo + at) = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
}
// Columns of row i that the products reading P and dS touch: all (ld), or up to the end of the row's 128-row tile.
__device__ __forceinline__ int row_extent(int i, int ld, int causal) { return causal ? min(ld, (i / tc::BM + 1) * tc::BM) : ld; }

// P = softmax(scale * S) over the keys j < seq (j <= i when causal), as planes, zeros in the row's other columns.  One
// warp per row, kept in registers (VPL float4s per lane) up to 1024 columns, else read twice more from L2.
template <int VPL>
__global__ void __launch_bounds__(256)
head_softmax_kernel(const float* __restrict__ s, float* __restrict__ hi, float* __restrict__ lo, long rows, int seq, int ld, int causal,
                    float scale) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31;
  for (long r = (long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long)gridDim.x * 8) {
    const int i = (int)(r % seq), live = causal ? i + 1 : seq, ext = row_extent(i, ld, causal);
    const float* src = s + (size_t)r * ld;
    float4 v[VPL];
    float mx = -INFINITY, sum = 0.0f;
    auto fetch = [&](int c) {   // four columns from c; -inf where there is no key
      float4 t = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
      if (c >= live) return t;
      t = *reinterpret_cast<const float4*>(src + c);
      t.x *= scale; t.y *= scale; t.z *= scale; t.w *= scale;
      if (c + 1 >= live) t.y = -INFINITY;
      if (c + 2 >= live) t.z = -INFINITY;
      if (c + 3 >= live) t.w = -INFINITY;
      return t;
    };
    auto exp4 = [&](float4 t) { return make_float4(expf(t.x - mx), expf(t.y - mx), expf(t.z - mx), expf(t.w - mx)); };
    if (VPL > 1 || ld <= 128) {
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        v[k] = fetch(4 * (lane + 32 * k));
        mx = fmaxf(mx, fmaxf(fmaxf(v[k].x, v[k].y), fmaxf(v[k].z, v[k].w)));
      }
      mx = wmax(mx);
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        v[k] = exp4(v[k]);
        sum += (v[k].x + v[k].y) + (v[k].z + v[k].w);
      }
      const float inv = 1.0f / wsum(sum);
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int c = 4 * (lane + 32 * k);
        if (c < ext) put_planes(hi, lo, (size_t)r * ld + c, make_float4(v[k].x * inv, v[k].y * inv, v[k].z * inv, v[k].w * inv));
      }
    } else {
      for (int c = 4 * lane; c < live; c += 128) {
        const float4 t = fetch(c);
        mx = fmaxf(mx, fmaxf(fmaxf(t.x, t.y), fmaxf(t.z, t.w)));
      }
      mx = wmax(mx);
      for (int c = 4 * lane; c < live; c += 128) {
        const float4 t = exp4(fetch(c));
        sum += (t.x + t.y) + (t.z + t.w);
      }
      const float inv = 1.0f / wsum(sum);
      for (int c = 4 * lane; c < ext; c += 128) {
        const float4 t = exp4(fetch(c));
        put_planes(hi, lo, (size_t)r * ld + c, make_float4(t.x * inv, t.y * inv, t.z * inv, t.w * inv));
      }
    }
  }
}

// dS = P o (dP - sum_j dP_j P_j) * scale as planes; P exact from its planes.  (Columns without a key have P = 0.)
template <int VPL>
__global__ void __launch_bounds__(256)
head_dsoftmax_kernel(const float* __restrict__ p_hi, const float* __restrict__ p_lo, const float* __restrict__ dp, float* __restrict__ hi,
                     float* __restrict__ lo, long rows, int seq, int ld, int causal, float scale) {
  NRS_PDL_PROLOGUE();
  const int lane = threadIdx.x & 31;
  for (long r = (long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long)gridDim.x * 8) {
    const int i = (int)(r % seq), live = causal ? i + 1 : seq, ext = row_extent(i, ld, causal);
    const size_t base = (size_t)r * ld;
    float dot = 0.0f;
    auto fetch = [&](int c, float4* p, float4* d) {
      *p = *d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c >= live) return;
      *p = *reinterpret_cast<const float4*>(p_hi + base + c);
      if (p_lo) {
        const float4 l = *reinterpret_cast<const float4*>(p_lo + base + c);
        p->x += l.x; p->y += l.y; p->z += l.z; p->w += l.w;
      }
      *d = *reinterpret_cast<const float4*>(dp + base + c);
      if (c + 1 >= live) d->y = 0.0f;   // (never written there)
      if (c + 2 >= live) d->z = 0.0f;
      if (c + 3 >= live) d->w = 0.0f;
    };
    auto dsoft = [&](float4 p, float4 d) {
      return make_float4(p.x * (d.x - dot) * scale, p.y * (d.y - dot) * scale, p.z * (d.z - dot) * scale, p.w * (d.w - dot) * scale);
    };
    if (VPL > 1 || ld <= 128) {
      float4 p[VPL], d[VPL];
#pragma unroll
      for (int k = 0; k < VPL; ++k) fetch(4 * (lane + 32 * k), &p[k], &d[k]);
#pragma unroll
      for (int k = 0; k < VPL; ++k) dot += (p[k].x * d[k].x + p[k].y * d[k].y) + (p[k].z * d[k].z + p[k].w * d[k].w);
      dot = wsum(dot);
#pragma unroll
      for (int k = 0; k < VPL; ++k) {
        const int c = 4 * (lane + 32 * k);
        if (c < ext) put_planes(hi, lo, base + c, dsoft(p[k], d[k]));
      }
    } else {
      float4 p, d;
      for (int c = 4 * lane; c < live; c += 128) {
        fetch(c, &p, &d);
        dot += (p.x * d.x + p.y * d.y) + (p.z * d.z + p.w * d.w);
      }
      dot = wsum(dot);
      for (int c = 4 * lane; c < ext; c += 128) {
        fetch(c, &p, &d);
        put_planes(hi, lo, base + c, dsoft(p, d));
      }
    }
  }
}

int row_blocks(const nrs_ctx* ctx, long rows) {
  const long b = (rows + 7) / 8, cap = (long)ctx->sm_count * 16;
  return (int)(b < cap ? b : cap);
}

// VPL by row length: 1 (128 columns), 2, 4, 8; 1 again, as the looping form, beyond 1024.
#define NRS_HEAD_VPL(ld, CALL)                              \
  do {                                                      \
    if ((ld) <= 128 || (ld) > 1024) { constexpr int V = 1; CALL; } \
    else if ((ld) <= 256) { constexpr int V = 2; CALL; }    \
    else if ((ld) <= 512) { constexpr int V = 4; CALL; }    \
    else { constexpr int V = 8; CALL; }                     \
  } while (0)

}  // namespace

bool nrs_mha_planes_applies(const nrs_ctx* ctx, int seq, int d_head) {
  return ctx->math_mode != NRS_MATH_FP32 && tc::tensor_map_encoder() && seq >= 1 && seq <= tc::kMaxChainK && d_head >= 8 && d_head % 8 == 0;
}

int nrs_mha_planes_fwd(nrs_ctx* ctx, const NrsMhaPlanes& a) {
  const int S = a.seq, dh = a.d_head, ld = nrs_plane_ld(S);
  const size_t ss = (size_t)S * ld;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  auto head = [&](int part) {   // 0 Q, 1 K, 2 V inside the projections' planes
    const size_t o = (size_t)part * a.heads * dh;
    return HeadMat{a.qkv_hi + o, split ? a.qkv_lo + o : nullptr, dh, S, (size_t)a.qkv_ld, (size_t)dh, (size_t)S * a.qkv_ld};
  };
  using P = HeadPolicy<false, false>;
  int st = product<false, false>(ctx, head(0), head(1), Out{a.scores, nullptr, nullptr, (size_t)ld, ss, ss * a.heads}, a.batch, a.heads, S, S, dh,
                                 a.causal ? P::kTiles : P::kDense);
  if (st != NRS_OK) return st;
  const long rows = (long)a.batch * a.heads * S;
  const float scale = 1.0f / sqrtf((float)dh);
  NRS_HEAD_VPL(ld, NRS_PDL_LAUNCH(head_softmax_kernel<V>, row_blocks(ctx, rows), 256, 0, ctx->stream, (const float*)a.scores, a.p_hi, a.p_lo, rows,
                                  S, ld, a.causal, scale));
  NRS_LAUNCHED(ctx);
  const HeadMat p{a.p_hi, a.p_lo, ld, S, (size_t)ld, ss, ss * a.heads};
  const size_t D = (size_t)a.heads * dh;
  return product<false, true>(ctx, p, head(2), Out{a.out, a.out_hi, a.out_lo, D, (size_t)dh, (size_t)S * D}, a.batch, a.heads, S, dh, S,
                              a.causal ? P::kUpTo : P::kDense);
}

int nrs_mha_planes_bwd(nrs_ctx* ctx, const NrsMhaPlanes& a) {
  const int S = a.seq, dh = a.d_head, ld = nrs_plane_ld(S);
  const size_t ss = (size_t)S * ld, D = (size_t)a.heads * dh;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  auto head = [&](int part) {
    const size_t o = (size_t)part * D;
    return HeadMat{a.qkv_hi + o, split ? a.qkv_lo + o : nullptr, dh, S, (size_t)a.qkv_ld, (size_t)dh, (size_t)S * a.qkv_ld};
  };
  auto grad = [&](int part) {
    const size_t o = (size_t)part * D;
    return Out{nullptr, a.dqkv_hi + o, split ? a.dqkv_lo + o : nullptr, 3 * D, (size_t)dh, (size_t)S * 3 * D};
  };
  using P = HeadPolicy<false, false>;
  const HeadMat dout{a.dout_hi, a.dout_lo, dh, S, D, (size_t)dh, (size_t)S * D};
  const HeadMat p{a.p_hi, a.p_lo, ld, S, (size_t)ld, ss, ss * a.heads};
  int st = product<false, false>(ctx, dout, head(2), Out{a.scores, nullptr, nullptr, (size_t)ld, ss, ss * a.heads}, a.batch, a.heads, S, S, dh,
                                 a.causal ? P::kTiles : P::kDense);
  if (st == NRS_OK) st = product<true, true>(ctx, p, dout, grad(2), a.batch, a.heads, S, dh, S, a.causal ? P::kFrom : P::kDense);
  if (st != NRS_OK) return st;
  const long rows = (long)a.batch * a.heads * S;
  const float scale = 1.0f / sqrtf((float)dh);
  NRS_HEAD_VPL(ld, NRS_PDL_LAUNCH(head_dsoftmax_kernel<V>, row_blocks(ctx, rows), 256, 0, ctx->stream, (const float*)a.p_hi, (const float*)a.p_lo,
                                  (const float*)a.scores, a.ds_hi, a.ds_lo, rows, S, ld, a.causal, scale));
  NRS_LAUNCHED(ctx);
  const HeadMat ds{a.ds_hi, a.ds_lo, ld, S, (size_t)ld, ss, ss * a.heads};
  st = product<false, true>(ctx, ds, head(1), grad(0), a.batch, a.heads, S, dh, S, a.causal ? P::kUpTo : P::kDense);
  if (st == NRS_OK) st = product<true, true>(ctx, ds, head(0), grad(1), a.batch, a.heads, S, dh, S, a.causal ? P::kFrom : P::kDense);
  return st;
}
