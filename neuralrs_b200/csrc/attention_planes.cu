// Multi-head attention over operand planes (f16 pairs, or TF32 values): any sequence length up to 4096 and any head size that is a
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
// and read per element of each of S, dP, P and dS (two halves of a pair, or a TF32 value), half of it when causal.
//
// Measured before f16 pairs, on the 512-wide model (6 sequences of 500, 8 heads of 64, causal, 3xTF32), one layer forward + backward:
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
  size_t ld, hs, bs;   // values
  const NrsRange* range;   // 3xTF32
};

// C[b][h] = scale * op(A) op(B).  AMN / BMN: that operand is stored with the reduction index slow.
template <bool AMN, bool BMN>
struct HeadPolicy {
  float* c;            // f32 result, or null
  float *hi, *lo;      // planes of the result, or null; same addressing
  size_t ldc, hs, bs;
  int M, N, heads;
  NrsFastDiv div_heads;
  bool vec;            // rows start on 16 bytes
  // Causal products: kTiles: result tiles above the diagonal do not exist.  kUpTo: K-slices beyond the tile's last row
  // are zero.  kFrom: K-slices before the tile's first row are zero.
  enum { kDense = tc::kRaster, kTiles = tc::kTriangle, kUpTo = tc::kLastFirst, kFrom = tc::kFirstFirst };
  int causal;
  // 3xTF32, planes: no result exceeds factor * the larger of r0 and r1 * r2 (null: 0)
  float factor;
  const NrsRange *r0, *r1, *r2;
  static constexpr bool kCanEmit = false, kMaySplit = false;
  static constexpr bool kAMnMajor = AMN, kBMnMajor = BMN;
  static constexpr int kEpiWarps = 16, kTeamWarps = 4;
  static constexpr bool kConv = false;
  static constexpr bool kSlab = false;
  int order() const { return causal; }   // the same numbers
  __device__ __forceinline__ float out_bound(float, float, int) const {
    return fminf(factor * fmaxf(r0 ? r0->top : 0.0f, r1 ? r1->top * r2->top : 0.0f), 3.0e38f);
  }

  __device__ __forceinline__ bool clip(int tile_m, int tile_n, int bn, int* kb_begin, int* kb_end) const {
    if (causal == kUpTo) *kb_end = min(*kb_end, (tile_m * tc::BM + tc::BM) / tc::BK);
    if (causal == kFrom) *kb_begin = tile_m * tc::BM / tc::BK;
    return *kb_begin < *kb_end;
  }
  __device__ __forceinline__ uint32_t a_slice_rows() const { return tc::BM; }
  struct Cursor { int k, row, h, b; };
  template <int KW>
  __device__ __forceinline__ Cursor cursor(int tile_m, int batch, int kb) const {
    const int b = (int)div_heads.div((uint32_t)batch);
    return Cursor{kb * tc::BK, tile_m * tc::BM, batch - b * heads, b};
  }
  template <int KW>
  __device__ __forceinline__ void advance(Cursor& c) const { c.k += KW; }
  template <bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_a(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c) const {
    if (AMN) {
#pragma unroll
      for (int i = 0; i < tc::BM / 32; ++i) tc::tma_load_4d_to<PAIR>((uint8_t*)dst + i * (32 * ROW_BYTES), tm, bar, c.row + 32 * i, c.k, c.h, c.b);
    } else {
      tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.k, c.row, c.h, c.b);
    }
  }
  template <int BN, bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_b(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c, int n0) const {
    if (BMN) {
#pragma unroll
      for (int i = 0; i < BN / 32; ++i) tc::tma_load_4d_to<PAIR>((uint8_t*)dst + i * (32 * ROW_BYTES), tm, bar, n0 + 32 * i, c.k, c.h, c.b);
    } else {
      tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.k, n0, c.h, c.b);
    }
  }
  __device__ __forceinline__ int row(int, int, int) const { return 0; }
  template <int W>
  __device__ __forceinline__ int fetch(int, int, bool) const { return 0; }
  template <bool SPLIT>
  __device__ __forceinline__ void store(int, int, int, int, float, float, uint32_t&) const {}   // no K-split
  template <bool SPLIT>
  __device__ __forceinline__ void epilogue(int tile_m, int batch, int row0, int n, float4 (&v)[4], float out_scale, uint32_t& top) const {
    const int b = (int)div_heads.div((uint32_t)batch), m0 = tile_m * tc::BM + row0, nn = N - n;
    const size_t at0 = (size_t)b * bs + (size_t)(batch - b * heads) * hs + (size_t)m0 * ldc + n;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (m0 + 8 * i >= M) continue;
      const size_t at = at0 + (size_t)(8 * i) * ldc;
      if (c) tc::store_guarded(c + at, v[i], nn, vec);
      if (SPLIT) {
        // (values of columns beyond the last and, causal, above the diagonal are of no tensor, but bound its own)
        top = pr::seen4(top, v[i]);
        if (hi && nn >= 4) pr::put4(hi, lo, at, v[i], out_scale);   // (planes: a multiple of 8 columns)
      } else if (hi) {
        const float4 h = make_float4(tc::tf32_rn(v[i].x), tc::tf32_rn(v[i].y), tc::tf32_rn(v[i].z), tc::tf32_rn(v[i].w));
        tc::store_guarded(hi + at, h, nn, vec);
      }
    }
  }
};

// mn: box {32 columns, 32 rows}; else {32 columns, `rows` rows}.
bool head_map(CUtensorMap* t, const float* p, const HeadMat& m, int heads, int batch, bool mn, int rows) {
  const uint64_t dim[4] = {(uint64_t)m.cols, (uint64_t)m.rows, (uint64_t)heads, (uint64_t)batch};
  const uint64_t str[3] = {m.ld, m.hs, m.bs};
  const uint32_t box[4] = {32, (uint32_t)(mn ? tc::BK : rows), 1, 1};
  return tc::encode_tmap(t, p, m.lo != nullptr, 4, dim, str, box, mn);
}

template <int BN, int NPLANES, bool AMN, bool BMN>
int run(nrs_ctx* ctx, const HeadMat& A, const HeadMat& B, const HeadPolicy<AMN, BMN>& pol, int batch, int k, NrsRange* out) {
  CUtensorMap a_hi, a_lo, b_hi, b_lo;
  bool ok = head_map(&a_hi, A.hi, A, pol.heads, batch, AMN, tc::BM) && head_map(&b_hi, B.hi, B, pol.heads, batch, BMN, BN);
  if (NPLANES == 2) ok = ok && head_map(&a_lo, A.lo, A, pol.heads, batch, AMN, tc::BM) && head_map(&b_lo, B.lo, B, pol.heads, batch, BMN, BN);
  else { a_lo = a_hi; b_lo = b_hi; }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "attention: cuTensorMapEncodeTiled failed");
  return tc::launch<BN, NPLANES, false, 32, HeadPolicy<AMN, BMN>>(ctx, a_hi, a_lo, b_hi, b_lo, pol, (pol.M + tc::BM - 1) / tc::BM, pol.N,
                                                       batch * pol.heads, (k + tc::BK - 1) / tc::BK, tc::Ranges{A.range, B.range, out});
}

struct Out {
  float *c, *hi, *lo;
  size_t ld, hs, bs;
  NrsRange* range;     // 3xTF32: of the planes, or the magnitudes of c
  float factor;        // its bound (see HeadPolicy)
  const NrsRange *r0, *r1, *r2;
};

template <bool AMN, bool BMN>
int product(nrs_ctx* ctx, const HeadMat& A, const HeadMat& B, const Out& o, int batch, int heads, int m, int n, int k, int causal) {
  auto ok16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  HeadPolicy<AMN, BMN> pol{o.c, o.hi, o.lo, o.ld, o.hs, o.bs, m, n, heads, NrsFastDiv(heads), false, causal, o.factor, o.r0, o.r1, o.r2};
  pol.vec = o.ld % 4 == 0 && o.hs % 4 == 0 && o.bs % 4 == 0 && ok16(o.c) && ok16(o.hi) && ok16(o.lo);
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  NrsProfScope prof(ctx, NRS_PROF_GEMM, 2.0 * batch * heads * m * n * k * (causal ? 0.5 : 1.0));
#define NRS_HEAD_RUN(BN_) (split ? run<BN_, 2, AMN, BMN>(ctx, A, B, pol, batch, k, o.range) : run<BN_, 1, AMN, BMN>(ctx, A, B, pol, batch, k, nullptr))
  if (n > 64) return NRS_HEAD_RUN(128);
  if (n > 32) return NRS_HEAD_RUN(64);
  return NRS_HEAD_RUN(32);
#undef NRS_HEAD_RUN
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
__device__ __forceinline__ void put_planes(float* hi, float* lo, size_t at, float4 v, float scale) {
  if (lo) pr::put4(hi, lo, at, v, scale);
  else *reinterpret_cast<float4*>(hi + at) = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
}
// Columns of row i that the products reading P and dS touch: all (ld), or up to the end of the row's 128-row tile.
__device__ __forceinline__ int row_extent(int i, int ld, int causal) { return causal ? min(ld, (i / tc::BM + 1) * tc::BM) : ld; }

// P = softmax(scale * S) over the keys j < seq (j <= i when causal), as planes, zeros in the row's other columns.  One
// warp per row, kept in registers (VPL float4s per lane) up to 1024 columns, else read twice more from L2.
template <int VPL>
__global__ void __launch_bounds__(256)
head_softmax_kernel(const float* __restrict__ s, float* __restrict__ hi, float* __restrict__ lo, long rows, int seq, int ld, int causal,
                    float scale, NrsRange* __restrict__ range) {
  NRS_PDL_PROLOGUE();
  const float pair_scale = pr::scale_of(1.0f);   // (a probability)
  if (range && blockIdx.x == 0 && threadIdx.x == 0) range->bound = range->top = 1.0f;
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
        if (c < ext) put_planes(hi, lo, (size_t)r * ld + c, make_float4(v[k].x * inv, v[k].y * inv, v[k].z * inv, v[k].w * inv), pair_scale);
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
        put_planes(hi, lo, (size_t)r * ld + c, make_float4(t.x * inv, t.y * inv, t.z * inv, t.w * inv), pair_scale);
      }
    }
  }
}

// dS = P o (dP - sum_j dP_j P_j) * scale as planes; P from its planes (TF32 mode: rounded to TF32; f16 pairs: to 2^-23 of
// itself, or to 2^-51).  |dS| <= 2 |dP| scale.  (Columns without a key have P = 0.)
template <int VPL>
__global__ void __launch_bounds__(256)
head_dsoftmax_kernel(const float* __restrict__ p_hi, const float* __restrict__ p_lo, const float* __restrict__ dp, float* __restrict__ hi,
                     float* __restrict__ lo, long rows, int seq, int ld, int causal, float scale, const NrsRange* __restrict__ range_dp,
                     NrsRange* __restrict__ range) {
  NRS_PDL_PROLOGUE();
  const float p_unscale = pr::pow2(-pr::scale_exp(1.0f));
  float pair_scale = 1.0f;
  uint32_t top = 0;
  if (lo) {
    const float bound = fminf(2.002f * range_dp->top * scale, 3.0e38f);
    if (blockIdx.x == 0 && threadIdx.x == 0) range->bound = bound;
    pair_scale = pr::scale_of(bound);
  }
  const int lane = threadIdx.x & 31;
  for (long r = (long)blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += (long)gridDim.x * 8) {
    const int i = (int)(r % seq), live = causal ? i + 1 : seq, ext = row_extent(i, ld, causal);
    const size_t base = (size_t)r * ld;
    float dot = 0.0f;
    auto fetch = [&](int c, float4* p, float4* d) {
      *p = *d = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c >= live) return;
      *p = p_lo ? pr::get4(p_hi, p_lo, base + c, p_unscale) : *reinterpret_cast<const float4*>(p_hi + base + c);
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
        if (c >= ext) continue;
        const float4 o = dsoft(p[k], d[k]);
        top = pr::seen4(top, o);
        put_planes(hi, lo, base + c, o, pair_scale);
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
        const float4 o = dsoft(p, d);
        top = pr::seen4(top, o);
        put_planes(hi, lo, base + c, o, pair_scale);
      }
    }
  }
  if (lo) pr::report_block(range, top);
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
  const NrsRange* qkv = nrs_range_of(ctx, a.qkv_hi);
  NrsRange *range_p = nullptr, *range_out = nullptr;
  int st = NRS_OK;
  if (split) st = nrs_range_renew(ctx, a.p_hi, &range_p);
  if (split && st == NRS_OK) st = nrs_range_renew(ctx, a.out_hi, &range_out);
  if (st != NRS_OK) return st;
  auto head = [&](int part) {   // 0 Q, 1 K, 2 V inside the projections' planes
    const size_t o = (size_t)part * a.heads * dh;
    return HeadMat{nrs_plane_at(a.qkv_hi, o, split), split ? nrs_plane_at(a.qkv_lo, o, true) : nullptr, dh, S, (size_t)a.qkv_ld, (size_t)dh,
                   (size_t)S * a.qkv_ld, qkv};
  };
  using P = HeadPolicy<false, false>;
  st = product<false, false>(ctx, head(0), head(1), Out{a.scores, nullptr, nullptr, (size_t)ld, ss, ss * a.heads, nullptr, 0.0f, nullptr, nullptr, nullptr},
                             a.batch, a.heads, S, S, dh, a.causal ? P::kTiles : P::kDense);
  if (st != NRS_OK) return st;
  const long rows = (long)a.batch * a.heads * S;
  const float scale = 1.0f / sqrtf((float)dh);
  NRS_HEAD_VPL(ld, NRS_PDL_LAUNCH(head_softmax_kernel<V>, row_blocks(ctx, rows), 256, 0, ctx->stream, (const float*)a.scores, a.p_hi, a.p_lo, rows,
                                  S, ld, a.causal, scale, range_p));
  NRS_LAUNCHED(ctx);
  const HeadMat p{a.p_hi, a.p_lo, ld, S, (size_t)ld, ss, ss * a.heads, range_p};
  const size_t D = (size_t)a.heads * dh;
  // a mean of rows of V under weights that sum to 1
  return product<false, true>(ctx, p, head(2), Out{a.out, a.out_hi, a.out_lo, D, (size_t)dh, (size_t)S * D, range_out, 1.01f, qkv, nullptr, nullptr},
                              a.batch, a.heads, S, dh, S, a.causal ? P::kUpTo : P::kDense);
}

int nrs_mha_planes_bwd(nrs_ctx* ctx, const NrsMhaPlanes& a) {
  const int S = a.seq, dh = a.d_head, ld = nrs_plane_ld(S);
  const size_t ss = (size_t)S * ld, D = (size_t)a.heads * dh;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  const NrsRange *qkv = nrs_range_of(ctx, a.qkv_hi), *range_p = nrs_range_of(ctx, a.p_hi), *range_dout = nrs_range_of(ctx, a.dout_hi);
  NrsRange *range_dp = nullptr, *range_ds = nullptr, *range_dqkv = nullptr;
  int st = NRS_OK;
  if (split) {
    NRS_REQUIRE(ctx, qkv && range_p && range_dout, NRS_ERR_ARG, "attention: planes without a range");
    st = nrs_range_renew(ctx, &ctx->scratch_range[0], &range_dp);
    if (st == NRS_OK) st = nrs_range_renew(ctx, a.ds_hi, &range_ds);
    if (st == NRS_OK) st = nrs_range_renew(ctx, a.dqkv_hi, &range_dqkv);
    if (st != NRS_OK) return st;
  }
  auto head = [&](int part) {
    const size_t o = (size_t)part * D;
    return HeadMat{nrs_plane_at(a.qkv_hi, o, split), split ? nrs_plane_at(a.qkv_lo, o, true) : nullptr, dh, S, (size_t)a.qkv_ld, (size_t)dh,
                   (size_t)S * a.qkv_ld, qkv};
  };
  // The three gradients are one tensor of planes with one exponent: sums over up to S keys or queries of P dO (P <= 1) and of
  // dS times a row of Q or K.
  auto grad = [&](int part) {
    const size_t o = (size_t)part * D;
    return Out{nullptr, nrs_plane_at(a.dqkv_hi, o, split), split ? nrs_plane_at(a.dqkv_lo, o, true) : nullptr, 3 * D, (size_t)dh, (size_t)S * 3 * D,
               range_dqkv, 1.001f * (float)S, range_dout, range_ds, qkv};
  };
  using P = HeadPolicy<false, false>;
  const HeadMat dout{a.dout_hi, a.dout_lo, dh, S, D, (size_t)dh, (size_t)S * D, range_dout};
  const HeadMat p{a.p_hi, a.p_lo, ld, S, (size_t)ld, ss, ss * a.heads, range_p};
  st = product<false, false>(ctx, dout, head(2), Out{a.scores, nullptr, nullptr, (size_t)ld, ss, ss * a.heads, range_dp, 0.0f, nullptr, nullptr, nullptr},
                             a.batch, a.heads, S, S, dh, a.causal ? P::kTiles : P::kDense);
  if (st != NRS_OK) return st;
  const long rows = (long)a.batch * a.heads * S;
  const float scale = 1.0f / sqrtf((float)dh);
  NRS_HEAD_VPL(ld, NRS_PDL_LAUNCH(head_dsoftmax_kernel<V>, row_blocks(ctx, rows), 256, 0, ctx->stream, (const float*)a.p_hi, (const float*)a.p_lo,
                                  (const float*)a.scores, a.ds_hi, a.ds_lo, rows, S, ld, a.causal, scale, (const NrsRange*)range_dp, range_ds));
  NRS_LAUNCHED(ctx);
  const HeadMat ds{a.ds_hi, a.ds_lo, ld, S, (size_t)ld, ss, ss * a.heads, range_ds};
  st = product<true, true>(ctx, p, dout, grad(2), a.batch, a.heads, S, dh, S, a.causal ? P::kFrom : P::kDense);
  if (st == NRS_OK) st = product<false, true>(ctx, ds, head(1), grad(0), a.batch, a.heads, S, dh, S, a.causal ? P::kUpTo : P::kDense);
  if (st == NRS_OK) st = product<true, true>(ctx, ds, head(0), grad(1), a.batch, a.heads, S, dh, S, a.causal ? P::kFrom : P::kDense);
  return st;
}
