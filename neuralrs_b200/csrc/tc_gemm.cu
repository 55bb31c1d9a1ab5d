// Dense / batched GEMM on the 5th-generation tensor cores (tcgen05), TF32 and
// 3xTF32:  C[b][m,n] = act(op(A[b]) . op(B[b]) + bias[n]) + beta * C.
//
// The main loop is tc_mainloop.cuh (TMA -> 128B-swizzled smem ring -> tcgen05.mma
// kind::tf32 -> TMEM -> tcgen05.ld epilogue); this file supplies the GEMM policy
// (dense K-major row slices, row-major store with bias/activation/accumulate) and
// operand preparation.  Both operands are consumed K-major: an operand stored
// the other way round is transposed by the staging pass, which for 3xTF32 also
// writes f16 pairs.  Plain TF32 reads untransposed, 16-byte
// aligned operands in place.
//
// Reference counterparts: matmul_nn / matmul_nt / matmul_tn, 64x64x16 FFMA tiles
// (src/cuda/graph/matmul.rs:44-198); bmm kernels (src/cuda/graph/bmm.rs:12-56).
#include "tc_mainloop.cuh"

namespace {

// MN: both operands are stored with the reduction index slow ([k][m] and [k][n], the planes of activations and of
// incoming gradients as they are): the slices arrive as 32-element column blocks, MN-major (see tc_wgrad.cu), and
// nothing is transposed.
template <bool MN>
struct GemmPolicy {
  float* C;
  const float* bias;
  int act;
  float beta;
  int M, N;
  size_t batch_stride;
  bool vec_ok;                 // rows of every output and epilogue input start on 16 bytes
  NrsGemmExtras x;
  float k_total;               // length of the reduction, for the result's bound
  // Several B matrices side by side ([Wq|Wk|Wv]): columns n0 of matrix n0 / seg_n, or reduction indices k of matrix
  // k / seg_k; 0 = one matrix.  The matrices are the batches of B's tensor map.
  int seg_n, seg_k;
  static constexpr bool kCanEmit = false;
  static constexpr bool kAMnMajor = MN, kBMnMajor = MN;
  static constexpr bool kMaySplit = true;
  __device__ __forceinline__ bool clip(int, int, int, int*, int*) const { return true; }
  // The epilogue is latency (TMEM, loads, GELU at about 66 instructions a value): four warps per lane quarter.  With two,
  // a 128 x 128 tile with GELU and three outputs took 27 thousand clocks, twice its main loop at K = 512.
  static constexpr int kEpiWarps = 16, kTeamWarps = 4;
  static constexpr bool kConv = false;
  static constexpr bool kSlab = false;
  int order() const { return tc::kRaster; }

  __device__ __forceinline__ uint32_t a_slice_rows() const { return tc::BM; }   // of A, that a load brings
  struct Cursor { int b_col, row, batch; };
  template <int KW>
  __device__ __forceinline__ Cursor cursor(int tile_m, int batch, int kb) const { return Cursor{kb * KW, tile_m * tc::BM, batch}; }
  template <int KW>
  __device__ __forceinline__ void advance(Cursor& c) const { c.b_col += KW; }
  template <bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_a(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c) const {
    if (MN) tc::tma_load_3d_to<PAIR>(dst, tm, bar, 0, c.b_col, c.row / KW);
    else tc::tma_load_3d_to<PAIR>(dst, tm, bar, c.b_col, c.row, c.batch);
  }
  template <int BN, bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_b(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c, int n0) const {
    if (MN) { tc::tma_load_3d_to<PAIR>(dst, tm, bar, 0, c.b_col, n0 / KW); return; }
    int b0 = c.b_col, b1 = n0, b2 = c.batch;
    if (seg_n) { b2 = n0 / seg_n; b1 = n0 - b2 * seg_n; }
    if (seg_k) { b2 = c.b_col / seg_k; b0 = c.b_col - b2 * seg_k; }
    tc::tma_load_3d_to<PAIR>(dst, tm, bar, b0, b1, b2);
  }
  __device__ __forceinline__ float dact(float src) const { return x.dact == NRS_ACT_RELU ? (src > 0.0f ? 1.0f : 0.0f) : nrs_gelu_d(src); }
  // No finished value exceeds this (a whole warp asks).
  __device__ __forceinline__ float out_bound(float top_a, float top_b, int lane) const {
    if (!x.hi) return 0.0f;   // only the largest magnitude is asked for
    uint32_t b = 0;
    if (bias)
      for (int n = lane; n < N; n += 32) b = pr::seen(b, bias[n]);
    const float bound = pr::product_bound(k_total, top_a, top_b, __uint_as_float(__reduce_max_sync(0xffffffffu, b)));
    return x.dact == NRS_ACT_GELU ? fminf(1.25f * bound, 3.0e38f) : bound;   // (GELU's derivative stays below 1.13, the activations within |v|)
  }
  // One element, from the pass that sums a K-split.
  template <bool SPLIT>
  __device__ __forceinline__ void store(int tile_m, int batch, int row, int n, float v, float out_scale, uint32_t& top) const {
    const int m = tile_m * tc::BM + row;
    if (m >= M || n >= N) return;
    const size_t at = (size_t)batch * batch_stride + (size_t)m * N + n;
    if (bias) v += bias[n];
    if (x.pre) x.pre[at] = v;
    v = nrs_apply_act(v, act);
    if (beta != 0.0f) v += beta * C[at];
    if (!x.skip_c) C[at] = v;
    if (SPLIT && !x.hi) top = pr::seen(top, v);
    if (!x.hi) return;
    if (x.dact != NRS_ACT_NONE) v *= dact(x.dact_src[at]);
    if (SPLIT) {
      top = pr::seen(top, v);
      pr::put(x.hi, x.lo, at, v, out_scale);
    } else {
      x.hi[at] = tc::tf32_rn(v);
    }
  }
  __device__ __forceinline__ int row(int, int, int) const { return 0; }
  template <int W>
  __device__ __forceinline__ int fetch(int, int, bool) const { return 0; }
  // Four row segments of a warp's 32 x 16 block: row r0 + 8*i of the tile, columns n..n+3 (see tc::rows_to_lines).  Blocks
  // that lie inside C on 16-byte boundaries, nearly all of them, take an instantiation without the checks.
  template <bool SPLIT>
  __device__ __forceinline__ void epilogue(int tile_m, int batch, int r0, int n, float4 (&v)[4], float out_scale, uint32_t& top) const {
    const int nb = n - (int)(threadIdx.x & 3) * 4;
    if (vec_ok && (tile_m + 1) * tc::BM <= M && nb + 16 <= N) finish<SPLIT, true>(tile_m, batch, r0, n, v, out_scale, top);
    else finish<SPLIT, false>(tile_m, batch, r0, n, v, out_scale, top);
  }
  template <bool SPLIT, bool INSIDE>
  __device__ __forceinline__ void finish(int tile_m, int batch, int r0, int n, float4 (&v)[4], float out_scale, uint32_t& top) const {
    const int m0 = tile_m * tc::BM + r0, nn = N - n;   // nn: how many of the four columns exist (four or more: all)
    const size_t at0 = (size_t)batch * batch_stride + (size_t)m0 * N + n;
    const uint32_t step = 8u * (uint32_t)N;
    auto row = [&](int i) { return INSIDE || m0 + 8 * i < M; };
    auto get = [&](const float* p) { return INSIDE ? *reinterpret_cast<const float4*>(p) : tc::load_guarded(p, nn, vec_ok); };
    auto put = [&](float* p, float4 q) {
      if (INSIDE) *reinterpret_cast<float4*>(p) = q;
      else tc::store_guarded(p, q, nn, vec_ok);
    };
    if (bias) {
      const float4 b = get(bias + n);
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[i].x += b.x; v[i].y += b.y; v[i].z += b.z; v[i].w += b.w; }
    }
    if (x.pre) {
      float* p = x.pre + at0;
#pragma unroll
      for (int i = 0; i < 4; ++i, p += step)
        if (row(i)) put(p, v[i]);
    }
    if (act != NRS_ACT_NONE) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[i].x = nrs_apply_act(v[i].x, act); v[i].y = nrs_apply_act(v[i].y, act);
        v[i].z = nrs_apply_act(v[i].z, act); v[i].w = nrs_apply_act(v[i].w, act);
      }
    }
    if (beta != 0.0f) {
      float4 o[4];
      const float* p = C + at0;
#pragma unroll
      for (int i = 0; i < 4; ++i, p += step) o[i] = row(i) ? get(p) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[i].x += beta * o[i].x; v[i].y += beta * o[i].y; v[i].z += beta * o[i].z; v[i].w += beta * o[i].w; }
    }
    if (!x.skip_c && !x.skip_c_unsplit) {
      float* p = C + at0;
#pragma unroll
      for (int i = 0; i < 4; ++i, p += step)
        if (row(i)) put(p, v[i]);
    }
    if (x.dact != NRS_ACT_NONE) {
      float4 s[4];
      const float* p = x.dact_src + at0;
#pragma unroll
      for (int i = 0; i < 4; ++i, p += step) s[i] = row(i) ? get(p) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) { v[i].x *= dact(s[i].x); v[i].y *= dact(s[i].y); v[i].z *= dact(s[i].z); v[i].w *= dact(s[i].w); }
    }
    if (SPLIT && x.range) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row(i)) top = pr::seen4(top, v[i]);
    }
    if (x.hi) {
      size_t at = at0;
#pragma unroll
      for (int i = 0; i < 4; ++i, at += step) {
        if (!row(i)) continue;
        if (SPLIT) {   // (n is a multiple of 8, so all four columns exist or none)
          if (INSIDE || nn >= 4) pr::put4(x.hi, x.lo, at, v[i], out_scale);
        } else {
          put(x.hi + at, make_float4(tc::tf32_rn(v[i].x), tc::tf32_rn(v[i].y), tc::tf32_rn(v[i].z), tc::tf32_rn(v[i].w)));
        }
      }
    }
    if (x.colsum) {   // sum over the warp's 32 rows, in a fixed order; lanes 0..3 write four columns each
      float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (row(i)) { s.x += v[i].x; s.y += v[i].y; s.z += v[i].z; s.w += v[i].w; }
#pragma unroll
      for (int d = 4; d <= 16; d <<= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, d); s.y += __shfl_xor_sync(0xffffffffu, s.y, d);
        s.z += __shfl_xor_sync(0xffffffffu, s.z, d); s.w += __shfl_xor_sync(0xffffffffu, s.w, d);
      }
      if ((threadIdx.x & 31) < 4) put(x.colsum + ((size_t)tile_m * 4 + (r0 >> 5)) * N + n, s);
    }
  }
};

struct Operand {
  const float* hi;
  const float* lo;
  int ld;          // leading dimension in floats
  int kdim;        // K extent given to the tensor map (TMA zero-fills beyond it)
  size_t bstride;  // values between batches
  const NrsRange* range;   // 3xTF32
};

// Brings one operand into K-major planes.  stored_kmajor: memory is [rows][K]; else [K][rows].  in_place: plain TF32
// may read a suitable source as it is (the tensor core truncates it); otherwise it is rounded into a plane.
int prepare_operand(nrs_ctx* ctx, const float* src, int rows, int K, int batch, bool stored_kmajor, bool split,
                    int ws, Operand* out, bool is_weight, bool in_place = true) {
  const int ldk = nrs_plane_ld(K);   // TMA zero-fills what a K-block reads beyond K
  if (batch == 1) {
    // a weight staged ahead with the rest of the model's (weight_set.cu) ...
    if (is_weight) {
      const NrsWeightPlanes* wp = nrs_weight_planes_find(ctx, src, stored_kmajor ? NRS_WF_LINEAR_ROWS : NRS_WF_LINEAR_T);
      if (wp && wp->rows == rows && wp->K == K) {
        const int ldw = (K + 31) / 32 * 32;
        *out = Operand{wp->hi, wp->lo, ldw, ldw, (size_t)rows * ldw, wp->range};
        return NRS_OK;
      }
    }
    // ... or an activation whose [rows][K] planes its producer or an earlier consumer left with the context
    if (stored_kmajor) {
      const NrsPlanes* ready = nrs_planes_find(ctx, src, split);
      if (ready && ready->rows == rows && ready->cols == K) {
        *out = Operand{ready->hi, ready->lo, ldk, K, (size_t)rows * ldk, nrs_range_of(ctx, ready->hi)};
        return NRS_OK;
      }
    }
  }
  const bool direct = in_place && !split && stored_kmajor && (K % 4 == 0) && ((reinterpret_cast<uintptr_t>(src) & 15) == 0);
  if (direct) {
    *out = Operand{src, nullptr, K, K, (size_t)rows * K, nullptr};
    return NRS_OK;
  }
  const size_t plane = (size_t)rows * ldk;
  void *phi = nullptr, *plo = nullptr;
  int st = nrs_ws_planes(ctx, ws, plane * batch, split, &phi, &plo);
  if (st != NRS_OK) return st;
  st = nrs_tc_stage(ctx, src, (float*)phi, (float*)plo, rows, K, ldk, batch, (size_t)rows * K, plane, !stored_kmajor);
  if (st != NRS_OK) return st;
  *out = Operand{(const float*)phi, (const float*)plo, ldk, K, plane, nrs_range_of(ctx, phi)};
  return NRS_OK;
}

bool make_operand_map(CUtensorMap* tm, const float* base, const Operand& op, int rows, int batch, int box_rows, int kw) {
  const uint64_t dim[3] = {(uint64_t)op.kdim, (uint64_t)rows, (uint64_t)batch};
  const uint64_t str[2] = {(uint64_t)op.ld, (uint64_t)op.bstride};
  const uint32_t box[3] = {(uint32_t)kw, (uint32_t)box_rows, 1};
  return tc::encode_tmap(tm, base, op.lo != nullptr, 3, dim, str, box);
}
// An operand stored [k][rows]: [row block][k][kw rows], one box = a K-slice of box_rows / kw blocks.
bool make_mn_operand_map(CUtensorMap* tm, const float* base, const Operand& op, int rows, int k, int box_rows, int kw) {
  const uint64_t dim[3] = {(uint64_t)kw, (uint64_t)k, (uint64_t)(rows / kw)};
  const uint64_t str[2] = {(uint64_t)op.ld, (uint64_t)kw};
  const uint32_t box[3] = {(uint32_t)kw, (uint32_t)kw, (uint32_t)(box_rows / kw)};
  return tc::encode_tmap(tm, base, op.lo != nullptr, 3, dim, str, box, true);
}

template <int BN, int NPLANES, bool PAIR, bool MN, int KW>
int run(nrs_ctx* ctx, const Operand& A, const Operand& B, int batch, int b_rows, int b_batch, int m, int n, int k,
        const GemmPolicy<MN>& pol, int* splits) {
  constexpr int kBRows = PAIR ? BN / 2 : BN;   // rows of B that one CTA brings
  CUtensorMap ta_hi, ta_lo, tb_hi, tb_lo;
  auto map_a = [&](CUtensorMap* t, const float* p) { return MN ? make_mn_operand_map(t, p, A, m, k, tc::BM, KW) : make_operand_map(t, p, A, m, batch, tc::BM, KW); };
  auto map_b = [&](CUtensorMap* t, const float* p) { return MN ? make_mn_operand_map(t, p, B, n, k, kBRows, KW) : make_operand_map(t, p, B, b_rows, b_batch, kBRows, KW); };
  bool ok = map_a(&ta_hi, A.hi) && map_b(&tb_hi, B.hi);
  if (NPLANES == 2) ok = ok && map_a(&ta_lo, A.lo) && map_b(&tb_lo, B.lo);
  else { ta_lo = ta_hi; tb_lo = tb_hi; }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "tc_gemm: cuTensorMapEncodeTiled failed (m=%d n=%d k=%d)", m, n, k);
  return tc::launch<BN, NPLANES, PAIR, KW, GemmPolicy<MN>>(ctx, ta_hi, ta_lo, tb_hi, tb_lo, pol, (m + tc::BM - 1) / tc::BM, n, batch,
                                                 (k + KW - 1) / KW, tc::Ranges{A.range, B.range, pol.x.range}, nullptr, nullptr, splits);
}

// `limit`: widest tile allowed (segmented B: the segment must be whole tiles).
tc::TilePlan tile_of(const nrs_ctx* ctx, int m, int n, int batch, int k, bool split, int limit = 128) {
  return tc::plan_tile(ctx, (m + tc::BM - 1) / tc::BM, n, batch, (k + tc::BK - 1) / tc::BK, split, 0.004, false, false, limit);
}

template <bool MN>
int dispatch(nrs_ctx* ctx, tc::TilePlan tile, bool split, const Operand& A, const Operand& B, int batch, int b_rows, int b_batch, int m, int n,
             int k, GemmPolicy<MN>& pol, NrsGemmExtras* extras) {
  auto aligned = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
  pol.k_total = (float)k;
  pol.vec_ok = n % 4 == 0 && ((size_t)m * n) % 4 == 0 && aligned(pol.C) && aligned(pol.bias);
  if (extras) {
    pol.x = *extras;
    pol.vec_ok = pol.vec_ok && aligned(extras->pre) && aligned(extras->dact_src);
    if (!split) pol.x.range = nullptr;
    if (split && extras->hi) {
      NRS_REQUIRE(ctx, pol.beta == 0.0f, NRS_ERR_ARG, "tc_gemm: no planes of an accumulated result");
      const int st = nrs_range_renew(ctx, extras->hi, &extras->range);
      if (st != NRS_OK) return st;
      pol.x.range = extras->range;
    }
    if (extras->colsum && (m + tc::BM - 1) / tc::BM * 4 > extras->colsum_cap) pol.x.colsum = nullptr;
  }
  int st, splits = 1;
  // f16 pairs: K-slices of 64, whose rows are 128 bytes, wherever they fit: TMA brings rows of 64 bytes at half the rate.
  // (MN-major blocks of 64 columns have to be whole, in a CTA's share of B too; a K-slice belongs to one matrix of B.)
  const bool wide = split && (MN ? m % 64 == 0 && n % 64 == 0 && tile.bn >= (tile.pair ? 128 : 64) : (k % 64 == 0 || k >= 256) && pol.seg_k % 64 == 0);
#define NRS_RUN_GEMM(BN_, PAIR_) (!split ? run<BN_, 1, PAIR_, MN, 32>(ctx, A, B, batch, b_rows, b_batch, m, n, k, pol, &splits)       \
                                  : wide ? run<BN_, 2, PAIR_, MN, MN && BN_ < (PAIR_ ? 128 : 64) ? 32 : 64>(ctx, A, B, batch, b_rows, b_batch, m, n, k, pol, &splits) \
                                         : run<BN_, 2, PAIR_, MN, 32>(ctx, A, B, batch, b_rows, b_batch, m, n, k, pol, &splits))
  if (tile.pair) st = tile.bn == 128 ? NRS_RUN_GEMM(128, true) : NRS_RUN_GEMM(64, true);
  else if (tile.bn == 128) st = NRS_RUN_GEMM(128, false);
  else if (tile.bn == 64) st = NRS_RUN_GEMM(64, false);
  else st = NRS_RUN_GEMM(32, false);
#undef NRS_RUN_GEMM
  if (extras && st == NRS_OK) {
    extras->honoured = true;
    extras->colsum_rows = pol.x.colsum && splits == 1 ? (m + tc::BM - 1) / tc::BM * 4 : 0;   // a K-split's second pass makes none
  }
  return st;
}

}  // namespace

namespace {
// Waits on an mbarrier nobody ever arrives on, with the kernels' own bounded-wait primitive and a
// short limit, and reports the expiry the way they do.
__global__ void bounded_wait_probe_kernel(long long limit_clocks, int* __restrict__ err_flag) {
  __shared__ uint64_t bar;
  if (threadIdx.x == 0) {
    tc::mbar_init(&bar, 1);
    tc::fence_barrier_init();
    if (!tc::mbar_wait_limit(&bar, 0, limit_clocks)) atomicExch(err_flag, tc::kErrMmaWait);
  }
}
}  // namespace

extern "C" int nrs_selftest_bounded_wait(nrs_ctx* ctx, int64_t limit_clocks) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, limit_clocks > 0 && limit_clocks <= 100000000, NRS_ERR_ARG,
              "nrs_selftest_bounded_wait: limit must be in (0, 1e8] clocks");
  int* err = nullptr;
  const int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  bounded_wait_probe_kernel<<<1, 32, 0, ctx->stream>>>((long long)limit_clocks, err);
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

namespace {
// Back-to-back tcgen05.mma (M = 128, N = 256, 32 bytes of K: 8 values of kind::tf32, 16 of kind::f16) on operands that never leave shared
// memory: the tensor pipe's own rate, with no TMA traffic and no epilogue.  One issuing thread per CTA,
// one CTA per SM; every wait is bounded.
template <bool HALF>
__global__ void __launch_bounds__(128, 1) umma_rate_kernel(int iters, int* __restrict__ err_flag) {
  extern __shared__ uint8_t umma_rate_smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(umma_rate_smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t bar;
  __shared__ uint32_t tmem_slot;
  for (int i = threadIdx.x; i < 48 * 1024 / 4; i += blockDim.x) reinterpret_cast<float*>(smem)[i] = 1.0f;
  if (threadIdx.x == 0) { tc::mbar_init(&bar, 1); tc::fence_barrier_init(); }
  if (threadIdx.x < 32) { tc::tmem_alloc(&tmem_slot, 512); tc::tmem_relinquish(); }
  tc::fence_proxy_async();
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem = tmem_slot;
  if (threadIdx.x == 0) {
    const uint32_t idesc = HALF ? tc::make_idesc_f16(128, 256, false, false) : tc::make_idesc_tf32(128, 256, false, false);
    const uint32_t a = tc::smem_u32(smem), b = a + 16384;     // A: 128 rows x 128 B; B: 256 rows x 128 B
    for (int i = 0; i < iters; ++i) {
      const uint32_t koff = (uint32_t)(i & 3) * 32u;            // the four K-steps of a row of 128 bytes
      const uint32_t d = tmem + ((i & 1) ? 256u : 0u);
      const uint64_t da = tc::make_smem_desc_sw128(a + koff, 16, 1024), db = tc::make_smem_desc_sw128(b + koff, 16, 1024);
      if (HALF) tc::umma_f16(d, da, db, idesc, 1);
      else tc::umma_tf32(d, da, db, idesc, 1);
    }
    tc::umma_commit(&bar);
    if (!tc::mbar_wait(&bar, 0)) atomicExch(err_flag, tc::kErrMmaWait);
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) { tc::tc_fence_after_sync(); tc::tmem_dealloc(tmem, 512); }
}

template <bool HALF>
int measure_umma_peak(nrs_ctx* ctx, const char* who, double* tflops_out) {
  NRS_REQUIRE_CTX(ctx);
  NRS_REQUIRE(ctx, tflops_out != nullptr, NRS_ERR_ARG, "%s: null output", who);
  *tflops_out = 0.0;
  int* err = nullptr;
  int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  constexpr int kSmem = 64 * 1024, kIters = 40000;          // ~2.6 ms at 128 clocks per UMMA
  static NrsSmemAttr attr;
  NRS_ENSURE_SMEM(ctx, attr, umma_rate_kernel<HALF>, kSmem);
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  NRS_CUDA(ctx, cudaEventCreate(&e0));
  NRS_CUDA(ctx, cudaEventCreate(&e1));
  float best_ms = 0.0f;
  for (int rep = 0; rep < 4; ++rep) {                        // the first launch warms up
    cudaEventRecord(e0, ctx->stream);
    umma_rate_kernel<HALF><<<ctx->sm_count, 128, kSmem, ctx->stream>>>(kIters, err);
    ctx->launches++;
    cudaEventRecord(e1, ctx->stream);
    if (cudaEventSynchronize(e1) != cudaSuccess) break;
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && (best_ms == 0.0f || ms < best_ms)) best_ms = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  NRS_CUDA(ctx, cudaGetLastError());
  st = nrs_check_device_error(ctx);
  if (st != NRS_OK) return st;
  if (best_ms > 0.0f) *tflops_out = 2.0 * 128 * 256 * (HALF ? 16 : 8) * (double)kIters * ctx->sm_count / (best_ms * 1e-3) / 1e12;
  return NRS_OK;
}
}  // namespace

extern "C" int nrs_measure_tf32_umma_peak(nrs_ctx* ctx, double* tflops_out) { return measure_umma_peak<false>(ctx, "nrs_measure_tf32_umma_peak", tflops_out); }
extern "C" int nrs_measure_f16_umma_peak(nrs_ctx* ctx, double* tflops_out) { return measure_umma_peak<true>(ctx, "nrs_measure_f16_umma_peak", tflops_out); }

int nrs_tc_gemm(nrs_ctx* ctx, int trans_a, int trans_b, int batch, int m, int n, int k, const float* a, const float* b,
                float* c, const float* bias, int act, float beta, NrsGemmExtras* extras) {
  if (!tc::tensor_map_encoder()) return NRS_ERR_UNSUPPORTED;
  // Fewer rows than a UMMA's smallest useful share of a 128-row tile stay on the FFMA kernels.
  if (m < 16 || n < 32 || k < 32) return NRS_ERR_UNSUPPORTED;
  if (batch > 65535) return NRS_ERR_UNSUPPORTED;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  Operand A, B;
  int st;
  if (trans_a && !trans_b && batch == 1 && m % 32 == 0 && n % 32 == 0) {   // A^T B on the operands' own rows
    st = prepare_operand(ctx, a, k, m, 1, true, split, NRS_WS_A, &A, false, false);
    if (st == NRS_OK) st = prepare_operand(ctx, b, k, n, 1, true, split, NRS_WS_B, &B, false, false);
    if (st != NRS_OK) return st;
    GemmPolicy<true> pol{c, bias, act, beta, m, n, (size_t)m * n, false, {}, 0.0f, 0, 0};
    return dispatch<true>(ctx, tile_of(ctx, m, n, 1, k, split), split, A, B, 1, n, 1, m, n, k, pol, extras);
  }
  st = prepare_operand(ctx, a, m, k, batch, /*stored_kmajor=*/!trans_a, split, NRS_WS_A, &A, false);
  if (st != NRS_OK) return st;
  st = prepare_operand(ctx, b, n, k, batch, /*stored_kmajor=*/trans_b != 0, split, NRS_WS_B, &B, true);
  if (st != NRS_OK) return st;
  // Batched operands read in place need 16-byte aligned batch strides.
  if (batch > 1 && ((A.bstride % (split ? 8 : 4)) || (B.bstride % (split ? 8 : 4)))) return NRS_ERR_UNSUPPORTED;
  GemmPolicy<false> pol{c, bias, act, beta, m, n, (size_t)m * n, false, {}, 0.0f, 0, 0};
  return dispatch<false>(ctx, tile_of(ctx, m, n, batch, k, split), split, A, B, batch, n, batch, m, n, k, pol, extras);
}

// x[m,k] times several weight matrices w[i] of one shape, in one product.  `reduce` == 0: c[m, count*n] = x . [w0|w1|..]
// (w[i]: [k][n] as stored).  `reduce` != 0: c[m,n] (+)= sum_i x_i . w[i]^T with x = [x_0|x_1|..] of `count` blocks of
// `n_i` columns, w[i]: [n][n_i].  The weights' planes come from the context's weight set when they lie there at equal
// distances (a trainer's), else they are staged side by side.
int nrs_tc_gemm_weights(nrs_ctx* ctx, int reduce, int count, int m, int n, int k, const float* x, const float* const* w, float* c,
                        float beta, NrsGemmExtras* extras) {
  if (ctx->math_mode == NRS_MATH_FP32 || !tc::tensor_map_encoder() || m < 16 || n < 32 || k < 32) return NRS_ERR_UNSUPPORTED;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  const int form = reduce ? NRS_WF_LINEAR_ROWS : NRS_WF_LINEAR_T;
  if (!reduce && n % 32 != 0) return NRS_ERR_UNSUPPORTED;   // a column tile belongs to one matrix
  if (reduce && k % 32 != 0) return NRS_ERR_UNSUPPORTED;    // and so does a K-slice
  Operand A, B{};
  int st = prepare_operand(ctx, x, m, reduce ? count * k : k, 1, true, split, NRS_WS_A, &A, false);
  if (st != NRS_OK) return st;
  bool found = true;
  for (int i = 0; i < count && found; ++i) {
    const NrsWeightPlanes* wp = nrs_weight_planes_find(ctx, w[i], form);
    found = wp && wp->rows == n && wp->K == k;
    if (!found) break;
    if (i == 0) { B.hi = wp->hi; B.lo = wp->lo; B.ld = (k + 31) / 32 * 32; B.kdim = B.ld; B.range = wp->range; }
    else if (i == 1) { found = wp->hi > B.hi; B.bstride = (size_t)((const uint8_t*)wp->hi - (const uint8_t*)B.hi) / (split ? 2 : 4); }
    found = found && wp->hi == nrs_plane_at(B.hi, i * B.bstride, split) && wp->range == B.range &&
            (!split || wp->lo == nrs_plane_at(B.lo, i * B.bstride, true));
  }
  if (!found) {
    const int ld = nrs_plane_ld(k);
    const size_t plane = (size_t)n * ld;
    void *hi = nullptr, *lo = nullptr;
    st = nrs_ws_planes(ctx, NRS_WS_B, plane * count, split, &hi, &lo);
    if (st == NRS_OK) st = nrs_tc_stage_each(ctx, w, count, (float*)hi, (float*)lo, n, k, ld, plane, !reduce);
    if (st != NRS_OK) return st;
    B = Operand{(const float*)hi, (const float*)lo, ld, k, plane, nrs_range_of(ctx, hi)};
  }
  const int cols = reduce ? n : count * n, kk = reduce ? count * k : k;
  GemmPolicy<false> pol{c, nullptr, NRS_ACT_NONE, beta, m, cols, (size_t)m * cols, false, {}, 0.0f, reduce ? 0 : n, reduce ? k : 0};
  const int limit = reduce ? 128 : n % 128 == 0 ? 128 : n % 64 == 0 ? 64 : 32;
  NrsProfScope prof(ctx, NRS_PROF_GEMM, 2.0 * m * cols * kk);
  return dispatch<false>(ctx, tile_of(ctx, m, cols, 1, kk, split, limit), split, A, B, 1, n, count, m, cols, kk, pol, extras);
}

extern "C" int nrs_has_tensor_core_path(void) { return 1; }
