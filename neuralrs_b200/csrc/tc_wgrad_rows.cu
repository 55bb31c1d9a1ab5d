// Weight gradient of 3x3 / stride 1 / pad 1 convolutions on tcgen05 (TF32 / 3xTF32), by slabs of image rows that serve
// all three vertical taps.
//
//   dw[co,ci,i,j] (+)= sum over (n,y,x) of dy[n,co,y,x] * x[n,ci,y+i-1,x+j-1]
//
// The general kernel (tc_wgrad.cu) loads one shifted x box per tap, so x crosses L2 -> shared memory nine times and dy
// once per tap group.  Here a CTA owns
//   128 output channels x one horizontal tap j x a chunk of input channels
// and walks tiles of R image rows x Wt columns.  A step brings in the tile's dy (R rows) and a slab of R + 2 rows of x
// (shifted by j - 1 through the TMA box origin; zero fill = padding, beyond the image on all sides).  Both lie in shared
// memory as [pixel][channels], pixels along K, so vertical tap i is the slab from its i-th row on: the same K-steps, Wt
// pixels further.  The taps are column blocks of ONE product: its B descriptor's block stride is Wt pixels, less than a
// block, so the blocks overlap in memory.  A UMMA thus covers 3 x 64 columns (f16 pairs; 3 x 32 of f32), there are no
// cases at the image's edges, and the issuing warp's part is one wait, a few UMMAs and one commit per step.  With 64
// output channels or fewer the 128 accumulator rows would be half empty, so a CTA takes TWO horizontal taps: the upper rows
// get a second copy of the dy tile fetched one pixel to the right, which turns the same x operand into the neighbouring tap
// (sum_p dy[p+1] x[p] = sum_p dy[p] x[p-1]); two kinds of CTA then cover the three taps instead of three.
//
// What bounds it: with 64-channel chunks the tensor pipe (288 clocks per 16 pixels) and the tiles' way through L2 (56 bytes
// a clock and SM at 32-pixel rows) are close.  Streaming one image row a step through separate rings of dy and x rows, as
// this kernel did before, took 1300 clocks per 32-pixel row, more than half of them bookkeeping of the issuing warp:
// x[256,64,32,32] -> 128 channels in 3xTF32 112 us, here 79 (1270 clocks per 64 pixels, of which the UMMAs are 1152).
//
// Tiles are split across CTAs (no accumulation chain longer than tc::kMaxChainPairs pixels in 3xTF32 mode); partial sums are
// added up in a fixed order by a second kernel, which also scatters into [co][ci][3][3].
//
// Replaces conv2d_im2col + conv2d_out2mm + matmul_nt_splitk (src/cuda/nn/conv.rs:
// 298-320) for the shapes it covers; everything else takes tc_wgrad.cu.
#include "fold.h"
#include "tc_mainloop.cuh"
#include "wgrad_queue.h"

namespace {

constexpr int kRowThreads = 192;
constexpr int kTaps = 3;          // vertical taps per CTA
constexpr int kMaxStages = 8;

struct RowParams {
  int co, ci;
  int Wt, R, P;                   // tile: columns (a multiple of 8), rows, and pixels = Wt * R (a multiple of a K-step)
  int tiles_x, tiles_y;           // tiles of an image
  int n_tiles, tiles_per_split;
  int chunk, n_chunks;            // input channels per CTA (multiple of wb) and how many chunks
  int wa, wb;                     // channels of a block of dy, of x: 32, or 64 (f16: rows of 128 bytes)
  int a_blocks;                   // blocks of dy one box brings (128 channels at most)
  int pack;                       // co <= 64: accumulator rows [0,h) and [h,2h), h = wa*a_blocks, hold two
                                  // horizontal taps (the second from a copy of the dy tile shifted one pixel)
  int jtypes;                     // CTA kinds along the horizontal taps: 3, or 2 when packed
  int m_blocks;                   // ceil(co / 128)
  int stages;
  float* partial;                 // [split][cta][128][3*chunk]
  int cross;                      // 3xTF32: accumulator columns between the hi*hi sums and the others
  const NrsRange *range_dy, *range_x;
  int ctas;                       // per split
  unsigned first_block;           // of this gradient's in the launch
};
// The gradients of one launch.
struct RowEntry {
  CUtensorMap dy_hi, dy_lo, x_hi, x_lo;
  RowParams p;
};
template <int CAP>
struct RowBatch {
  RowEntry e[CAP];
  int n;
  int independent;                // reads nothing the kernel launched just before it wrote (NRS_PDL_PROLOGUE)
};
constexpr int kRowBatch = 12;

// Bytes of one plane of a stage's operands.  (A UMMA reads 128 channels of dy whatever there are: the slab of x behind
// them is at least as long as what that reads beyond.)
__host__ __device__ inline uint32_t dy_bytes(const RowParams& p, int value) { return (uint32_t)((p.pack ? 2 : 1) * p.a_blocks * p.wa * p.P * value); }
__host__ __device__ inline uint32_t x_bytes(const RowParams& p, int value) { return (uint32_t)(p.chunk * (p.R + 2) * p.Wt * value); }

template <int NPLANES, int CAP>
__global__ void __launch_bounds__(kRowThreads, 1)
tc_wgrad_rows_kernel(const __grid_constant__ RowBatch<CAP> batch, int* __restrict__ err_flag) {
  extern __shared__ uint8_t smem_raw[];
  int entry = 0;
  while (CAP > 1 && entry + 1 < batch.n && batch.e[entry + 1].p.first_block <= blockIdx.x) ++entry;
  const RowEntry& en = batch.e[entry];
  const RowParams& p = en.p;
  const CUtensorMap &tm_dy_hi = en.dy_hi, &tm_dy_lo = en.dy_lo, &tm_x_hi = en.x_hi, &tm_x_lo = en.x_lo;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  constexpr int kValue = NPLANES == 2 ? 2 : 4;
  constexpr int kStepPixels = NPLANES == 2 ? 16 : 8;
  const uint32_t a_blk = (uint32_t)(p.P * p.wa * kValue), b_blk = (uint32_t)((p.R + 2) * p.Wt * p.wb * kValue);
  const uint32_t a_box = (uint32_t)p.a_blocks * a_blk, a_plane = dy_bytes(p, kValue), b_plane = x_bytes(p, kValue);
  const uint32_t stage_bytes = NPLANES * (a_plane + b_plane);   // [dy hi][x hi][dy lo][x lo]
  const uint32_t over = 128u * p.P * kValue;                    // of dy that a UMMA may read
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + (size_t)p.stages * stage_bytes + over);
  uint64_t* empty = full + p.stages;
  uint64_t* accum_bar = empty + p.stages;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum_bar + 1);

  const int warp = (int)tc::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  // A block is (split, m block, horizontal tap kind, channel chunk).  Unpacked: kind = tap j, x shifted by
  // j - 1.  Packed: kind 0 shifts x by 0 and holds taps j = 1 (plain dy) and j = 0 (dy shifted one
  // pixel: sum_p dy[p+1] x[p] = sum_p dy[p] x[p-1]); kind 1 shifts x by +1 and holds j = 2 alone.
  const int local = (int)(blockIdx.x - p.first_block), split = local / p.ctas, cta = local - split * p.ctas;
  const int cc = cta % p.n_chunks;
  const int jk = (cta / p.n_chunks) % p.jtypes;
  const int mb = cta / (p.n_chunks * p.jtypes);
  const int x_shift = p.pack ? jk : jk - 1;
  const bool two_taps = p.pack && jk == 0;
  const int t0 = split * p.tiles_per_split, steps = min(p.n_tiles - t0, p.tiles_per_split);
  const uint32_t tmem_cols = (NPLANES == 2 ? 2u : 1u) * (kTaps * p.chunk <= 128 ? 128u : (kTaps * p.chunk <= 256 ? 256u : 512u));

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tm_dy_hi);
    tc::prefetch_tmap(&tm_x_hi);
    if (NPLANES == 2) { tc::prefetch_tmap(&tm_dy_lo); tc::prefetch_tmap(&tm_x_lo); }
    for (int s = 0; s < p.stages; ++s) { tc::mbar_init(&full[s], 1); tc::mbar_init(&empty[s], 1); }
    tc::mbar_init(accum_bar, 1);
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, tmem_cols);
    tc::tmem_relinquish();
  }
  tc::tc_fence_before_sync();
  __syncthreads();
  tc::tc_fence_after_sync();
  const uint32_t tmem_base = tc::uniform(*tmem_slot);
  if (!batch.independent) NRS_PDL_WAIT();   // set-up above may overlap the previous kernel's tail; its results are needed from here
  NRS_PDL_TRIGGER();

  // (Both issuing roles run as whole warps and elect a lane for the instructions themselves: tc::elect_one.)
  if (warp == 0) {
    // ---------------- TMA producer
    const uint32_t tx = NPLANES * ((two_taps ? 2u : 1u) * a_box + b_plane);
    int tx0 = t0 % p.tiles_x, ty = t0 / p.tiles_x;   // the tile's place, stepped along
    int n = ty / p.tiles_y;
    ty -= n * p.tiles_y;
    int s = 0, it = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (; it < steps; ++it) {
      if (!tc::mbar_wait_warp(&empty[s], ph ^ 1u)) { ok = false; break; }
      uint8_t* st = smem + (size_t)s * stage_bytes;
      const int x0 = tx0 * p.Wt, y0 = ty * p.R;
      if (tc::elect_one()) {
        tc::mbar_expect_tx(&full[s], tx);
#pragma unroll
        for (int pl = 0; pl < NPLANES; ++pl) {
          const CUtensorMap* tdy = pl == 0 ? &tm_dy_hi : &tm_dy_lo;
          uint8_t* a = st + pl * (a_plane + b_plane);
          tc::tma_load_5d(a, tdy, &full[s], 0, x0, y0, n, mb * 128 / p.wa);
          if (two_taps) tc::tma_load_5d(a + a_box, tdy, &full[s], 0, x0 + 1, y0, n, mb * 128 / p.wa);
          tc::tma_load_5d(a + a_plane, pl == 0 ? &tm_x_hi : &tm_x_lo, &full[s], 0, x0 + x_shift, y0 - 1, n, cc * (p.chunk / p.wb));
        }
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1u; }
      if (++tx0 == p.tiles_x) {
        tx0 = 0;
        if (++ty == p.tiles_y) { ty = 0; ++n; }
      }
    }
    if (!ok) {
      if (lane == 0) atomicExch(err_flag, tc::kErrProducerWait);
      // Loads already issued still land in this CTA's shared memory: wait for them (bounded) before the CTA may retire.
      for (int u = it > p.stages ? it - p.stages : 0; u < it; ++u)
        if (!tc::mbar_wait_warp(&full[u % p.stages], (uint32_t)(u / p.stages) & 1u)) {
          if (lane == 0) atomicExch(err_flag, tc::kErrDrainWait);
          break;
        }
    }
  } else if (warp == 1) {
    // ---------------- UMMA issuer: per K-step and block of x one product of three taps (a column block each)
    bool ok = true;
    const uint32_t idesc = NPLANES == 2 ? tc::make_idesc_f16(128, kTaps * p.wb, true, true) : tc::make_idesc_tf32(128, kTaps * p.wb, true, true);
    auto desc = [](int w, uint32_t lbo) {   // every field but the start address (bytes >> 4)
      return NPLANES == 1 ? tc::make_smem_desc_sw128_32b(0, lbo, 512) : w == 64 ? tc::make_smem_desc_sw128(0, lbo, 1024) : tc::make_smem_desc_sw64(0, lbo, 512);
    };
    const uint64_t da = desc(p.wa, a_blk), db = desc(p.wb, (uint32_t)(p.Wt * p.wb * kValue));
    const uint32_t step_a = (uint32_t)(kStepPixels * p.wa * kValue) >> 4, step_b = (uint32_t)(kStepPixels * p.wb * kValue) >> 4;
    const uint32_t a16 = a_plane >> 4, b16 = b_plane >> 4, blk16 = b_blk >> 4;
    const int ksteps = p.P / kStepPixels, x_blocks = p.chunk / p.wb;
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < steps; ++it) {
      if (!tc::mbar_wait_warp(&full[s], ph)) { ok = false; break; }
      const uint32_t a_hi = tc::smem_u32(smem + (size_t)s * stage_bytes) >> 4, b_hi = a_hi + a16;
      const uint32_t a_lo = b_hi + b16, b_lo = a_lo + a16;
      if (tc::elect_one()) {
#pragma unroll 2
        for (int k = 0; k < ksteps; ++k) {
          const uint32_t ka = (uint32_t)k * step_a, more = (it | k) != 0;
#pragma unroll 1
          for (int b = 0; b < x_blocks; ++b) {
            const uint32_t kb = (uint32_t)k * step_b + (uint32_t)b * blk16, d = tmem_base + (uint32_t)(b * kTaps * p.wb);
            const uint64_t ah = da + (a_hi + ka), bh = db + (b_hi + kb);
            if (NPLANES == 2) {
              tc::umma_f16(d, ah, bh, idesc, more);
              tc::umma_f16(d + (uint32_t)p.cross, ah, db + (b_lo + kb), idesc, more);
              tc::umma_f16(d + (uint32_t)p.cross, da + (a_lo + ka), bh, idesc, 1);
            } else {
              tc::umma_tf32(d, ah, bh, idesc, more);
            }
          }
        }
        tc::umma_commit(&empty[s]);
      }
      __syncwarp();
      if (++s == p.stages) { s = 0; ph ^= 1u; }
    }
    if (ok && tc::elect_one()) tc::umma_commit(accum_bar);
    if (!ok && lane == 0) atomicExch(err_flag, tc::kErrMmaWait);
    __syncwarp();
  } else {
    // ---------------- epilogue: raw partial tile to the workspace
    const int q = warp & 3;
    const bool ok = tc::mbar_wait(accum_bar, 0);
    if (!ok && lane == 0) atomicExch(err_flag, tc::kErrEpilogueWait);
    if (ok) {
      tc::tc_fence_after_sync();
      const int row = q * 32 + lane;
      const int cols = kTaps * p.chunk;
      float* dst = p.partial + ((size_t)local * 128 + row) * cols;
      // packed: rows [0,h) are tap j = 1 or 2, rows [h,2h) tap j = 0 (kind 0 only)
      const int half = p.wa * p.a_blocks;
      const bool row_live = p.pack ? (row < half || (two_taps && row < 2 * half)) : (mb * 128 + row < p.co);
      const pr::Unscale unscale(NPLANES == 2 ? p.range_dy->bound : 1.0f, NPLANES == 2 ? p.range_x->bound : 1.0f);
#pragma unroll 1
      for (int b = 0; b < p.chunk / p.wb; ++b)
#pragma unroll 1
        for (int i = 0; i < kTaps; ++i)
#pragma unroll 1
          for (int c = 0; c < p.wb; c += 32) {   // columns of the accumulator: [block of x][tap][channel]
            uint32_t r[32];
            const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)((b * kTaps + i) * p.wb + c);
            tc::tmem_ld_32x32(at, r);
            if constexpr (NPLANES == 2) {
              uint32_t x[32];
              tc::tmem_ld_32x32(at + (uint32_t)p.cross, x);
              tc::tmem_ld_wait();
#pragma unroll
              for (int e = 0; e < 32; ++e) r[e] = __float_as_uint(unscale(__uint_as_float(r[e]), __uint_as_float(x[e])));
            } else {
              tc::tmem_ld_wait();
            }
            if (!row_live) continue;
            float* out = dst + i * p.chunk + b * p.wb + c;
#pragma unroll
            for (int e = 0; e < 32; e += 4)
              *reinterpret_cast<float4*>(out + e) =
                  make_float4(__uint_as_float(r[e]), __uint_as_float(r[e + 1]), __uint_as_float(r[e + 2]), __uint_as_float(r[e + 3]));
          }
    }
  }

  if (batch.independent) NRS_PDL_WAIT();   // nothing after this kernel may run ahead of its predecessor
  __syncwarp();
  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, tmem_cols);
  }
}

// The tile: the Wt x R rectangle that walks the image in the least time, by what a step costs: its UMMAs or its bytes
// through L2 (60 a clock), whichever is more, and about 150 clocks besides (118 of them measured, above); rings of two
// stages lose about a sixth (forced to two: 256 images, 64 -> 128 channels, 32 x 32 73 -> 95 us, 256 -> 128, 12 x 12 55 -> 68,
// 64 of 64 x 24 x 24 16.2 -> 16.7).
bool plan_row_tile(RowParams* p, int h, int w, int planes) {
  const int value = planes == 2 ? 2 : 4, step = planes == 2 ? 16 : 8;
  const double step_clk = (planes == 2 ? 3 : 1) * (p->chunk / p->wb) * kTaps * p->wb * 0.5;
  double best = -1.0;
  RowParams q = *p;
  for (q.Wt = 8; q.Wt <= 64; q.Wt += 8) {
    if (q.Wt - w >= 8) break;
    for (q.R = 1; q.R <= h + 1 && q.Wt * q.R <= 128; ++q.R) {
      q.P = q.Wt * q.R;
      if (q.P % step != 0) continue;
      const size_t bytes = (size_t)planes * (dy_bytes(q, value) + x_bytes(q, value));
      const int stages = (int)((size_t)(204 * 1024 - 128 * q.P * value) / bytes);
      if (stages < 2) continue;
      q.tiles_x = (w + q.Wt - 1) / q.Wt;
      q.tiles_y = (h + q.R - 1) / q.R;
      const double umma = q.P / step * step_clk, fill = bytes / 60.0;
      const double cost = (double)q.tiles_x * q.tiles_y * ((umma > fill ? umma : fill) + 150.0) * (stages < 3 ? 1.17 : 1.0);
      if (best < 0.0 || cost < best) {
        best = cost;
        q.stages = stages < kMaxStages ? stages : kMaxStages;
        *p = q;
      }
    }
  }
  return best >= 0.0;
}

// A weight gradient that may wait.
struct RowJob {
  RowEntry e;
  int planes;
  long most;   // tiles of an accumulation chain
  double flop;
  float* dw;
  int accumulate;
};
size_t smem_of(const RowParams& p, int planes) {
  const int value = planes == 2 ? 2 : 4;
  return (size_t)p.stages * planes * (dy_bytes(p, value) + x_bytes(p, value)) + (size_t)128 * p.P * value + (size_t)(2 * p.stages + 1) * 8 + 16 + 1024;
}
long max_tiles(const RowParams& p, int planes) { return planes == 2 ? tc::kMaxChainPairs / p.P : 1 << 30; }
size_t split_floats(const RowParams& p) { return (size_t)p.ctas * 128 * kTaps * p.chunk; }

template <int NPLANES, int CAP>
int launch_rows(nrs_ctx* ctx, RowJob* jobs, int n, bool independent) {
  static NrsSmemAttr attr;
  RowBatch<CAP> b{};
  size_t smem = 0;
  unsigned blocks = 0;
  b.n = n;
  b.independent = independent ? 1 : 0;
  for (int i = 0; i < n; ++i) {
    RowParams& p = jobs[i].e.p;
    const int splits = (p.n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
    const int st = nrs_fold_partial(ctx, NRS_WS_WGRAD_PARTIAL, splits * split_floats(p) * sizeof(float), &p.partial);
    if (st != NRS_OK) return st;
    p.first_block = blocks;
    blocks += (unsigned)(p.ctas * splits);
    smem = std::max(smem, smem_of(p, NPLANES));
    b.e[i] = jobs[i].e;
  }
  NRS_ENSURE_SMEM(ctx, attr, (tc_wgrad_rows_kernel<NPLANES, CAP>), smem);
  int* err = nullptr;
  int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  NRS_PDL_LAUNCH((tc_wgrad_rows_kernel<NPLANES, CAP>), blocks, kRowThreads, smem, ctx->stream, b, err);
  NRS_LAUNCHED(ctx);
  // dw[co][ci][i][j] (+)= sum over splits of the partial accumulators
  for (int i = 0; i < n && st == NRS_OK; ++i) {
    const RowParams& p = jobs[i].e.p;
    NrsFoldJob jb{};
    jb.kind = NRS_FOLD_WGRAD_ROWS;
    jb.src = p.partial; jb.dst = jobs[i].dw;
    jb.accumulate = jobs[i].accumulate;
    jb.splits = (p.n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
    jb.lanes = reduce_lanes(jb.splits);
    jb.co = p.co; jb.ci = p.ci; jb.taps = 9;
    jb.chunk = p.chunk; jb.n_chunks = p.n_chunks; jb.jtypes = p.jtypes; jb.a_blocks = p.a_blocks * p.wa / 32; jb.pack = p.pack;
    jb.split_stride = split_floats(p);
    st = nrs_fold_submit(ctx, jb);
  }
  return st;
}
template <int CAP>
int launch_rows(nrs_ctx* ctx, RowJob* jobs, int n, bool independent) {
  return jobs[0].planes == 2 ? launch_rows<2, CAP>(ctx, jobs, n, independent) : launch_rows<1, CAP>(ctx, jobs, n, independent);
}

}  // namespace

// NRS_ERR_UNSUPPORTED (no error text) for anything but 3x3 / stride 1 / pad 1 with channel counts
// that are multiples of 32.
int nrs_tc_conv_wgrad_rows(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co,
                           int kh, int kw, int stride, int pad, int accumulate) {
  if (!tc::tensor_map_encoder()) return NRS_ERR_UNSUPPORTED;
  if (kh != 3 || kw != 3 || stride != 1 || pad != 1 || ci % 32 != 0 || co % 32 != 0 || n < 1 || h < 1 || wd < 1) return NRS_ERR_UNSUPPORTED;
  const bool split3 = ctx->math_mode == NRS_MATH_3XTF32;
  const int planes = split3 ? 2 : 1;
  // A TF32 gradient on its own: rows of 16, 32 or 64 pixels, of which a tile wastes nothing.  At other widths the general
  // kernel is faster or as fast (us here / there: 8 pixels 30 / 23, 12 58 / 39, 14 20 / 17, 24 16 / 14, 28 41 / 34, 40 28 / 30,
  // 48 78 / 74, 56 61 / 62; 64 to 256 channels).  Among others of a backward pass all of them (CIFAR CNN with batch
  // normalisation: a step 1.35 ms, 1.38 without).
  if (!split3 && wd != 16 && wd != 32 && wd != 64 && !ctx->folds.active) return NRS_ERR_UNSUPPORTED;

  RowParams p{};
  p.co = co; p.ci = ci;
  p.wa = split3 && co % 64 == 0 ? 64 : 32;
  p.wb = split3 && ci % 64 == 0 ? 64 : 32;
  // (f16 pairs: two accumulators of 3 * chunk columns each in 512)
  p.chunk = split3 ? p.wb : ci % 128 == 0 ? 128 : (ci <= 128 ? ci : (ci % 96 == 0 ? 96 : (ci % 64 == 0 ? 64 : 32)));
  p.cross = kTaps * p.chunk <= 128 ? 128 : 256;
  p.n_chunks = ci / p.chunk;
  p.a_blocks = (co < 128 ? co : 128) / p.wa;
  p.pack = co <= 64 ? 1 : 0;
  p.jtypes = p.pack ? 2 : 3;
  p.m_blocks = (co + 127) / 128;
  p.ctas = p.m_blocks * p.jtypes * p.n_chunks;
  if (!plan_row_tile(&p, h, wd, planes)) return NRS_ERR_UNSUPPORTED;
  const long tiles = (long)n * p.tiles_x * p.tiles_y;
  if (tiles > 2000000000L) return NRS_ERR_UNSUPPORTED;
  p.n_tiles = (int)tiles;
  if (smem_of(p, planes) > 227 * 1024) return NRS_ERR_UNSUPPORTED;

  // tile split (of a gradient that does not wait): fill the GPU, bound the accumulation chain in 3xTF32 mode, amortise the
  // partial tile
  const int most = (int)std::min(max_tiles(p, planes), 1L << 30);
  int min_tiles = (512 + p.P - 1) / p.P;
  if (min_tiles > most) min_tiles = most;
  p.tiles_per_split = tc::plan_units_per_cta(ctx->sm_count, p.ctas, p.n_tiles, min_tiles, most, 2 + 256 / p.P);
  if ((long)p.ctas * ((p.n_tiles + p.tiles_per_split - 1) / p.tiles_per_split) > 2147483647L) return NRS_ERR_UNSUPPORTED;

  // workspaces: NHWC planes of dy and x (or the caller's registered planes).  Staged by image tiles: by transposed 32 x 32
  // tiles, as they were here, 64 images of 128 x 48 x 48 and as many of their gradient took 195 us in 3xTF32, 252 for 256 of
  // 64 and 128 x 32 x 32 (the whole gradient 309 -> 180 us, 360 -> 207).
  const size_t dy_plane = (size_t)n * h * wd * co, x_plane = (size_t)n * h * wd * ci;
  void *dy_hi = nullptr, *dy_lo = nullptr, *x_hi = nullptr, *x_lo = nullptr;
  int st = NRS_OK;
  bool may_overlap = ctx->independent_next;   // withdrawn below if this call stages an operand itself
  if (const NrsPlanes* ready = nrs_planes_find(ctx, dy, split3)) {
    dy_hi = ready->hi;
    dy_lo = ready->lo;
  } else {
    may_overlap = false;
    st = nrs_ws_planes(ctx, NRS_WS_A, dy_plane, split3, &dy_hi, &dy_lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, dy, (float*)dy_hi, (float*)dy_lo, n, co, h * wd);
    if (st != NRS_OK) return st;
  }
  if (const NrsPlanes* ready = nrs_planes_find(ctx, x, split3)) {
    x_hi = ready->hi;
    x_lo = ready->lo;
  } else {
    may_overlap = false;
    st = nrs_ws_planes(ctx, NRS_WS_B, x_plane, split3, &x_hi, &x_lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, x, (float*)x_hi, (float*)x_lo, n, ci, h * wd);
    if (st != NRS_OK) return st;
  }

  // planes viewed as [channel block][n][h][w][channels of a block]; a box is some rows of some blocks
  RowJob job{};
  auto encode = [&](CUtensorMap* m, const void* base, int c, int w, int rows, int blocks) {
    const uint64_t dim[5] = {(uint64_t)w, (uint64_t)wd, (uint64_t)h, (uint64_t)n, (uint64_t)(c / w)};
    const uint64_t str[4] = {(uint64_t)c, (uint64_t)wd * c, (uint64_t)h * wd * c, (uint64_t)w};
    const uint32_t box[5] = {(uint32_t)w, (uint32_t)p.Wt, (uint32_t)rows, 1, (uint32_t)blocks};
    return tc::encode_tmap(m, base, split3, 5, dim, str, box, true);
  };
  RowEntry& e = job.e;
  bool ok = encode(&e.dy_hi, dy_hi, co, p.wa, p.R, p.a_blocks) && encode(&e.x_hi, x_hi, ci, p.wb, p.R + 2, p.chunk / p.wb);
  if (split3) ok = ok && encode(&e.dy_lo, dy_lo, co, p.wa, p.R, p.a_blocks) && encode(&e.x_lo, x_lo, ci, p.wb, p.R + 2, p.chunk / p.wb);
  else { e.dy_lo = e.dy_hi; e.x_lo = e.x_hi; }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "tc_wgrad_rows: cuTensorMapEncodeTiled failed");
  p.range_dy = nrs_range_of(ctx, dy_hi);
  p.range_x = nrs_range_of(ctx, x_hi);
  e.p = p;
  job.planes = planes;
  job.most = split3 ? max_tiles(p, planes) : std::max((long)p.tiles_per_split, (long)tc::kMaxChainK / p.P);   // (see wgrad_queue.h)
  job.flop = 18.0 * n * h * wd * co * ci;
  job.dw = dw;
  job.accumulate = accumulate;
  if (nrs_wgrad_may_wait(ctx, dy_hi, x_hi)) {
    st = nrs_folds_limit_kept(ctx);
    if (st != NRS_OK) return st;
    NrsFolds& f = ctx->folds;
    if (!f.waiting_rows) f.waiting_rows = std::make_shared<std::vector<RowJob>>();
    static_cast<std::vector<RowJob>*>(f.waiting_rows.get())->push_back(job);
    f.waiting.push_back({dw, (size_t)co * ci * 9});
    ++f.queued;
    return NRS_OK;
  }
  return launch_rows<1>(ctx, &job, 1, may_overlap);
}

int nrs_wgrad_rows_run(nrs_ctx* ctx) {
  auto all = std::static_pointer_cast<std::vector<RowJob>>(ctx->folds.waiting_rows);
  ctx->folds.waiting_rows.reset();
  if (!all) return NRS_OK;
  constexpr double kMostPartial = 256.0 * (1 << 20);   // bytes of partial tiles in one launch
  for (size_t i = 0, e; i < all->size(); i = e) {
    RowJob* jobs = all->data() + i;
    const int planes = jobs[0].planes;
    std::vector<wgq::Piece> pieces;
    double least = 0.0, flop = 0.0;
    for (e = i; e < all->size() && (int)(e - i) < kRowBatch; ++e) {
      const RowParams& p = (*all)[e].e.p;
      const long most = (*all)[e].most;
      const double bytes = (double)split_floats(p) * sizeof(float), umma = (planes == 2 ? 3 : 1) * (p.chunk / p.wb) * kTaps * p.wb * 0.5;
      const double need = bytes * ((p.n_tiles + most - 1) / most);
      if ((*all)[e].planes != planes || (e > i && least + need > kMostPartial)) break;
      least += need;
      flop += (*all)[e].flop;
      const double fill = planes * (dy_bytes(p, planes == 2 ? 2 : 4) + x_bytes(p, planes == 2 ? 2 : 4)) / 60.0;
      pieces.push_back({p.ctas, p.n_tiles, std::max(p.P / (planes == 2 ? 16.0 : 8.0) * umma, fill) + 110.0, 4000.0, most, bytes, 0});
    }
    wgq::share_out(pieces, ctx->sm_count);
    const int n = (int)(e - i);
    for (int k = 0; k < n; ++k) jobs[k].e.p.tiles_per_split = (int)pieces[k].per;
    NrsProfScope prof(ctx, NRS_PROF_CONV_WGRAD, flop);
    const int st = n == 1 ? launch_rows<1>(ctx, jobs, 1, false) : launch_rows<kRowBatch>(ctx, jobs, n, false);
    if (st != NRS_OK) return st;
  }
  return NRS_OK;
}
