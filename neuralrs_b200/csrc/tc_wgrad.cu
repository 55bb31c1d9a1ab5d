// Convolution weight gradient as implicit GEMM on tcgen05 (TF32 / 3xTF32).
//
//   dw[co,ci,i,j] (+)= sum over (n,oy,ox) of dy[n,co,oy,ox] * x[n,ci,oy+i-p,ox+j-p]
//
// GEMM view: rows = 128 output channels, columns = (tap, ci) for a group of taps
// (up to 256 columns), reduction over output pixels.  Both operands come from
// the NHWC planes the forward / data-gradient kernels also use, so along the
// reduction (pixels) they are MN-major: a TMA box {32 channels, Wt, Ht, Nt}
// lands in shared memory as [pixel][32 channels = 128 B] (f16 pairs: 64 channels, or 32 in 64 B).  For 32-bit operands
// kind::tf32 takes MN-major data only in the 128-byte swizzle with 32-byte atoms
// (4 pixels x 128 B per swizzle group), which TMA produces with
// CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B.  A K-step of 8 pixels is two groups (SBO =
// 512 B apart); 32-channel blocks sit LBO bytes apart.  The x operand of
// tap (i,j) is the same box shifted by (i-p, j-p) with TMA zero fill as padding; a stride s
// makes it take every s-th pixel (the tensor map's element strides).  A box may reach beyond
// the image: dy is zero there, so those pixels add nothing, and rows of any width are cut into
// boxes of a multiple of 8 pixels.  Channel counts that are no multiple of 32 are fetched one
// 32-channel block at a time, with zeros beyond the last channel.
//
// The reduction is long (batch x H x W pixels) and the output tiny, so pixels
// are split across CTAs; each CTA writes its partial tile and a second kernel
// sums the partials in a fixed order (deterministic, unlike the reference's
// atomicAdd split-K, src/cuda/graph/matmul.rs:207-261) and scatters into the
// [co][ci][kh][kw] layout.  In 3xTF32 mode no CTA accumulates more than
// tc::kMaxChainPairs pixels (the tensor core's f32 accumulation error grows with the
// chain length); for TF32 mode see wgrad_queue.h.
//
// Replaces conv2d_im2col + conv2d_out2mm + matmul_nt_splitk (src/cuda/nn/conv.rs:
// 298-320).
#include "fold.h"
#include "tc_mainloop.cuh"
#include "wgrad_queue.h"

namespace {

constexpr int kWgThreads = 192;
constexpr int kMaxN = 256;        // widest UMMA

struct WgradParams {
  int Wt, Ht, Nt, tiles_y, tiles_x;  // pixel tile (box) geometry in dy space
  int kp;                         // pixels per tile = Wt*Ht*Nt (multiple of 8)
  int n_tiles;                    // pixel tiles in all
  int tiles_per_split;
  int co, ci, kh, kw, pad, stride;
  int taps_per_group, n_groups;   // taps handled by one CTA
  int wa, wb;                     // channels of a block of dy, of x: 32, or 64 (f16: rows of 128 bytes)
  int cblocks;                    // ceil(ci / wb)
  int a_box_blocks;               // blocks of dy one box brings (128 channels at most)
  int ragged_a, ragged_x;         // channel count no multiple of 32: one 4-D box per block instead of one 5-D box for all
  int m_blocks;                   // ceil(co / 128)
  float* partial;                 // [split][m_block][group][col_block][128][group_cols]
  int group_cols;                 // taps_per_group * cblocks * wb; in column blocks: the width of one (64, 128 or 256)
  int col_blocks;                 // column blocks of the input channels, each its own CTA (more than 256 channels, or 1x1)
  int stages;
  int ctas;                       // per split
  unsigned first_block;           // of this gradient's in the launch
  const NrsRange *range_dy, *range_x;   // 3xTF32
  float* direct;                  // 1x1, one split, no accumulation: the tile is the result; written straight to dw[co][ci]
};

// The gradients of one launch.
struct WgradEntry {
  CUtensorMap dy_hi, dy_lo, x_hi, x_lo;
  WgradParams p;
};
template <int CAP>
struct WgradBatch {
  WgradEntry e[CAP];
  int n;
  int independent;                // reads nothing the kernel launched just before it wrote (NRS_PDL_PROLOGUE)
};
constexpr int kWgBatch = 16;

template <int NPLANES, int CAP>
__global__ void __launch_bounds__(kWgThreads, 1)
tc_wgrad_kernel(const __grid_constant__ WgradBatch<CAP> batch, int* __restrict__ err_flag) {
  extern __shared__ uint8_t smem_raw[];
  int entry = 0;
  while (CAP > 1 && entry + 1 < batch.n && batch.e[entry + 1].p.first_block <= blockIdx.x) ++entry;
  const WgradEntry& en = batch.e[entry];
  const WgradParams& p = en.p;
  const CUtensorMap &tm_dy_hi = en.dy_hi, &tm_dy_lo = en.dy_lo, &tm_x_hi = en.x_hi, &tm_x_lo = en.x_lo;
  const int STAGES = p.stages, n_cols = p.group_cols /*UMMA N, multiple of 16*/;
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const uint32_t value = NPLANES == 2 ? 2u : 4u;
  const uint32_t a_blk = (uint32_t)(p.kp * p.wa) * value, b_blk = (uint32_t)(p.kp * p.wb) * value;   // one block of one plane
  const uint32_t a_bytes = (uint32_t)(p.kp * 128) * value;         // per plane
  const uint32_t b_bytes = (uint32_t)(p.kp * p.group_cols) * value;
  const uint32_t stage_bytes = NPLANES * (a_bytes + b_bytes);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + STAGES * stage_bytes);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* accum_bar = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(accum_bar + 1);

  const int warp = (int)tc::uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int local = (int)(blockIdx.x - p.first_block), split = local / p.ctas, cta = local - split * p.ctas;
  const int cbk = (int)tc::uniform(cta % p.col_blocks);
  const int mg = cta / p.col_blocks;
  const int mb = (int)tc::uniform(mg / p.n_groups), grp = mg - mb * p.n_groups;
  // blocks of x this CTA's columns cover (a column block of a wide layer may be ragged)
  const int most = p.group_cols / p.wb, cblocks = p.col_blocks > 1 ? min(most, p.cblocks - cbk * most) : p.cblocks;
  const int t_begin = split * p.tiles_per_split;
  const int t_end = min(p.n_tiles, t_begin + p.tiles_per_split);
  const int ntiles = t_end - t_begin;
  const int tap0 = grp * p.taps_per_group;
  const int ntaps = min(p.taps_per_group, p.kh * p.kw - tap0);

  if (warp == 0 && lane == 0) {
    tc::prefetch_tmap(&tm_dy_hi);
    tc::prefetch_tmap(&tm_x_hi);
    if (NPLANES == 2) { tc::prefetch_tmap(&tm_dy_lo); tc::prefetch_tmap(&tm_x_lo); }
    for (int s = 0; s < STAGES; ++s) { tc::mbar_init(&full_bar[s], 1); tc::mbar_init(&empty_bar[s], 1); }
    tc::mbar_init(accum_bar, 1);
    tc::fence_barrier_init();
  }
  if (warp == 1) {
    tc::tmem_alloc(tmem_slot, NPLANES * kMaxN);
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
    // ---------------- TMA producer: one pixel tile per ring slot
    // One 5-D box per operand plane brings all 32-channel blocks of a pixel tile at once
    // (the channel-block index is the outermost box dimension), so a tile costs
    // planes x (1 + taps) TMA instructions instead of one per block.
    // (a ragged last column block still receives a full box: TMA zero-fills the blocks beyond the tensor)
    // The warp's own instructions bound layers with many loads a tile: places are stepped along, and what comes out of a
    // division goes through tc::uniform, so that operands stay in uniform registers.  (Multiplied out per load from the job's
    // parameters: 135 us instead of 117 for 48 -> 128 channels, 5x5, 118 x 29 x 26 in TF32, 199 instead of 152 in 3xTF32; 48
    // instead of 39 for 256 -> 128, 3x3, 256 x 12 x 12.)
    const int x_blocks = p.col_blocks > 1 ? most : p.cblocks;
    const uint32_t tx = NPLANES * ((uint32_t)p.a_box_blocks * a_blk + (uint32_t)(ntaps * x_blocks) * b_blk);
    const int i_first = (int)tc::uniform(tap0 / p.kw), j_first = tap0 - i_first * p.kw;
    int xt = (int)tc::uniform(t_begin % p.tiles_x), yt = (int)tc::uniform(t_begin / p.tiles_x);   // the tile's place, stepped along
    int nt = (int)tc::uniform(yt / p.tiles_y);
    yt -= nt * p.tiles_y;
    const int x_first = cbk * most * p.wb, a_first = mb * 128;   // channels; the boxes of whole counts go by blocks
    const int x_block = cbk * most, a_block = p.wa == 64 ? mb * 2 : mb * 4;
    const uint32_t tap_bytes = (uint32_t)p.cblocks * b_blk;
    int issued = 0, s = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int it = 0; it < ntiles; ++it, ++issued) {
      if (!tc::mbar_wait_warp(&empty_bar[s], ph ^ 1u)) { ok = false; break; }
      const int n0 = nt * p.Nt, y0 = yt * p.Ht, x0 = xt * p.Wt;
      const int xx0 = x0 * p.stride - p.pad, xy0 = y0 * p.stride - p.pad;
      uint8_t* st = smem + (size_t)s * stage_bytes;
      uint64_t* bar = &full_bar[s];
      if (tc::elect_one()) {
        tc::mbar_expect_tx(bar, tx);
#pragma unroll
        for (int pl = 0; pl < NPLANES; ++pl) {
          const CUtensorMap* tdy = pl == 0 ? &tm_dy_hi : &tm_dy_lo;
          const CUtensorMap* txm = pl == 0 ? &tm_x_hi : &tm_x_lo;
          uint8_t* a_dst = st + pl * (a_bytes + b_bytes);
          uint8_t* dst = a_dst + a_bytes;
          if (p.ragged_a) {
            int ch = a_first;
#pragma unroll 1
            for (int b = 0; b < p.a_box_blocks; ++b, a_dst += a_blk, ch += p.wa) tc::tma_load_4d(a_dst, tdy, bar, ch, x0, y0, n0);
          } else {
            tc::tma_load_5d(a_dst, tdy, bar, 0, x0, y0, n0, a_block);
          }
          int tj = j_first, xx = xx0 + j_first, xy = xy0 + i_first;
#pragma unroll 1
          for (int t = 0; t < ntaps; ++t) {
            if (p.ragged_x) {
              uint8_t* d = dst;
              int ch = x_first;
#pragma unroll 1
              for (int b = 0; b < x_blocks; ++b, d += b_blk, ch += p.wb) tc::tma_load_4d(d, txm, bar, ch, xx, xy, n0);
            } else {
              tc::tma_load_5d(dst, txm, bar, 0, xx, xy, n0, x_block);
            }
            dst += tap_bytes;
            ++xx;
            if (++tj == p.kw) { tj = 0; xx = xx0; ++xy; }
          }
        }
      }
      __syncwarp();
      if (++s == STAGES) { s = 0; ph ^= 1u; }
      if (++xt == p.tiles_x) {
        xt = 0;
        if (++yt == p.tiles_y) { yt = 0; ++nt; }
      }
    }
    if (!ok) {
      if (lane == 0) atomicExch(err_flag, tc::kErrProducerWait);
      for (int it = (issued > STAGES ? issued - STAGES : 0); it < issued; ++it) {
        const int sj = it % STAGES;
        if (!tc::mbar_wait_warp(&full_bar[sj], (uint32_t)(it / STAGES) & 1u)) {
          if (lane == 0) atomicExch(err_flag, tc::kErrDrainWait);
          break;
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- UMMA issuer: both operands MN-major, K-step = 8 pixels (f16: 16) = 1024 B
    const uint32_t idesc = NPLANES == 2 ? tc::make_idesc_f16(128, n_cols, true, true) : tc::make_idesc_tf32(128, n_cols, true, true);
    // every field but the start address (bytes >> 4), and a K-step's bytes >> 4
    auto desc = [](int w, uint32_t blk) {
      return NPLANES == 1 ? tc::make_smem_desc_sw128_32b(0, blk, 512) : w == 64 ? tc::make_smem_desc_sw128(0, blk, 1024) : tc::make_smem_desc_sw64(0, blk, 512);
    };
    const uint64_t da = desc(p.wa, a_blk), db = desc(p.wb, b_blk);
    const uint32_t step_a = NPLANES == 2 && p.wa == 64 ? 128u : 64u, step_b = NPLANES == 2 && p.wb == 64 ? 128u : 64u;
    bool ok = true;
    const int ksteps = p.kp / (NPLANES == 2 ? 16 : 8);
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < ntiles; ++it) {
      if (!tc::mbar_wait_warp(&full_bar[s], ph)) { ok = false; break; }
      const uint32_t a_hi = tc::smem_u32(smem + (size_t)s * stage_bytes) >> 4;
      const uint32_t b_hi = a_hi + (a_bytes >> 4);
      const uint32_t a_lo = b_hi + (b_bytes >> 4);
      const uint32_t b_lo = a_lo + (a_bytes >> 4);
      if (tc::elect_one()) {
#pragma unroll 2
        for (int k = 0; k < ksteps; ++k) {
          const uint64_t ah = da + (a_hi + (uint32_t)k * step_a), bh = db + (b_hi + (uint32_t)k * step_b);
          const uint32_t more = (it | k) != 0;
          if (NPLANES == 2) {
            tc::umma_f16(tmem_base, ah, bh, idesc, more);
            tc::umma_f16(tmem_base + kMaxN, ah, db + (b_lo + (uint32_t)k * step_b), idesc, more);
            tc::umma_f16(tmem_base + kMaxN, da + (a_lo + (uint32_t)k * step_a), bh, idesc, 1);
          } else {
            tc::umma_tf32(tmem_base, ah, bh, idesc, more);
          }
        }
        tc::umma_commit(&empty_bar[s]);
      }
      __syncwarp();
      if (++s == STAGES) { s = 0; ph ^= 1u; }
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
      const int live_cols = (p.col_blocks > 1 ? cblocks : ntaps * p.cblocks) * p.wb;
      float* dst = p.direct ? p.direct + (size_t)(mb * 128 + row) * p.ci + (size_t)cbk * p.group_cols
                            : p.partial + (((((size_t)split * p.m_blocks + mb) * p.n_groups + grp) * p.col_blocks + cbk) * 128 + row) *
                                              p.group_cols;
      const bool row_live = mb * 128 + row < p.co;
      const pr::Unscale unscale(NPLANES == 2 ? p.range_dy->bound : 1.0f, NPLANES == 2 ? p.range_x->bound : 1.0f);
#pragma unroll 1
      for (int c = 0; c < (live_cols + 31) / 32; ++c) {
        uint32_t r[32];
        const uint32_t at = tmem_base + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 32);
        tc::tmem_ld_32x32(at, r);
        if constexpr (NPLANES == 2) {
          uint32_t x[32];
          tc::tmem_ld_32x32(at + kMaxN, x);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; ++j) r[j] = __float_as_uint(unscale(__uint_as_float(r[j]), __uint_as_float(x[j])));
        } else {
          tc::tmem_ld_wait();
        }
        if (row_live) {
#pragma unroll
          for (int j = 0; j < 32; j += 4)
            if (c * 32 + j < live_cols)
              *reinterpret_cast<float4*>(dst + c * 32 + j) =
                  make_float4(__uint_as_float(r[j]), __uint_as_float(r[j + 1]), __uint_as_float(r[j + 2]), __uint_as_float(r[j + 3]));
        }
      }
    }
  }

  if (batch.independent) NRS_PDL_WAIT();   // nothing after this kernel may run ahead of its predecessor
  __syncwarp();
  tc::tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::tc_fence_after_sync();
    tc::tmem_dealloc(tmem_base, NPLANES * kMaxN);
  }
}

// Pixel tile = one TMA box {32 channels, Wt, Ht, Nt} of kp = Wt*Ht*Nt pixels, a multiple of 8 (a K-step) up to 64.
// Boxes of whole rows, or of a multiple of 8 pixels of a row; the one that walks the fewest pixels, padding included,
// is taken, where every tile costs half a pixel's worth per TMA load (measured: 3000 x 2048 x 512 in 3xTF32 35.8 us with
// slots of 16 pixels, 39.2 with two slots of 32; but with the 12 loads of five taps a slot of 16 costs 24.7 us against
// 18.6), and a ring of fewer than three slots a few percent.  A box may reach past the last image too (a few 1x1 "images").
void plan_pixel_box(WgradParams* p, int n, int oh, int ow, int planes, size_t bytes_per_pixel) {
  const int step = planes == 2 ? 16 : 8, most = planes == 2 ? 128 : 64;   // pixels of a K-step; of a box
  const int loads = planes * ((p->ragged_a ? 128 / p->wa : 1) + p->taps_per_group * (p->ragged_x ? p->cblocks : 1));
  const double per_tile = loads > 4 ? 0.5 * loads : 2.0;
  double best = -1.0;
  for (int c = 0; c <= most / 8; ++c) {
    const int Wt = c == 0 ? ow : 8 * c;
    if (Wt > most || Wt * p->stride > 256 || (c > 0 && Wt - ow >= 8)) continue;
    for (int Ht = 1; Ht <= (c > 0 && planes == 2 ? oh + 1 : oh) && Wt * Ht <= most && Ht * p->stride <= 256; ++Ht) {
      const bool whole = Ht == oh && Wt >= ow;
      for (int Nt = 1; Nt <= (whole ? n + step - 1 : 1) && Wt * Ht * Nt <= most; ++Nt) {
        const int kp = Wt * Ht * Nt;
        if (kp % step != 0) continue;
        const int stages = (int)((200 * 1024) / (bytes_per_pixel * kp));
        if (stages < 2) continue;
        const long tiles = (long)((ow + Wt - 1) / Wt) * ((oh + Ht - 1) / Ht) * ((n + Nt - 1) / Nt);
        const double cost = (double)tiles * (kp + per_tile) * (stages < 3 ? 1.06 : 1.0);
        if (best < 0.0 || cost < best) {
          best = cost;
          p->Wt = Wt; p->Ht = Ht; p->Nt = Nt; p->kp = kp;
        }
      }
    }
  }
}

}  // namespace

namespace {

// A weight gradient that may wait.
struct WgradJob {
  WgradEntry e;
  int planes;
  long most;   // tiles of an accumulation chain
  double flop;
  bool linear;
  float* dw;
  int accumulate, out_cols;
  bool can_be_direct;
};
size_t pixel_bytes_of(const WgradParams& p) { return (size_t)(128 + p.group_cols) * 4; }   // both operands, all planes
size_t split_floats(const WgradParams& p) { return (size_t)p.ctas * 128 * p.group_cols; }
long max_tiles(const WgradParams& p, int planes) { return planes == 2 ? std::max(1, tc::kMaxChainPairs / p.kp) : 1 << 30; }

template <int NPLANES, int CAP>
int launch_wgrad(nrs_ctx* ctx, WgradJob* jobs, int n, bool independent) {
  static NrsSmemAttr attr;
  WgradBatch<CAP> b{};
  size_t smem = 0;
  unsigned blocks = 0;
  b.n = n;
  b.independent = independent ? 1 : 0;
  for (int i = 0; i < n; ++i) {
    WgradParams& p = jobs[i].e.p;
    const int splits = (p.n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
    // a single split of a 1x1 "convolution" (A^T B) that overwrites its output needs no second pass
    p.direct = splits == 1 && jobs[i].can_be_direct ? jobs[i].dw : nullptr;
    const int st = p.direct ? NRS_OK : nrs_fold_partial(ctx, NRS_WS_WGRAD_PARTIAL, splits * split_floats(p) * sizeof(float), &p.partial);
    if (st != NRS_OK) return st;
    p.first_block = blocks;
    blocks += (unsigned)(p.ctas * splits);
    smem = std::max(smem, p.stages * pixel_bytes_of(p) * p.kp + 1024 + 256);
    b.e[i] = jobs[i].e;
  }
  NRS_ENSURE_SMEM(ctx, attr, (tc_wgrad_kernel<NPLANES, CAP>), smem);
  int* err = nullptr;
  int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  NRS_PDL_LAUNCH((tc_wgrad_kernel<NPLANES, CAP>), blocks, kWgThreads, smem, ctx->stream, b, err);
  NRS_LAUNCHED(ctx);
  // dw[co][ci][tap] (+)= sum over splits of partial[split][mb][grp][col block][row][t*cblocks*wb + c]
  for (int i = 0; i < n && st == NRS_OK; ++i) {
    const WgradParams& p = jobs[i].e.p;
    if (p.direct) continue;
    NrsFoldJob j{};
    j.kind = NRS_FOLD_WGRAD;
    j.src = p.partial; j.dst = jobs[i].dw;
    j.accumulate = jobs[i].accumulate;
    j.splits = (p.n_tiles + p.tiles_per_split - 1) / p.tiles_per_split;
    j.lanes = reduce_lanes(j.splits);
    j.co = p.co; j.ci = p.ci; j.taps = p.kh * p.kw;
    j.taps_per_group = p.taps_per_group; j.n_groups = p.n_groups; j.col_blocks = p.col_blocks; j.cblocks = p.cblocks * p.wb / 32;
    j.group_cols = p.group_cols;
    j.out_cols = jobs[i].out_cols;
    j.split_stride = split_floats(p);
    st = nrs_fold_submit(ctx, j);
  }
  return st;
}
template <int CAP>
int launch_wgrad(nrs_ctx* ctx, WgradJob* jobs, int n, bool independent) {
  return jobs[0].planes == 2 ? launch_wgrad<2, CAP>(ctx, jobs, n, independent) : launch_wgrad<1, CAP>(ctx, jobs, n, independent);
}

}  // namespace

int nrs_tc_conv_wgrad(nrs_ctx* ctx, const float* x, const float* dy, float* dw, int n, int ci, int h, int wd, int co,
                      int kh, int kw, int stride, int pad, int accumulate, int out_cols) {
  if (!tc::tensor_map_encoder()) return NRS_ERR_UNSUPPORTED;
  if (n < 1 || stride > 8) return NRS_ERR_UNSUPPORTED;
  const int oh = (h + 2 * pad - kh) / stride + 1, ow = (wd + 2 * pad - kw) / stride + 1;
  if (ow < 1 || oh < 1) return NRS_ERR_UNSUPPORTED;
  const bool split3 = ctx->math_mode == NRS_MATH_3XTF32;
  const int planes = split3 ? 2 : 1;

  WgradParams p{};
  p.co = co; p.ci = ci; p.kh = kh; p.kw = kw; p.pad = pad; p.stride = stride;
  // f16: blocks of 64 channels, unless that pads much more (TMA brings rows of 64 bytes at half the rate of 128)
  auto padded = [](int c, int w) { return (c + w - 1) / w * w; };
  p.wa = split3 && co > 32 ? 64 : 32;
  p.wb = split3 && 20 * padded(ci, 64) <= 23 * padded(ci, 32) ? 64 : 32;
  p.cblocks = padded(ci, p.wb) / p.wb;
  p.ragged_a = co % p.wa != 0;
  p.ragged_x = ci % p.wb != 0;
  p.m_blocks = (co + 127) / 128;
  const int taps = kh * kw;
  const int tap_cols = p.cblocks * p.wb;
  int tpg = tap_cols <= kMaxN ? kMaxN / tap_cols : 1;
  if (tpg > taps) tpg = taps;
  p.n_groups = (taps + tpg - 1) / tpg;
  p.taps_per_group = (taps + p.n_groups - 1) / p.n_groups;
  p.group_cols = p.taps_per_group * tap_cols;
  p.col_blocks = 1;
  if (tap_cols > kMaxN) {     // the input channels are cut into column blocks of 256, one CTA each
    p.col_blocks = (ci + kMaxN - 1) / kMaxN;
    p.n_groups = taps;
    p.taps_per_group = 1;
    p.group_cols = kMaxN;
  }
  const bool can_be_direct = taps == 1 && ci % p.wb == 0 && !accumulate && !out_cols && (reinterpret_cast<uintptr_t>(dw) & 15) == 0;
  // The pixel box of a plan, and the ring its operands allow; false where there is none.
  auto box = [&](WgradParams* q) {
    const size_t pixel_bytes = pixel_bytes_of(*q);
    q->kp = 0;
    plan_pixel_box(q, n, oh, ow, planes, pixel_bytes);
    if (q->kp == 0) return false;
    q->tiles_x = (ow + q->Wt - 1) / q->Wt;
    q->tiles_y = (oh + q->Ht - 1) / q->Ht;
    const long n_tiles = (long)((n + q->Nt - 1) / q->Nt) * q->tiles_y * q->tiles_x;
    if (n_tiles > 2147483647L) return false;
    q->n_tiles = (int)n_tiles;
    q->stages = std::min(6, (int)((200 * 1024) / (pixel_bytes * q->kp)));
    q->ctas = q->m_blocks * q->n_groups * q->col_blocks;
    return q->stages >= 2;
  };
  const NrsPlanes *dy_ready = nrs_planes_find(ctx, dy, split3), *x_ready = nrs_planes_find(ctx, x, split3);
  const bool waits = dy_ready && x_ready && nrs_wgrad_may_wait(ctx, dy_ready->hi, x_ready->hi);
  int tps = 0;   // pixel tiles per CTA
  // The split that fills the GPU with this product alone, and bounds the accumulation chain in 3xTF32 mode.
  auto alone = [&](const WgradParams& q) {
    const int most = (int)std::min(max_tiles(q, planes), 1L << 30);
    int min_tiles = 512 / q.kp;   // amortise the prologue and the partial-tile store
    // ... unless that leaves most of the GPU idle
    while (min_tiles > 4 && (long)(q.n_tiles / min_tiles) * q.ctas < ctx->sm_count / 2) min_tiles /= 2;
    if (min_tiles > most) min_tiles = most;
    return tc::plan_units_per_cta(ctx->sm_count, q.ctas, q.n_tiles, min_tiles, most, 8);
  };
  if (waits) {   // shared out with the others; wide column blocks, which read the least
    if (tap_cols > kMaxN) {
      p.col_blocks = (tap_cols + kMaxN - 1) / kMaxN;
      p.n_groups = taps;
      p.taps_per_group = 1;
      p.group_cols = kMaxN;
    }
    if (!box(&p)) return NRS_ERR_UNSUPPORTED;
    tps = p.n_tiles;
  } else if (taps == 1) {
    // A^T B: columns per CTA and pixel split together, by what a CTA takes (its UMMAs, 46 clocks at least, or its operands'
    // way at about 60 bytes a clock; 2500 clocks and the store of its tile besides) and the second pass, which reads
    // splits + 1 times the output at about 1.1 KB a clock.  No split is longer than an accumulation chain may be.
    // (dW of 256 x 256 over 4096 rows: with 256 columns eight splits of two CTAs.)
    const WgradParams base = p;
    double best = -1.0;
    for (int cols : {256, 128, 64}) {
      WgradParams q = base;
      if (cols < tap_cols || tap_cols > kMaxN) {
        q.col_blocks = (tap_cols + cols - 1) / cols;
        q.n_groups = q.taps_per_group = 1;
        q.group_cols = cols;
      } else if (cols != 256) {
        continue;   // one CTA takes all columns as it is
      }
      if (!box(&q)) continue;
      const int ctas = q.ctas;
      const long most = max_tiles(q, planes);
      const double umma = (split3 ? 3.0 : 2.0) * std::max(q.group_cols / 2, 47), fill = 16.0 * pixel_bytes_of(q) / 60.0;   // per 16 pixels
      for (int i = 1, last = 0; i <= 96; ++i) {   // up to 64 splits, then whole waves
        const long s = i <= 64 ? i : (long)(i - 64) * ctx->sm_count / ctas;
        if (s < 1 || (i > 64 && s <= 64)) continue;
        const int per = (int)((q.n_tiles + s - 1) / s);
        if (per > most || per == last) continue;
        last = per;
        const long splits = (q.n_tiles + per - 1) / per;
        const double rounds = (double)((ctas * splits + ctx->sm_count - 1) / ctx->sm_count);
        const double fold = s == 1 && can_be_direct ? 0.0 : (splits + 1.0) * co * ci * 4 / 1100.0;
        const double cost = rounds * (per * (q.kp / 16.0) * std::max(umma, fill) + 2500.0 + 4.0 * q.group_cols) + fold;
        if (best < 0.0 || cost < best) {
          best = cost;
          tps = per;
          p = q;
        }
      }
    }
    // (a reduction that needs more splits by the chain limit alone)
    if (best < 0.0 && box(&p)) tps = (int)std::min((long)p.n_tiles, max_tiles(p, planes));
    if (tps == 0 || !box(&p)) return NRS_ERR_UNSUPPORTED;
  } else {
    if (!box(&p)) return NRS_ERR_UNSUPPORTED;
    tps = alone(p);
  }
  p.tiles_per_split = tps;
  if ((long)p.ctas * ((p.n_tiles + tps - 1) / tps) > 2147483647L) return NRS_ERR_UNSUPPORTED;

  // workspaces: NHWC planes of dy and x
  const int dy_ld = nrs_plane_ld(co), x_ld = nrs_plane_ld(ci);
  const size_t dy_plane = (size_t)n * oh * ow * dy_ld, x_plane = (size_t)n * h * wd * x_ld;
  void *dy_hi = nullptr, *dy_lo = nullptr, *x_hi = nullptr, *x_lo = nullptr;
  int st = NRS_OK;
  bool may_overlap = ctx->independent_next;   // withdrawn below if this call stages an operand itself
  if (dy_ready) {
    dy_hi = dy_ready->hi;
    dy_lo = dy_ready->lo;
  } else {
    may_overlap = false;
    st = nrs_ws_planes(ctx, NRS_WS_A, dy_plane, split3, &dy_hi, &dy_lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, dy, (float*)dy_hi, (float*)dy_lo, n, co, oh * ow);
    if (st != NRS_OK) return st;
  }
  if (x_ready) {
    x_hi = x_ready->hi;
    x_lo = x_ready->lo;
  } else {
    may_overlap = false;
    st = nrs_ws_planes(ctx, NRS_WS_B, x_plane, split3, &x_hi, &x_lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, x, (float*)x_hi, (float*)x_lo, n, ci, h * wd);
    if (st != NRS_OK) return st;
  }

  // Planes viewed as [channel block][n][h][w][32 or 64 channels], the block index outermost, so that one box brings all
  // blocks; with a ragged channel count as [n][h][w][channels], one block per box.
  WgradJob job{};
  CUtensorMap maps[4];
  p.a_box_blocks = std::min(padded(co, p.wa), 128) / p.wa;
  auto encode = [&](CUtensorMap* m, void* base, bool ragged, int c, int w, int ld, int img_h, int img_w, int step, int blocks) {
    const uint64_t dim[5] = {(uint64_t)(ragged ? c : w), (uint64_t)img_w, (uint64_t)img_h, (uint64_t)n, (uint64_t)(c / w)};
    const uint64_t str[4] = {(uint64_t)ld, (uint64_t)img_w * ld, (uint64_t)img_h * img_w * ld, (uint64_t)w};
    const uint32_t box[5] = {(uint32_t)w, (uint32_t)p.Wt, (uint32_t)p.Ht, (uint32_t)p.Nt, (uint32_t)blocks};
    const uint32_t es[5] = {1, (uint32_t)step, (uint32_t)step, 1, 1};
    return tc::encode_tmap(m, base, split3, ragged ? 4 : 5, dim, str, box, true, es);
  };
  const int x_blocks = p.col_blocks > 1 ? p.group_cols / p.wb : p.cblocks;
  bool ok = encode(&maps[0], dy_hi, p.ragged_a, co, p.wa, dy_ld, oh, ow, 1, p.a_box_blocks) &&
            encode(&maps[2], x_hi, p.ragged_x, ci, p.wb, x_ld, h, wd, stride, x_blocks);
  if (split3) ok = ok && encode(&maps[1], dy_lo, p.ragged_a, co, p.wa, dy_ld, oh, ow, 1, p.a_box_blocks) &&
                   encode(&maps[3], x_lo, p.ragged_x, ci, p.wb, x_ld, h, wd, stride, x_blocks);
  else { maps[1] = maps[0]; maps[3] = maps[2]; }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "tc_wgrad: cuTensorMapEncodeTiled failed");
  p.range_dy = nrs_range_of(ctx, dy_hi);
  p.range_x = nrs_range_of(ctx, x_hi);
  job.e = WgradEntry{maps[0], maps[1], maps[2], maps[3], p};
  job.planes = planes;
  job.most = split3 ? max_tiles(p, planes) : std::max((long)alone(p), (long)tc::kMaxChainK / p.kp);   // (see wgrad_queue.h)
  job.flop = 2.0 * n * oh * ow * co * ci * taps;
  job.linear = oh * ow == 1;
  job.dw = dw;
  job.accumulate = accumulate;
  job.out_cols = out_cols;
  job.can_be_direct = can_be_direct;
  if (!waits) return launch_wgrad<1>(ctx, &job, 1, may_overlap);
  st = nrs_folds_limit_kept(ctx);
  if (st != NRS_OK) return st;
  NrsFolds& f = ctx->folds;
  if (!f.waiting_tiles) f.waiting_tiles = std::make_shared<std::vector<WgradJob>>();
  static_cast<std::vector<WgradJob>*>(f.waiting_tiles.get())->push_back(job);
  f.waiting.push_back({dw, (size_t)co * ci * taps});
  ++f.queued;
  return NRS_OK;
}

int nrs_wgrad_tiles_run(nrs_ctx* ctx) {
  auto all = std::static_pointer_cast<std::vector<WgradJob>>(ctx->folds.waiting_tiles);
  ctx->folds.waiting_tiles.reset();
  if (!all) return NRS_OK;
  constexpr double kMostPartial = 256.0 * (1 << 20);   // bytes of partial tiles in one launch
  for (size_t i = 0, e; i < all->size(); i = e) {
    WgradJob* jobs = all->data() + i;
    const int planes = jobs[0].planes;
    std::vector<wgq::Piece> pieces;
    double least = 0.0, flop = 0.0, linear = 0.0;
    for (e = i; e < all->size() && (int)(e - i) < kWgBatch; ++e) {
      const WgradParams& p = (*all)[e].e.p;
      const long most = (*all)[e].most;
      const double bytes = (double)split_floats(p) * sizeof(float), need = bytes * ((p.n_tiles + most - 1) / most);
      if ((*all)[e].planes != planes || (e > i && least + need > kMostPartial)) break;
      least += need;
      flop += (*all)[e].flop;
      if ((*all)[e].linear) linear += (*all)[e].flop;
      const double umma = p.kp / 16.0 * (planes == 2 ? 3.0 : 2.0) * std::max(p.group_cols / 2, 47), fill = p.kp * pixel_bytes_of(p) / 60.0;
      pieces.push_back({p.ctas, p.n_tiles, std::max(umma, fill), 2500.0 + 4.0 * p.group_cols, most, bytes, 0});
    }
    wgq::share_out(pieces, ctx->sm_count);
    const int n = (int)(e - i);
    for (int k = 0; k < n; ++k) jobs[k].e.p.tiles_per_split = (int)pieces[k].per;
    NrsProfScope prof(ctx, 2.0 * linear > flop ? NRS_PROF_GEMM : NRS_PROF_CONV_WGRAD, flop);   // (a launch of both: by the larger part)
    const int st = n == 1 ? launch_wgrad<1>(ctx, jobs, 1, false) : launch_wgrad<kWgBatch>(ctx, jobs, n, false);
    if (st != NRS_OK) return st;
  }
  return NRS_OK;
}

// C[m,n] (+)= A^T B for A stored [k][m] and B stored [k][n] (both row-major) without transposing either:
// the reduction index k is the slow index of both operands, which is what the weight-gradient kernel above
// consumes (a 1x1 convolution over k "pixels": rows = A's columns, columns = B's columns).  The weight
// gradient of a Linear layer, dW = x^T dz, is this product on the activations' own row-major planes.
// NRS_ERR_UNSUPPORTED (no error text) for products too thin for a 128-row tile.
int nrs_tc_gemm_tn(nrs_ctx* ctx, int m, int n, int k, const float* a, const float* b, float* c, int accumulate) {
  if (m < 32 || n < 32 || k < 8) return NRS_ERR_UNSUPPORTED;
  // Outputs of up to 4 M elements (the Linear layers of the CNN and transformer configurations).  Larger ones
  // (4096 x 4096 hidden layers) stay on the persistent GEMM kernel, which reads both operands as stored too
  // (transposed while they are staged where m or n is no multiple of 32) and whose rastered tiles reuse them through L2.
  if ((long)m * n > (4L << 20)) return NRS_ERR_UNSUPPORTED;
  return nrs_tc_conv_wgrad(ctx, /*x=*/b, /*dy=*/a, /*dw=*/c, /*n=*/k, /*ci=*/n, 1, 1, /*co=*/m, 1, 1, 1, 0, accumulate);
}
