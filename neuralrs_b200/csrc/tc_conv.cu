// Convolution forward and data gradient as implicit GEMM on tcgen05 (TF32 / 3xTF32).
//
// No im2col matrix exists anywhere.  The activation is staged once as NHWC
// (channels innermost) planes; output pixels are GEMM rows (a tile is Wt x Ht x Nt
// = up to 128 pixels of Nt images), output channels are GEMM columns, and the
// reduction runs over (tap, 32-channel block).  For every tap the A slice is ONE
// 4-D TMA box {32 channels, Wt, Ht, Nt} whose spatial origin is shifted by the
// tap offset; rows or columns that fall outside the image are zero-filled by TMA,
// which is exactly the zero padding, and so are the channels beyond the last one of
// a ragged channel block.  (The shift lands on the W/H coordinates; the innermost,
// 16-byte-aligned coordinate is the channel block.)  The B slice is a plain 2-D box
// of the re-laid-out weights [out_ch][(tap, in_ch padded to 32)].
//
//   forward        y[n,co,oy,ox]  = act(b[co] + sum x[n,ci,oy*s+i-p,ox*s+j-p] w[co,ci,i,j])
//   data gradient  dx[n,ci,y,x] (+)= sum dy[n,co,(y+p-i)/s,(x+p-j)/s] w[co,ci,i,j]
// are the same kernel with the tap sign flipped and the roles of the channel
// counts exchanged.  A stride s makes the forward box take every s-th pixel (the
// tensor map's element strides).  The data gradient of a strided layer falls into
// s*s independent stride-1 problems, one per residue of (y+p, x+p) modulo s: each
// reads the taps of its own residue only (no multiplication by the zeros between
// the pixels of dy) and writes every s-th pixel of dx.  The epilogue writes NCHW
// directly: for a fixed channel the 32 lanes of a warp hold 32 consecutive pixels,
// so every store of a stride-1 problem is a full 128-byte line.
//
// Measured (x[64,48,57,57] -> 80 channels, 3x3, stride 2, 3xTF32): forward 220 us as an FFMA implicit GEMM, 61 here;
// data gradient 1706 us (three quarters of its products were with zeros), 97 in its four residues.
//
// Reference counterparts: conv2d_im2col + matmul_nn + conv2d_col2out (forward),
// conv2d_out2mm + matmul_tn + conv2d_col2im (data gradient) — src/cuda/nn/conv.rs:27-149,
// 244-312.
#include <cstring>

#include "tc_mainloop.cuh"

namespace {

template <int EPI, bool SLAB>
struct ConvPolicyOf {
  static constexpr bool kConv = true;
  static constexpr bool kSlab = SLAB;
  // A tile's pixels in the order of its box: (x, y, image), in slabs (x, image, y), so that a row of all its images is one
  // stretch of the slab and the next vertical tap starts Wt * Nt pixels on.
  NrsFastDiv div_Wt, div_mid /*Ht; slabs: Nt*/, div_tiles_x, div_tiles_y, div_cblocks;
  int Wt, Ht, Nt, tiles_x, tiles_y;   // pixel tile in the space of (u, v), the pixels this launch computes
  int sub_h, sub_w;                   // extents of that space
  int out_h, out_w;                   // the tensor written: pixel (u, v) is (u*out_step + out_y0, v*out_step + out_x0)
  int out_step, out_y0, out_x0;
  int n_img, n_ch_out;
  int cblocks, tap_cols;              // channel blocks (of KW) per tap; taps per kernel row that take part
  int in_step;                        // pixels of the activation per step of (u, v)
  int sgn, base_y, base_x;
  int w_tap0, w_tap_row, w_tap_col;   // weight tap of (0, 0), and its steps along both tap axes
  float* out;
  const float* bias;
  int act, accumulate;
  int taps_y;                         // slabs: vertical taps that one serves
  uint32_t slice_rows;                // pixels of a tile's box
  float k_total;                      // terms of a sum, for the result's bound
  // optional: ReLU mask taken from an NCHW tensor of the output's shape, and NHWC operand planes of
  // the result for the next tensor-core kernel
  const float* mask_src;
  float* out_hi;
  float* out_lo;
  // optional: [tiles_m * 4][n_ch_out] sums of the finished values over each epilogue warp's 32 rows
  float* colsum_partial;
  bool bias_vec;   // bias starts on 16 bytes
  bool skip_out;   // the finished values leave as planes and channel sums only (a K-split's second pass writes them still)

  __device__ __forceinline__ uint32_t a_slice_rows() const { return slice_rows; }
  __device__ __forceinline__ uint32_t slab_rows() const { return (uint32_t)(Wt * Nt * (Ht + taps_y - 1)); }
  __device__ __forceinline__ int slab_taps() const { return taps_y; }
  __device__ __forceinline__ uint32_t slab_tap_row(int i) const { return (uint32_t)((sgn > 0 ? i : taps_y - 1 - i) * Wt * Nt); }
  template <class Cur>
  __device__ __forceinline__ int slab_weight(const Cur& c, int i) const { return (w_tap0 + i * w_tap_row + c.j * w_tap_col) * cblocks + c.cb; }
  template <int KW, class Cur>
  __device__ __forceinline__ int slab_column(const Cur& c, int i) const { return slab_weight(c, i) * KW; }
  // No finished value exceeds this (a whole warp asks).
  __device__ __forceinline__ float out_bound(float top_a, float top_b, int lane) const {
    if (!out_hi) return 0.0f;   // only the largest magnitude is asked for
    uint32_t b = 0;
    if (bias)
      for (int n = lane; n < n_ch_out; n += 32) b = pr::seen(b, bias[n]);
    return pr::product_bound(k_total, top_a, top_b, __uint_as_float(__reduce_max_sync(0xffffffffu, b)));
  }
  __device__ __forceinline__ void origin(int tile_m, int* x0, int* y0, int* n0) const {
    uint32_t t, tx, n, ty;
    div_tiles_x.divmod((uint32_t)tile_m, t, tx);
    div_tiles_y.divmod(t, n, ty);
    *x0 = (int)tx * Wt;
    *y0 = (int)ty * Ht;
    *n0 = (int)n * Nt;
  }
  // Position of a K-slice: tap (i, j), channel block cb; the box origin of tap (i, j) and the weight column.
  struct Cursor { int b_col, cb, i, j, x, y, n, x_first; };
  template <int KW>
  __device__ __forceinline__ Cursor cursor(int tile_m, int, int kb) const {
    Cursor c;
    const int tap = (int)div_cblocks.div((uint32_t)kb);
    c.cb = kb - tap * cblocks;
    c.i = SLAB || tap == 0 ? 0 : tap / tap_cols;
    c.j = tap - c.i * tap_cols;
    int x0, y0;
    origin(tile_m, &x0, &y0, &c.n);
    c.x_first = x0 * in_step + base_x;
    c.x = c.x_first + sgn * c.j;
    c.y = y0 * in_step + base_y + (SLAB ? (sgn > 0 ? 0 : 1 - taps_y) : sgn * c.i);
    c.b_col = SLAB ? 0 : weight_column<KW>(c);
    return c;
  }
  template <int KW>
  __device__ __forceinline__ int weight_column(const Cursor& c) const {
    return ((w_tap0 + c.i * w_tap_row + c.j * w_tap_col) * cblocks + c.cb) * KW;
  }
  template <int KW>
  __device__ __forceinline__ void advance(Cursor& c) const {
    c.b_col += KW;
    if (++c.cb < cblocks) return;
    c.cb = 0;
    c.x += sgn;
    if (SLAB) {
      ++c.j;
      return;
    }
    if (++c.j == tap_cols) {
      c.j = 0;
      c.x = c.x_first;
      c.y += sgn;
      ++c.i;
    }
    c.b_col = weight_column<KW>(c);
  }
  template <int BN, bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_b(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c, int n0) const {
    tc::tma_load_3d_to<PAIR>(dst, tm, bar, c.b_col, n0, 0);
  }
  template <bool PAIR, int KW, int ROW_BYTES>
  __device__ __forceinline__ void load_a(void* dst, const CUtensorMap* tm, uint32_t bar, const Cursor& c) const {
    if (SLAB) tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.cb * KW, c.x, c.n, c.y);
    else tc::tma_load_4d_to<PAIR>(dst, tm, bar, c.cb * KW, c.x, c.y, c.n);
  }
  // NCHW offset of channel 0 of the pixel behind accumulator row `row`, and the pixel's linear index.
  __device__ __forceinline__ bool locate(int tile_m, int row, size_t* nchw_off, size_t* pixel) const {
    if (row >= Wt * Ht * Nt) return false;
    int x0, y0, n0;
    origin(tile_m, &x0, &y0, &n0);
    const int t = (int)div_Wt.div((uint32_t)row);
    const int hi = (int)div_mid.div((uint32_t)t), lo = t - hi * (int)div_mid.d;
    const int v = x0 + row - t * Wt, u = y0 + (SLAB ? hi : lo), n = n0 + (SLAB ? lo : hi);
    if (n >= n_img || u >= sub_h || v >= sub_w) return false;
    const int y = u * out_step + out_y0, x = v * out_step + out_x0;
    *nchw_off = (size_t)n * n_ch_out * out_h * out_w + (size_t)y * out_w + x;
    *pixel = ((size_t)n * out_h + y) * out_w + x;
    return true;
  }
  template <bool SPLIT>
  __device__ __forceinline__ void store(int tile_m, int, int row, int ch, float v, float out_scale, uint32_t& top) const {
    size_t off, pixel;
    if (ch >= n_ch_out || !locate(tile_m, row, &off, &pixel)) return;
    off += (size_t)ch * out_h * out_w;
    if (bias) v += bias[ch];
    v = nrs_apply_act(v, act);
    if (accumulate) v += out[off];
    if (mask_src && !(mask_src[off] > 0.0f)) v = 0.0f;
    out[off] = v;
    if (SPLIT) top = pr::seen(top, v);
    if (!out_hi) return;
    if (SPLIT) pr::put(out_hi, out_lo, pixel * n_ch_out + ch, v, out_scale);
    else out_hi[pixel * n_ch_out + ch] = tc::tf32_rn(v);
  }
  static constexpr bool kCanEmit = true;
  static constexpr bool kAMnMajor = false, kBMnMajor = false;
  static constexpr bool kMaySplit = true;
  __device__ __forceinline__ bool clip(int, int, int, int*, int*) const { return true; }
  int order() const { return tc::kRaster; }
  static constexpr int kEpiWarps = EPI, kTeamWarps = EPI == 16 ? 8 : 4;   // see takes_sixteen_warps
  __device__ __forceinline__ float* colsum_row(int tile_m, int q) const {
    return colsum_partial ? colsum_partial + ((size_t)tile_m * 4 + q) * n_ch_out : nullptr;
  }
  // An accumulator row: does it hold a pixel, the NCHW offset of that pixel in channel 0, and the origin of its tile's
  // box (x, y, image), which is where the TMA store of the tile's planes goes (out_step == 1).
  struct Row { bool live; size_t off; int x0, y0, n0; };
  __device__ __forceinline__ Row row(int tile_m, int, int r) const {
    Row w;
    size_t pixel;
    w.off = 0;
    w.live = locate(tile_m, r, &w.off, &pixel);
    origin(tile_m, &w.x0, &w.y0, &w.n0);
    return w;
  }
  // One accumulator row, channels [nb, nb + W) as far as they exist: bias, activation, accumulate, mask,
  // NCHW store; the finished values come back in v (zeros for rows and channels outside the tensor) so the
  // caller can emit them as planes.  Loads are issued in batches ahead of the stores.
  // The mask of W channels from nb on, of one pixel, a bit each.
  template <int W>
  __device__ __forceinline__ uint32_t fetch(const Row& rw, int nb, bool any) const {
    uint32_t keep = ~0u;
    if (mask_src && any && rw.live && nb < n_ch_out) {   // (whole channel blocks only)
      const size_t plane = (size_t)out_h * out_w;
      const float* m = mask_src + rw.off + (size_t)nb * plane;
      float mv[W];
#pragma unroll
      for (int j = 0; j < W; ++j) mv[j] = __ldg(m + (size_t)j * plane);
      keep = 0;
#pragma unroll
      for (int j = 0; j < W; ++j) keep |= mv[j] > 0.0f ? 1u << j : 0u;
    }
    return keep;
  }
  template <int W>
  __device__ __forceinline__ void epilogue(const Row& rw, int nb, const uint32_t (&r)[W], uint32_t keep, float (&v)[W]) const {
    if (!rw.live) {
#pragma unroll
      for (int j = 0; j < W; ++j) v[j] = 0.0f;
      return;
    }
    // Whole channel blocks take their own instantiation: with per-channel conditions the loads of a block no longer
    // issue together (measured on the 64-channel data gradient with mask and planes: 69 -> 217 us).
    if (n_ch_out - nb >= W) finish<true>(rw.off, nb, r, keep, v);
    else finish<false>(rw.off, nb, r, keep, v);
  }
  template <bool FULL, int W>
  __device__ __forceinline__ void finish(size_t off, int nb, const uint32_t (&r)[W], uint32_t keep, float (&v)[W]) const {
    const size_t plane = (size_t)out_h * out_w;
    float* dst = out + off + (size_t)nb * plane;
    const int nch = FULL ? W : n_ch_out - nb;   // channels of this block that exist
#pragma unroll
    for (int j = 0; j < W; ++j) v[j] = (FULL || j < nch) ? __uint_as_float(r[j]) : 0.0f;
    if (bias && FULL && bias_vec) {
#pragma unroll
      for (int j = 0; j < W; j += 4) {
        const float4 b = __ldg(reinterpret_cast<const float4*>(bias + nb + j));
        v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
      }
    } else if (bias) {
#pragma unroll
      for (int j = 0; j < W; ++j)
        if (FULL || j < nch) v[j] += __ldg(bias + nb + j);
    }
    if (act != NRS_ACT_NONE) {
#pragma unroll
      for (int j = 0; j < W; ++j) v[j] = nrs_apply_act(v[j], act);
    }
    if (accumulate) {
      float o[W];
#pragma unroll
      for (int j = 0; j < W; ++j) o[j] = (FULL || j < nch) ? dst[(size_t)j * plane] : 0.0f;
#pragma unroll
      for (int j = 0; j < W; ++j) v[j] += o[j];
    }
    if (FULL && mask_src) {
#pragma unroll
      for (int j = 0; j < W; ++j) v[j] = (keep >> j) & 1u ? v[j] : 0.0f;
    }
    if (FULL && skip_out) return;
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (FULL || j < nch) dst[(size_t)j * plane] = v[j];
  }
};

using ConvPolicy = ConvPolicyOf<4, false>;

// 3xTF32 launches take four epilogue warps per lane quarter, 16 columns at a time: with the products at the f16 rate the
// epilogue (activation or mask, NCHW store, split and staging) is the longer part of most tiles, and it is latency: one
// warp with 32 columns took 2 thousand clocks a block and spilled.  TF32 keeps one (two: 1.5 % slower).
constexpr bool takes_sixteen_warps(int nplanes) { return nplanes == 2; }

// One axis of a (sub-)problem: `len` output pixels at positions u*step + first, `taps` kernel taps tap0,
// tap0 + tap_step, ..., and the activation coordinate of tap t for pixel u: u * in_step + base + sgn * t.
struct ConvAxis {
  int len, step, first;
  int taps, tap0, tap_step;
  int in_step, base;
};

struct ConvPlan {
  // activation read by the A operand: [n_img][a_h][a_w] pixels of a_ch channels, NHWC planes (pixel stride
  // nrs_plane_ld(a_ch) floats) staged from NCHW `act_src`
  const float* act_src;
  int n_img, a_ch, a_h, a_w;
  // weights and which re-layout
  const float* w;
  int co, ci, kh, kw, for_dgrad;
  const float *w_hi, *w_lo;   // its planes once staged (the residues of a strided data gradient share them)
  const NrsRange* w_range;
  // output NCHW [n_img][n_ch_out][out_h][out_w]
  float* out;
  int n_ch_out, out_h, out_w;
  int sgn;
  ConvAxis ay, ax;
  const float* bias;
  int act, accumulate;
};

template <int BN, int NPLANES, bool PAIR, int KW, bool SLAB>
int run_conv(nrs_ctx* ctx, const ConvPlan& p, const float* a_hi, const float* a_lo, const ConvPolicy& base, const tc::Ranges& rg, int tiles_m,
             int* splits_out) {
  constexpr bool kHalf = NPLANES == 2;
  using Policy = ConvPolicyOf<takes_sixteen_warps(NPLANES) ? 16 : 4, SLAB>;
  Policy pol;
  static_assert(sizeof(pol) == sizeof(base), "the same fields");
  std::memcpy((void*)&pol, &base, sizeof(pol));
  const int a_ld = nrs_plane_ld(p.a_ch);
  const int kdim = p.kh * p.kw * pol.cblocks * KW;
  CUtensorMap ta_hi, ta_lo, tb_hi, tb_lo;
  // An activation-shaped tensor of `c` channels, ld apart, as [n][h][w][c] or (slabs) [h][n][w][c], in boxes of a tile and
  // `more` rows above it.
  auto image_map = [&](CUtensorMap* m, const float* at, int c, int ld, int h, int w, int box_c, int more, int step) {
    const uint64_t row = (uint64_t)w * ld, img = (uint64_t)h * row;
    const uint64_t dim[4] = {(uint64_t)c, (uint64_t)w, (uint64_t)(SLAB ? p.n_img : h), (uint64_t)(SLAB ? h : p.n_img)};
    const uint64_t str[3] = {(uint64_t)ld, SLAB ? img : row, SLAB ? row : img};
    const uint32_t box[4] = {(uint32_t)box_c, (uint32_t)pol.Wt, (uint32_t)(SLAB ? pol.Nt : pol.Ht), (uint32_t)(SLAB ? pol.Ht + more : pol.Nt)};
    const uint32_t es[4] = {1, (uint32_t)step, (uint32_t)step, 1};
    return tc::encode_tmap(m, at, kHalf, 4, dim, str, box, false, SLAB ? nullptr : es);
  };
  const uint64_t bdim[3] = {(uint64_t)kdim, (uint64_t)p.n_ch_out, 1};
  const uint64_t bstr[2] = {(uint64_t)kdim, (uint64_t)kdim * p.n_ch_out};
  const uint32_t bbox[3] = {(uint32_t)KW, (uint32_t)(PAIR ? BN / 2 : BN), 1};
  const int more = pol.taps_y - 1;
  bool ok = image_map(&ta_hi, a_hi, p.a_ch, a_ld, p.a_h, p.a_w, KW, more, pol.in_step) && tc::encode_tmap(&tb_hi, p.w_hi, kHalf, 3, bdim, bstr, bbox);
  if (kHalf) ok = ok && image_map(&ta_lo, a_lo, p.a_ch, a_ld, p.a_h, p.a_w, KW, more, pol.in_step) && tc::encode_tmap(&tb_lo, p.w_lo, true, 3, bdim, bstr, bbox);
  else { ta_lo = ta_hi; tb_lo = tb_hi; }
  // Output planes (optional): the same box geometry as an activation load, in output space.
  CUtensorMap to_hi, to_lo;
  if (pol.out_hi) {
    ok = ok && image_map(&to_hi, pol.out_hi, p.n_ch_out, p.n_ch_out, p.out_h, p.out_w, 32, 0, 1);
    if (pol.out_lo) ok = ok && image_map(&to_lo, pol.out_lo, p.n_ch_out, p.n_ch_out, p.out_h, p.out_w, 32, 0, 1);
  }
  NRS_REQUIRE(ctx, ok, NRS_ERR_CUDA, "tc_conv: cuTensorMapEncodeTiled failed");
  return tc::launch<BN, NPLANES, PAIR, KW, Policy>(ctx, ta_hi, ta_lo, tb_hi, tb_lo, pol, tiles_m, p.n_ch_out, 1,
                                                   (SLAB ? 1 : p.ay.taps) * p.ax.taps * pol.cblocks, rg, pol.out_hi ? &to_hi : nullptr,
                                                   pol.out_lo ? &to_lo : nullptr, splits_out, SLAB ? KW * p.ay.taps : KW);
}

// Pixel tile: the Wt x Ht x Nt box of at most 128 pixels (a box side times the activation step may not exceed
// TMA's 256) that covers the output in the fewest tiles; among equals the widest, whose stores have the longest runs.
void plan_pixel_tile(const ConvPlan& p, ConvPolicy* pol) {
  const int lim = 256 / p.ax.in_step < tc::BM ? 256 / p.ax.in_step : tc::BM;
  const int lim_y = 256 / p.ay.in_step;
  long best = -1;
  for (int tx = (p.ax.len + lim - 1) / lim, end = tx + 3; tx < end && tx <= p.ax.len; ++tx) {
    const int Wt = (p.ax.len + tx - 1) / tx;
    int Ht = tc::BM / Wt;
    if (Ht > p.ay.len) Ht = p.ay.len;
    if (Ht > lim_y) Ht = lim_y;
    int Nt = 1;
    if (Ht == p.ay.len && Wt == p.ax.len) {
      Nt = tc::BM / (Wt * Ht);
      if (Nt > p.n_img) Nt = p.n_img;
    }
    const int nx = (p.ax.len + Wt - 1) / Wt, ny = (p.ay.len + Ht - 1) / Ht;
    const long tiles = (long)nx * ny * ((p.n_img + Nt - 1) / Nt);
    if (best < 0 || tiles < best) {
      best = tiles;
      pol->Wt = Wt; pol->Ht = Ht; pol->Nt = Nt; pol->tiles_x = nx; pol->tiles_y = ny;
    }
  }
}

// The same for slabs: rows of 8, 16, 24 or 32 pixels (a slab's taps have to start on whole swizzle patterns, and it has
// room for tc::kSlabRows pixels).  Taken where that costs at most a tenth more tiles.
bool plan_slab_tile(const ConvPlan& p, ConvPolicy* pol) {
  if (p.ax.in_step != 1 || p.ay.in_step != 1 || p.ay.taps < 2) return false;
  const long plain = (long)pol->tiles_x * pol->tiles_y * ((p.n_img + pol->Nt - 1) / pol->Nt);
  long best = plain + plain / 10;
  bool found = false;
  for (int Wt = 8; Wt <= 32 && Wt < p.ax.len + 8; Wt += 8) {
    int Ht = tc::BM / Wt;
    if (Ht > p.ay.len) Ht = p.ay.len;
    int Nt = 1;
    if (Ht == p.ay.len && Wt >= p.ax.len) Nt = std::max(1, std::min(p.n_img, tc::BM / (Wt * Ht)));
    while (Nt > 1 && Wt * Nt * (Ht + p.ay.taps - 1) > tc::kSlabRows) --Nt;
    while (Ht > 1 && Wt * Nt * (Ht + p.ay.taps - 1) > tc::kSlabRows) --Ht;
    if (Wt * Nt * (Ht + p.ay.taps - 1) > tc::kSlabRows) continue;
    const int nx = (p.ax.len + Wt - 1) / Wt, ny = (p.ay.len + Ht - 1) / Ht;
    const long tiles = (long)nx * ny * ((p.n_img + Nt - 1) / Nt);
    if (tiles <= best) {   // (among equals the widest rows)
      best = tiles;
      pol->Wt = Wt; pol->Ht = Ht; pol->Nt = Nt; pol->tiles_x = nx; pol->tiles_y = ny;
      found = true;
    }
  }
  return found;
}

int conv_common(nrs_ctx* ctx, ConvPlan& p) {
  if (p.ax.len < 1 || p.ay.len < 1 || p.ax.taps < 1 || p.ay.taps < 1) return NRS_OK;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  ConvPolicy pol{};
  plan_pixel_tile(p, &pol);
  const bool slab = split && plan_slab_tile(p, &pol);   // (TF32: 5 % slower with slabs on most layers, 256 x 200 x 9 x 8 -> 200 205 us, without 186)
  pol.taps_y = slab ? p.ay.taps : 1;
  const long tiles_m = (long)((p.n_img + pol.Nt - 1) / pol.Nt) * pol.tiles_y * pol.tiles_x;
  if (tiles_m > 2147483647L) return NRS_ERR_UNSUPPORTED;
  pol.sub_h = p.ay.len; pol.sub_w = p.ax.len;
  pol.out_h = p.out_h; pol.out_w = p.out_w; pol.n_img = p.n_img; pol.n_ch_out = p.n_ch_out;
  pol.out_step = p.ay.step; pol.out_y0 = p.ay.first; pol.out_x0 = p.ax.first;
  const int blocks32 = (p.a_ch + 31) / 32;
  const bool wide = split && blocks32 % 2 == 0;   // K-slices of 64 channels: TMA brings rows of 64 bytes at half the rate
  pol.cblocks = wide ? blocks32 / 2 : blocks32; pol.tap_cols = p.ax.taps;
  pol.in_step = p.ay.in_step;
  pol.sgn = p.sgn; pol.base_y = p.ay.base; pol.base_x = p.ax.base;
  pol.w_tap0 = p.ay.tap0 * p.kw + p.ax.tap0; pol.w_tap_row = p.ay.tap_step * p.kw; pol.w_tap_col = p.ax.tap_step;
  pol.out = p.out; pol.bias = p.bias; pol.act = p.act; pol.accumulate = p.accumulate;
  pol.div_Wt = NrsFastDiv(pol.Wt); pol.div_mid = NrsFastDiv(slab ? pol.Nt : pol.Ht);
  pol.div_cblocks = NrsFastDiv(pol.cblocks);
  pol.div_tiles_x = NrsFastDiv(pol.tiles_x); pol.div_tiles_y = NrsFastDiv(pol.tiles_y);
  pol.slice_rows = (uint32_t)(pol.Wt * pol.Ht * pol.Nt);
  pol.bias_vec = (reinterpret_cast<uintptr_t>(p.bias) & 15) == 0;
  pol.k_total = (float)p.a_ch * p.ay.taps * p.ax.taps;
  // Requests of the caller are honoured where this launch writes every pixel of the output (planes: whole
  // 32-channel blocks); the caller finds the others still registered and does the work itself.
  const bool whole = pol.out_step == 1 && p.n_ch_out % 32 == 0;
  NrsRange* out_range = nullptr;
  auto extras = pol.out_step == 1 ? ctx->out_extras.find(p.out) : ctx->out_extras.end();
  if (extras != ctx->out_extras.end()) {
    const NrsOutExtras& e = extras->second;
    if (((e.relu_mask_src || e.hi) && !whole) ||
        (e.relu_mask_src && p.accumulate) ||   // the mask would hit the old content too
        ((e.hi || e.measure) && split && p.accumulate) ||   // no bound of the old content
        (e.hi && (e.lo != nullptr) != split) || (e.measure && !split)) {
      extras = ctx->out_extras.end();
    } else {
      pol.mask_src = e.relu_mask_src; pol.out_hi = e.hi; pol.out_lo = e.lo;
      out_range = e.measure;
      if (split && e.hi) {
        const int got = nrs_range_renew(ctx, e.hi, &out_range);
        if (got != NRS_OK) return got;
      }
    }
  }
  auto colsum = ctx->colsum_requests.find(p.out);
  if (whole && colsum != ctx->colsum_requests.end() && !p.accumulate && tiles_m * 4 <= colsum->second.cap_rows)
    pol.colsum_partial = colsum->second.partial;
  pol.skip_out = pol.colsum_partial && pol.out_hi && extras->second.planes_suffice;

  // stage the activation: per image [C][H*W] -> [H*W][C] planes
  void *a_hi = nullptr, *a_lo = nullptr;
  int st = NRS_OK;
  const NrsPlanes* ready = nrs_planes_find(ctx, p.act_src, split);
  if (ready) {
    a_hi = ready->hi;
    a_lo = ready->lo;
  } else {
    const size_t a_plane = (size_t)p.n_img * p.a_h * p.a_w * nrs_plane_ld(p.a_ch);
    st = nrs_ws_planes(ctx, NRS_WS_A, a_plane, split, &a_hi, &a_lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, p.act_src, (float*)a_hi, (float*)a_lo, p.n_img, p.a_ch, p.a_h * p.a_w);
    if (st != NRS_OK) return st;
  }
  const NrsWeightPlanes* wp = nrs_weight_planes_find(ctx, p.w, p.for_dgrad ? NRS_WF_CONV_DGRAD : NRS_WF_CONV_FWD);
  if (p.w_hi) {
  } else if (wp && wp->co == p.co && wp->ci == p.ci && wp->taps == p.kh * p.kw) {   // staged ahead with the rest of the model's weights
    p.w_hi = wp->hi;
    p.w_lo = wp->lo;
    p.w_range = wp->range;
  } else {
    void *w_hi = nullptr, *w_lo = nullptr;
    const size_t w_plane = (size_t)p.n_ch_out * p.kh * p.kw * blocks32 * 32;
    st = nrs_ws_planes(ctx, NRS_WS_B, w_plane, split, &w_hi, &w_lo);
    if (st != NRS_OK) return st;
    st = nrs_tc_stage_conv_weight(ctx, p.w, (float*)w_hi, (float*)w_lo, p.co, p.ci, p.kh, p.kw, p.for_dgrad);
    if (st != NRS_OK) return st;
    p.w_hi = (const float*)w_hi;
    p.w_lo = (const float*)w_lo;
    p.w_range = nrs_range_of(ctx, w_hi);
  }
  const tc::Ranges rg{nrs_range_of(ctx, a_hi), p.w_range, out_range};

  if (extras != ctx->out_extras.end()) ctx->out_extras.erase(extras);   // honoured from here on
  int splits = 0;
  const tc::TilePlan tile = tc::plan_tile(ctx, tiles_m, p.n_ch_out, 1, p.ay.taps * p.ax.taps * blocks32, split, 0.025, true, slab);
#define NRS_RUN_AS(BN_, PAIR_, SLAB_)                                                                                          \
  st = wide ? run_conv<BN_, 2, PAIR_, 64, SLAB_>(ctx, p, (const float*)a_hi, (const float*)a_lo, pol, rg, (int)tiles_m, &splits) \
            : run_conv<BN_, 2, PAIR_, 32, SLAB_>(ctx, p, (const float*)a_hi, (const float*)a_lo, pol, rg, (int)tiles_m, &splits)
#define NRS_RUN(BN_, PAIR_)                                                                                                    \
  {                                                                                                                            \
    if (!split) st = run_conv<BN_, 1, PAIR_, 32, false>(ctx, p, (const float*)a_hi, nullptr, pol, rg, (int)tiles_m, &splits);   \
    else if (slab) NRS_RUN_AS(BN_, PAIR_, true);                                                                               \
    else NRS_RUN_AS(BN_, PAIR_, false);                                                                                        \
  }
  if (tile.pair && tile.bn == 128) NRS_RUN(128, true)
  else if (tile.pair) NRS_RUN(64, true)
  else if (tile.bn == 128) NRS_RUN(128, false)
  else if (tile.bn == 64) NRS_RUN(64, false)
  else NRS_RUN(32, false)
#undef NRS_RUN
#undef NRS_RUN_AS
  // channel sums come from the direct epilogue only (a K-split stores through the reduce kernel)
  if (st == NRS_OK && pol.colsum_partial && splits == 1) colsum->second.rows = (int)tiles_m * 4;
  return st;
}

// Strides beyond TMA's element-stride limit keep the FFMA kernels.
bool tensor_core_conv(int stride) { return tc::tensor_map_encoder() && stride <= 8; }

}  // namespace

// y = act(conv(x, w) + b); NRS_ERR_UNSUPPORTED when the shape is outside this kernel's range.
int nrs_tc_conv_fwd(nrs_ctx* ctx, const float* x, const float* w, const float* b, float* y, int n, int ci, int h,
                    int wd, int co, int kh, int kw, int stride, int pad, int act) {
  if (!tensor_core_conv(stride)) return NRS_ERR_UNSUPPORTED;
  ConvPlan p{};
  p.act_src = x; p.n_img = n; p.a_ch = ci; p.a_h = h; p.a_w = wd;
  p.w = w; p.co = co; p.ci = ci; p.kh = kh; p.kw = kw; p.for_dgrad = 0;
  p.out = y; p.n_ch_out = co; p.out_h = (h + 2 * pad - kh) / stride + 1; p.out_w = (wd + 2 * pad - kw) / stride + 1;
  p.sgn = 1;
  p.ay = ConvAxis{p.out_h, 1, 0, kh, 0, 1, stride, -pad};
  p.ax = ConvAxis{p.out_w, 1, 0, kw, 0, 1, stride, -pad};
  p.bias = b; p.act = act; p.accumulate = 0;
  return conv_common(ctx, p);
}

// dx (+)= conv_transpose(dy, w)
int nrs_tc_conv_dgrad(nrs_ctx* ctx, const float* w, const float* dy, float* dx, int n, int ci, int h, int wd, int co,
                      int kh, int kw, int stride, int pad, int accumulate) {
  if (!tensor_core_conv(stride)) return NRS_ERR_UNSUPPORTED;
  ConvPlan p{};
  p.act_src = dy; p.n_img = n; p.a_ch = co; p.a_h = (h + 2 * pad - kh) / stride + 1; p.a_w = (wd + 2 * pad - kw) / stride + 1;
  p.w = w; p.co = co; p.ci = ci; p.kh = kh; p.kw = kw; p.for_dgrad = 1;
  p.out = dx; p.n_ch_out = ci; p.out_h = h; p.out_w = wd;
  p.sgn = -1;
  p.bias = nullptr; p.act = NRS_ACT_NONE; p.accumulate = accumulate;
  // Residue r = (y + pad) % stride: its pixels are y = u*stride + first, its taps r, r + stride, ..., and tap t of
  // them reads dy row u + (first + pad - r)/stride - t.
  auto axis = [&](int r, int extent, int k) {
    const int first = ((r - pad) % stride + stride) % stride;
    return ConvAxis{first < extent ? (extent - first + stride - 1) / stride : 0, stride, first,
                    r < k ? (k - r + stride - 1) / stride : 0, r, stride, 1, (first + pad - r) / stride};
  };
  if (stride > kh || stride > kw) {   // some residues meet no tap: their pixels receive no gradient
    if (!accumulate) NRS_CUDA(ctx, cudaMemsetAsync(dx, 0, (size_t)n * ci * h * wd * sizeof(float), ctx->stream));
  }
  // the residues share dy's planes: staged once here unless the caller left them with the context
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  bool lent = false;
  if (stride > 1 && !nrs_planes_find(ctx, dy, split)) {
    void *hi = nullptr, *lo = nullptr;
    const size_t plane = (size_t)n * p.a_h * p.a_w * nrs_plane_ld(co);
    int st = nrs_ws_planes(ctx, NRS_WS_A, plane, split, &hi, &lo);
    if (st == NRS_OK) st = nrs_tc_stage_image(ctx, dy, (float*)hi, (float*)lo, n, co, p.a_h * p.a_w);
    if (st != NRS_OK) return st;
    ctx->plane_hints[dy] = NrsPlanes{(float*)hi, (float*)lo, split ? 1 : 0};
    lent = true;
  }
  int st = NRS_OK;
  for (int ry = 0; ry < stride && st == NRS_OK; ++ry)
    for (int rx = 0; rx < stride && st == NRS_OK; ++rx) {
      p.ay = axis(ry, h, kh);
      p.ax = axis(rx, wd, kw);
      st = conv_common(ctx, p);
    }
  if (lent) ctx->plane_hints.erase(dy);
  return st;
}

namespace {

// Columns [n, n + width) that the epilogue warps read ahead of a layer's accumulators: checks that failed.
template <int BN, bool SLAB>
int check_reads_ahead(int n_ch, int* ragged) {
  using E = tc::EpiBlocks<BN, ConvPolicyOf<16, SLAB>>;
  int bad = 0;
  for (int n0 = 0; n0 < n_ch; n0 += BN) {
    if (n_ch - n0 < BN) ++*ragged;
    for (int warp = 0; warp < 16; ++warp) {
      const int c = E::first(warp), n = n0 + c * E::kW;
      const bool reads = E::reads_first(c, n0, n_ch, 1);
      bad += reads == (c < E::kBlocks && n < n_ch) && !(reads && n + E::kW > n_ch) ? 0 : 1;
      bad += E::reads_first(c, n0, n_ch, 2) ? 1 : 0;   // (a K-split's results do not pass through here)
    }
  }
  return bad;
}

}  // namespace

// Host-only: over layers of whole 32-channel blocks (those whose data gradient may apply a mask) on images of several sizes, the
// plan that their data gradient takes never has an epilogue warp read a channel that the layer does not have.
extern "C" int nrs_selftest_conv_reads_ahead(void) {
  static const struct { int n, hw; } kImages[] = {{1, 32}, {9, 32}, {64, 32}, {64, 16}, {100, 8}, {13, 10}, {256, 4}, {1024, 32}};
  nrs_ctx ctx;   // (only its SM count is asked for)
  int bad = 0, ragged = 0;
  for (const auto& im : kImages)
    for (int ch = 32; ch <= 512; ch += 32)
      for (int co : {32, 128, 200}) {
        ConvPlan p{};
        p.n_img = im.n; p.a_ch = co;
        p.ay = p.ax = ConvAxis{im.hw, 1, 0, 3, 0, 1, 1, 1};
        ConvPolicy pol{};
        plan_pixel_tile(p, &pol);
        const bool slab = plan_slab_tile(p, &pol);
        const long tiles_m = (long)((im.n + pol.Nt - 1) / pol.Nt) * pol.tiles_y * pol.tiles_x;
        const tc::TilePlan tile = tc::plan_tile(&ctx, tiles_m, ch, 1, 9 * ((co + 31) / 32), true, 0.025, true, slab);
        if (tile.bn == 128) bad += slab ? check_reads_ahead<128, true>(ch, &ragged) : check_reads_ahead<128, false>(ch, &ragged);
        else if (tile.bn == 64) bad += slab ? check_reads_ahead<64, true>(ch, &ragged) : check_reads_ahead<64, false>(ch, &ragged);
        else bad += slab ? check_reads_ahead<32, true>(ch, &ragged) : check_reads_ahead<32, false>(ch, &ragged);
      }
  return bad + (ragged > 0 ? 0 : 1);   // (layers with a ragged last column tile are among them)
}
