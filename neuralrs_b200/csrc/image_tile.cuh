// A block's tile of an NCHW image batch: 32 channels x 128 pixels, the pixels counted through the batch (images smaller
// than 128 pixels share a tile).  Read in 128-byte row segments, 16 independent loads per thread (warp w: channels w,
// w + 8, w + 16, w + 24, four segments each), written as NHWC operand planes in full 128-byte lines (32 channels of a
// pixel, 128-bit stores).
#pragma once

#include "igemm_problems.cuh"
#include "nrs_internal.h"
#include "pair.cuh"
#include "tc_common.cuh"

namespace img {

constexpr int kTileCh = 32, kTilePx = 128;
using Tile = float[kTileCh][kTilePx + 1];

struct Grid {
  int c, hw;
  uint32_t pixels;   // in the batch
  int ld;            // pixel stride of the planes, floats
  NrsFastDiv div_hw;
  Grid(int n, int c_, int hw_) : c(c_), hw(hw_), pixels((uint32_t)n * (uint32_t)hw_), ld(nrs_plane_ld(c_)), div_hw(hw_) {}
  dim3 blocks() const { return dim3((pixels + kTilePx - 1) / kTilePx, (unsigned)((ld + kTileCh - 1) / kTileCh)); }
};

// Where this thread's four pixels (segments) lie in NCHW, channel 0: offsets from the tile's first image, which fit 32
// bits (a tile touches two images, or 128 pixels of smaller ones).
struct Pixels {
  size_t base;
  uint32_t at[4];
  bool live[4];
  __device__ __forceinline__ Pixels(const Grid& g, uint32_t p0) {
    const uint32_t im0 = g.div_hw.div(p0), plane = (uint32_t)g.c * (uint32_t)g.hw;
    base = (size_t)im0 * plane;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const uint32_t p = p0 + s * 32 + (threadIdx.x & 31);
      uint32_t im, px;
      g.div_hw.divmod(p < g.pixels ? p : p0, im, px);
      live[s] = p < g.pixels;
      at[s] = (im - im0) * plane + px;
    }
  }
};

template <bool SPLIT>
__device__ __forceinline__ void tile_to_planes(const Tile& tile, const Grid& g, uint32_t p0, int c0, float* __restrict__ hi, float* __restrict__ lo,
                                               float scale = 1.0f) {
  const int cq = (threadIdx.x & 7) * 4;
  if (c0 + cq >= g.ld) return;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const int pl = k * 32 + (threadIdx.x >> 3);
    if (p0 + pl >= g.pixels) break;
    const float4 f = make_float4(tile[cq][pl], tile[cq + 1][pl], tile[cq + 2][pl], tile[cq + 3][pl]);
    const size_t o = (size_t)(p0 + pl) * g.ld + c0 + cq;
    if (SPLIT) pr::put4(hi, lo, o, f, scale);
    else *reinterpret_cast<float4*>(hi + o) = make_float4(tc::tf32_rn(f.x), tc::tf32_rn(f.y), tc::tf32_rn(f.z), tc::tf32_rn(f.w));
  }
}

}  // namespace img
