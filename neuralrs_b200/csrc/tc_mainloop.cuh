// Shared tcgen05 main loop: D[128 x BN] (TMEM, f32) = sum over K-slices of
// A[128 x KW] . B[BN x KW]^T, operands K-major (or MN-major) in swizzled shared
// memory, fed by TMA, consumed by tcgen05.mma kind::tf32 (TF32 mode) or kind::f16 (3xTF32).
//
// Persistent CTAs (one per SM) walk a list of output tiles (row tile, column tile,
// batch x K-split).  Six to nineteen warps, fixed roles:
//   warp 0     TMA producer: per K-slice, one mbarrier-tracked ring
//              slot holding the A and B slices (for 3xTF32 both halves of the pairs);
//              the ring runs ahead across tile boundaries
//   warp 1     TMEM allocation; issues the UMMAs (M=128, K=8 or 16) and commits
//              ring slots back to the producer, then the accumulator to the epilogue
//   warps 2..  epilogue (4, 8 or 16 warps, the policy's choice): tcgen05.ld (thread = accumulator row),
//              policy-defined store
// TMEM holds two accumulators, so the epilogue of tile i runs under the main loop of
// tile i+1.
// A Policy supplies how an A slice is fetched (dense rows for GEMM, a shifted
// NHWC window for convolution), which K-slices of a tile count and whether the tile
// exists at all (clip: triangular products), and what the epilogue does with a row of results.
// A policy with kCanEmit may also hand the finished values back: the epilogue warps then
// write them as operand planes ([row][32 columns], swizzled) into a
// staging tile and one thread sends each tile to global memory with a TMA store — the
// operand planes of the next tensor-core kernel, written in full lines without a pass of
// their own.
//
// 3xTF32 (NPLANES == 2): operands are f16 pairs (pair.cuh), multiplied by kind::f16 at twice the rate of kind::tf32.  The
// low halves carry a factor 2^11, so hi*hi and the sum of hi*lo and lo*hi have accumulators of their own (columns [0,BN) and
// [BN,2BN)); the epilogue adds them and takes the operands' exponents out.  In shared memory B_lo sits directly behind B_hi,
// so one UMMA of width 2*BN computes A_hi.[B_hi ; B_lo] and a second of width BN adds A_lo.B_hi onto the second half; a pair
// of CTAs, each holding half of B_hi and of B_lo, takes three UMMAs of width BN.  A K-slice is 64 values wide where the
// operands allow (rows of 128 bytes; TMA brings rows of 64 at a lower rate: 138 -> 119 us on the data gradient below).
// Against three kind::tf32 products of a TF32 value and its f32 residual: 16384 x 4096 x 4096 in 787 clocks per 64 values of
// K (1640), of which the UMMAs alone are 768; x[256,64,32,32] -> 128 channels, 3x3: forward 172 -> 110 us, data gradient
// 170 -> 119 us.
//
// Policy::kSlab (convolutions over a pixel grid): a ring slot of A holds a slab of the activation, some image rows more than
// the tile has, that serves all vertical taps of a horizontal one: tap i is the same operand some pixels further.  B comes
// through a ring and a producing warp of its own.  A 3x3 layer thus brings 3 slabs of 1.25 to 1.5 tiles per channel block
// instead of 9 tiles.
//
// What bounds a tile: with 128 columns the tensor pipe, with 64 the way of A through L2 (40 KB per 64 values of K at about
// 60 bytes a clock) and the 46 clocks that a UMMA takes at least; short reductions the epilogue.  With PAIR the
// two CTAs of a cluster work on two row tiles of one column tile: each brings its own A rows and half of the B rows, and
// one warp issues UMMAs of 256 rows that read B from both (cta_group::2), which halves B's share of that traffic.  The
// ring, the accumulators and the epilogue stay per CTA.
//
// The tensor core's f32 accumulation is not round-to-nearest; its error grows
// linearly with the length of one accumulation chain (about 7e-9 relative per K
// element), so no chain is longer than kMaxChainK: a tile with more is walked in
// chunks of K, whose sums the epilogue adds up in f32, in order, in a buffer of the
// CTA's own that stays in L2 (a second pass over partial tiles took 135 us for a
// 4096 x 4096 result).  Products with too few tiles to fill the GPU split K across
// CTAs, and tc_splitk_reduce_kernel sums their partial results in a fixed order.
//
// Every mbarrier wait is bounded: on expiry the kernel records an error code,
// waits (bounded) for TMA loads it already issued, frees its TMEM and returns.
#pragma once

#include <algorithm>

#include "igemm_problems.cuh"
#include "nrs_internal.h"
#include "pair.cuh"
#include "tc_common.cuh"

namespace tc {

constexpr int BM = 128, BK = 32;   // 32 values: 128 bytes of f32, 64 of f16: one swizzle row
constexpr int kMaxChainK = 4096;   // longest single accumulation chain in 3xTF32 mode
// The same of a convolution with few pixels (at most half a wave of 128-column tiles).  With TF32 pairs such a product was
// split over the CTAs there are, down to chains of 512; f16 pairs err a third as much per value, are fast enough in narrow
// tiles not to be split, and are to err no more.
constexpr int kFewChainK = 1536;
constexpr int kMaxChainPairs = 8192;   // the same of weight gradients: at this length f16 pairs err as much as TF32 pairs did at half
constexpr int kGroupM = 16;        // row tiles per raster group (see TileMap)
constexpr int kSlabRows = 192;     // most pixels of a slab of A (see Policy::kSlab)

// KW: values of K in a K-slice, and in a row of it (MN-major operands: columns of a block): 32, or 64 of f16.
template <int BN, int NPLANES, int EMIT_BYTES, bool PAIR, int KW, bool SLAB>
struct SmemLayout {
  static_assert(KW == 32 || (KW == 64 && NPLANES == 2), "a row is at most 128 bytes");
  static constexpr int kRowBytes = KW * (NPLANES == 2 ? 2 : 4);
  static constexpr int kATile = BM * kRowBytes;                // per plane
  static constexpr int kBTile = BN / (PAIR ? 2 : 1) * kRowBytes;   // this CTA's rows of B
  static constexpr int kSlice = NPLANES * (kATile + kBTile);   // [A_hi][B_hi][B_lo][A_lo]
  static constexpr int kSlices = KW == 64 ? 1 : 2;             // K-slices per ring slot
  static constexpr int kStage = kSlices * kSlice;
  static constexpr int kExtra = EMIT_BYTES /*plane staging tile*/ + 1024 /*align*/ + 512 /*barriers*/;
  static constexpr int kRing = 227 * 1024 - kExtra;
  static constexpr int kStages = kRing / kStage >= 8 ? 8 : kRing / kStage;
  // Slabs (Policy::kSlab): a ring of A slabs and a ring of B slices.
  static constexpr int kSlabPlane = kSlabRows * kRowBytes, kSlab = NPLANES * kSlabPlane;
  // A pair's f16 pairs: a third block in a slice of B, B_hi again (see kTwice in tc_kernel).
  static constexpr bool kTwice = SLAB && PAIR && NPLANES == 2 && BN >= 64;
  static constexpr int kBSlice = (kTwice ? 3 : NPLANES) * kBTile;
  static constexpr int kMostA = kSlab > 24 * 1024 ? (BN == 128 ? 2 : 3) : 4;   // (128 columns: more slices of B instead)
  static constexpr int kSlabsA = kRing - kMostA * kSlab >= 3 * kBSlice ? kMostA : 2;
  static constexpr int kSlicesB = (kRing - kSlabsA * kSlab) / kBSlice >= 8 ? 8 : (kRing - kSlabsA * kSlab) / kBSlice;
  static constexpr int kRingBytes = SLAB ? kSlabsA * kSlab + kSlicesB * kBSlice : kStages * kStage;
  static constexpr int kBytes = kRingBytes + kExtra;
  static constexpr int kAccCols = NPLANES * BN;                 // one accumulator
  static constexpr int kTmemCols = 2 * kAccCols < 32 ? 32 : 2 * kAccCols;   // two of them
  static_assert((kTmemCols & (kTmemCols - 1)) == 0 && kTmemCols <= 512, "TMEM allocation must be a power of two <= 512");
};

// 3xTF32: ranges of both operands, and of the result where its planes or its largest magnitude are wanted (else null).
struct Ranges {
  const NrsRange* a;
  const NrsRange* b;
  NrsRange* out;
};

struct SplitInfo {
  int splits;          // K-splits per (tile, batch)
  int kb_per_split;    // K-slices per split, or per chunk
  int chunks;          // > 1 (splits == 1 then): K-chunks that a CTA takes one after the other
  int kb_total;        // K-slices in all
  int batches;
  NrsFastDiv div_splits;
  float* partial;      // [split][batch][tiles_m*128][n_total] when splits > 1; [CTA][128][BN] when chunks > 1
  int n_total;
  int rows_total;      // tiles_m * 128
};

// Tile list of one launch.  Within a (batch, split) plane tiles are visited in groups of
// kGroupM row tiles x all column tiles, row tile fastest, so the tiles in flight at any
// moment cover a compact block of the output and share operand slices through L2.
// Causal products have lists of their own, walked back and forth (round 0 of the grid from its first CTA, round 1 from
// its last, ...): with the plain list the tiles a CTA meets are a fixed stride apart, which for four row tiles gave some
// CTAs nothing but empty tiles and others nothing but the longest.
enum TileOrder { kRaster = 0, kTriangle = 1 /* only tiles that touch the diagonal or lie below */, kLastFirst = 2, kFirstFirst = 3 /* by row tile,
                 the one with the most K-slices first, all planes of it before the next */ };
struct TileMap {
  int tiles_m, tiles_n;
  long total;          // tiles_m * tiles_n * batches * splits (kTriangle: the tiles that exist)
  int order, planes, per_plane;
  NrsFastDiv div_planes, div_plane, div_group, div_tiles_n, div_last;   // (integer divisions took each role 2 thousand clocks a tile)
  void finish() {
    div_planes = NrsFastDiv(planes);
    div_plane = NrsFastDiv(per_plane);
    div_group = NrsFastDiv(kGroupM * tiles_n);
    div_tiles_n = NrsFastDiv(tiles_n);
    div_last = NrsFastDiv(tiles_m % kGroupM ? tiles_m % kGroupM : kGroupM);   // row tiles of the last group
  }
  template <int BN>
  __device__ __forceinline__ void decode(long t, int* tile_m, int* tile_n, int* z) const {
    const uint32_t u = (uint32_t)t;   // (launch() checks the range)
    uint32_t a, b;
    if (order >= kLastFirst) {
      div_planes.divmod(u, a, b);
      *z = (int)b;
      const uint32_t m = div_tiles_n.div(a);
      *tile_n = (int)(a - m * (uint32_t)tiles_n);
      *tile_m = order == kLastFirst ? tiles_m - 1 - (int)m : (int)m;
      return;
    }
    div_plane.divmod(u, a, b);
    *z = (int)a;
    const int r = (int)b;
    if (order == kTriangle) {
      int m = 0, left = r;
      for (int cnt; left >= (cnt = min(tiles_n, (m * BM + BM - 1) / BN + 1)); ++m) left -= cnt;
      *tile_m = m;
      *tile_n = left;
      return;
    }
    const int group = (int)div_group.div((uint32_t)r), first = group * kGroupM, rr = r - group * kGroupM * tiles_n;
    const int gm = min(kGroupM, tiles_m - first);
    *tile_n = (int)(gm == kGroupM ? (uint32_t)rr / kGroupM : div_last.div((uint32_t)rr));
    *tile_m = first + (rr - *tile_n * gm);
  }
  // The tile that CTA `me` of `step` takes in the round that starts at `base`; -1: none.
  __device__ __forceinline__ long at(long base, long me, long step, bool odd) const {
    const long t = base + (order != kRaster && odd ? step - 1 - me : me);
    return t < total ? t : -1;
  }
};

// Shared memory of the epilogue: a plane-emission staging tile per team of warps (which take 32 columns together), [128 rows][128 B] (pairs: [128 rows][64 B] of
// hi, then of lo), or (row-major results) a 32 x 16 transpose tile per warp.
template <int NPLANES, class Policy>
__host__ __device__ constexpr int emit_bytes() { return Policy::kCanEmit ? Policy::kEpiWarps / Policy::kTeamWarps * BM * 128 : Policy::kEpiWarps * 2048; }
template <class Policy>
__host__ __device__ constexpr int threads() { return 64 + 32 * Policy::kEpiWarps + (Policy::kSlab ? 32 : 0); }

// Four consecutive values of which `n` (or more: all) exist; `vec`: dst is 16-byte aligned when all four do.
__device__ __forceinline__ void store_guarded(float* dst, float4 v, int n, bool vec) {
  if (vec && n >= 4) { *reinterpret_cast<float4*>(dst) = v; return; }
  if (n > 0) dst[0] = v.x;
  if (n > 1) dst[1] = v.y;
  if (n > 2) dst[2] = v.z;
  if (n > 3) dst[3] = v.w;
}
__device__ __forceinline__ float4 load_guarded(const float* src, int n, bool vec) {
  if (vec && n >= 4) return *reinterpret_cast<const float4*>(src);
  return make_float4(n > 0 ? src[0] : 0.0f, n > 1 ? src[1] : 0.0f, n > 2 ? src[2] : 0.0f, n > 3 ? src[3] : 0.0f);
}

// A warp's 32 rows x 16 columns, one row per lane, turned into four float4s per lane that lie along the rows: lane l
// gets row 8*i + l/4, columns 4*(l%4)..+3 in v[i].  A global access of the warp then covers eight 64-byte row segments
// instead of 16 bytes in each of 32 rows (which took the store unit 32 cycles an instruction: 2 us per 128 x 128 tile and
// output).  The tile is 16 lines of 128 bytes, two rows a line, its 16-byte chunks XORed by the line: conflict-free both ways.
__device__ __forceinline__ void rows_to_lines(float* tile, int lane, const uint32_t (&r)[16], float4 (&v)[4]) {
  float4* t4 = reinterpret_cast<float4*>(tile);
  auto chunk = [](int row, int c) { return row * 4 + (c ^ ((row >> 1) & 3)); };
  __syncwarp();   // the previous block's values have been read
#pragma unroll
  for (int g = 0; g < 4; ++g)
    t4[chunk(lane, g)] = make_float4(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]), __uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = t4[chunk(8 * i + (lane >> 2), lane & 3)];
}

// The column blocks of an epilogue warp: block c of a tile is its columns [c * kW, (c + 1) * kW); a warp takes c_first,
// c_first + kStep, ...
template <int BN, class Policy>
struct EpiBlocks {
  static constexpr int kW = Policy::kCanEmit && Policy::kTeamWarps == 4 ? 32 : 16, kBlocks = BN / kW, kStep = Policy::kEpiWarps / 4;
  // (a team of eight: 2 * team + half)
  __host__ __device__ static constexpr int first(int warp /*from 0, of the epilogue*/) { return kStep == 1 ? 0 : warp >> 2; }
  // Does the epilogue of the tile whose columns start at n0 read what belongs to the warp's first block?  The tile has that
  // block, the output has columns in it (a ragged last column tile may not), and the results leave here, not through a
  // K-split's second pass.
  __host__ __device__ static constexpr bool reads_first(int c_first, int n0, int n_total, int splits) {
    return c_first < kBlocks && n0 + c_first * kW < n_total && splits == 1;
  }
};

template <int BN, int NPLANES, class Policy, bool PAIR, int KW>
__global__ void __launch_bounds__(threads<Policy>(), 1)
tc_kernel(const __grid_constant__ CUtensorMap tm_a_hi, const __grid_constant__ CUtensorMap tm_a_lo,
          const __grid_constant__ CUtensorMap tm_b_hi, const __grid_constant__ CUtensorMap tm_b_lo,
          const __grid_constant__ CUtensorMap tm_out_hi, const __grid_constant__ CUtensorMap tm_out_lo,
          const Policy pol, const SplitInfo sp, const TileMap tmap, const int emit /*planes to emit: 0, 1 or 2*/,
          const Ranges rg, int* __restrict__ err_flag) {
  constexpr int kEmitBytes = emit_bytes<NPLANES, Policy>();
  using L = SmemLayout<BN, NPLANES, kEmitBytes, PAIR, KW, Policy::kSlab>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* emit_tile = smem + L::kRingBytes;   // [four warps][planes][128 rows][128 B], 1024-byte aligned
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(emit_tile + kEmitBytes);
  constexpr int kBars = Policy::kSlab ? L::kSlabsA + L::kSlicesB : L::kStages;   // (slabs of A, then slices of B)
  uint64_t* empty_bar = full_bar + kBars;
  uint64_t* acc_full = empty_bar + kBars;   // [2] accumulator ready for the epilogue
  uint64_t* acc_empty = acc_full + 2;            // [2] accumulator drained by the epilogue
  uint64_t* emit_bars = acc_empty + 2;           // [four warps][2] staging tile free / staging tile written
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(emit_bars + 4);

  const int warp = (int)uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
  // A pair walks the tile list together: its CTA of rank r takes row tile 2*i + r of every pair of row tiles i.
  const int rank = PAIR ? (int)cluster_rank() : 0;
  const long t_first = PAIR ? blockIdx.x / 2 : blockIdx.x, t_step = PAIR ? gridDim.x / 2 : gridDim.x;

  if (warp == 0 && lane == 0) {
    prefetch_tmap(&tm_a_hi);
    prefetch_tmap(&tm_b_hi);
    if (NPLANES == 2) { prefetch_tmap(&tm_a_lo); prefetch_tmap(&tm_b_lo); }
    if (emit >= 1) prefetch_tmap(&tm_out_hi);
    if (emit == 2) prefetch_tmap(&tm_out_lo);
    for (int s = 0; s < kBars; ++s) { mbar_init(&full_bar[s], 1); mbar_init(&empty_bar[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], Policy::kEpiWarps * (PAIR ? 2 : 1)); for (int t = 0; t < 2; ++t) mbar_init(&emit_bars[2 * t + b], Policy::kTeamWarps * 32); }
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc<PAIR>(tmem_slot, L::kTmemCols);
    tmem_relinquish<PAIR>();
  }
  tc_fence_before_sync();
  if constexpr (PAIR) cluster_sync(); else __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = uniform(*tmem_slot);
  // Everything above (barriers, tensor memory, descriptor prefetch) may overlap the tail of the kernel
  // before this one in the stream; from here on its results are needed.
  NRS_PDL_WAIT();
  NRS_PDL_TRIGGER();   // the next kernel may be scheduled as this grid's SMs free up

  if constexpr (Policy::kSlab) {
    // ---------------- TMA producers: slabs of A (warp 0) and slices of B (the last warp) through rings of their own
    if (warp == 0 || warp == 2 + Policy::kEpiWarps) {
      const bool of_a = warp == 0;
      const uint32_t bytes = (uint32_t)(PAIR ? 2 : 1) * (of_a ? NPLANES * pol.slab_rows() * (uint32_t)L::kRowBytes : (uint32_t)L::kBSlice);
      const int slots = of_a ? L::kSlabsA : L::kSlicesB, first_bar = of_a ? 0 : L::kSlabsA, per_slab = of_a ? 1 : pol.slab_taps();
      uint32_t s = 0, ph = 0, issued = 0;
      bool ok = true;
      for (long base = 0; base < tmap.total && ok; base += t_step) {
        const long t = tmap.at(base, t_first, t_step, false);
        if (t < 0) break;
        int tile_m, tile_n, z;
        tmap.template decode<BN>(t, &tile_m, &tile_n, &z);
        if (PAIR) tile_m = 2 * tile_m + rank;
        const int batch = (int)sp.div_splits.div((uint32_t)z), split = z - batch * sp.splits;
        const int kb_begin = split * sp.kb_per_split;
        const int kb_end = sp.chunks > 1 ? sp.kb_total : min(sp.kb_total, kb_begin + sp.kb_per_split);
        const int n0 = tile_n * BN + (PAIR ? rank * (BN / 2) : 0);
        typename Policy::Cursor cur = pol.template cursor<KW>(tile_m, batch, kb_begin);
        for (int kb = kb_begin; kb < kb_end && ok; ++kb) {
          for (int i = 0; i < per_slab; ++i) {
            if (!mbar_wait_warp(&empty_bar[first_bar + s], ph ^ 1u)) { ok = false; break; }
            uint32_t bar;
            if constexpr (PAIR) bar = cluster_addr(&full_bar[first_bar + s], 0); else bar = smem_u32(&full_bar[first_bar + s]);
            if (elect_one()) {
              if (rank == 0) mbar_expect_tx(&full_bar[first_bar + s], bytes);
              if (of_a) {
                uint8_t* dst = smem + s * L::kSlab;
                pol.template load_a<PAIR, KW, L::kRowBytes>(dst, &tm_a_hi, bar, cur);
                if (NPLANES == 2) pol.template load_a<PAIR, KW, L::kRowBytes>(dst + L::kSlabPlane, &tm_a_lo, bar, cur);
              } else {
                uint8_t* dst = smem + L::kSlabsA * L::kSlab + s * L::kBSlice;
                const int col = pol.template slab_column<KW>(cur, i);
                if constexpr (L::kTwice) {   // rank 0: hi lo hi, rank 1: lo hi hi
                  tma_load_3d_to<PAIR>(dst + rank * L::kBTile, &tm_b_hi, bar, col, n0, 0);
                  tma_load_3d_to<PAIR>(dst + (1 - rank) * L::kBTile, &tm_b_lo, bar, col, n0, 0);
                  tma_load_3d_to<PAIR>(dst + 2 * L::kBTile, &tm_b_hi, bar, col, n0, 0);
                } else {
                  tma_load_3d_to<PAIR>(dst, &tm_b_hi, bar, col, n0, 0);
                  if (NPLANES == 2) tma_load_3d_to<PAIR>(dst + L::kBTile, &tm_b_lo, bar, col, n0, 0);
                }
              }
            }
            __syncwarp();
            ++issued;
            if (++s == (uint32_t)slots) { s = 0; ph ^= 1u; }
          }
          pol.template advance<KW>(cur);
        }
      }
      if (!ok) {   // (as below)
        if (lane == 0) atomicExch(err_flag, kErrProducerWait);
        if (rank == 0) for (uint32_t j = (issued > (uint32_t)slots ? issued - slots : 0); j < issued; ++j)
          if (!mbar_wait_warp(&full_bar[first_bar + j % slots], (j / slots) & 1u)) {
            if (lane == 0) atomicExch(err_flag, kErrDrainWait);
            break;
          }
      }
    }
  }
  if (warp == 0) {
    if constexpr (!Policy::kSlab) {
    // ---------------- TMA producer
    // Both CTAs of a pair count their bytes on the barrier of rank 0, which expects the sum.
    const uint32_t slice_bytes = (uint32_t)(PAIR ? 2 : 1) * NPLANES * (pol.a_slice_rows() * (uint32_t)L::kRowBytes + (uint32_t)L::kBTile);
    uint32_t s = 0, ph = 0, issued = 0;   // ring slot, its use's parity, slices so far: run on across tiles
    bool ok = true;
    bool odd = false;
    for (long base = 0; base < tmap.total && ok; base += t_step, odd = !odd) {
      const long t = tmap.at(base, t_first, t_step, odd);
      if (t < 0) break;
      int tile_m, tile_n, z;
      tmap.template decode<BN>(t, &tile_m, &tile_n, &z);
      if (PAIR) tile_m = 2 * tile_m + rank;   // beyond the last row tile: TMA fills zeros
      const int batch = (int)sp.div_splits.div((uint32_t)z), split = z - batch * sp.splits;
      int kb_begin = split * sp.kb_per_split;
      int kb_end = sp.chunks > 1 ? sp.kb_total : min(sp.kb_total, kb_begin + sp.kb_per_split);
      if (!pol.clip(tile_m, tile_n, BN, &kb_begin, &kb_end)) continue;
      const int n0 = tile_n * BN + (PAIR ? rank * (BN / 2) : 0);
      // Where the K-slices of this tile lie, stepped along instead of recomputed (the divisions of a recomputation per
      // slice and plane made the producer the bottleneck: 58 -> 72 us on a 64-channel convolution).
      typename Policy::Cursor cur = pol.template cursor<KW>(tile_m, batch, kb_begin);
      for (int kb = kb_begin; kb < kb_end; kb += L::kSlices) {
        if (!mbar_wait_warp(&empty_bar[s], ph ^ 1u)) { ok = false; break; }
        const bool two = L::kSlices == 2 && kb + 1 < kb_end;
        uint8_t* st = smem + s * L::kStage;
        uint32_t bar;
        if constexpr (PAIR) bar = cluster_addr(&full_bar[s], 0); else bar = smem_u32(&full_bar[s]);
        auto bring = [&](uint8_t* dst) {
          pol.template load_a<PAIR, KW, L::kRowBytes>(dst, &tm_a_hi, bar, cur);
          pol.template load_b<BN, PAIR, KW, L::kRowBytes>(dst + L::kATile, &tm_b_hi, bar, cur, n0);
          if (NPLANES == 2) {
            pol.template load_b<BN, PAIR, KW, L::kRowBytes>(dst + L::kATile + L::kBTile, &tm_b_lo, bar, cur, n0);
            pol.template load_a<PAIR, KW, L::kRowBytes>(dst + L::kATile + 2 * L::kBTile, &tm_a_lo, bar, cur);
          }
        };
        const bool leader = elect_one();
        if (leader) {
          if (rank == 0) mbar_expect_tx(&full_bar[s], two ? 2 * slice_bytes : slice_bytes);
          bring(st);
        }
        pol.template advance<KW>(cur);
        if (two) {
          if (leader) bring(st + L::kSlice);
          pol.template advance<KW>(cur);
        }
        __syncwarp();
        ++issued;
        if (++s == (uint32_t)L::kStages) { s = 0; ph ^= 1u; }
      }
    }
    if (!ok) {
      if (lane == 0) atomicExch(err_flag, kErrProducerWait);
      // Loads already issued still land in this CTA's shared memory: wait for them
      // (bounded) before the CTA may retire.  (Rank 1 of a pair has no barrier of its own to ask; its last load was
      // issued a full wait limit, a second, ago.)
      if (rank == 0) for (uint32_t j = (issued > (uint32_t)L::kStages ? issued - L::kStages : 0); j < issued; ++j) {
        const int sj = j % L::kStages;
        if (!mbar_wait_warp(&full_bar[sj], (j / L::kStages) & 1u)) {
          if (lane == 0) atomicExch(err_flag, kErrDrainWait);
          break;
        }
      }
    }
    }
  } else if (warp == 1) {
    if (rank == 0) {
      // ---------------- UMMA issuer
      constexpr bool kAMn = Policy::kAMnMajor, kBMn = Policy::kBMnMajor;
      constexpr int kRows = PAIR ? 2 * BM : BM;
      constexpr uint32_t idesc_wide = NPLANES == 2 ? make_idesc_f16(kRows, 2 * BN, kAMn, kBMn) : make_idesc_tf32(kRows, BN, kAMn, kBMn);
      constexpr uint32_t idesc_half = make_idesc_f16(kRows, BN, kAMn, kBMn);
      // K-major: a UMMA's K (8 values of f32, 16 of f16) is 32 bytes inside the swizzle row.  MN-major: 32-column blocks of
      // [32 k][row], so a K-step is 1024 bytes and blocks are a whole slice apart (the blocks of B_lo follow those of B_hi).
      auto desc = [](bool mn, uint32_t addr, int k) {
        if (KW == 64) return mn ? make_smem_desc_sw128(addr + (uint32_t)k * 2048u, KW * 128, 1024) : make_smem_desc_sw128(addr + (uint32_t)k * 32u, 16, 1024);
        if (NPLANES == 2) return mn ? make_smem_desc_sw64(addr + (uint32_t)k * 1024u, BK * 64, 512) : make_smem_desc_sw64(addr + (uint32_t)k * 32u, 16, 512);
        return mn ? make_smem_desc_sw128_32b(addr + (uint32_t)k * 1024u, BK * 128, 512) : make_smem_desc_sw128(addr + (uint32_t)k * 32u, 16, 1024);
      };
      // The products of one K-slice.
      auto multiply = [&](uint32_t d, uint32_t a_hi, uint32_t a_lo, uint32_t b_hi, bool first) {
#pragma unroll
        for (int k = 0; k < (NPLANES == 2 ? KW / 16 : BK / 8); ++k) {
          const uint64_t da_hi = desc(kAMn, a_hi, k), db_hi = desc(kBMn, b_hi, k);
          const uint32_t more = !(first && k == 0);
          if constexpr (NPLANES == 1) {
            umma_tf32<PAIR>(d, da_hi, db_hi, idesc_wide, more);
          } else {
            if constexpr (L::kTwice) {
              // A_hi read once instead of twice: shared memory is what bounds these tiles (and a UMMA of 64 columns takes
              // 46 clocks instead of 32).  With B laid out [hi0 lo0 hi0] in one CTA and [lo1 hi1 hi1] in the other (halves 0
              // and 1 of the columns), the wide product's columns are hh0 hl0 hl1 hh1, and the narrow one (lh0 lh1, of the
              // third blocks) lands on hl0 hl1.  1014 -> 909 clocks per slice of a 64 -> 128 layer, 895 -> 830 of 128 -> 128.
              umma_f16<PAIR>(d, da_hi, db_hi, idesc_wide, more);
              umma_f16<PAIR>(d + BN / 2, desc(kAMn, a_lo, k), desc(kBMn, b_hi + 2 * L::kBTile, k), idesc_half, 1);
              continue;
            }
            if constexpr (PAIR) {   // (each CTA holds its half of B_hi and of B_lo: no one product over both)
              umma_f16<PAIR>(d, da_hi, db_hi, idesc_half, more);
              umma_f16<PAIR>(d + BN, da_hi, desc(kBMn, b_hi + L::kBTile, k), idesc_half, more);
            } else {
              umma_f16<PAIR>(d, da_hi, db_hi, idesc_wide, more);   // hi*hi | hi*lo
            }
            umma_f16<PAIR>(d + BN, desc(kAMn, a_lo, k), db_hi, idesc_half, 1);   // + lo*hi
          }
        }
      };
      [[maybe_unused]] uint32_t sb = 0, phb = 0;   // slabs: the ring of B
      uint32_t s = 0, ph = 0, local = 0;
      bool ok = true;
      bool odd = false;
      for (long base = 0; base < tmap.total && ok; base += t_step, odd = !odd) {
        const long t = tmap.at(base, t_first, t_step, odd);
        if (t < 0) break;
        int tile_m, tile_n, z;
        tmap.template decode<BN>(t, &tile_m, &tile_n, &z);
        const int split = z - (int)sp.div_splits.div((uint32_t)z) * sp.splits;
        int kb_begin = split * sp.kb_per_split, kb_end = sp.chunks > 1 ? sp.kb_total : min(sp.kb_total, kb_begin + sp.kb_per_split);
        if (!pol.clip(tile_m, tile_n, BN, &kb_begin, &kb_end)) continue;
        for (int k0 = kb_begin; k0 < kb_end && ok; k0 += sp.kb_per_split) {
          const int nkb = min(sp.kb_per_split, kb_end - k0);   // >= 1 by construction
          const uint32_t buf = local & 1u, use = local >> 1;
          ++local;
          if (!(PAIR ? mbar_wait_warp_cluster(&acc_empty[buf], (use & 1u) ^ 1u) : mbar_wait_warp(&acc_empty[buf], (use & 1u) ^ 1u))) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t d = tmem_base + buf * (uint32_t)L::kAccCols;
          // (No tcgen05 fence after a wait: the mbarrier's complete_tx orders the TMA writes before the
          // UMMAs, and a fence would make the issuing thread wait out the UMMAs in flight.)
          if constexpr (Policy::kSlab) {
            for (int i = 0; i < nkb && ok; ++i) {
              if (!mbar_wait_warp(&full_bar[s], ph)) { ok = false; break; }
              const uint32_t slab = smem_u32(smem + s * L::kSlab);
              for (int tap = 0; tap < pol.slab_taps(); ++tap) {
                if (!mbar_wait_warp(&full_bar[L::kSlabsA + sb], phb)) { ok = false; break; }
                const uint32_t b_hi = smem_u32(smem + L::kSlabsA * L::kSlab + sb * L::kBSlice);
                const uint32_t a_hi = slab + pol.slab_tap_row(tap) * (uint32_t)L::kRowBytes;
                if (elect_one()) {
                  multiply(d, a_hi, a_hi + L::kSlabPlane, b_hi, (i | tap) == 0);
                  umma_commit<PAIR>(&empty_bar[L::kSlabsA + sb]);
                }
                __syncwarp();
                if (++sb == (uint32_t)L::kSlicesB) { sb = 0; phb ^= 1u; }
              }
              if (ok && elect_one()) umma_commit<PAIR>(&empty_bar[s]);
              __syncwarp();
              if (++s == (uint32_t)L::kSlabsA) { s = 0; ph ^= 1u; }
            }
          } else {
            for (int i = 0; i < nkb; i += L::kSlices) {
              if (!mbar_wait_warp(&full_bar[s], ph)) { ok = false; break; }
              const uint32_t slot = smem_u32(smem + s * L::kStage);
              if (elect_one()) {
#pragma unroll
                for (int sl = 0; sl < L::kSlices; ++sl) {
                  if (sl > 0 && i + sl >= nkb) break;
                  const uint32_t a_hi = slot + sl * L::kSlice, b_hi = a_hi + L::kATile;   // B_lo follows B_hi directly
                  multiply(d, a_hi, b_hi + 2 * L::kBTile, b_hi, (i | sl) == 0);
                }
                umma_commit<PAIR>(&empty_bar[s]);  // slot reusable once these UMMAs have read it
              }
              __syncwarp();
              if (++s == (uint32_t)L::kStages) { s = 0; ph ^= 1u; }
            }
          }
          if (ok && elect_one()) umma_commit<PAIR>(&acc_full[buf]);
          __syncwarp();
        }
      }
      if (!ok && lane == 0) atomicExch(err_flag, kErrMmaWait);
    }
  } else if (!Policy::kSlab || warp < 2 + Policy::kEpiWarps) {
    // ---------------- epilogue: warp w owns TMEM lanes [32*(w%4), +32)
    const int q = warp & 3;
    const int row = q * 32 + lane;   // row inside the tile
    // (kCanEmit: every team of warps takes 32-column blocks of its own, with a staging tile and an issuing thread; four
    // warps have a whole block each for their lanes' rows, eight half of one)
    const int team = (warp - 2) / Policy::kTeamWarps, half = Policy::kTeamWarps == 8 ? ((warp - 2) >> 2) & 1 : 0;
    const bool emit_issuer = (warp - 2) % Policy::kTeamWarps == 0 && lane == 0;
    uint64_t* emit_bar = emit_bars + (Policy::kCanEmit ? 2 * team : 0);
    uint8_t* team_tile = emit_tile + (Policy::kCanEmit ? team * BM * 128 : 0);
    [[maybe_unused]] float out_scale = 1.0f;
    [[maybe_unused]] uint32_t top = 0;
    [[maybe_unused]] const pr::Unscale unscale(NPLANES == 2 ? rg.a->bound : 1.0f, NPLANES == 2 ? rg.b->bound : 1.0f);
    if constexpr (NPLANES == 2) {
      if (rg.out) {
        const float bound = pol.out_bound(rg.a->top, rg.b->top, lane);
        out_scale = pr::scale_of(bound);
        if (blockIdx.x == 0 && warp == 2 && lane == 0) rg.out->bound = bound;   // (a K-split's second pass and the readers)
      }
    }
    uint32_t local = 0, emitted = 0;
    bool ok = true;
    bool odd = false;
    for (long base = 0; base < tmap.total && ok; base += t_step, odd = !odd) {
      const long t = tmap.at(base, t_first, t_step, odd);
      if (t < 0) break;
      int tile_m, tile_n, z;
      tmap.template decode<BN>(t, &tile_m, &tile_n, &z);
      if (PAIR) tile_m = 2 * tile_m + rank;
      const int batch = (int)sp.div_splits.div((uint32_t)z), split = z - batch * sp.splits;
      int kb_begin = split * sp.kb_per_split, kb_end = sp.chunks > 1 ? sp.kb_total : min(sp.kb_total, kb_begin + sp.kb_per_split);
      if (!pol.clip(tile_m, tile_n, BN, &kb_begin, &kb_end)) continue;   // the same verdict in all three roles
      const int n0 = tile_n * BN;
      [[maybe_unused]] const auto rw = pol.row(tile_m, batch, row);   // index arithmetic under the main loop
      using E = EpiBlocks<BN, Policy>;
      constexpr int kW = E::kW, kBlocks = E::kBlocks, kStep = E::kStep;
      const int c_first = E::first(warp - 2);
      // What the first block reads besides the accumulator is under way before that is full.
      [[maybe_unused]] auto extra = pol.template fetch<kW>(rw, n0 + c_first * kW, E::reads_first(c_first, n0, sp.n_total, sp.splits));
      for (int k0 = kb_begin; k0 < kb_end && ok; k0 += sp.kb_per_split) {
        const uint32_t buf = local & 1u, use = local >> 1;
        ++local;
        if (!mbar_wait(&acc_full[buf], use & 1u)) {
          if (lane == 0) atomicExch(err_flag, kErrEpilogueWait);
          ok = false;
          break;
        }
        tc_fence_after_sync();
        auto hand_back = [&]() {   // to the issuing thread, which a pair has in rank 0
          __syncwarp();
          if (lane != 0) return;
          if constexpr (PAIR) mbar_arrive_cluster(cluster_addr(&acc_empty[buf], 0)); else mbar_arrive(&acc_empty[buf]);
        };
        // The warps of a lane quarter share its column blocks out; those without one just hand the accumulator back, and so
        // do all of a pair's second CTA beyond the last row tile.
        if (c_first >= kBlocks || (PAIR && tile_m * BM >= sp.rows_total)) {
          hand_back();
          continue;
        }
        const uint32_t acc = tmem_base + buf * (uint32_t)L::kAccCols + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
        for (int c = c_first; c < kBlocks; c += kStep) {
          uint32_t r[kW];
          const int main_col = L::kTwice && c * kW >= BN / 2 ? BN + c * kW : c * kW;   // (kTwice: hh0 hl0 hl1 hh1)
          tmem_ld_32(acc + (uint32_t)main_col, r);
          if (NPLANES == 2) {
            uint32_t r2[kW];
            tmem_ld_32(acc + (uint32_t)((L::kTwice ? BN / 2 : BN) + c * kW), r2);
            tmem_ld_wait();
            unscale.apply(r, r2);
          } else {
            tmem_ld_wait();
          }
          if (c + kStep >= kBlocks) {
            // Everything this warp needs is in registers: hand the accumulator back.
            tc_fence_before_sync();
            hand_back();
          }
          if (sp.chunks > 1) {   // rows along the lanes: 512 bytes an access; a thread reads what it wrote itself
            float4* sum = reinterpret_cast<float4*>(sp.partial) + ((size_t)blockIdx.x * (BN / 4) + c * (kW / 4)) * BM + row;
#pragma unroll
            for (int g = 0; g < kW / 4; ++g) {
              if (k0 != kb_begin) {
                const float4 o = sum[g * BM];
                r[4 * g] = __float_as_uint(o.x + __uint_as_float(r[4 * g]));
                r[4 * g + 1] = __float_as_uint(o.y + __uint_as_float(r[4 * g + 1]));
                r[4 * g + 2] = __float_as_uint(o.z + __uint_as_float(r[4 * g + 2]));
                r[4 * g + 3] = __float_as_uint(o.w + __uint_as_float(r[4 * g + 3]));
              }
              if (k0 + sp.kb_per_split < kb_end)
                sum[g * BM] = make_float4(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]), __uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
            }
            if (k0 + sp.kb_per_split < kb_end) continue;
          }
          if (n0 + c * kW >= sp.n_total) continue;   // padding columns of a ragged last tile
          if constexpr (!Policy::kCanEmit) {
            float4 v[4];
            rows_to_lines(reinterpret_cast<float*>(emit_tile) + (warp - 2) * 512, lane, r, v);
            const int r0 = q * 32 + (lane >> 2), n = n0 + c * kW + (lane & 3) * 4;
            if (sp.splits > 1) {
              float* dst = sp.partial + (((size_t)split * sp.batches + batch) * sp.rows_total + (size_t)tile_m * BM + r0) * sp.n_total + n;
#pragma unroll
              for (int i = 0; i < 4; ++i, dst += (size_t)8 * sp.n_total) store_guarded(dst, v[i], sp.n_total - n, sp.n_total % 4 == 0);
            } else {
              pol.template epilogue<NPLANES == 2>(tile_m, batch, r0, n, v, out_scale, top);
            }
          } else if (sp.splits > 1) {
            float* dst = sp.partial + (((size_t)split * sp.batches + batch) * sp.rows_total + (size_t)tile_m * BM + row) * sp.n_total;
#pragma unroll
            for (int j = 0; j < kW; ++j) {
              const int n = n0 + c * kW + j;
              if (n < sp.n_total) dst[n] = __uint_as_float(r[j]);
            }
          } else {
            float v[kW];
            if (c != c_first || k0 + sp.kb_per_split < kb_end) extra = pol.template fetch<kW>(rw, n0 + c * kW, true);
            pol.epilogue(rw, n0 + c * kW, r, extra, v);
            if (NPLANES == 2 && rg.out) top = pr::seen_all(top, v);
            if (float* cs = pol.colsum_row(tile_m, q)) {
              // Sum over this warp's 32 rows, one channel per lane: a transpose-reduce (each stage halves the values a lane
              // holds; fixed order, deterministic): 31 shuffles for 32 channels, 16 for 16.
              float s[kW];
#pragma unroll
              for (int j = 0; j < kW; ++j) s[j] = v[j];
#pragma unroll
              for (int d = kW / 2; d >= 1; d >>= 1) {
                const bool up = (lane & d) != 0;
#pragma unroll
                for (int i = 0; i < d; ++i) {
                  const float keep = up ? s[i + d] : s[i];
                  const float send = up ? s[i] : s[i + d];
                  s[i] = keep + __shfl_xor_sync(0xffffffffu, send, d);
                }
              }
              if (kW == 16) s[0] += __shfl_xor_sync(0xffffffffu, s[0], 16);
              if (lane < kW) cs[n0 + c * kW + lane] = s[0];
            }
            if (emit) {
              // The staging tile is free once the previous TMA store has read it; the issuer
              // arrives on emit_bar[0] only after that.
              const uint32_t ph = emitted & 1u;
              ++emitted;
              if (emit_issuer) bulk_wait_read();
              mbar_arrive(&emit_bar[0]);
              if (!mbar_wait(&emit_bar[0], ph)) { atomicExch(err_flag, kErrEpilogueWait); ok = false; break; }
              if constexpr (NPLANES == 2) {
                uint8_t* row_hi = team_tile + row * 64;
#pragma unroll
                for (int g = 0; g < kW / 8; ++g) {   // eight values
                  const int chunk = ((g + 2 * half) ^ ((row >> 1) & 3)) * 16;   // 64-byte swizzle
                  uint2 h0, l0, h1, l1;
                  pr::split4(make_float4(v[8 * g], v[8 * g + 1], v[8 * g + 2], v[8 * g + 3]), out_scale, &h0, &l0);
                  pr::split4(make_float4(v[8 * g + 4], v[8 * g + 5], v[8 * g + 6], v[8 * g + 7]), out_scale, &h1, &l1);
                  *reinterpret_cast<uint4*>(row_hi + chunk) = make_uint4(h0.x, h0.y, h1.x, h1.y);
                  *reinterpret_cast<uint4*>(row_hi + BM * 64 + chunk) = make_uint4(l0.x, l0.y, l1.x, l1.y);
                }
              } else if constexpr (kW == 32) {
                uint8_t* row_hi = team_tile + row * 128;
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                  const int chunk = (g ^ (row & 7)) * 16;   // 128-byte swizzle: 16-byte chunk index XOR row % 8
                  *reinterpret_cast<float4*>(row_hi + chunk) = make_float4(tf32_rn(v[4 * g]), tf32_rn(v[4 * g + 1]), tf32_rn(v[4 * g + 2]), tf32_rn(v[4 * g + 3]));
                }
              }
              fence_proxy_async();   // generic-proxy writes -> visible to the TMA engine
              mbar_arrive(&emit_bar[1]);
              if (emit_issuer) {
                if (!mbar_wait(&emit_bar[1], ph)) { atomicExch(err_flag, kErrEpilogueWait); ok = false; break; }
                tma_store_4d(&tm_out_hi, team_tile, n0 + c / (32 / kW) * 32, rw.x0, Policy::kSlab ? rw.n0 : rw.y0, Policy::kSlab ? rw.y0 : rw.n0);
                if (NPLANES == 2) tma_store_4d(&tm_out_lo, team_tile + BM * 64, n0 + c / (32 / kW) * 32, rw.x0, Policy::kSlab ? rw.n0 : rw.y0, Policy::kSlab ? rw.y0 : rw.n0);
                bulk_commit();
              }
            }
          }
        }
      }
    }
    if constexpr (NPLANES == 2) {
      __syncwarp();
      if (rg.out && sp.splits == 1) pr::report(rg.out, top);
    }
    if (emit_issuer) bulk_wait_all();   // shared memory must outlive the stores that read it
  }

  tc_fence_before_sync();
  // (a pair: neither CTA may leave while the other's UMMAs read its memory or arrive on its barriers)
  __syncwarp();
  if constexpr (PAIR) cluster_sync(); else __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc<PAIR>(tmem_base, L::kTmemCols);
  }
}

// out(row, n) = policy.store(sum over splits of partial), fixed summation order.
template <bool SPLIT, class Policy>
__global__ void __launch_bounds__(256)
tc_splitk_reduce_kernel(const Policy pol, const SplitInfo sp, NrsRange* __restrict__ out_range) {
  NRS_PDL_PROLOGUE();
  const size_t per = (size_t)sp.batches * sp.rows_total * sp.n_total;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t top = 0;
  if (idx < per) {
    float s = 0.0f;
    for (int z = 0; z < sp.splits; ++z) s += sp.partial[(size_t)z * per + idx];
    const int n = (int)(idx % sp.n_total);
    const size_t t = idx / sp.n_total;
    const int row_lin = (int)(t % sp.rows_total);
    const int b = (int)(t / sp.rows_total);
    const float out_scale = SPLIT && out_range ? pr::scale_of(out_range->bound) : 1.0f;
    pol.template store<SPLIT>(row_lin / BM, b, row_lin % BM, n, s, out_scale, top);
  }
  if (SPLIT && out_range) {
    __syncwarp();
    pr::report(out_range, top);
  }
}

// Chooses the K-split: enough CTAs to fill the GPU, and no accumulation chain longer than kMaxChainK (kFewChainK) values when
// `limit_chain` (chunks where the tiles fill the GPU anyway).
inline void plan_split(const nrs_ctx* ctx, long tiles, long out_elems, int kb_total, int kw, bool limit_chain, bool conv, SplitInfo* sp) {
  const int longest = conv && 2 * out_elems <= (long)ctx->sm_count * BM * 128 ? kFewChainK : kMaxChainK;
  int s = 1;
  // (More than half a wave of tiles runs unsplit: the second pass over the partial tiles costs more
  // than the idle SMs.)
  if (2 * tiles <= ctx->sm_count && kb_total * kw >= 1024) {
    s = (int)(ctx->sm_count / tiles);
    // a split shorter than 16 K-blocks is all prologue and second pass, except where the output is so small (a Linear
    // layer at a batch of a few dozen) that the second pass is nothing: there down to 4
    const int shortest = std::max(1, (out_elems <= (1 << 15) ? 4 : 16) * BK / kw);
    if (s > kb_total / shortest) s = kb_total / shortest;
    if (s < 1) s = 1;
  }
  const int need = limit_chain ? (int)(((long)kb_total * kw + longest - 1) / longest) : 1;
  const bool in_chunks = s == 1 && need > 1;
  if (s < need) s = need;
  int per = (kb_total + s - 1) / s;
  if (per < 1) per = 1;
  if (in_chunks) per += per & 1;   // (a ring slot's two K-slices belong to one chunk)
  s = (kb_total + per - 1) / per;
  sp->kb_per_split = per;
  sp->splits = in_chunks ? 1 : s;
  sp->chunks = in_chunks ? s : 1;
}

// The tile of a launch: its columns, and whether CTAs work in pairs.  kPlans holds clocks per 32 values of K (3xTF32; 3xTF32
// in slabs; TF32), and per tile what the accumulator's way out takes (3xTF32: of each round it is hidden behind the next;
// TF32: adds to each).  The tile with the least time is taken, a K-split's second pass counted in: wide tiles for large
// outputs, narrower ones where they fill SMs that would idle or where a ragged column count would pad, pairs where there
// are enough row tiles.  `reduce_clk`: what the second pass over a K-split costs per output value, on top of its launch
// (measured: 3.6 us for 51 thousand values of a GEMM, 13.4 us for 819 thousand of a convolution, whose pixels lie strided).
// A convolution's 64-column pair is slower than the single tile in TF32 (30.1 us against 27.4 for 64 channels on 100 images
// of 32 x 32).  `limit`: widest tile allowed.
struct TilePlan { int bn; bool pair; };
inline TilePlan plan_tile(const nrs_ctx* ctx, long tiles_m, int n, long batches, int kblocks, bool split_planes, double reduce_clk, bool conv, bool slab,
                          int limit = 128) {
  static const struct { int bn; bool pair; int kb_clk[3], tile_clk[2]; } kPlans[] = {{128, true, {395, 395, 345}, {5500, 2600}},
                                                                                     {64, true, {315, 235, 317}, {3500, 1700}},
                                                                                     {128, false, {530, 420, 428}, {5500, 2600}},
                                                                                     {64, false, {400, 280, 369}, {3500, 1700}},
                                                                                     {32, false, {330, 210, 352}, {2600, 1300}}};
  TilePlan best{32, false};
  double best_t = -1.0;
  for (const auto& c : kPlans) {
    if (c.bn > limit || (c.bn > 32 && c.bn / 2 >= n)) continue;   // half of the tile or more would be padding
    const long tiles_n = (n + c.bn - 1) / c.bn;
    SplitInfo sp{};
    plan_split(ctx, tiles_m * tiles_n * batches, tiles_m * BM * n * batches, kblocks, BK, split_planes, conv, &sp);
    const int splits = sp.splits, per = sp.kb_per_split * sp.chunks;
    const long units = (c.pair ? (tiles_m + 1) / 2 : tiles_m) * tiles_n * batches * splits, slots = ctx->sm_count / (c.pair ? 2 : 1);
    const double rounds = (double)((units + slots - 1) / slots);
    double t;
    if (split_planes) {
      t = rounds * std::max((double)per * c.kb_clk[slab ? 1 : 0], (double)c.tile_clk[0]) + c.tile_clk[0];
    } else {
      t = rounds * ((double)per * (c.pair && c.bn == 64 && conv ? 400 : c.kb_clk[2]) + c.tile_clk[1]);
    }
    if (splits > 1) t += 4000.0 + reduce_clk * (double)tiles_m * BM * n * batches;
    if (best_t < 0.0 || t < best_t) { best_t = t; best = TilePlan{c.bn, c.pair}; }
  }
  return best;
}

// Work units (pixel tiles, image rows) per CTA for a reduction that is split across CTAs, `ctas`
// CTAs per split and one CTA per SM at a time.  Candidates put the CTA count just under a whole
// number of waves (a count just over one costs a whole extra round); a CTA's fixed cost
// (prologue, partial-tile store) is weighed in as `overhead_units`; more than max_units per CTA
// (the accumulation-chain limit) is not allowed, fewer than min_units not worthwhile.
inline int plan_units_per_cta(int sm_count, int ctas, long units, int min_units, int max_units, int overhead_units) {
  if (units < 1) return 1;
  long best_u = -1, best_cost = 0;
  for (int w = 1; w <= 64; ++w) {
    const long splits = (long)w * sm_count / ctas;
    if (splits < 1) continue;
    long u = (units + splits - 1) / splits;
    if (u < min_units) u = min_units;
    if (u > units) u = units;
    if (u > max_units) continue;
    const long actual = (units + u - 1) / u;
    const long rounds = (actual * ctas + sm_count - 1) / sm_count;
    const long cost = rounds * (u + overhead_units);
    if (best_u < 0 || cost < best_cost) { best_u = u; best_cost = cost; }
  }
  if (best_u < 0) best_u = max_units < units ? max_units : units;
  return (int)(best_u < 1 ? 1 : best_u);
}

template <int BN, int NPLANES, bool PAIR, int KW, class Policy>
int launch(nrs_ctx* ctx, const CUtensorMap& ta_hi, const CUtensorMap& ta_lo, const CUtensorMap& tb_hi,
           const CUtensorMap& tb_lo, const Policy& pol, int tiles_m, int n_total, int batches, int kb_total,
           const Ranges& rg, const CUtensorMap* out_hi = nullptr, const CUtensorMap* out_lo = nullptr, int* splits_out = nullptr,
           int k_per_block = KW /*values of K in one of the kb_total blocks*/) {
  using L = SmemLayout<BN, NPLANES, emit_bytes<NPLANES, Policy>(), PAIR, KW, Policy::kSlab>;
  constexpr int kSmem = L::kBytes;
  static_assert(kSmem <= 227 * 1024 && L::kStages >= 2 && (!Policy::kSlab || L::kSlicesB >= 3), "shared memory budget");
  static NrsSmemAttr attr;
  NRS_ENSURE_SMEM(ctx, attr, (tc_kernel<BN, NPLANES, Policy, PAIR, KW>), kSmem);
  const int tiles_n = (n_total + BN - 1) / BN;
  SplitInfo sp{};
  if (Policy::kMaySplit) {
    plan_split(ctx, (long)tiles_m * tiles_n * batches, (long)tiles_m * BM * n_total * batches, kb_total, k_per_block, NPLANES == 2, Policy::kConv, &sp);
  } else {   // tiles whose K ranges differ
    sp.splits = sp.chunks = 1;
    sp.kb_per_split = kb_total;
  }
  sp.kb_total = kb_total;
  sp.div_splits = NrsFastDiv(sp.splits);
  sp.batches = batches;
  sp.n_total = n_total;
  sp.rows_total = tiles_m * BM;
  sp.partial = nullptr;
  if (splits_out) *splits_out = sp.splits;
  if (sp.splits > 1 || sp.chunks > 1) {
    void* ws = nullptr;
    const size_t floats = sp.splits > 1 ? (size_t)sp.splits * batches * sp.rows_total * n_total : (size_t)ctx->sm_count * BM * BN;
    const int st = nrs_ws_slot(ctx, NRS_WS_PARTIAL, floats * sizeof(float), &ws);
    if (st != NRS_OK) return st;
    sp.partial = (float*)ws;
  }
  int* err = nullptr;
  int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  const int units_m = PAIR ? (tiles_m + 1) / 2 : tiles_m;
  TileMap tmap{};
  tmap.tiles_m = units_m; tmap.tiles_n = tiles_n; tmap.order = pol.order(); tmap.planes = batches * sp.splits; tmap.per_plane = units_m * tiles_n;
  if (tmap.order == kTriangle) {
    tmap.per_plane = 0;
    for (int m = 0; m < tiles_m; ++m) tmap.per_plane += std::min(tiles_n, (m * BM + BM - 1) / BN + 1);
  }
  tmap.finish();
  tmap.total = (long)tmap.per_plane * tmap.planes;
  NRS_REQUIRE(ctx, (long)units_m * tiles_n <= 0x7fffffffL && tmap.total <= 0x7fffffffL, NRS_ERR_SHAPE, "tensor-core product: too many tiles");
  const long slots = PAIR ? ctx->sm_count / 2 : ctx->sm_count;
  const unsigned grid = (unsigned)((tmap.total < slots ? tmap.total : slots) * (PAIR ? 2 : 1));
  // Planes can only be emitted by the direct epilogue; with a K-split the policy's store() writes them.
  const int emit = (Policy::kCanEmit && out_hi && sp.splits == 1) ? (out_lo && NPLANES == 2 ? 2 : 1) : 0;
  (void)nrs_pdl_launch_cluster(PAIR ? 2 : 1, tc_kernel<BN, NPLANES, Policy, PAIR, KW>, dim3(grid), dim3(threads<Policy>()), (size_t)kSmem, ctx->stream,
                               ta_hi, ta_lo, tb_hi, tb_lo, out_hi ? *out_hi : ta_hi, out_lo ? *out_lo : ta_hi, pol, sp, tmap, emit, rg, err);
  NRS_LAUNCHED(ctx);
  if (sp.splits > 1) {
    const size_t per = (size_t)batches * sp.rows_total * n_total;
    NRS_PDL_LAUNCH((tc_splitk_reduce_kernel<NPLANES == 2, Policy>), nrs_blocks(per, 256), 256, 0, ctx->stream, pol, sp, rg.out);
    NRS_LAUNCHED(ctx);
  }
  return NRS_OK;
}

}  // namespace tc

// Operand staging (tc_stage.cu).  Planes are [batch][rows][ldk] f32 with ldk a multiple of
// 8 and zeros beyond K; `lo == nullptr` means no split (hi = the values themselves).
// src_k_by_rows: the source is stored [K][rows] (transposed) instead of [rows][K].
// Masked gradient staging (see stage_masked_kernel): mode 0 = ReLU mask of dy[n,c,h,w] by y;
// mode 1 = gradient of a k x k / stride-k max-pool (g[n,c,h/k,w/k], argmax) followed by the ReLU
// mask, taken from the pooled output y[n,c,h/k,w/k].  nchw_out and the planes are each optional
// (lo only with hi).  chan_partial (optional, nrs_stage_masked_partial_rows(...) x c floats): per-block
// channel sums of the result, for the bias gradient; *chan_partial_rows receives how many rows
// were written (0: this path does not produce them and the caller sums the NCHW gradient).
int nrs_tc_stage_masked(nrs_ctx* ctx, int mode, const float* g, const float* y, const int32_t* argmax, int n, int c,
                        int h, int w, int k, float* nchw_out, float* hi, float* lo, float* chan_partial = nullptr,
                        int* chan_partial_rows = nullptr, const NrsRange* g_range = nullptr);
// 2x2 / stride-2 max-pool forward that also writes the NHWC planes of the pooled output
// (NRS_ERR_UNSUPPORTED for odd image sizes).
int nrs_tc_pool2_fwd_planes(nrs_ctx* ctx, const float* x, float* y, int32_t* argmax, float* hi, float* lo, int n, int c,
                            int h, int w, const NrsRange* x_range = nullptr);
inline size_t nrs_stage_masked_partial_rows(int n, int h, int w) { return ((size_t)n * (h / 2) * (w / 2) + 31) / 32; }
// Conv weights w[co][ci][kh][kw] -> K-major planes; the channels of a tap are padded with zeros to a multiple of 32.
//  for_dgrad == 0: out[co][(i*kw + j)*ceil32(ci) + ci]   (forward B operand)
//  for_dgrad == 1: out[ci][(i*kw + j)*ceil32(co) + co]   (data-gradient B operand)
int nrs_tc_stage_conv_weight(nrs_ctx* ctx, const float* w, float* hi, float* lo, int co, int ci, int kh, int kw,
                             int for_dgrad);
