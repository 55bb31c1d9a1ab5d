// Row-wise operators (LayerNorm, softmax, cross-entropy) on tensors large enough to be bound by HBM, and on
// rows of any width: an asynchronous pipeline through shared memory.
//
// The rows of a dense [rows][f] tensor are one contiguous range, so a group of rows is fetched with one bulk
// copy (cp.async.bulk) whatever f is, and sent out with one; a row of odd width costs no misaligned or partial
// vector access.  A team of warps (one warp up to 512 columns, else one per 512) owns a private ring of
// slots, so nothing ever waits for another team: wait for the slot's copy, work on its rows in place (the
// values of a row sit in registers between its reductions), hand the slot to the bulk store, refill it once
// the store has read it.  Two slots of every team are on their way while one is worked on: some 100 KB in
// flight per SM against the 44 KB that 6.5 TB/s at one microsecond of latency need, with one block of 8 to 16
// warps per SM and no dependence on occupancy.  (The register kernels it replaces at these sizes keep a row per
// warp in flight: 80 to 160 registers per thread left them latency-bound.)
//
// Measured on [16384][1000] (us, the kernel it replaces -> this one; 40, 30 at the measured copy rate): LayerNorm
// backward with parameters 104 -> 41, dx alone 96 -> 34, LayerNorm forward 42 -> 36, cross-entropy 52 -> 48.  It is not the
// better kernel at every width: what decides is how many warps' worth of columns an SM works on (live_warps below) and how
// much a row costs besides its bytes (a barrier wait, a proxy fence, two team syncs and a store issued by one lane: at
// 256 columns a row is 1 KB, and LayerNorm backward takes 56 us for 16 M elements against 44 in registers).  The
// operators state their own lines with both sides measured.
#pragma once

#include "nrs_internal.h"
#include "tc_common.cuh"

namespace rowpipe {

constexpr int kMaxIn = 2, kMaxOut = 3;

struct Params {
  const float* in[kMaxIn];     // [rows][f] each; in[k] lands in buffer k
  float* out[kMaxOut];         // [rows][f] each (null: not wanted)
  int out_buf[kMaxOut];        // buffer that holds the result of out[k]
  int out_add[kMaxOut];        // add to the destination instead of overwriting it
  int n_in, n_buf;
  int rows, f;
  int group_rows;              // rows per slot (a multiple that keeps slots 16-byte aligned)
  int team_warps, slots;       // warps per team; ring depth
};

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(tc::smem_u32(dst)), "l"(src), "r"(bytes), "r"(tc::smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void bulk_store(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst), "r"(tc::smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_add(void* dst, const void* src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;"
               ::"l"(dst), "r"(tc::smem_u32(src)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bulk_wait_read_1() { asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory"); }

// A team's view of itself: reductions over all its lanes (fixed order: butterfly inside a warp, warps in order).
struct Team {
  int lane, warp, warps, bar_id;
  float* scratch;              // [warps][4] of shared memory
  __device__ __forceinline__ void sync() const {
    if (warps == 1) __syncwarp();
    else tc::named_barrier(bar_id, warps * 32);
  }
  template <int N>
  __device__ __forceinline__ void sum(float (&v)[N]) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
    if (warps == 1) return;
    sync();                    // the previous reduction's values have been read
    if (lane == 0)
#pragma unroll
      for (int i = 0; i < N; ++i) scratch[warp * 4 + i] = v[i];
    sync();
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = 0.0f;
    for (int w = 0; w < warps; ++w)
#pragma unroll
      for (int i = 0; i < N; ++i) v[i] += scratch[w * 4 + i];
  }
  __device__ __forceinline__ float max(float v) const {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (warps == 1) return v;
    sync();
    if (lane == 0) scratch[warp * 4] = v;
    sync();
    for (int w = 0; w < warps; ++w) v = fmaxf(v, scratch[w * 4]);
    return v;
  }
};

// The columns a lane owns: NPL of them, in NPL / VEC vectors of VEC; first(k) is the column of vector k.
template <int NPL, int VEC>
struct Cols {
  static constexpr int kVecs = NPL / VEC;
  int base, f;
  __device__ __forceinline__ Cols(const Team& t, int f_) : base(t.warp * NPL * 32 + t.lane * VEC), f(f_) {}
  __device__ __forceinline__ int first(int k) const { return base + k * 32 * VEC; }
  __device__ __forceinline__ bool live(int k) const { return first(k) < f; }
  __device__ __forceinline__ void load(const float* row, float (&v)[NPL], float fill = 0.0f) const {
#pragma unroll
    for (int k = 0; k < kVecs; ++k) {
      if (VEC == 4) {
        const float4 q = live(k) ? *reinterpret_cast<const float4*>(row + first(k)) : make_float4(fill, fill, fill, fill);
        v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
      } else {
        v[k] = live(k) ? row[first(k)] : fill;
      }
    }
  }
  __device__ __forceinline__ void store(float* row, const float (&v)[NPL]) const {
#pragma unroll
    for (int k = 0; k < kVecs; ++k) {
      if (!live(k)) continue;
      if (VEC == 4) *reinterpret_cast<float4*>(row + first(k)) = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      else row[first(k)] = v[k];
    }
  }
};

constexpr int kThreads = 512;

// Op: `State` (per-thread, over all rows), start(cols, state), row(team, cols, state, buffers of the row, row index), finish().
template <int NPL, int VEC, class Op>
__global__ void __launch_bounds__(kThreads, 1)
row_pipe_kernel(const Params p, const Op op, int* __restrict__ err_flag) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int teams = (blockDim.x >> 5) / p.team_warps, team = warp / p.team_warps;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem_raw) + team * p.slots;
  float* scratch = reinterpret_cast<float*>(smem_raw + 1024) + team * p.team_warps * 4;
  const uint32_t buf_bytes = (uint32_t)p.group_rows * p.f * 4u, slot_bytes = buf_bytes * p.n_buf;
  uint8_t* ring = smem_raw + 2048 + (size_t)team * p.slots * slot_bytes;
  const Team tm{lane, warp - team * p.team_warps, p.team_warps, 1 + team, scratch};
  const Cols<NPL, VEC> cols(tm, p.f);
  const bool leader = tm.warp == 0 && lane == 0;
  if (threadIdx.x == 0) {
    uint64_t* all = reinterpret_cast<uint64_t*>(smem_raw);
    for (int i = 0; i < teams * p.slots; ++i) tc::mbar_init(all + i, 1);
    tc::fence_barrier_init();
  }
  __syncthreads();
  NRS_PDL_PROLOGUE();
  typename Op::template State<NPL> state;
  op.start(cols, state);

  const int groups = (p.rows + p.group_rows - 1) / p.group_rows;
  const int first = blockIdx.x * teams + team, step = gridDim.x * teams;
  auto group_bytes = [&](int grp) { return (uint32_t)min(p.group_rows, p.rows - grp * p.group_rows) * p.f * 4u; };
  auto fetch = [&](int grp, int slot) {   // by the leader; at most 12 bytes of the last group stay for plain loads
    const uint32_t bytes = group_bytes(grp) & ~15u;
    if (bytes == 0) { tc::mbar_arrive(&full[slot]); return; }
    tc::mbar_expect_tx(&full[slot], bytes * p.n_in);
    for (int k = 0; k < p.n_in; ++k)
      bulk_load(ring + (size_t)slot * slot_bytes + k * buf_bytes, p.in[k] + (size_t)grp * p.group_rows * p.f, bytes, &full[slot]);
  };
  if (leader)
    for (int s = 0; s < p.slots; ++s)
      if ((long)first + (long)s * step < groups) fetch(first + s * step, s);
  int slot = 0, prev_slot = 0, prev_next = -1;   // prev_next: the group to fetch into prev_slot
  uint32_t ph = 0;
  bool ok = true;
  for (long gl = first; gl < groups; gl += step) {
    const int grp = (int)gl;
    if (!tc::mbar_wait(&full[slot], ph)) {
      if (lane == 0) atomicExch(err_flag, tc::kErrMmaWait);
      ok = false;
      break;
    }
    float* buf0 = reinterpret_cast<float*>(ring + (size_t)slot * slot_bytes);
    float* buf1 = buf0 + buf_bytes / 4;
    const uint32_t bytes = group_bytes(grp);
    const size_t at = (size_t)grp * p.group_rows * p.f;
    const int tail0 = (int)((bytes & ~15u) >> 2), tail = (int)(bytes >> 2) - tail0;   // floats the bulk copies leave
    if (tail) {
      if (tm.warp == 0 && lane < tail)
        for (int k = 0; k < p.n_in; ++k) (k == 0 ? buf0 : buf1)[tail0 + lane] = p.in[k][at + tail0 + lane];
      tm.sync();
    }
    const int nrows = (int)(bytes / (p.f * 4u));
    for (int r = 0; r < nrows; ++r)
      op.template row<NPL, VEC>(tm, cols, state, buf0 + (size_t)r * p.f, buf1 + (size_t)r * p.f, grp * p.group_rows + r);
    tc::fence_proxy_async();   // results -> visible to the bulk engine
    tm.sync();
    if (leader) {
      for (int k = 0; k < kMaxOut; ++k) {
        if (!p.out[k]) continue;
        const float* src = p.out_buf[k] == 0 ? buf0 : buf1;
        if (bytes & ~15u) {
          if (p.out_add[k]) bulk_add(p.out[k] + at, src, bytes & ~15u);
          else bulk_store(p.out[k] + at, src, bytes & ~15u);
        }
        for (int i = 0; i < tail; ++i) {
          float* d = p.out[k] + at + tail0 + i;
          *d = p.out_add[k] ? *d + src[tail0 + i] : src[tail0 + i];
        }
      }
      tc::bulk_commit();
      // refill the slot before this one: its stores have had a whole group's time to read it
      if (prev_next >= 0) { bulk_wait_read_1(); fetch(prev_next, prev_slot); }
    }
    const long nxt = gl + (long)p.slots * step;
    prev_next = nxt < groups ? (int)nxt : -1;
    prev_slot = slot;
    if (++slot == p.slots) { slot = 0; ph ^= 1u; }
  }
  if (!ok && leader) {   // copies already issued land in this block's shared memory: wait for them (bounded)
    for (int s = 0; s < p.slots; ++s) (void)tc::mbar_wait_limit(&full[s], ph ^ (s < slot ? 1u : 0u), tc::kWaitClocks);
  }
  if (leader) tc::bulk_wait_all();   // shared memory must outlive the stores that read it
  __syncthreads();
  op.template finish<NPL, VEC>(tm, cols, state, reinterpret_cast<float*>(smem_raw + 2048), team, teams);
}

// Elements per lane by width: 8 up to 256 columns, else 16, a row of more than 512 columns being shared by a team of
// warps (with 32 per lane, one warp per row of 1000 columns, shared memory had room for eight or nine warps and the
// exponentials of a softmax ran at a third of the rate: 65 us).
struct Plan {
  int npl, team_warps, group_rows, teams;   // teams: 0 when three slots of one team do not fit
  size_t slot;
};
constexpr size_t kHead = 2048, kBudget = 220 * 1024 - kHead;
constexpr int kMaxColumns = 8192;   // one slot of two buffers is then 64 KB
inline Plan plan(int f, int n_buf) {
  Plan q{};
  if (f > kMaxColumns) return q;
  q.npl = f <= 256 ? 8 : 16;
  q.team_warps = (f + q.npl * 32 - 1) / (q.npl * 32);
  // rows per slot: whole 16-byte groups, and at least 1 KB per copy
  const int unit = f % 4 == 0 ? 1 : f % 2 == 0 ? 2 : 4;
  q.group_rows = unit;
  while (q.group_rows * f * 4 < 1024) q.group_rows += unit;
  q.slot = (size_t)q.group_rows * f * 4 * n_buf;
  int warps = kThreads / 32;
  while (warps > q.team_warps && (size_t)(warps / q.team_warps) * 3 * q.slot > kBudget) --warps;
  q.teams = warps / q.team_warps;
  if (q.teams > 0 && kBudget / (q.slot * q.teams) < 3) q.teams = 0;
  return q;
}
// Share of a row's lanes x elements that hold columns.
inline double fill(int f) {
  if (f > kMaxColumns) return 0.0;
  const int unit = 32 * (f <= 256 ? 8 : 16);
  return (double)f / ((f + unit - 1) / unit * unit);
}
// Warps' worth of columns an SM works on: the warps whose slots fit into shared memory (16 at most; groups of four rows
// of an odd width leave 3 of 1401 columns) times their fill.  With few of them the work inside a row is not hidden.
inline double live_warps(int f, int n_buf) {
  const Plan q = plan(f, n_buf);   // (no teams beyond kMaxColumns)
  return q.teams * q.team_warps * fill(f);
}
// Whether a tensor set can take this path: 16-byte aligned bases, rows of at most kMaxColumns, 128 K elements (below, a
// shorter prologue wins: [64][10] 4 us against 20).  The operators add their own lines against the register kernels
// (widths of whole float4s) and the scalar loops (other widths).
inline bool applies(int rows, int f, std::initializer_list<const void*> ptrs) {
  if (f > kMaxColumns || rows < 1) return false;
  for (const void* q : ptrs)
    if (reinterpret_cast<uintptr_t>(q) & 15) return false;
  return (size_t)rows * f >= (size_t)1 << 17;
}

template <int NPL, int VEC, class Op>
int launch_one(nrs_ctx* ctx, Params p, const Op& op, int* blocks_out) {
  const Plan q = plan(p.f, p.n_buf);
  if (q.teams == 0) return NRS_ERR_UNSUPPORTED;
  p.team_warps = q.team_warps;
  p.group_rows = q.group_rows;
  const size_t slot = q.slot;
  int teams = q.teams;
  // fewer rows than teams: spread them over the SMs
  const long groups = ((long)p.rows + p.group_rows - 1) / p.group_rows;
  while (teams > 1 && (long)(teams - 1) * ctx->sm_count >= groups) --teams;
  p.slots = (int)(kBudget / (slot * teams));
  if (p.slots > 6) p.slots = 6;
  long blocks = (groups + teams - 1) / teams;
  if (blocks > ctx->sm_count) blocks = ctx->sm_count;
  size_t smem = kHead + (size_t)teams * p.slots * slot;
  const size_t fin = kHead + Op::finish_bytes(teams, p.f);
  if (smem < fin) smem = fin;
  if (smem > 227 * 1024) return NRS_ERR_UNSUPPORTED;
  static NrsSmemAttr attr;
  NRS_ENSURE_SMEM(ctx, attr, (row_pipe_kernel<NPL, VEC, Op>), smem);
  int* err = nullptr;
  const int st = nrs_err_flag(ctx, &err);
  if (st != NRS_OK) return st;
  NRS_PDL_LAUNCH((row_pipe_kernel<NPL, VEC, Op>), (unsigned)blocks, teams * p.team_warps * 32, smem, ctx->stream, p, op, err);
  NRS_LAUNCHED(ctx);
  if (blocks_out) *blocks_out = (int)blocks;
  return NRS_OK;
}

// Rows whose width is a multiple of four move through registers as float4s.
template <class Op>
int launch(nrs_ctx* ctx, const Params& p, const Op& op, int* blocks_out = nullptr) {
  if (p.f % 4 == 0) return p.f <= 256 ? launch_one<8, 4>(ctx, p, op, blocks_out) : launch_one<16, 4>(ctx, p, op, blocks_out);
  return p.f <= 256 ? launch_one<8, 1>(ctx, p, op, blocks_out) : launch_one<16, 1>(ctx, p, op, blocks_out);
}

}  // namespace rowpipe
