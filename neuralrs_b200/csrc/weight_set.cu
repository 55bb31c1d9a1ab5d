// Batched staging of a model's weights for the tensor-core kernels.
//
// Every contraction reads its weight operand as K-major TF32 planes (a high plane rounded to nearest
// and, for 3xTF32, an f32 residual plane), re-laid out per use: convolution forward and data gradient
// want two different tap-major layouts, x@W wants W transposed, dz@W^T wants W as stored.  Staged per
// call that is one small launch per layer and pass; a training loop knows all its weights in advance,
// so they are staged here in ONE launch per step from a job table resident on the device, and the
// contraction entry points pick the planes up by (weight pointer, form).  The reference has no
// counterpart (its GEMMs read f32 weights directly, src/cuda/graph/matmul.rs:44-261).
#include "tc_mainloop.cuh"

namespace {

// One weight, read once for both of its forms (either may be absent).
struct WeightJob {
  const float* src;
  float *a_hi, *a_lo;    // x@W: W^T, [cols][ceil32(rows)]; convolution forward: [co][taps][ceil32(ci)]
  float *b_hi, *b_lo;    // dz@W^T: W, [rows][ceil32(cols)]; data gradient: [ci][taps][ceil32(co)]
  int conv, vec;         // vec: rows of a linear weight start on 16 bytes
  int rows, cols;        // as stored, [rows][cols]; a convolution's [co][ci][taps]
  int taps;
  unsigned first_block;  // this job's first block in the launch
};

constexpr int kTile = 64;          // linear: 64 x 64 values per block
constexpr int kConvCo = 16;        // convolution: 16 output x 32 input channels x up to kConvTaps taps per block (with 32 x 32 a
constexpr int kConvCi = 32;        // model's few such blocks last longer than all the others)
constexpr int kConvTaps = 9;

__host__ __device__ inline int ceil_div(int a, int b) { return (a + b - 1) / b; }
__host__ __device__ inline int ceil32(int a) { return (a + 31) / 32 * 32; }
inline unsigned job_blocks(const WeightJob& j) {
  if (j.conv) return (unsigned)(ceil32(j.rows) / kConvCo) * ceil_div(j.cols, kConvCi) * ceil_div(j.taps, kConvTaps);
  return (unsigned)ceil_div(j.rows, kTile) * ceil_div(j.cols, kTile);
}

__device__ __forceinline__ void put(float* hi, float* lo, size_t i, float v) {
  const float h = tc::tf32_rn(v);
  hi[i] = h;
  if (lo) lo[i] = v - h;
}
__device__ __forceinline__ void put4(float* hi, float* lo, size_t i, float4 v) {
  const float4 h = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
  *reinterpret_cast<float4*>(hi + i) = h;
  if (lo) *reinterpret_cast<float4*>(lo + i) = make_float4(v.x - h.x, v.y - h.y, v.z - h.z, v.w - h.w);
}

// HBM / L2-bound: 4 B read and 8 B (TF32: 4) written per value and form.  A block takes a tile that both forms want in
// runs of whole sectors and turns it in shared memory.
__global__ void __launch_bounds__(256)
weight_stage_batch_kernel(const WeightJob* __restrict__ jobs, int n_jobs, unsigned block_offset) {
  NRS_PDL_PROLOGUE();
  constexpr int kPitch = kConvCi * kConvTaps + 1;
  __shared__ float tile[kConvCo * kPitch > kTile * (kTile + 1) ? kConvCo * kPitch : kTile * (kTile + 1)];
  // the job this block belongs to: the last one whose first_block <= its index in the full launch
  const unsigned bid = blockIdx.x + block_offset;
  int lo_j = 0, hi_j = n_jobs - 1;
  while (lo_j < hi_j) {
    const int mid = (lo_j + hi_j + 1) >> 1;
    if (jobs[mid].first_block <= bid) lo_j = mid; else hi_j = mid - 1;
  }
  const WeightJob j = jobs[lo_j];
  const int blk = (int)(bid - j.first_block);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!j.conv) {
    const int tiles_c = ceil_div(j.cols, kTile);
    const int r0 = blk / tiles_c * kTile, c0 = (blk % tiles_c) * kTile;
    const int ld_b = ceil32(j.cols), ld_a = ceil32(j.rows);
    const int cq = (threadIdx.x & 15) * 4, c = c0 + cq;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = (threadIdx.x >> 4) + 16 * i, r = r0 + rr;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r < j.rows) {
        const float* s = j.src + (size_t)r * j.cols + c;
        if (j.vec && c < j.cols) v = *reinterpret_cast<const float4*>(s);
        else if (!j.vec) v = make_float4(c < j.cols ? s[0] : 0.f, c + 1 < j.cols ? s[1] : 0.f, c + 2 < j.cols ? s[2] : 0.f, c + 3 < j.cols ? s[3] : 0.f);
        if (j.b_hi && c < ld_b) put4(j.b_hi, j.b_lo, (size_t)r * ld_b + c, v);
      }
      float* t = tile + rr * (kTile + 1) + cq;
      t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w;
    }
    if (!j.a_hi) return;
    __syncthreads();
    const int kq = (lane & 7) * 4;   // 8 quads of rows x 4 columns per warp: no bank is asked twice
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = kq + 32 * (i & 1), cc = warp * 4 + (lane >> 3) + 32 * (i >> 1);
      if (c0 + cc >= j.cols || r0 + rr >= ld_a) continue;
      const float* t = tile + rr * (kTile + 1) + cc;
      put4(j.a_hi, j.a_lo, (size_t)(c0 + cc) * ld_a + r0 + rr, make_float4(t[0], t[kTile + 1], t[2 * (kTile + 1)], t[3 * (kTile + 1)]));
    }
    return;
  }
  const int tiles_i = ceil_div(j.cols, kConvCi), tiles_o = ceil32(j.rows) / kConvCo;
  const int ci0 = blk % tiles_i * kConvCi, co0 = blk / tiles_i % tiles_o * kConvCo, t0 = blk / tiles_i / tiles_o * kConvTaps;
  const int nt = min(kConvTaps, j.taps - t0), nci = min(kConvCi, j.cols - ci0), nco = min(kConvCo, j.rows - co0);
  // tile[co][ci * nt + tap], zeros beyond the channels; nearly always nt == taps, and a row of it is one run of memory
#pragma unroll
  for (int oo = 0; oo < kConvCo / 8; ++oo) {
    const int o = warp + 8 * oo;
    const float* s = j.src + ((size_t)(co0 + o) * j.cols + ci0) * j.taps + t0;
    float* t = tile + o * kPitch;
#pragma unroll
    for (int u = 0; u < kConvTaps; ++u) {   // kConvCi values a step, so that all loads of a row are under way together
      const int e = lane + 32 * u;
      if (u >= nt) break;
      if (nt == j.taps) {
        t[e] = o < nco && e < nci * nt ? s[e] : 0.0f;
      } else {
        const int ci = e / nt;
        t[e] = o < nco && ci < nci ? s[(size_t)ci * j.taps + (e - ci * nt)] : 0.0f;
      }
    }
  }
  __syncthreads();
  if (j.a_hi) {
    const int ld = ceil32(j.cols);
    for (int o = warp; o < nco; o += 8)
#pragma unroll
      for (int t = 0; t < kConvTaps; ++t)
        if (t < nt) put(j.a_hi, j.a_lo, ((size_t)(co0 + o) * j.taps + t0 + t) * ld + ci0 + lane, tile[o * kPitch + lane * nt + t]);
  }
  if (j.b_hi) {
    const int ld = ceil32(j.rows), o = lane & 15;
    for (int i = warp; i < nci; i += 8)
#pragma unroll
      for (int t2 = 0; t2 < kConvTaps; t2 += 2) {   // the two halves of a warp take neighbouring taps
        const int t = t2 + (lane >> 4);
        if (t < nt) put(j.b_hi, j.b_lo, ((size_t)(ci0 + i) * j.taps + t0 + t) * ld + co0 + o, tile[o * kPitch + i * nt + t]);
      }
  }
}

size_t plane_floats(const NrsWeightDesc& d) {
  if (d.form == NRS_WF_LINEAR_ROWS || d.form == NRS_WF_LINEAR_T) return (size_t)d.rows * ceil32(d.K);
  return d.form == NRS_WF_CONV_FWD ? (size_t)d.co * ceil32(d.ci) * d.taps : (size_t)d.ci * ceil32(d.co) * d.taps;
}

}  // namespace

void nrs_weight_set_clear(nrs_ctx* ctx) {
  NrsWeightSet& ws = ctx->weight_set;
  if (ws.storage || ws.jobs_dev) cudaStreamSynchronize(ctx->stream);
  if (ws.storage) cudaFree(ws.storage);
  if (ws.jobs_dev) cudaFree(ws.jobs_dev);
  ws = NrsWeightSet();
}

int nrs_weight_set_build(nrs_ctx* ctx, const NrsWeightDesc* descs, int count) {
  nrs_weight_set_clear(ctx);
  if (count <= 0 || ctx->math_mode == NRS_MATH_FP32) return NRS_OK;
  NrsWeightSet& ws = ctx->weight_set;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  size_t total = 0;
  for (int i = 0; i < count; ++i) total += (plane_floats(descs[i]) + 63) / 64 * 64 * (split ? 2 : 1);
  const int got = nrs_device_alloc(ctx, "weight planes", total * sizeof(float), &ws.storage);
  if (got != NRS_OK) return got;
  std::vector<WeightJob> jobs;
  float* cursor = (float*)ws.storage;
  for (int i = 0; i < count; ++i) {
    const NrsWeightDesc& d = descs[i];
    const size_t n = (plane_floats(d) + 63) / 64 * 64;
    float* hi = cursor;
    cursor += n;
    float* lo = split ? cursor : nullptr;
    if (split) cursor += n;
    const bool conv = d.form == NRS_WF_CONV_FWD || d.form == NRS_WF_CONV_DGRAD, a = d.form == NRS_WF_CONV_FWD || d.form == NRS_WF_LINEAR_T;
    const int rows = conv ? d.co : a ? d.K : d.rows, cols = conv ? d.ci : a ? d.rows : d.K, taps = conv ? d.taps : 1;
    // the other form of a weight already met joins its job
    WeightJob* job = nullptr;
    for (WeightJob& o : jobs)
      if (o.src == d.w && o.conv == (int)conv && o.rows == rows && o.cols == cols && o.taps == taps && !(a ? o.a_hi : o.b_hi)) job = &o;
    if (!job) {
      WeightJob j{};
      j.src = d.w;
      j.conv = conv;
      j.vec = cols % 4 == 0 && (reinterpret_cast<uintptr_t>(d.w) & 15) == 0;
      j.rows = rows; j.cols = cols; j.taps = taps;
      jobs.push_back(j);
      job = &jobs.back();
    }
    (a ? job->a_hi : job->b_hi) = hi;
    (a ? job->a_lo : job->b_lo) = lo;
    ws.planes[std::make_pair((const void*)d.w, d.form)] = NrsWeightPlanes{hi, lo, d.rows, d.K, d.co, d.ci, d.taps};
  }
  unsigned block = 0;
  for (WeightJob& j : jobs) {
    j.first_block = block;
    block += job_blocks(j);
    ws.job_src.push_back(j.src);
    ws.job_first.push_back(j.first_block);
  }
  cudaError_t e = cudaMalloc(&ws.jobs_dev, jobs.size() * sizeof(WeightJob));
  if (e == cudaSuccess) e = cudaMemcpyAsync(ws.jobs_dev, jobs.data(), jobs.size() * sizeof(WeightJob), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // `jobs` is a local
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    nrs_weight_set_clear(ctx);
    return nrs_fail(ctx, NRS_ERR_ALLOC, "weight planes: job table upload failed: %s", cudaGetErrorString(e));
  }
  ws.n_jobs = (int)jobs.size();
  ws.blocks = block;
  ws.job_first.push_back(block);
  ws.split = split;
  ws.fresh = false;
  return NRS_OK;
}

int nrs_weight_set_refresh(nrs_ctx* ctx) {
  NrsWeightSet& ws = ctx->weight_set;
  if (ws.n_jobs == 0) return NRS_OK;
  NRS_PDL_LAUNCH(weight_stage_batch_kernel, ws.blocks, 256, 0, ctx->stream, (const WeightJob*)ws.jobs_dev, ws.n_jobs, 0u);
  NRS_LAUNCHED(ctx);
  ws.fresh = true;
  ws.refreshed_jobs = 0;
  return NRS_OK;
}

int nrs_weight_set_refresh_range(nrs_ctx* ctx, const float* lo, const float* hi) {
  NrsWeightSet& ws = ctx->weight_set;
  // one launch per run of consecutive jobs whose weight lies in the range (jobs follow the layer order, so
  // a bucket of adjacent parameters is one run)
  int j = 0;
  while (j < ws.n_jobs) {
    if (ws.job_src[j] < lo || ws.job_src[j] >= hi) { ++j; continue; }
    int e = j;
    while (e < ws.n_jobs && ws.job_src[e] >= lo && ws.job_src[e] < hi) ++e;
    const unsigned first = ws.job_first[j], count = ws.job_first[e] - first;
    if (count > 0) {
      NRS_PDL_LAUNCH(weight_stage_batch_kernel, count, 256, 0, ctx->stream, (const WeightJob*)ws.jobs_dev, ws.n_jobs, first);
      NRS_LAUNCHED(ctx);
    }
    ws.refreshed_jobs += e - j;
    j = e;
  }
  return NRS_OK;
}
