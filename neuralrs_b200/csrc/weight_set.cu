// Batched staging of a model's weights for the tensor-core kernels.
//
// Every contraction reads its weight operand as K-major planes (values rounded to TF32 or, for 3xTF32,
// f16 pairs), re-laid out per use: convolution forward and data gradient
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
  // 3xTF32: the range its planes share with those of its group, and the blocks that measure it
  NrsRange* range;
  unsigned first_scan, group_scans;
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

template <bool SPLIT>
__device__ __forceinline__ void put(float* hi, float* lo, size_t i, float v, float scale) {
  if (SPLIT) pr::put(hi, lo, i, v, scale);
  else hi[i] = tc::tf32_rn(v);
}
template <bool SPLIT>
__device__ __forceinline__ void put4(float* hi, float* lo, size_t i, float4 v, float scale) {
  if (SPLIT) pr::put4(hi, lo, i, v, scale);
  else *reinterpret_cast<float4*>(hi + i) = make_float4(tc::tf32_rn(v.x), tc::tf32_rn(v.y), tc::tf32_rn(v.z), tc::tf32_rn(v.w));
}

constexpr int kScan = 4096;   // values per block
inline unsigned job_scans(const WeightJob& j) { return (unsigned)(((size_t)j.rows * j.cols * j.taps + kScan - 1) / kScan); }

// Both kernels last a few microseconds, most of it latency.  What a block works on is therefore one load away
// (`job_of_block`, made with the table; a binary search over the jobs is four loads, each waiting for the one before), is
// looked up before the wait for the kernel ahead (the tables never change), and all loads of a thread are under way
// before the first value is used.  Measured in a training step, scan and staging together: small CNN 16 -> 11 us, language
// model of 32 x 128 tokens 13 -> 8.

// The largest magnitude of every weight (group), for its planes' exponent.  L2-bound: the optimizer has just written them.
// A group's last block to arrive turns what all of them left in the range's scratch words into the range, and clears those.
__global__ void __launch_bounds__(256)
weight_scan_kernel(const WeightJob* __restrict__ jobs, const int* __restrict__ job_of_block, unsigned scan_offset) {
  __shared__ uint32_t part[8];
  const unsigned bid = blockIdx.x + scan_offset;
  const WeightJob j = jobs[job_of_block[bid]];
  NRS_PDL_PROLOGUE();
  const size_t count = (size_t)j.rows * j.cols * j.taps, begin = (size_t)(bid - j.first_scan) * kScan;
  const int n = (int)min((size_t)kScan, count - begin);
  const float* src = j.src + begin;
  uint32_t top = 0;
  if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
    float4 v[kScan / 1024];
#pragma unroll
    for (int u = 0; u < kScan / 1024; ++u) {
      const int i = 4 * (int)threadIdx.x + 1024 * u;
      v[u] = i + 3 < n ? *reinterpret_cast<const float4*>(src + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if ((n & 3) != 0 && threadIdx.x < (unsigned)(n & 3)) top = pr::seen(top, src[(n & ~3) + (int)threadIdx.x]);
#pragma unroll
    for (int u = 0; u < kScan / 1024; ++u) top = pr::seen4(top, v[u]);
  } else {
    for (int i = threadIdx.x; i < n; i += 256) top = pr::seen(top, src[i]);
  }
  top = __reduce_max_sync(0xffffffffu, top);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = top;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < 8; ++w) top = max(top, part[w]);
  unsigned* scratch = reinterpret_cast<unsigned*>(j.range->pad);   // largest so far; blocks that have arrived
  atomicMax(&scratch[0], top);
  __threadfence();
  if (atomicAdd(&scratch[1], 1u) + 1u != j.group_scans) return;
  __threadfence();
  const float bound = __uint_as_float(atomicExch(&scratch[0], 0u));
  scratch[1] = 0;
  j.range->bound = j.range->top = bound;
}

// HBM / L2-bound: 4 B read and 4 B written per value and form.  A block takes a tile that both forms want in
// runs of whole sectors and turns it in shared memory.
template <bool SPLIT>
__global__ void __launch_bounds__(256)
weight_stage_batch_kernel(const WeightJob* __restrict__ jobs, const int* __restrict__ job_of_block, unsigned block_offset) {
  constexpr int kPitch = kConvCi * kConvTaps + 1;
  __shared__ float tile[kConvCo * kPitch > kTile * (kTile + 1) ? kConvCo * kPitch : kTile * (kTile + 1)];
  const unsigned bid = blockIdx.x + block_offset;
  const WeightJob j = jobs[job_of_block[bid]];
  NRS_PDL_PROLOGUE();
  const float scale = SPLIT ? pr::scale_of(j.range->bound) : 1.0f;
  const int blk = (int)(bid - j.first_block);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (!j.conv) {
    const int tiles_c = ceil_div(j.cols, kTile);
    const int r0 = blk / tiles_c * kTile, c0 = (blk % tiles_c) * kTile;
    const int ld_b = ceil32(j.cols), ld_a = ceil32(j.rows);
    const int cq = (threadIdx.x & 15) * 4, c = c0 + cq;
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = r0 + (threadIdx.x >> 4) + 16 * i;
      const float* s = j.src + (size_t)r * j.cols + c;
      v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (r >= j.rows) continue;
      if (j.vec && c < j.cols) v[i] = *reinterpret_cast<const float4*>(s);
      else if (!j.vec) v[i] = make_float4(c < j.cols ? s[0] : 0.f, c + 1 < j.cols ? s[1] : 0.f, c + 2 < j.cols ? s[2] : 0.f, c + 3 < j.cols ? s[3] : 0.f);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = (threadIdx.x >> 4) + 16 * i, r = r0 + rr;
      if (j.b_hi && r < j.rows && c < ld_b) put4<SPLIT>(j.b_hi, j.b_lo, (size_t)r * ld_b + c, v[i], scale);
      float* t = tile + rr * (kTile + 1) + cq;
      t[0] = v[i].x; t[1] = v[i].y; t[2] = v[i].z; t[3] = v[i].w;
    }
    if (!j.a_hi) return;
    __syncthreads();
    const int kq = (lane & 7) * 4;   // 8 quads of rows x 4 columns per warp: no bank is asked twice
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = kq + 32 * (i & 1), cc = warp * 4 + (lane >> 3) + 32 * (i >> 1);
      if (c0 + cc >= j.cols || r0 + rr >= ld_a) continue;
      const float* t = tile + rr * (kTile + 1) + cc;
      put4<SPLIT>(j.a_hi, j.a_lo, (size_t)(c0 + cc) * ld_a + r0 + rr, make_float4(t[0], t[kTile + 1], t[2 * (kTile + 1)], t[3 * (kTile + 1)]), scale);
    }
    return;
  }
  const int tiles_i = ceil_div(j.cols, kConvCi), tiles_o = ceil32(j.rows) / kConvCo;
  const int ci0 = blk % tiles_i * kConvCi, co0 = blk / tiles_i % tiles_o * kConvCo, t0 = blk / tiles_i / tiles_o * kConvTaps;
  const int nt = min(kConvTaps, j.taps - t0), nci = min(kConvCi, j.cols - ci0), nco = min(kConvCo, j.rows - co0);
  // tile[co][ci * nt + tap], zeros beyond the channels; nearly always nt == taps, and a row of it is one run of memory
  float v[kConvCo / 8][kConvTaps];
#pragma unroll
  for (int oo = 0; oo < kConvCo / 8; ++oo) {
    const int o = warp + 8 * oo;
    const float* s = j.src + ((size_t)(co0 + o) * j.cols + ci0) * j.taps + t0;
#pragma unroll
    for (int u = 0; u < kConvTaps; ++u) {   // kConvCi values a step
      const int e = lane + 32 * u;
      v[oo][u] = 0.0f;
      if (u >= nt || o >= nco) continue;
      if (nt == j.taps) {
        if (e < nci * nt) v[oo][u] = s[e];
      } else {
        const int ci = e / nt;
        if (ci < nci) v[oo][u] = s[(size_t)ci * j.taps + (e - ci * nt)];
      }
    }
  }
#pragma unroll
  for (int oo = 0; oo < kConvCo / 8; ++oo)
#pragma unroll
    for (int u = 0; u < kConvTaps; ++u)
      if (u < nt) tile[(warp + 8 * oo) * kPitch + lane + 32 * u] = v[oo][u];
  __syncthreads();
  if (j.a_hi) {
    const int ld = ceil32(j.cols);
    for (int o = warp; o < nco; o += 8)
#pragma unroll
      for (int t = 0; t < kConvTaps; ++t)
        if (t < nt) put<SPLIT>(j.a_hi, j.a_lo, ((size_t)(co0 + o) * j.taps + t0 + t) * ld + ci0 + lane, tile[o * kPitch + lane * nt + t], scale);
  }
  if (j.b_hi) {
    const int ld = ceil32(j.rows), o = lane & 15;
    for (int i = warp; i < nci; i += 8)
#pragma unroll
      for (int t2 = 0; t2 < kConvTaps; t2 += 2) {   // the two halves of a warp take neighbouring taps
        const int t = t2 + (lane >> 4);
        if (t < nt) put<SPLIT>(j.b_hi, j.b_lo, ((size_t)(ci0 + i) * j.taps + t0 + t) * ld + co0 + o, tile[o * kPitch + i * nt + t], scale);
      }
  }
}

size_t plane_values(const NrsWeightDesc& d) {
  if (d.form == NRS_WF_LINEAR_ROWS || d.form == NRS_WF_LINEAR_T) return (size_t)d.rows * ceil32(d.K);
  return d.form == NRS_WF_CONV_FWD ? (size_t)d.co * ceil32(d.ci) * d.taps : (size_t)d.ci * ceil32(d.co) * d.taps;
}

}  // namespace

void nrs_weight_set_clear(nrs_ctx* ctx) {
  NrsWeightSet& ws = ctx->weight_set;
  if (ws.storage || ws.jobs_dev) cudaStreamSynchronize(ctx->stream);
  if (ws.storage) cudaFree(ws.storage);
  if (ws.jobs_dev) cudaFree(ws.jobs_dev);
  if (ws.ranges) nrs_free(ctx, ws.ranges);
  ws = NrsWeightSet();
}

int nrs_weight_set_build(nrs_ctx* ctx, const NrsWeightDesc* descs, int count) {
  nrs_weight_set_clear(ctx);
  if (count <= 0 || ctx->math_mode == NRS_MATH_FP32) return NRS_OK;
  NrsWeightSet& ws = ctx->weight_set;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  size_t total = 0;
  for (int i = 0; i < count; ++i) total += (plane_values(descs[i]) + 63) / 64 * 64 * sizeof(float);
  int got = nrs_device_alloc(ctx, "weight planes", total, &ws.storage);
  if (got == NRS_OK && split) got = nrs_alloc(ctx, count * sizeof(NrsRange), 1, (void**)&ws.ranges);   // (one per job at most)
  if (got != NRS_OK) return got;
  std::vector<WeightJob> jobs;
  std::vector<int> groups;   // per job
  uint8_t* cursor = (uint8_t*)ws.storage;
  for (int i = 0; i < count; ++i) {
    const NrsWeightDesc& d = descs[i];
    const size_t n = (plane_values(d) + 63) / 64 * 64;
    float* hi = (float*)cursor;
    cursor += n * (split ? 2 : 4);
    float* lo = split ? (float*)cursor : nullptr;
    if (split) cursor += n * 2;
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
      j.range = ws.ranges;
      if (split && !jobs.empty()) j.range = jobs.back().range + (d.group != 0 && d.group == groups.back() ? 0 : 1);
      groups.push_back(d.group);
      jobs.push_back(j);
      job = &jobs.back();
    }
    (a ? job->a_hi : job->b_hi) = hi;
    (a ? job->a_lo : job->b_lo) = lo;
    ws.planes[std::make_pair((const void*)d.w, d.form)] = NrsWeightPlanes{hi, lo, job->range, d.rows, d.K, d.co, d.ci, d.taps};
  }
  unsigned block = 0, scan = 0;
  for (size_t i = 0, e; i < jobs.size(); i = e) {
    unsigned total_scans = 0;
    for (e = i; e < jobs.size() && (e == i || (split && jobs[e].range == jobs[i].range)); ++e) total_scans += job_scans(jobs[e]);
    for (size_t k = i; k < e; ++k) { jobs[k].group_scans = total_scans; ws.job_group.push_back((int)i); }
  }
  for (WeightJob& j : jobs) {
    j.first_block = block;
    j.first_scan = scan;
    block += job_blocks(j);
    scan += job_scans(j);
    ws.job_scan.push_back(j.first_scan);
    ws.job_src.push_back(j.src);
    ws.job_first.push_back(j.first_block);
  }
  std::vector<int> job_of_block, job_of_scan;
  for (size_t i = 0; i < jobs.size(); ++i) {
    job_of_block.insert(job_of_block.end(), job_blocks(jobs[i]), (int)i);
    job_of_scan.insert(job_of_scan.end(), job_scans(jobs[i]), (int)i);
  }
  const size_t jobs_bytes = jobs.size() * sizeof(WeightJob);
  cudaError_t e = cudaMalloc(&ws.jobs_dev, jobs_bytes + (block + scan) * sizeof(int));
  if (e == cudaSuccess) e = cudaMemcpyAsync(ws.jobs_dev, jobs.data(), jobs_bytes, cudaMemcpyHostToDevice, ctx->stream);
  int* maps = (int*)((uint8_t*)ws.jobs_dev + jobs_bytes);
  if (e == cudaSuccess) e = cudaMemcpyAsync(maps, job_of_block.data(), block * sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(maps + block, job_of_scan.data(), scan * sizeof(int), cudaMemcpyHostToDevice, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);   // the sources are locals
  if (e != cudaSuccess) {
    (void)cudaGetLastError();
    nrs_weight_set_clear(ctx);
    return nrs_fail(ctx, NRS_ERR_ALLOC, "weight planes: job table upload failed: %s", cudaGetErrorString(e));
  }
  ws.n_jobs = (int)jobs.size();
  ws.blocks = block;
  ws.job_first.push_back(block);
  ws.job_scan.push_back(scan);
  ws.job_group.push_back((int)jobs.size());
  ws.split = split;
  ws.fresh = false;
  return NRS_OK;
}

// Jobs [first, last), whole groups.
static int refresh_jobs(nrs_ctx* ctx, int first, int last) {
  NrsWeightSet& ws = ctx->weight_set;
  const unsigned block = ws.job_first[first], blocks = ws.job_first[last] - block, scan = ws.job_scan[first], scans = ws.job_scan[last] - scan;
  if (blocks == 0) return NRS_OK;
  const WeightJob* jobs = (const WeightJob*)ws.jobs_dev;
  const int* job_of_block = (const int*)(jobs + ws.n_jobs);
  if (ws.split) {
    NRS_PDL_LAUNCH(weight_scan_kernel, scans, 256, 0, ctx->stream, jobs, job_of_block + ws.job_first[ws.n_jobs], scan);
    NRS_LAUNCHED(ctx);
    NRS_PDL_LAUNCH((weight_stage_batch_kernel<true>), blocks, 256, 0, ctx->stream, jobs, job_of_block, block);
  } else {
    NRS_PDL_LAUNCH((weight_stage_batch_kernel<false>), blocks, 256, 0, ctx->stream, jobs, job_of_block, block);
  }
  NRS_LAUNCHED(ctx);
  return NRS_OK;
}

int nrs_weight_set_refresh(nrs_ctx* ctx) {
  NrsWeightSet& ws = ctx->weight_set;
  if (ws.n_jobs == 0) return NRS_OK;
  const int st = refresh_jobs(ctx, 0, ws.n_jobs);
  if (st != NRS_OK) return st;
  ws.fresh = true;
  ws.refreshed_jobs = 0;
  return NRS_OK;
}

int nrs_weight_set_refresh_range(nrs_ctx* ctx, const float* lo, const float* hi) {
  NrsWeightSet& ws = ctx->weight_set;
  // one launch per run of consecutive jobs whose weight lies in the range (jobs follow the layer order, so
  // a bucket of adjacent parameters is one run); what shares its range with one of them is restaged too
  int j = 0;
  while (j < ws.n_jobs) {
    if (ws.job_src[j] < lo || ws.job_src[j] >= hi) { ++j; continue; }
    int e = j;
    while (e < ws.n_jobs && ws.job_src[e] >= lo && ws.job_src[e] < hi) ++e;
    int first = ws.job_group[j], last = e;
    while (last < ws.n_jobs && ws.job_group[last] == ws.job_group[e - 1]) ++last;
    const int st = refresh_jobs(ctx, first, last);
    if (st != NRS_OK) return st;
    ws.refreshed_jobs += e - j;
    j = e;
  }
  return NRS_OK;
}
