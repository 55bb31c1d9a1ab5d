// Transformer-side operators of the graph layer: embedding, positional encoding,
// batched attention, multi-head attention, the post-LN transformer block.
// They are written the way the reference writes them — compositions of the
// resident graph ops (src/cuda/nn/attention.rs:23-32, multihead.rs:57-85,
// transformer_block.rs:28-60) — plus the embedding gather/scatter kernels and
// the causal mask, which need their own backward closures.
#include <cmath>
#include <cstring>

#include "attention_planes.h"
#include "fold.h"
#include "host/graph.h"

namespace nrs {
namespace cuda {

static void fail(int code, const std::string& m) { throw Error(code, m); }

NodeP causal_mask(const NodeP& scores) {
  if (!scores || !scores->on_gpu()) fail(NRS_ERR_ARG, "cuda causal_mask: input not on GPU");
  const size_t nd = scores->shape.size();
  if (nd < 2 || scores->shape[nd - 1] != scores->shape[nd - 2]) fail(NRS_ERR_SHAPE, "cuda causal_mask: last two dims must be equal");
  nrs_ctx* ctx = scores->ctx;
  const int s = (int)scores->shape[nd - 1];
  const int batch = (int)(scores->len() / ((size_t)s * s));
  NodeP out = make_result(ctx, scores->shape, {scores});
  check(ctx, nrs_causal_mask(ctx, scores->data, out->data, batch, s, 0, 0));
  Node* self = out.get();
  out->backward_fn = [self, scores, batch, s]() {
    if (!scores->requires_grad) return;
    const float* g = grad_view(self);
    GradSlot t = grad_slot(scores);
    check(self->ctx, nrs_causal_mask(self->ctx, g, t.ptr, batch, s, 1, t.accumulate));
  };
  return out;
}

// softmax(q k^T / sqrt(d_head)) v for every head of [batch, seq, heads*d_head] tensors in one kernel
// (shapes inside nrs_attention_supported only).
static NodeP fused_attention(const NodeP& q, const NodeP& k, const NodeP& v, size_t heads, bool causal) {
  nrs_ctx* ctx = q->ctx;
  const size_t batch = q->shape[0], seq = q->shape[1], d = q->shape[2], d_head = d / heads;
  if (k->shape != q->shape || v->shape != q->shape) fail(NRS_ERR_SHAPE, "cuda attention: q, k, v shapes differ");
  NodeP out = make_result(ctx, q->shape, {q, k, v});
  void* probs = nullptr;
  check(ctx, nrs_alloc(ctx, std::max<size_t>(1, batch * heads * seq * seq) * sizeof(float), 0, &probs));
  out->saved.push_back(probs);
  check(ctx, nrs_attention_fwd(ctx, q->data, k->data, v->data, out->data, (float*)probs, (int)batch, (int)seq, (int)heads,
                               (int)d_head, causal ? 1 : 0));
  Node* self = out.get();
  out->backward_fn = [self, q, k, v, probs, batch, seq, heads, d_head]() {
    nrs_ctx* ctx = self->ctx;
    const float* g = grad_view(self);
    // a tensor that needs no gradient still gets a scratch target: the kernel computes all three
    const size_t len = self->len();
    auto target = [&](const NodeP& n, float** scratch) {
      if (n->requires_grad) return grad_slot(n);
      void* p = nullptr;
      check(ctx, nrs_alloc(ctx, std::max<size_t>(1, len) * sizeof(float), 0, &p));
      *scratch = (float*)p;
      return GradSlot{(float*)p, 0};
    };
    float *sq = nullptr, *sk = nullptr, *sv = nullptr;
    GradSlot tq = target(q, &sq), tk = target(k, &sk), tv = target(v, &sv);
    check(ctx, nrs_attention_bwd(ctx, q->data, k->data, v->data, (const float*)probs, g, tq.ptr, tk.ptr, tv.ptr, (int)batch,
                                 (int)seq, (int)heads, (int)d_head, tq.accumulate, tk.accumulate, tv.accumulate));
    for (float* s : {sq, sk, sv})
      if (s) nrs_free(ctx, s);
  };
  return out;
}

NodeP attention_batch(const NodeP& q, const NodeP& k, const NodeP& v, bool causal) {
  if (!q || q->shape.size() != 3) fail(NRS_ERR_SHAPE, "cuda attention_batch: q must be [batch, seq, d_head]");
  if (k && v && k->on_gpu() && v->on_gpu() && q->on_gpu() && nrs_attention_supported((int)q->shape[1], (int)q->shape[2]))
    return fused_attention(q, k, v, 1, causal);
  const float scale_factor = 1.0f / std::sqrt((float)q->shape[2]);
  NodeP scores = scale(bmm(q, transpose(k)), scale_factor);
  if (causal) scores = causal_mask(scores);
  return bmm(softmax(scores), v);
}

NodeP Linear::forward(const NodeP& x) const { return add(matmul(x, weights), bias); }

NodeP LayerNorm::forward(const NodeP& x) const { return layernorm(x, gamma, beta, eps); }

// Gather (+ positional table) from indices already on the device; the node does not own `idx_dev`.
static NodeP embed_resident(const Embedding& e, const int32_t* idx_dev, size_t count, const std::vector<size_t>& out_shape,
                            const NodeP& pos_table, size_t seq) {
  nrs_ctx* ctx = e.weight->ctx;
  const int dim = (int)e.embedding_dim, vocab = (int)e.vocab_size;
  NodeP out = make_result(ctx, out_shape, {e.weight});
  check(ctx, nrs_embedding_pos_fwd(ctx, e.weight->data, idx_dev, pos_table ? pos_table->data : nullptr, out->data, (int)count,
                                   (int)seq, dim, vocab));
  Node* self = out.get();
  const NodeP w = e.weight;
  out->backward_fn = [self, w, idx_dev, count, dim, vocab]() {
    if (!w->requires_grad) return;
    const float* g = grad_view(self);
    GradSlot t = grad_slot(w);
    check(self->ctx, nrs_embedding_bwd(self->ctx, g, idx_dev, t.ptr, (int)count, dim, vocab, t.accumulate));
  };
  return out;
}

static NodeP embed(const Embedding& e, const int32_t* indices, size_t count, const std::vector<size_t>& out_shape) {
  if (!e.weight || !e.weight->on_gpu()) fail(NRS_ERR_ARG, "cuda embedding: weight not on GPU");
  if (!indices && count) fail(NRS_ERR_ARG, "cuda embedding: null indices");
  for (size_t i = 0; i < count; ++i)
    if (indices[i] < 0 || (size_t)indices[i] >= e.vocab_size) fail(NRS_ERR_ARG, "embedding: token index out of vocab range");
  nrs_ctx* ctx = e.weight->ctx;
  void* idx_dev = nullptr;
  check(ctx, nrs_alloc(ctx, (count ? count : 1) * sizeof(int32_t), 0, &idx_dev));
  NodeP out;
  try {
    check(ctx, nrs_h2d(ctx, idx_dev, indices, count * sizeof(int32_t)));
    check(ctx, nrs_sync(ctx));  // the caller's index buffer may go away
    out = embed_resident(e, (const int32_t*)idx_dev, count, out_shape, nullptr, 1);
  } catch (...) {
    nrs_free(ctx, idx_dev);
    throw;
  }
  out->saved.push_back(idx_dev);
  return out;
}

NodeP Embedding::forward_resident(const int32_t* idx_dev, size_t batch, size_t seq, const NodeP& pos_table) const {
  if (!weight || !weight->on_gpu()) fail(NRS_ERR_ARG, "cuda embedding: weight not on GPU");
  if (!idx_dev && batch * seq) fail(NRS_ERR_ARG, "cuda embedding: null indices");
  if (pos_table) {
    if (!pos_table->on_gpu() || pos_table->shape.size() != 2 || pos_table->shape[1] != embedding_dim)
      fail(NRS_ERR_SHAPE, "cuda embedding: positional table must be a resident [max_len, dim] tensor");
    if (seq > pos_table->shape[0]) fail(NRS_ERR_SHAPE, "sequence longer than max_len");
  }
  return embed_resident(*this, idx_dev, batch * seq, {batch, seq, embedding_dim}, pos_table, seq);
}

NodeP Embedding::forward(const int32_t* indices, size_t count) const {
  return embed(*this, indices, count, {count, embedding_dim});
}

NodeP Embedding::forward_batch(const int32_t* indices, size_t batch, size_t seq) const {
  return embed(*this, indices, batch * seq, {batch, seq, embedding_dim});
}

PositionalEncoding PositionalEncoding::make(nrs_ctx* ctx, size_t d_model, size_t max_len) {
  // The table is computed on the host in f32 exactly as the reference does
  // (src/cuda/nn/positional.rs:24-33), once, and stays resident.
  std::vector<float> pe(max_len * d_model);
  for (size_t pos = 0; pos < max_len; ++pos)
    for (size_t i = 0; i < d_model; ++i) {
      const float exponent = (float)(2 * (i / 2)) / (float)d_model;
      const float freq = 1.0f / std::pow(10000.0f, exponent);
      const float angle = (float)pos * freq;
      pe[pos * d_model + i] = (i % 2 == 0) ? std::sin(angle) : std::cos(angle);
    }
  PositionalEncoding p;
  p.d_model = d_model;
  p.max_len = max_len;
  p.table = node_new(ctx, pe.data(), {max_len, d_model});
  p.table->requires_grad = false;
  to_cuda(p.table);
  synchronize(ctx);
  return p;
}

NodeP PositionalEncoding::forward(const NodeP& x) const {
  if (!x || !x->on_gpu()) fail(NRS_ERR_ARG, "cuda positional: input not on GPU");
  const size_t nd = x->shape.size();
  if (nd != 2 && nd != 3) fail(NRS_ERR_SHAPE, "cuda positional: input must be [seq, d] or [batch, seq, d]");
  const size_t seq = x->shape[nd - 2], d = x->shape[nd - 1];
  if (d != d_model) fail(NRS_ERR_SHAPE, "cuda positional: feature size differs from d_model");
  if (seq > max_len) fail(NRS_ERR_SHAPE, "sequence longer than max_len");
  nrs_ctx* ctx = x->ctx;
  const size_t batch = nd == 3 ? x->shape[0] : 1;
  // out[b, i] = x[b, i] + pe[i] over the first seq*d entries of the table: a row-broadcast add.
  NodeP out = make_result(ctx, x->shape, {x});
  check(ctx, nrs_bias_add(ctx, x->data, table->data, out->data, (int)batch, (int)(seq * d)));
  Node* self = out.get();
  const size_t len = x->len();
  out->backward_fn = [self, x, len]() {
    if (!x->requires_grad) return;
    const float* g = grad_view(self);
    GradSlot t = grad_slot(x);
    if (t.accumulate) check(self->ctx, nrs_accumulate(self->ctx, t.ptr, g, len));
    else check(self->ctx, nrs_d2d(self->ctx, t.ptr, g, len * sizeof(float)));
  };
  return out;
}

// [batch, seq, heads*d_head] <-> [batch*heads, seq, d_head]; the backward pass is the opposite permutation.
static NodeP permute_heads(const NodeP& x, size_t batch, size_t seq, size_t heads, size_t d_head, bool to_heads) {
  nrs_ctx* ctx = x->ctx;
  NodeP out = make_result(ctx, to_heads ? std::vector<size_t>{batch * heads, seq, d_head}
                                        : std::vector<size_t>{batch, seq, heads * d_head}, {x});
  check(ctx, nrs_permute_heads(ctx, x->data, out->data, (int)batch, (int)seq, (int)heads, (int)d_head, to_heads ? 1 : 0, 0));
  Node* self = out.get();
  out->backward_fn = [self, x, batch, seq, heads, d_head, to_heads]() {
    if (!x->requires_grad) return;
    const float* g = grad_view(self);
    GradSlot t = grad_slot(x);
    check(self->ctx, nrs_permute_heads(self->ctx, g, t.ptr, (int)batch, (int)seq, (int)heads, (int)d_head, to_heads ? 0 : 1,
                                       t.accumulate));
  };
  return out;
}

// Projections and attention core over operand planes (attention_planes.cu) as one node: x [tokens, d] -> [tokens, d], the
// heads' results side by side.  One product makes Q, K and V, one sums the three shares of x's gradient, one makes the
// three weight gradients.
static NodeP planes_attention(const MultiHeadAttention& m, const NodeP& x, size_t batch, size_t seq) {
  nrs_ctx* ctx = x->ctx;
  const size_t tokens = batch * seq, d = m.d_model, heads = m.num_heads, d_head = d / heads;
  const bool split = ctx->math_mode == NRS_MATH_3XTF32;
  const NodeP wq = m.w_q, wk = m.w_k, wv = m.w_v;
  NodeP out = make_result(ctx, {tokens, d}, {x, wq, wk, wv});
  auto block = [ctx](size_t floats) {
    void* p = nullptr;
    check(ctx, nrs_alloc(ctx, floats * sizeof(float), 0, &p));
    return (float*)p;
  };
  auto plane = [block, split](size_t values) { return block(split ? (values + 1) / 2 : values); };
  auto saved_plane = [&](size_t values) {
    float* p = plane(values);
    out->saved.push_back(p);
    return p;
  };
  cache_row_planes(x, tokens, d);   // read again by the weight gradients
  NrsGemmExtras e;
  e.skip_c = true;
  e.hi = saved_plane(tokens * 3 * d);
  e.lo = split ? saved_plane(tokens * 3 * d) : nullptr;
  const float* w[3] = {wq->data, wk->data, wv->data};
  check(ctx, nrs_tc_gemm_weights(ctx, 0, 3, (int)tokens, (int)d, (int)d, x->data, w, nullptr, 0.0f, &e));
  const size_t square = batch * heads * seq * (size_t)nrs_plane_ld((int)seq);
  NrsMhaPlanes a{};
  a.batch = (int)batch; a.seq = (int)seq; a.heads = (int)heads; a.d_head = (int)d_head; a.causal = m.causal ? 1 : 0;
  a.qkv_hi = e.hi; a.qkv_lo = e.lo; a.qkv_ld = (int)(3 * d);
  a.p_hi = saved_plane(square);
  a.p_lo = split ? saved_plane(square) : nullptr;
  out->internal = true;
  out->planes_only = values_as_planes_only(ctx, tokens, d, d);   // read by the output projection alone
  a.out = out->planes_only ? nullptr : out->data;
  a.out_hi = plane(tokens * d);
  a.out_lo = split ? plane(tokens * d) : nullptr;
  out->planes_hi = a.out_hi;        // the output projection reads them (and its weight gradient)
  out->planes_lo = a.out_lo;
  NrsPlanes pl{a.out_hi, a.out_lo, split ? 1 : 0};
  pl.rows = (int)tokens;
  pl.cols = (int)d;
  ctx->plane_hints[out->data] = pl;
  a.scores = block(square);
  const int st = nrs_mha_planes_fwd(ctx, a);
  nrs_free(ctx, a.scores);
  check(ctx, st);
  out->row_planes_wanted = true;
  Node* self = out.get();
  out->backward_fn = [self, x, wq, wk, wv, a, tokens, d, square, split, block, plane]() mutable {
    nrs_ctx* ctx = self->ctx;
    struct Mode {   // the saved planes are those of the forward pass's mode
      nrs_ctx* c; const int was;
      Mode(nrs_ctx* c_, int m) : c(c_), was(c_->math_mode) { c->math_mode = m; }
      ~Mode() { c->math_mode = was; }
    } mode{ctx, split ? NRS_MATH_3XTF32 : NRS_MATH_TF32};
    const float* g = grad_view(self);
    // the gradient's row planes: left by the output projection's input-gradient kernel, else staged here (also where that
    // kernel ran in another mode than the forward pass: the f32 values that f16 pairs stand for may not have been written)
    float *ghi = self->gplanes_hi, *glo = self->gplanes_lo;
    if (ghi) {
      ctx->plane_hints.erase(g);
      self->gplanes_hi = self->gplanes_lo = nullptr;
    }
    if (ghi && split != (glo != nullptr)) {
      if (glo) check(ctx, nrs_pair_unpack(ctx, ghi, glo, const_cast<float*>(g), tokens * d));
      nrs_free(ctx, ghi);
      if (glo) nrs_free(ctx, glo);
      ghi = glo = nullptr;
    }
    if (!ghi) {
      ghi = plane(tokens * d);
      if (split) glo = plane(tokens * d);
      check(ctx, nrs_tc_stage(ctx, g, ghi, glo, (int)tokens, (int)d, (int)d, 1, 0, 0, false));
    }
    a.dout_hi = ghi; a.dout_lo = split ? glo : nullptr;
    a.scores = block(square);
    a.ds_hi = plane(square);
    a.ds_lo = split ? plane(square) : nullptr;
    a.dqkv_hi = plane(tokens * 3 * d);
    a.dqkv_lo = split ? plane(tokens * 3 * d) : nullptr;
    struct Release {   // (the weight gradient may wait: it reads dqkv, and nothing else of these)
      nrs_ctx* c; std::vector<float*> now, later; const float* key;
      void free_now() {
        for (float* q : now) if (q) nrs_free(c, q);
        now.clear();
      }
      ~Release() {
        if (key) c->plane_hints.erase(key);
        free_now();
        for (float* q : later) if (q) nrs_free_after_wgrads(c, q);
      }
    } release{ctx, {ghi, glo, a.scores, a.ds_hi, a.ds_lo}, {a.dqkv_hi, a.dqkv_lo}, nullptr};
    check(ctx, nrs_mha_planes_bwd(ctx, a));
    release.free_now();
    NrsPlanes pl{a.dqkv_hi, a.dqkv_lo, split ? 1 : 0};
    pl.rows = (int)tokens;
    pl.cols = (int)(3 * d);
    ctx->plane_hints[a.dqkv_hi] = pl;
    release.key = a.dqkv_hi;
    if (x->requires_grad) {
      GradSlot t = grad_slot(x);
      const float* w[3] = {wq->data, wk->data, wv->data};
      NrsGemmExtras e;
      TopP top = new_top(ctx);   // (the layer below makes planes of the sum)
      if (top) e.range = top->range;
      check(ctx, nrs_tc_gemm_weights(ctx, 1, 3, (int)tokens, (int)d, (int)d, a.dqkv_hi, w, t.ptr, t.accumulate ? 1.0f : 0.0f, &e));
      set_grad_top(x, std::move(top));
    }
    GradSlot s[3] = {grad_slot(wq), grad_slot(wk), grad_slot(wv)};
    const size_t dd = d * d;
    const bool side_by_side = s[1].ptr == s[0].ptr + dd && s[2].ptr == s[0].ptr + 2 * dd && s[0].accumulate == s[1].accumulate &&
                              s[0].accumulate == s[2].accumulate;   // a trainer's flat block: one write for all three
    float* dst = side_by_side ? s[0].ptr : block(3 * dd);
    NrsIndependentNext overlap(ctx, x->requires_grad);   // reads nothing that dX wrote
    check(ctx, nrs_tc_conv_wgrad(ctx, a.dqkv_hi, x->data, dst, (int)tokens, (int)(3 * d), 1, 1, (int)d, 1, 1, 1, 0,
                                 side_by_side ? s[0].accumulate : 0, (int)d));
    if (!side_by_side) {
      release.now.push_back(dst);
      check(ctx, nrs_folds_flush(ctx));
      for (int i = 0; i < 3; ++i)
        check(ctx, s[i].accumulate ? nrs_accumulate(ctx, s[i].ptr, dst + i * dd, dd)
                                   : nrs_d2d(ctx, s[i].ptr, dst + i * dd, dd * sizeof(float)));
    }
  };
  return out;
}

// Which form attention takes in a TF32 mode.  (The kernels of attention_tc.cu stay for nrs_attention_fwd / _bwd, whose
// callers hold q, k, v as separate f32 tensors.)
static bool planes_attention_applies(const MultiHeadAttention& m, const NodeP& x, size_t batch, size_t seq) {
  const size_t d = m.d_model, tokens = batch * seq;
  if (!operand_planes_possible(x->ctx) || d % 32 != 0 || tokens < 16 || tokens > 2147483647u / 3 / d) return false;
  for (const NodeP& w : {m.w_q, m.w_k, m.w_v})
    if (!w || !w->on_gpu() || !w->requires_grad || w->view_of || w->shape.size() != 2 || w->shape[0] != d || w->shape[1] != d) return false;
  return nrs_mha_planes_applies(x->ctx, (int)seq, (int)(d / m.num_heads));
}

NodeP MultiHeadAttention::forward_batch(const NodeP& x) const {
  if (!x || x->shape.size() != 3) fail(NRS_ERR_SHAPE, "cuda mha: input must be [batch, seq, d_model]");
  const size_t batch = x->shape[0], seq = x->shape[1], d = x->shape[2];
  if (d != d_model || num_heads == 0 || d_model % num_heads != 0) fail(NRS_ERR_SHAPE, "cuda mha: d_model / num_heads mismatch");
  if (x->on_gpu() && planes_attention_applies(*this, x, batch, seq)) {
    NodeP flat = reshape(x, {batch * seq, d});
    return reshape(matmul(planes_attention(*this, flat, batch, seq), w_o), {batch, seq, d});
  }
  auto proj = [&](const NodeP& w) { return reshape(matmul(reshape(x, {batch * seq, d}), w), {batch, seq, d}); };
  NodeP q = proj(w_q), k = proj(w_k), v = proj(w_v);
  // The reference slices the heads out column by column, runs attention_batch per head and
  // concatenates (multihead.rs:94-107).  The same arithmetic in one pass: heads become extra
  // batch entries, attention_batch runs once over [batch*heads, seq, d_head].
  const size_t d_head = d_model / num_heads;
  if (nrs_attention_supported((int)seq, (int)d_head))   // short sequences: the whole core in one kernel, heads in place
    return reshape(matmul(reshape(fused_attention(q, k, v, num_heads, causal), {batch * seq, d}), w_o), {batch, seq, d});
  auto split = [&](const NodeP& t) { return permute_heads(t, batch, seq, num_heads, d_head, true); };
  NodeP attended = attention_batch(split(q), split(k), split(v), causal);
  NodeP concat = permute_heads(attended, batch, seq, num_heads, d_head, false);
  return reshape(matmul(reshape(concat, {batch * seq, d}), w_o), {batch, seq, d});
}

static NodeP block_body(const TransformerBlock& b, const NodeP& x, bool final_norm) {
  if (!x || x->shape.size() != 3) fail(NRS_ERR_SHAPE, "cuda transformer block: input must be [batch, seq, d_model]");
  const size_t batch = x->shape[0], seq = x->shape[1], d = x->shape[2];
  NodeP attn_out = b.mha.forward_batch(x);
  NodeP x1 = b.fused_epilogues ? layernorm_residual(x, attn_out, b.norm1.gamma, b.norm1.beta, b.norm1.eps, true)
                               : b.norm1.forward(add(x, attn_out));
  NodeP flat = reshape(x1, {batch * seq, d});
  NodeP h, ff;
  if (b.fused_epilogues) {
    h = linear_act(flat, b.ff1.weights, b.ff1.bias, b.act, true, b.ff2.weights ? b.ff2.weights->shape.back() : 0);
    ff = linear_act(h, b.ff2.weights, b.ff2.bias, NRS_ACT_NONE);
  } else {
    h = b.ff1.forward(flat);
    h = b.act == NRS_ACT_GELU ? gelu(h) : relu(h);
    ff = b.ff2.forward(h);
  }
  NodeP ff_out = reshape(ff, {batch, seq, d});
  if (final_norm && b.fused_epilogues) return layernorm_residual(x1, ff_out, b.norm2.gamma, b.norm2.beta, b.norm2.eps, true);
  NodeP x2 = add(x1, ff_out);
  return final_norm ? b.norm2.forward(x2) : x2;
}

NodeP TransformerBlock::forward(const NodeP& x) const { return block_body(*this, x, true); }
NodeP TransformerBlock::forward_no_final_norm(const NodeP& x) const { return block_body(*this, x, false); }

}  // namespace cuda
}  // namespace nrs
