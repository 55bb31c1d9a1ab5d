// Multi-head attention over operand planes (attention_planes.cu).
#pragma once

#include "nrs_internal.h"

// D = heads * d_head; ld = nrs_plane_ld(seq).  The lo pointers are null unless 3xTF32.
struct NrsMhaPlanes {
  int batch, seq, heads, d_head, causal;
  const float *qkv_hi, *qkv_lo;   // [batch*seq][qkv_ld]: Q, K, V side by side, D columns each
  int qkv_ld;
  float* scores;                  // [batch*heads][seq][ld] scratch (S forward, dP backward)
  float *p_hi, *p_lo;             // [batch*heads][seq][ld] probabilities, written forward, read backward
  float *out, *out_hi, *out_lo;   // [batch*seq][D]: f32 result (may be null) and its planes
  const float *dout_hi, *dout_lo; // [batch*seq][D]
  float *ds_hi, *ds_lo;           // [batch*heads][seq][ld] scratch
  float *dqkv_hi, *dqkv_lo;       // [batch*seq][3*D]
};
bool nrs_mha_planes_applies(const nrs_ctx* ctx, int seq, int d_head);
int nrs_mha_planes_fwd(nrs_ctx* ctx, const NrsMhaPlanes& a);
int nrs_mha_planes_bwd(nrs_ctx* ctx, const NrsMhaPlanes& a);
