// Second stages of split reductions, run one by one or collected into one launch (fold.cu).
#pragma once

#include "nrs_internal.h"

// While on, submitted folds wait for nrs_folds_flush (a backward pass's end) or nrs_folds_settle.
void nrs_folds_begin(nrs_ctx* ctx);
int nrs_folds_flush(nrs_ctx* ctx);   // (and the weight gradients that wait, before them)
// nrs_free, or, while weight gradients wait that may read it, once they have run.
void nrs_free_after_wgrads(nrs_ctx* ctx, void* p);
// Launches the weight gradients that wait and lets go of what was kept for them: ahead of another one where more than
// kNrsKeptBytes are (nrs_wgrad_may_wait's callers), and where the driver has no memory left (at any point of a pass).
constexpr size_t kNrsKeptBytes = (size_t)1 << 30;
int nrs_folds_relieve(nrs_ctx* ctx);
inline int nrs_folds_limit_kept(nrs_ctx* ctx) { return ctx->folds.kept_bytes > kNrsKeptBytes ? nrs_folds_relieve(ctx) : NRS_OK; }
void nrs_folds_end(nrs_ctx* ctx);    // leaves the collecting mode; what is still queued is dropped (a failed pass)
void nrs_folds_free(nrs_ctx* ctx);
// Runs what is queued if it writes any of the `len` floats at `dst`: called by whoever is about to read, overwrite or
// add to a gradient.
int nrs_folds_settle(nrs_ctx* ctx, const float* dst, size_t len);
// Memory for a fold's partial sums that lives until the fold has run; outside of the collecting mode the given
// workspace slot (-1: the context's workspace).
int nrs_fold_partial(nrs_ctx* ctx, int ws_slot, size_t bytes, float** out);
int nrs_fold_submit(nrs_ctx* ctx, NrsFoldJob job);
// dst[c] (+)= sum over rows of src[r*stride + c]; src must stay as it is until the fold has run.
int nrs_fold_columns(nrs_ctx* ctx, const float* src, float* dst, int rows, int cols, int stride, int accumulate);
// The same for two results side by side: columns [0, cols) to dst, [cols, 2*cols) to dst2.
int nrs_fold_column_pair(nrs_ctx* ctx, const float* src, float* dst, float* dst2, int rows, int cols, int stride, int accumulate);
