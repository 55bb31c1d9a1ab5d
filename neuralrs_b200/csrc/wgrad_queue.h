// Weight gradients of a backward pass, collected into one launch per kernel at its end.
//
// A layer's weight gradient is a reduction over all pixels into a small result: alone it fills the GPU only by splitting the
// pixels among all SMs, pays a launch, a ramp and a partial tile of 98 KB from every SM, and the partial tiles are read again
// by the folds.  Nothing in a pass reads a parameter's gradient, so the layers' products wait until its end and share one
// launch: every CTA takes a longer run of pixels of one layer, and there are as many partial tiles as SMs in all instead of
// per layer.  No accumulation chain becomes longer for it than it may be: in 3xTF32 the mode's limit, in TF32, which has none
// of its own, what the product would have alone, or tc::kMaxChainK values.  Collected while folds are (NrsFolds::active), where both operands' planes are there and stay: their owners
// release them through nrs_free_after_wgrads.
#pragma once

#include <algorithm>

#include "fold.h"
#include "nrs_internal.h"

// May the weight gradient of these planes wait?
inline bool nrs_wgrad_may_wait(const nrs_ctx* ctx, const void* dy_hi, const void* x_hi) {
  if (!ctx->folds.active) return false;
  for (const void* s : ctx->ws_slot)
    if (s == dy_hi || s == x_hi) return false;   // scratch that the next layer overwrites
  return true;
}
// The kernels' queues (tc_wgrad_rows.cu, tc_wgrad.cu).
int nrs_wgrad_rows_run(nrs_ctx* ctx);
int nrs_wgrad_tiles_run(nrs_ctx* ctx);

namespace wgq {

// One weight gradient as work to be shared out: `units` of pixels for each of `ctas` output tiles.
struct Piece {
  int ctas;
  long units;
  double unit_clk, fixed_clk;   // a CTA's time: units * unit_clk + fixed_clk
  long max_units;               // an accumulation chain's
  double split_bytes;           // partial tiles of one split
  long per;                     // out: units per CTA
};

// Units per CTA of every piece so that the launch ends early: CTAs of about the same length T, T from a sweep around the mean.
// Up to one CTA per SM the longest one decides, beyond that the sum and half of the longest; partial tiles are written and
// read again at about 1.1 KB a clock.
inline void share_out(std::vector<Piece>& pieces, int sm_count) {
  double total = 0.0;
  for (const Piece& q : pieces) total += q.ctas * (q.units * q.unit_clk + q.fixed_clk);
  double best = -1.0, best_t = 0.0;
  auto per_of = [](const Piece& q, double t) {
    long per = (long)((t - q.fixed_clk) / q.unit_clk);
    per = std::max(1L, std::min({per, q.max_units, q.units}));
    const long splits = (q.units + per - 1) / per;
    return (q.units + splits - 1) / splits;
  };
  for (int i = 0; i < 64; ++i) {
    const double t = total / sm_count * (0.15 + 0.04 * i);
    double sum = 0.0, longest = 0.0, bytes = 0.0;
    long ctas = 0;
    for (const Piece& q : pieces) {
      const long per = per_of(q, t), splits = (q.units + per - 1) / per;
      const double one = per * q.unit_clk + q.fixed_clk;
      ctas += q.ctas * splits;
      sum += (double)q.ctas * splits * one;
      longest = std::max(longest, one);
      bytes += q.split_bytes * splits;
    }
    const double cost = (ctas <= sm_count ? longest : std::max(longest, sum / sm_count + 0.5 * longest)) + 2.0 * bytes / 1100.0;
    if (best < 0.0 || cost < best) { best = cost; best_t = t; }
  }
  for (Piece& q : pieces) q.per = per_of(q, best_t);
}

}  // namespace wgq
