// Quantised T-LoKr linear and MLP as native autograd nodes.
#pragma once

#include "common.h"

namespace anima_host {

// One adapted linear: the frozen quantised base, the factors, their MXFP8 / bf16 forms, the rank mask.
struct TLinear {
  Op w_row, w_col;          // w_col may be missing where no input gradient is made
  OptTensor bias;
  Kept w1, a, b;            // parameters: [8, 8], [vp, r], [r, vq]
  OptTensor mask;           // [batch, r]
  Kept mask_in;             // the mask as it was given; like the parameters it may not change before backward
  double alpha;
  Tensor c;                 // w1 in bf16
  Op aq, aq_col, bq, bq_col, a_scaled;   // a_scaled: row form of alpha * a (folded delta only)
  bool fold, fuse_mix;      // switches of tlokr.py

  int64_t n_out() const { return w_row.rows; }
  int64_t k_in() const { return w_row.k; }
  int64_t vp() const { return a.t.size(0); }
  int64_t rank() const { return a.t.size(1); }
  void check_unchanged() const {
    for (const Kept* k : {&w1, &a, &b, &mask_in}) k->get();
  }
  bool can_fold(int64_t rows, int64_t cols, int64_t batch) const;
};

Tensor tlokr_linear(const Tensor& x, Op x_row, TLinear t, bool first);
Tensor tlokr_mlp(const Tensor& x, Op x_row, TLinear t1, TLinear t2, bool first);

// The two halves without autograd, on existing operands (kernel_bench times them): x as [rows, K] and grouped
Tensor tlokr_forward_only(const Op& x_row, const Op& gq, at::IntArrayRef lead, const TLinear& t);
std::vector<Tensor> tlokr_backward_only(const Op& gbq, const Op& gbq_col, const Op& gq, const Op& gq_col,
                                        at::IntArrayRef lead, const TLinear& t);

}  // namespace anima_host
