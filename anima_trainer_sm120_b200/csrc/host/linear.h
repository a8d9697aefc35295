// Quantised linears and the LoKr MLP as native autograd nodes. Operands of the input come from the caller (the
// activation memo of fp8_quant.py decides whether they have to be made).
#pragma once

#include "common.h"

namespace anima_host {

// y = x (W + alpha * kron(w1, w2))^T + bias. `first`: a pass whose saved tensors a checkpoint drops.
Tensor lokr_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& W, const OptTensor& bias, const Tensor& w1,
                   const Tensor& w2, double alpha, bool first);
// y = x merged^T + bias with the gradient of merged
Tensor merged_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& merged, const OptTensor& bias, bool first);
// y = x W^T + bias, W frozen and quantised; `w_bf16` serves backward when W has no column form. `save_weight`: the column
// form is a saved tensor (hooks, version check, released by backward) instead of the caller's to keep as it is.
Tensor frozen_linear(const Tensor& x, Op x_row, Op w_row, Op w_col, const OptTensor& w_bf16,
                     const OptTensor& bias, bool save_weight);
// layer2(gelu(layer1(x))) with both layers LoKr linears
Tensor lokr_mlp(const Tensor& x, Op x_row, Op x_col, const Tensor& W1, const OptTensor& b1, const Tensor& w1a,
                const Tensor& w2a, double alpha1, const Tensor& W2, const OptTensor& b2, const Tensor& w1b,
                const Tensor& w2b, double alpha2, bool first);

}  // namespace anima_host
