// AdaLN, gated residual, and q / k RMSNorm + rotary embedding as native autograd nodes.
#pragma once

#include "common.h"

namespace anima_host {

// Activations (B, T, H, W, D), modulation (B, T, 1, 1, D). `quant`: also the row-wise operand of y.
std::tuple<Tensor, Op> adaln(const Tensor& x, const Tensor& scale, const Tensor& shift, double eps, bool quant);
Tensor gated_add(const Tensor& x, const Tensor& gate, const Tensor& y);
std::tuple<Tensor, Tensor, Op> gated_add_adaln(const Tensor& x, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                                               const Tensor& shift, double eps, bool quant);
// x (B, L, H, 128) bf16; cos / sin fp32 [L, 128] or undefined
Tensor rmsnorm_rope(const Tensor& x, const Tensor& weight, const OptTensor& cos, const OptTensor& sin, double eps);

}  // namespace anima_host
