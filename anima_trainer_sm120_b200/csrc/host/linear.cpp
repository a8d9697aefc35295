#include "linear.h"

namespace anima_host {

using torch::autograd::Function;

namespace {

struct OutBias {           // bias as the GEMM reads it
  Tensor t;
  explicit OutBias(const OptTensor& b) : t(b && b->defined() ? bf16_contiguous(*b) : Tensor()) {}
  const void* ptr() const { return t.defined() ? t.data_ptr() : nullptr; }
};

// [*lead, N] in bf16, then in the dtype of the input
Tensor project(const Launch& l, const Tensor& x, const Op& x_row, const Op& w_row, const OptTensor& bias) {
  const int64_t n = w_row.rows();
  const OutBias b(bias);
  TORCH_CHECK_VALUE(!b.t.defined() || b.t.numel() == n, "bias must be of length N");
  Tensor y = empty(with_last(x.sizes(), n), BF16, l.dev);
  if (x_row.rows()) gemm(l, x_row, w_row, {y.data_ptr(), n, false}, b.ptr());
  return cast(y, x.scalar_type());
}

Tensor input_grad(const Launch& l, const Tensor& gy, const Op& g_row, const Op& w_col) {
  Tensor gx = empty(with_last(gy.sizes(), w_col.rows()), BF16, l.dev);
  if (g_row.rows()) gemm(l, g_row, w_col, {gx.data_ptr(), w_col.rows(), false});
  return cast(gx, gy.scalar_type());
}

Tensor bias_grad(const Tensor& gy) { return gy.reshape({-1, gy.size(-1)}).sum(0); }

// ------------------------------------------------------------------------------------------------ LoKr linear
struct LokrCall {
  const Tensor* W;
  Op x_row, x_col;
  double alpha;
  bool first, need_x, train, need_bias;
};
struct LokrHeld {
  double alpha;
  bool need_x, train, need_bias;
};

Tensor lokr_fwd(const Launch& l, const Tensor& x, const OptTensor& bias, const Tensor& w1, const Tensor& w2, LokrCall& c,
                Op& w_col) {
  auto [w_row, col] = merge_quantize(l, *c.W, w1, w2, c.alpha, true, c.need_x && !c.first);
  w_col = col;
  return project(l, x, c.x_row, w_row, bias);
}

struct LokrLinear : Function<LokrLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& bias, const Tensor& w1, const Tensor& w2,
                        LokrCall* c) {
    const Launch l(x);
    Op w_col;
    Tensor y = lokr_fwd(l, x, bias, w1, w2, *c, w_col);
    const int64_t n = c->W->size(0), k = c->W->size(1);
    if (c->first) {
      if (c->need_x) w_col = placeholder(k, n, l.dev);
      if (c->train) c->x_col = placeholder(k, c->x_row.rows(), l.dev);
    }
    variable_list keep;
    if (c->train) keep = {w1, w2};
    push(keep, c->x_col);
    push(keep, w_col);
    ctx->save_for_backward(std::move(keep));
    hold(ctx, LokrHeld{c->alpha, c->need_x, c->train, c->need_bias});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const LokrHeld h = held<LokrHeld>(ctx);
    const variable_list saved = ctx->get_saved_variables();     // once: checkpointing unpacks on access
    size_t at = h.train ? 2 : 0;
    const Op x_col = pop(saved, at, h.train), w_col = pop(saved, at, h.need_x);
    const Tensor& gy = grads[0];
    const Launch l(gy);
    auto [g_row, g_col] = quantize(l, as_matrix(gy, gy.size(-1)), h.need_x, h.train);
    variable_list out(5);
    if (h.need_x) out[0] = input_grad(l, gy, g_row, w_col);
    if (h.train) std::tie(out[2], out[3]) = kron_backward(l, gemm_f32(l, g_col, x_col), saved[0], saved[1], h.alpha);
    if (h.need_bias) out[1] = bias_grad(gy);
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ merged linear
struct MergedCall {
  Op x_row, x_col;
  bool first, need_x, train, need_bias;
};
struct MergedHeld {
  bool need_x, train, need_bias;
  at::ScalarType w_dtype;
};

std::pair<Op, Op> quantize_merged(const Launch& l, const Tensor& merged, bool col) {
  return quantize(l, as_matrix(merged, merged.size(1)), true, col);
}

struct MergedLinear : Function<MergedLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& merged, const OptTensor& bias, MergedCall* c) {
    const Launch l(x);
    auto [w_row, w_col] = quantize_merged(l, merged, c->need_x && !c->first);
    Tensor y = project(l, x, c->x_row, w_row, bias);
    if (c->first) {
      if (c->need_x) w_col = placeholder(merged.size(1), merged.size(0), l.dev);
      if (c->train) c->x_col = placeholder(merged.size(1), c->x_row.rows(), l.dev);
    }
    variable_list keep;
    push(keep, c->x_col);
    push(keep, w_col);
    ctx->save_for_backward(std::move(keep));
    hold(ctx, MergedHeld{c->need_x, c->train, c->need_bias, merged.scalar_type()});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const MergedHeld h = held<MergedHeld>(ctx);
    const variable_list saved = ctx->get_saved_variables();
    size_t at = 0;
    const Op x_col = pop(saved, at, h.train), w_col = pop(saved, at, h.need_x);
    const Tensor& gy = grads[0];
    const Launch l(gy);
    auto [g_row, g_col] = quantize(l, as_matrix(gy, gy.size(-1)), h.need_x, h.train);
    variable_list out(4);
    if (h.need_x) out[0] = input_grad(l, gy, g_row, w_col);
    if (h.train) {
      Tensor gw = empty({g_col.rows(), x_col.rows()}, BF16, l.dev);
      gemm(l, g_col, x_col, {gw.data_ptr(), x_col.rows(), false});
      out[1] = cast(gw, h.w_dtype);
    }
    if (h.need_bias) out[2] = bias_grad(gy);
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ frozen linear
struct FrozenCall {
  Op x_row, w_row, w_col;
  Tensor w_bf16;
  bool need_x, need_bias;
};
struct FrozenHeld {
  Op w_col;
  Tensor w_bf16;
  bool need_x, need_bias;
};

struct FrozenLinear : Function<FrozenLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor& bias, FrozenCall* c) {
    const Launch l(x);
    hold(ctx, FrozenHeld{c->w_col, c->w_bf16, c->need_x, c->need_bias});
    return project(l, x, c->x_row, c->w_row, bias);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const FrozenHeld& h = held<FrozenHeld>(ctx);
    const Tensor& gy = grads[0];
    variable_list out(3);
    if (h.need_x) {
      const Launch l(gy);
      const Mat g = as_matrix(gy, gy.size(-1));
      if (h.w_col.defined()) {
        out[0] = input_grad(l, gy, quantize(l, g, true, false).first, h.w_col);
      } else {
        Tensor gx = at::matmul(g.keep.reshape({g.rows, g.cols}), h.w_bf16.to(BF16));
        out[0] = cast(gx.reshape(with_last(gy.sizes(), h.w_bf16.size(1))), gy.scalar_type());
      }
    }
    if (h.need_bias) out[1] = bias_grad(gy);
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ LoKr MLP
struct MlpCall {
  Op x_row, x_col;
  const Tensor *W1, *W2;
  OptTensor b1, b2;
  double alpha1, alpha2;
  bool first, need_x, train;
  bool back() const { return need_x || train; }
};
struct MlpHeld {
  double alpha1, alpha2;
  bool need_x, train;
};
struct MlpKept {
  Tensor h;
  Op a_col, W1_col, W2_col;
};

Tensor mlp_fwd(const Launch& l, const Tensor& x, const Tensor& w1a, const Tensor& w2a, const Tensor& w1b,
               const Tensor& w2b, const MlpCall& c, MlpKept& kept) {
  const bool back = c.back() && !c.first;
  const int64_t rows = c.x_row.rows(), hid = c.W1->size(0);
  Op W1_row, W2_row, a_row;
  std::tie(W1_row, kept.W1_col) = merge_quantize(l, *c.W1, w1a, w2a, c.alpha1, true, back && c.need_x);
  const OutBias b1(c.b1);
  kept.h = empty({rows, hid}, BF16, l.dev);
  if (rows) gemm(l, c.x_row, W1_row, {kept.h.data_ptr(), hid, false}, b1.ptr());
  std::tie(a_row, kept.a_col) = quantize_gelu(l, kept.h, Tensor(), rows, hid, true, back && c.train);
  std::tie(W2_row, kept.W2_col) = merge_quantize(l, *c.W2, w1b, w2b, c.alpha2, true, back);
  return project(l, x, a_row, W2_row, c.b2);
}

struct LokrMlp : Function<LokrMlp> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1a, const Tensor& w2a, const Tensor& w1b,
                        const Tensor& w2b, MlpCall* c) {
    const Launch l(x);
    MlpKept k;
    Tensor y = mlp_fwd(l, x, w1a, w2a, w1b, w2b, *c, k);
    if (c->first) {
      const int64_t rows = c->x_row.rows(), hid = c->W1->size(0), k_in = c->W1->size(1), n_out = c->W2->size(0);
      if (c->need_x) k.W1_col = placeholder(k_in, hid, l.dev);
      k.W2_col = placeholder(hid, n_out, l.dev);
      if (c->train) {
        c->x_col = placeholder(k_in, rows, l.dev);
        k.a_col = placeholder(hid, rows, l.dev);
      }
    }
    variable_list keep{k.h, w1a, w2a, w1b, w2b};
    for (const Op* o : {&c->x_col, &k.a_col, &k.W1_col, &k.W2_col}) push(keep, *o);
    ctx->save_for_backward(std::move(keep));
    hold(ctx, MlpHeld{c->alpha1, c->alpha2, c->need_x, c->train});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const MlpHeld m = held<MlpHeld>(ctx);
    const variable_list saved = ctx->get_saved_variables();
    size_t at = 5;
    const Op x_col = pop(saved, at, m.train), a_col = pop(saved, at, m.train), W1_col = pop(saved, at, m.need_x),
             W2_col = pop(saved, at, true);
    const Tensor &h = saved[0], &gy = grads[0];
    const Launch l(gy);
    const int64_t rows = h.size(0), hid = h.size(1);
    auto [g_row, g_col] = quantize(l, as_matrix(gy, gy.size(-1)), true, m.train);
    Tensor grad_act = empty({rows, hid}, BF16, l.dev);
    gemm(l, g_row, W2_col, {grad_act.data_ptr(), hid, false});
    variable_list out(6);
    if (m.train) std::tie(out[3], out[4]) = kron_backward(l, gemm_f32(l, g_col, a_col), saved[3], saved[4], m.alpha2);
    auto [dh_row, dh_col] = quantize_gelu(l, h, grad_act, rows, hid, m.need_x, m.train);
    grad_act.reset();
    if (m.need_x) out[0] = input_grad(l, gy, dh_row, W1_col);
    if (m.train) std::tie(out[1], out[2]) = kron_backward(l, gemm_f32(l, dh_col, x_col), saved[1], saved[2], m.alpha1);
    return out;
  }
};

}  // namespace

Tensor lokr_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& W, const OptTensor& bias, const Tensor& w1,
                   const Tensor& w2, double alpha, bool first) {
  LokrCall c{&W, std::move(x_row), std::move(x_col), alpha, first, wants(x), wants(w1) || wants(w2), wants(bias)};
  if (c.need_x || c.train || c.need_bias) return LokrLinear::apply(x, bias, w1, w2, &c);
  const Launch l(x);
  Op unused;
  return lokr_fwd(l, x, bias, w1, w2, c, unused);
}

Tensor merged_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& merged, const OptTensor& bias, bool first) {
  MergedCall c{std::move(x_row), std::move(x_col), first, wants(x), wants(merged), wants(bias)};
  if (c.need_x || c.train || c.need_bias) return MergedLinear::apply(x, merged, bias, &c);
  const Launch l(x);
  return project(l, x, c.x_row, quantize_merged(l, merged, false).first, bias);
}

Tensor frozen_linear(const Tensor& x, Op x_row, Op w_row, Op w_col, const OptTensor& w_bf16, int64_t k_in,
                     const OptTensor& bias) {
  TORCH_CHECK_VALUE(x.size(-1) == k_in, "input of width ", x.size(-1), " for a weight with ", k_in, " columns");
  FrozenCall c{std::move(x_row), std::move(w_row), std::move(w_col), w_bf16.value_or(Tensor()), wants(x), wants(bias)};
  if (c.need_x || c.need_bias) return FrozenLinear::apply(x, bias, &c);
  const Launch l(x);
  return project(l, x, c.x_row, c.w_row, bias);
}

Tensor lokr_mlp(const Tensor& x, Op x_row, Op x_col, const Tensor& W1, const OptTensor& b1, const Tensor& w1a,
                const Tensor& w2a, double alpha1, const Tensor& W2, const OptTensor& b2, const Tensor& w1b,
                const Tensor& w2b, double alpha2, bool first) {
  const bool train = wants(w1a) || wants(w2a) || wants(w1b) || wants(w2b);
  MlpCall c{std::move(x_row), std::move(x_col), &W1, &W2, b1, b2, alpha1, alpha2, first, wants(x), train};
  if (c.back()) return LokrMlp::apply(x, w1a, w2a, w1b, w2b, &c);
  const Launch l(x);
  MlpKept unused;
  return mlp_fwd(l, x, w1a, w2a, w1b, w2b, c, unused);
}

}  // namespace anima_host
