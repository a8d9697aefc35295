#include "linear.h"

namespace anima_host {

namespace {

using torch::autograd::set_history;

// [*lead, N] in bf16, then in the dtype of the input
Tensor project(const Launch& l, const Tensor& x, const Op& x_row, const Op& w_row, const OptTensor& bias) {
  const int64_t n = w_row.rows;
  const Tensor b = bias_rows(bias);
  Tensor y = empty(with_last(x.sizes(), n), BF16, l.dev);
  if (x_row.rows) gemm(l, x_row, w_row, {y.data_ptr(), n, false}, ptr(b));
  return cast(y, x.scalar_type());
}

Tensor input_grad(const Launch& l, const Tensor& gy, const Op& g_row, const Op& w_col) {
  Tensor gx = empty(with_last(gy.sizes(), w_col.rows), BF16, l.dev);
  if (g_row.rows) gemm(l, g_row, w_col, {gx.data_ptr(), w_col.rows, false});
  return cast(gx, gy.scalar_type());
}

Tensor bias_grad(const Tensor& gy) { return gy.reshape({-1, gy.size(-1)}).sum(0); }

Op shape_of(int64_t rows, int64_t k) {      // of an operand saved as one store
  Op o;
  o.rows = rows;
  o.k = k;
  return o;
}
Op shape_of(const Op& o) {
  Op s = shape_of(o.rows, o.k);
  s.other = o.other.defined() ? o.other : Tensor();
  return s;
}

// ------------------------------------------------------------------------------------------------ LoKr linear
struct LokrNode : public HostNode {
  Kept w1, w2;
  Op x_col, w_col;      // shapes
  double alpha;
  bool need_x, train, need_bias;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor gy = grad_of(g, 0);
    const Launch l(gy);
    size_t at = 0;
    const Op xc = get_op(at, x_col), wc = get_op(at, w_col);
    Op g_row, g_col;
    if (need_x || train) std::tie(g_row, g_col) = quantize(l, as_matrix(gy, gy.size(-1)), need_x, train);
    variable_list out(4);
    if (need_x) out[0] = input_grad(l, gy, g_row, wc);
    if (train) std::tie(out[2], out[3]) = kron_backward(l, gemm_f32(l, g_col, xc), w1.get(), w2.get(), alpha);
    if (need_bias) out[1] = bias_grad(gy);
    return out;
  }
  std::string name() const override { return "LoKrLinearFusedBackward"; }
};

// ------------------------------------------------------------------------------------------------ merged linear
struct MergedNode : public HostNode {
  Op x_col, w_col;
  bool need_x, train, need_bias;
  at::ScalarType w_dtype;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor gy = grad_of(g, 0);
    const Launch l(gy);
    size_t at = 0;
    const Op xc = get_op(at, x_col), wc = get_op(at, w_col);
    Op g_row, g_col;
    if (need_x || train) std::tie(g_row, g_col) = quantize(l, as_matrix(gy, gy.size(-1)), need_x, train);
    variable_list out(3);
    if (need_x) out[0] = input_grad(l, gy, g_row, wc);
    if (train) {
      Tensor gw = empty({g_col.rows, xc.rows}, BF16, l.dev);
      gemm(l, g_col, xc, {gw.data_ptr(), xc.rows, false});
      out[1] = cast(gw, w_dtype);
    }
    if (need_bias) out[2] = bias_grad(gy);
    return out;
  }
  std::string name() const override { return "MXFP8LoKrLinearBackward"; }
};

// ------------------------------------------------------------------------------------------------ frozen linear
struct FrozenNode : public HostNode {
  Op w_col;                // its shape alone where it is a saved tensor
  Tensor w_bf16;
  bool need_x, need_bias, w_saved;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor gy = grad_of(g, 0);
    variable_list out(2);
    size_t at = 0;
    const Op w = w_saved ? get_op(at, w_col) : w_col;
    if (need_x) {
      const Launch l(gy);
      const Mat m = as_matrix(gy, gy.size(-1));
      if (w.defined()) {
        out[0] = input_grad(l, gy, quantize(l, m, true, false).first, w);
      } else {
        Tensor gx = at::matmul(m.keep.reshape({m.rows, m.cols}), w_bf16.to(BF16));
        out[0] = cast(gx.reshape(with_last(gy.sizes(), w_bf16.size(1))), gy.scalar_type());
      }
    }
    if (need_bias) out[1] = bias_grad(gy);
    return out;
  }
  std::string name() const override { return "MXFP8FrozenLinearBackward"; }
};

// ------------------------------------------------------------------------------------------------ LoKr MLP
struct MlpNode : public HostNode {
  Kept w1a, w2a, w1b, w2b;
  Op x_col, a_col, W1_col, W2_col;
  double alpha1, alpha2;
  bool need_x, train;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!need_x && !train) return variable_list(5);
    const Tensor gy = grad_of(g, 0);
    const Launch l(gy);
    const Tensor h = get(0);
    size_t at = 1;
    const Op xc = get_op(at, x_col), ac = get_op(at, a_col), W1 = get_op(at, W1_col), W2 = get_op(at, W2_col);
    const int64_t rows = h.size(0), hid = h.size(1);
    auto [g_row, g_col] = quantize(l, as_matrix(gy, gy.size(-1)), true, train);
    Tensor grad_act = empty({rows, hid}, BF16, l.dev);
    if (rows) gemm(l, g_row, W2, {grad_act.data_ptr(), hid, false});
    variable_list out(5);
    if (train) std::tie(out[3], out[4]) = kron_backward(l, gemm_f32(l, g_col, ac), w1b.get(), w2b.get(), alpha2);
    auto [dh_row, dh_col] = quantize_gelu(l, h, grad_act, rows, hid, need_x, train);
    grad_act.reset();
    if (need_x) out[0] = input_grad(l, gy, dh_row, W1);
    if (train) std::tie(out[1], out[2]) = kron_backward(l, gemm_f32(l, dh_col, xc), w1a.get(), w2a.get(), alpha1);
    return out;
  }
  std::string name() const override { return "LoKrMLPFusedBackward"; }
};

}  // namespace

Tensor lokr_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& W, const OptTensor& bias, const Tensor& w1,
                   const Tensor& w2, double alpha, bool first) {
  const bool need_x = wants(x), train = wants(w1) || wants(w2), need_bias = wants(bias);
  check_bias(bias, W.size(0));
  const Launch l(x);
  admit(l, x, W, bias, w1, w2);
  Tensor y;
  Op w_col;
  {
    Below below;
    Op w_row;
    std::tie(w_row, w_col) = merge_quantize(l, W, w1, w2, alpha, true, need_x && !first);
    y = project(l, x, x_row, w_row, bias);
    if (first) {
      if (need_x) w_col = placeholder(W.size(1), W.size(0), l.dev);
      if (train) x_col = placeholder(W.size(1), x_row.rows, l.dev);
    }
  }
  if (any_wants(x, W, bias, w1, w2)) {
    auto n = make_node<LokrNode>(x, bias, w1, w2);
    if (train) {
      n->w1 = Kept(w1);
      n->w2 = Kept(w2);
      n->save(x_col);
      n->x_col = shape_of(x_col);
    }
    if (need_x) {
      n->save(w_col);
      n->w_col = shape_of(w_col);
    }
    n->alpha = alpha;
    n->need_x = need_x;
    n->train = train;
    n->need_bias = need_bias;
    set_history(y, n);
  }
  return y;
}

Tensor merged_linear(const Tensor& x, Op x_row, Op x_col, const Tensor& merged, const OptTensor& bias, bool first) {
  const bool need_x = wants(x), train = wants(merged), need_bias = wants(bias);
  check_bias(bias, merged.size(0));
  const Launch l(x);
  admit(l, x, merged, bias);
  Tensor y;
  Op w_col;
  {
    Below below;
    Op w_row;
    std::tie(w_row, w_col) = quantize(l, as_matrix(merged, merged.size(1)), true, need_x && !first);
    y = project(l, x, x_row, w_row, bias);
    if (first) {
      if (need_x) w_col = placeholder(merged.size(1), merged.size(0), l.dev);
      if (train) x_col = placeholder(merged.size(1), x_row.rows, l.dev);
    }
  }
  if (need_x || train || need_bias) {
    auto n = make_node<MergedNode>(x, merged, bias);
    if (train) {
      n->save(x_col);
      n->x_col = shape_of(x_col);
    }
    if (need_x) {
      n->save(w_col);
      n->w_col = shape_of(w_col);
    }
    n->need_x = need_x;
    n->train = train;
    n->need_bias = need_bias;
    n->w_dtype = merged.scalar_type();
    set_history(y, n);
  }
  return y;
}

Tensor frozen_linear(const Tensor& x, Op x_row, Op w_row, Op w_col, const OptTensor& w_bf16, const OptTensor& bias,
                     bool save_weight) {
  TORCH_CHECK_VALUE(x.size(-1) == w_row.k, "input of width ", x.size(-1), " for a weight with ", w_row.k, " columns");
  const bool need_x = wants(x), need_bias = wants(bias);
  TORCH_CHECK_VALUE(!need_x || !w_col.defined() || (w_col.rows == w_row.k && w_col.k == w_row.rows),
                    "the backward operand [", w_col.rows, ", ", w_col.k, "] is not the transpose of the weight [", w_row.rows, ", ",
                    w_row.k, "]");
  check_bias(bias, w_row.rows);
  const Launch l(x);
  admit(l, x, bias, x_row.store, x_row.other, w_row.store, w_row.other, w_col.store, w_col.other);
  Tensor y;
  {
    Below below;
    y = project(l, x, x_row, w_row, bias);
  }
  if (any_wants(x, w_bf16, bias)) {
    auto n = make_node<FrozenNode>(x, bias);
    n->w_saved = save_weight && w_col.defined();
    if (n->w_saved) n->save(w_col);
    n->w_col = n->w_saved ? shape_of(w_col) : std::move(w_col);
    n->w_bf16 = w_bf16.value_or(Tensor());
    n->need_x = need_x;
    n->need_bias = need_bias;
    set_history(y, n);
  }
  return y;
}

Tensor lokr_mlp(const Tensor& x, Op x_row, Op x_col, const Tensor& W1, const OptTensor& b1, const Tensor& w1a,
                const Tensor& w2a, double alpha1, const Tensor& W2, const OptTensor& b2, const Tensor& w1b,
                const Tensor& w2b, double alpha2, bool first) {
  const bool train = wants(w1a) || wants(w2a) || wants(w1b) || wants(w2b), need_x = wants(x), back = need_x || train;
  const bool keep = back && !first;
  check_bias(b1, W1.size(0));
  check_bias(b2, W2.size(0));
  const Launch l(x);
  admit(l, x, W1, b1, w1a, w2a, W2, b2, w1b, w2b);
  const int64_t rows = x_row.rows, hid = W1.size(0);
  Tensor y, h;
  Op a_col, W1_col, W2_col;
  {
    Below below;
    Op W1_row, W2_row, a_row;
    std::tie(W1_row, W1_col) = merge_quantize(l, W1, w1a, w2a, alpha1, true, keep && need_x);
    const Tensor b = bias_rows(b1);
    h = empty({rows, hid}, BF16, l.dev);
    if (rows) gemm(l, x_row, W1_row, {h.data_ptr(), hid, false}, ptr(b));
    std::tie(a_row, a_col) = quantize_gelu(l, h, Tensor(), rows, hid, true, keep && train);
    std::tie(W2_row, W2_col) = merge_quantize(l, W2, w1b, w2b, alpha2, true, keep);
    y = project(l, x, a_row, W2_row, b2);
    if (back && first) {
      if (need_x) W1_col = placeholder(W1.size(1), hid, l.dev);
      W2_col = placeholder(hid, W2.size(0), l.dev);
      if (train) {
        x_col = placeholder(W1.size(1), rows, l.dev);
        a_col = placeholder(hid, rows, l.dev);
      }
    }
  }
  if (any_wants(x, W1, b1, w1a, w2a, W2, b2, w1b, w2b)) {
    auto n = make_node<MlpNode>(x, w1a, w2a, w1b, w2b);
    if (back) n->save(h);
    for (auto [op, shape] : {std::pair{&x_col, &n->x_col}, {&a_col, &n->a_col}, {&W1_col, &n->W1_col}, {&W2_col, &n->W2_col}}) {
      if (op == &x_col && !train) continue;
      n->save(*op);
      *shape = shape_of(*op);
    }
    if (train) {
      n->w1a = Kept(w1a);
      n->w2a = Kept(w2a);
      n->w1b = Kept(w1b);
      n->w2b = Kept(w2b);
    }
    n->alpha1 = alpha1;
    n->alpha2 = alpha2;
    n->need_x = need_x;
    n->train = train;
    set_history(y, n);
  }
  return y;
}

}  // namespace anima_host
