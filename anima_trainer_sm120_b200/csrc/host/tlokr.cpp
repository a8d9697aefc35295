#include "tlokr.h"

namespace anima_host {

using torch::autograd::set_history;

bool TLinear::can_fold(int64_t rows, int64_t cols, int64_t batch) const {
  return fold && c.size(0) == 8 && rows > 128 && cols > 128 && rows % 128 == 0 && cols % 8 == 0 && (cols / 8) % 64 == 0 &&
         rows % batch == 0 && rank() == 128;
}

namespace {

const void* mask_ptr(const OptTensor& m) { return m && m->defined() ? m->data_ptr() : nullptr; }

// Shapes for which the mix kernel can write the row-wise operand of its output itself.
bool can_quantise_mix(int64_t items, int64_t rank) {
  return (rank == 128 || rank == 256 || rank == 512) && items > 0 && items % 16 == 0;
}

Tensor mix(const Launch& l, const Tensor& hidden, const TLinear& t, int64_t batch, bool transpose) {
  const int64_t r = t.rank(), items = hidden.size(0) / 8;
  TORCH_CHECK_NOT_IMPLEMENTED(r % 8 == 0, "rank ", r, " must be a multiple of 8");
  Tensor out = at::detail::empty_cuda(hidden.sizes(), BF16, l.dev, std::nullopt);
  check(anima_tlokr_rank_mix(hidden.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, items / batch, r,
                             transpose ? 1 : 0, out.data_ptr(), l.stream));
  return out;
}

// Operands of the mixed tensor viewed as [rows * 8, rank]. Where the shape allows, the mix writes them itself: at
// [8, 4096, 8, 128] 42.0 (row), 42.1 (column), 57.3 us (both) against 30.8 + 22.6 / 24.6 / 32.8 for mix and quantiser.
std::pair<Op, Op> mix_operands(const Launch& l, const Tensor& hidden, const TLinear& t, int64_t batch, bool transpose,
                               bool row, bool col) {
  const int64_t r = t.rank(), R = hidden.size(0), items = R / 8;
  if (can_quantise_mix(items, r)) {
    Op ro, co;
    if (row) ro = empty_op(R, r, l.dev);
    if (col) co = empty_op(r, R, l.dev);
    check(anima_tlokr_rank_mix_quant(hidden.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, items / batch, r,
                                     transpose ? 1 : 0, nullptr, ro.codes, ro.scales, co.codes, co.scales, l.stream));
    return {ro, co};
  }
  return quantize(l, as_matrix(mix(l, hidden, t, batch, transpose), r), row, col);
}

Tensor gemm_bf16(const Launch& l, const Op& a, const Op& b, double alpha = 1.0) {
  Tensor c = empty({a.rows, b.rows}, BF16, l.dev);
  gemm(l, a, b, {c.data_ptr(), b.rows, false}, nullptr, nullptr, 0, alpha);
  return c;
}

// y = x W^T + bias + alpha * delta(x) into `y` [rows, n_out]. x_row and gq are the same codes as [rows, K] and as the
// grouped [rows * 8, K / 8]. Foldable shapes take two kernels: hidden = grouped . B^T with the 8x8 mix, the mask and
// the quantisation in its epilogue (hidden never leaves the SM), then ONE GEMM in which those planes times alpha * A
// are extra K-blocks of the base projection. Other shapes add alpha * delta in the last GEMM's stores.
void linear_fwd(const Launch& l, const Op& x_row, const Op& gq, int64_t batch, const TLinear& t, void* y) {
  const int64_t rows = x_row.rows, n = t.n_out(), vp = t.vp(), r = t.rank();
  const Tensor b = bias_rows(t.bias);
  if (t.can_fold(rows, n, batch) && n == 8 * vp) {
    Op planes = empty_op(rows * 8, r, l.dev);
    if (t.fuse_mix) {
      check(anima_tlokr_hidden_mix_planes(gq.codes, gq.scales, t.bq.codes, t.bq.scales,
                                          t.c.data_ptr(), mask_ptr(t.mask), batch, rows / batch, gq.k, 0, nullptr,
                                          planes.codes, planes.scales, status_word(l.dev), l.stream));
    } else {
      const Tensor hidden = gemm_bf16(l, gq, t.bq);
      check(anima_tlokr_rank_mix_quant_planes(hidden.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, rows / batch, r,
                                              0, planes.codes, planes.scales, nullptr, nullptr, l.stream));
    }
    gemm_delta(l, x_row, t.w_row, planes, t.a_scaled, y, ptr(b));
    return;
  }
  const Tensor hidden = gemm_bf16(l, gq, t.bq);
  gemm(l, x_row, t.w_row, {y, n, false}, ptr(b));
  const Op mq = mix_operands(l, hidden, t, batch, false, true, false).first;
  gemm(l, mq, t.aq, {y, vp, false}, nullptr, y, vp, t.alpha);
}

struct LinearGrads {
  Tensor x, w1, a, b;
};

// `g` / `g_col`: operands of the incoming gradient viewed as [rows * 8, vp]; gq / gq_col those of the grouped input.
LinearGrads linear_bwd(const Launch& l, const Op& gbq, const Op& gbq_col, const Op& gq, const Op& gq_col,
                       at::IntArrayRef lead, const TLinear& t, bool need_x) {
  const int64_t batch = lead[0], rows = gbq.rows / 8, K = t.k_in(), vp = t.vp(), r = t.rank(), vq = K / 8;
  TORCH_CHECK_VALUE(!need_x || t.w_col.defined(), "the base weight has no column form: quantise it with its input-gradient operand");
  LinearGrads g;
  const bool fold = t.can_fold(rows, K, batch);
  if (need_x) {
    std::vector<int64_t> shape(lead.begin(), lead.end());
    shape.push_back(K);
    g.x = empty(shape, BF16, l.dev);
    if (!fold) gemm(l, regroup(l, gbq, rows, 8 * vp), t.w_col, {g.x.data_ptr(), K, false});   // base input gradient
  }
  const Tensor hidden = gemm_bf16(l, gq, t.bq);
  const Op mq_col = mix_operands(l, hidden, t, batch, false, false, true).second;
  Tensor ga = gemm_f32(l, gbq_col, mq_col, t.alpha);                   // alpha * grad^T @ mixed  [vp, r]
  const Tensor g_mixed = gemm_bf16(l, gbq, t.aq_col, t.alpha);         // alpha * grad @ A
  Tensor gc = empty({8, 8}, F32, l.dev);
  {
    const int64_t bytes = check(anima_tlokr_rank_mix_wgrad_workspace_bytes(batch, rows / batch, r));
    Tensor ws = empty({bytes}, U8, l.dev);
    check(anima_tlokr_rank_mix_wgrad(g_mixed.data_ptr(), hidden.data_ptr(), mask_ptr(t.mask), batch, rows / batch, r,
                                     gc.data_ptr<float>(), ws.data_ptr(), bytes, l.stream));
  }
  Tensor gb;
  if (fold && need_x) {
    // grad_hidden leaves as eight planes + its column form; base dgrad and + grad_hidden @ B are one GEMM
    Op planes = empty_op(rows * 8, r, l.dev), col = empty_op(r, rows * 8, l.dev);
    check(anima_tlokr_rank_mix_quant_planes(g_mixed.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, rows / batch, r, 1,
                                            planes.codes, planes.scales, col.codes, col.scales,
                                            l.stream));
    gb = gemm_f32(l, col, gq_col);                                     // grad_hidden^T @ grouped [r, vq]
    gemm_delta(l, regroup(l, gbq, rows, 8 * vp), t.w_col, planes, t.bq_col, g.x.data_ptr(), nullptr);
  } else {
    auto [ghq, ghq_col] = mix_operands(l, g_mixed, t, batch, true, need_x, true);
    gb = gemm_f32(l, ghq_col, gq_col);
    if (need_x) gemm(l, ghq, t.bq_col, {g.x.data_ptr(), vq, false}, nullptr, g.x.data_ptr(), vq);
  }
  g.w1 = cast(gc, t.w1.t.scalar_type());
  g.a = cast(ga, t.a.t.scalar_type());
  g.b = cast(gb, t.b.t.scalar_type());
  return g;
}

struct Needs {
  bool x, factors, bias;
  bool any() const { return x || factors || bias; }
};
Needs needs_of(const Tensor& x, const TLinear& t) {
  return {wants(x), wants(t.w1.t) || wants(t.a.t) || wants(t.b.t), wants(t.bias)};
}

// Operands of a layer input. With `keep` the grouped view is quantised in both forms by one pass and its row codes
// serve the base GEMM too; otherwise only the row form exists (`x_row`).
struct Input {
  Op x_row, gq, gq_col;
};
template <class Quantise>
Input input_operands(const Launch& l, const Op& x_row, int64_t rows, int64_t K, bool keep, Quantise&& q) {
  Input in;
  if (keep) {
    std::tie(in.gq, in.gq_col) = q(rows * 8, K / 8);
    in.x_row = regroup(l, in.gq, rows, K);
  } else {
    in.x_row = x_row;
    in.gq = regroup(l, x_row, rows * 8, K / 8);
  }
  return in;
}
// what a node saves of it: the grouped operands, or stand-ins for them
void save_input(HostNode& n, const Launch& l, Input& in, int64_t rows, int64_t K, bool keep) {
  if (!keep) {
    in.gq = placeholder(rows * 8, K / 8, l.dev);
    in.gq_col = placeholder(K / 8, rows * 8, l.dev);
  }
  n.save(in.gq);
  n.save(in.gq_col);
}
std::pair<Op, Op> saved_input(HostNode& n, size_t& at, int64_t rows, int64_t K) {
  Op g, c;
  g.rows = c.k = rows * 8;
  g.k = c.rows = K / 8;
  Op gq = n.get_op(at, g), gq_col = n.get_op(at, c);
  return {gq, gq_col};
}

// The kernels index by these shapes: a mismatch must not reach them.
void check_linear(const Launch& l, const Tensor& x, int64_t k_in, const TLinear& t) {
  admit(l, t.bias, t.w1.t, t.a.t, t.b.t, t.mask, t.c, t.w_row.store, t.w_row.other, t.w_col.store, t.w_col.other);
  TORCH_CHECK_NOT_IMPLEMENTED(t.c.dim() == 2 && t.c.size(0) == 8 && t.c.size(1) == 8,
                              "rank_mix supports an 8x8 factor; got ", t.c.sizes());
  TORCH_CHECK_VALUE(t.a.t.dim() == 2 && t.b.t.dim() == 2 && t.b.t.size(0) == t.rank() && t.n_out() == 8 * t.vp() &&
                        t.k_in() == 8 * t.b.t.size(1) &&
                        (!t.w_col.defined() || (t.w_col.rows == t.k_in() && t.w_col.k == t.n_out())),
                    "factors ", t.a.t.sizes(), " and ", t.b.t.sizes(), " do not match a weight [", t.n_out(), ", ", t.k_in(), "]");
  TORCH_CHECK_VALUE(x.dim() >= 2 && k_in == t.k_in(), "input of width ", k_in, " for a weight with ", t.k_in(), " columns");
  if (t.mask && t.mask->defined())
    TORCH_CHECK_VALUE(t.mask->dim() == 2 && t.mask->size(0) == x.size(0) && t.mask->size(1) == t.rank(), "mask ",
                      t.mask->sizes(), " does not match batch ", x.size(0), " and rank ", t.rank());
}

std::vector<int64_t> lead_of(const Tensor& x) { return {x.sizes().begin(), x.sizes().end() - 1}; }
int64_t product(at::IntArrayRef v) { return c10::multiply_integers(v); }
Tensor grad_bias(const Tensor& gy) { return gy.reshape({-1, gy.size(-1)}).sum(0); }

// ------------------------------------------------------------------------------------------------ one linear
// ``x W^T + bias + alpha * delta(x)`` as one node: x is quantised once (base GEMM and delta contract the same codes
// under two scale tilings), so is the incoming gradient; saved are the MXFP8 operands of x in its grouped view, the
// rank-space intermediates are recomputed in backward.
struct TlokrNode : public HostNode {
  TLinear t;
  Needs need;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor gy = grad_of(g, 0);
    const Launch l(gy);
    const auto lead = lead_of(gy);
    size_t at = 0;
    const auto [gq, gq_col] = saved_input(*this, at, product(lead), t.k_in());
    t.check_unchanged();
    auto [gbq, gbq_col] = quantize(l, as_matrix(gy, t.vp()), true, true);
    LinearGrads r = linear_bwd(l, gbq, gbq_col, gq, gq_col, lead, t, need.x);
    return {r.x, need.bias ? grad_bias(gy) : Tensor(), r.w1, r.a, r.b};
  }
  std::string name() const override { return "MXTLoKrLinearBackward"; }
};

// ------------------------------------------------------------------------------------------------ MLP
// ``layer2(gelu(layer1(x)))``: the activation and its derivative are evaluated inside the quantiser, so neither
// gelu(h) nor grad * gelu'(h) is written as a bf16 tensor.
struct TlokrMlpNode : public HostNode {
  TLinear t1, t2;
  bool need_x, back;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!back) return variable_list(7);
    const Tensor gy = grad_of(g, 0);
    const Launch l(gy);
    const auto lead = lead_of(gy);
    const int64_t rows = product(lead);
    const Tensor h = get(0);
    size_t at = 1;
    const auto [gq1, gq1_col] = saved_input(*this, at, rows, t1.k_in());
    const auto [gq2, gq2_col] = saved_input(*this, at, rows, t2.k_in());
    t1.check_unchanged();
    t2.check_unchanged();
    LinearGrads g2, g1;
    {
      auto [gbq, gbq_col] = quantize(l, as_matrix(gy, t2.vp()), true, true);
      g2 = linear_bwd(l, gbq, gbq_col, gq2, gq2_col, lead, t2, true);
    }
    {
      const int64_t vp = t1.vp();
      auto [gbq, gbq_col] = quantize_gelu(l, h, g2.x, h.numel() / vp, vp, true, true);
      g2.x.reset();
      g1 = linear_bwd(l, gbq, gbq_col, gq1, gq1_col, lead, t1, need_x);
    }
    return {g1.x, g1.w1, g1.a, g1.b, g2.w1, g2.a, g2.b};
  }
  std::string name() const override { return "MXTLoKrMLPBackward"; }
};

}  // namespace

Tensor tlokr_linear(const Tensor& x, Op x_row, TLinear t, bool first) {
  const Needs need = needs_of(x, t);
  check_bias(t.bias, t.n_out());
  const Launch l(x);
  admit(l, x);
  check_linear(l, x, x.size(-1), t);
  const int64_t K = t.k_in(), rows = x.numel() / K;
  const bool keep = need.any() && !first;
  Tensor y;
  Input in;
  {
    Below below;
    in = input_operands(l, x_row, rows, K, keep, [&](int64_t, int64_t k) { return quantize(l, as_matrix(x, k), true, true); });
    y = empty(with_last(x.sizes(), t.n_out()), BF16, l.dev);
    linear_fwd(l, in.x_row, in.gq, x.size(0), t, y.data_ptr());
  }
  if (need.any()) {
    auto n = make_node<TlokrNode>(x, t.bias, t.w1.t, t.a.t, t.b.t);
    save_input(*n, l, in, rows, K, keep);
    n->need = need;
    n->t = std::move(t);
    set_history(y, n);
  }
  return y;
}

Tensor tlokr_mlp(const Tensor& x, Op x_row, TLinear t1, TLinear t2, bool first) {
  const Needs n1 = needs_of(x, t1), n2 = needs_of(x, t2);
  const bool back = n1.x || n1.factors || n2.factors, keep = back && !first;
  check_bias(t1.bias, t1.n_out());
  check_bias(t2.bias, t2.n_out());
  const Launch l(x);
  admit(l, x);
  check_linear(l, x, x.size(-1), t1);
  check_linear(l, x, t1.n_out(), t2);
  const int64_t K = t1.k_in(), rows = x.numel() / K, hid = t1.n_out();
  Tensor y, h;
  Input in1, in2;
  {
    Below below;
    in1 = input_operands(l, x_row, rows, K, keep, [&](int64_t, int64_t k) { return quantize(l, as_matrix(x, k), true, true); });
    h = empty(with_last(x.sizes(), hid), BF16, l.dev);
    linear_fwd(l, in1.x_row, in1.gq, x.size(0), t1, h.data_ptr());
    Op act_row;
    if (!keep) act_row = quantize_gelu(l, h, Tensor(), rows, hid, true, false).first;
    in2 = input_operands(l, act_row, rows, hid, keep,
                         [&](int64_t r, int64_t k) { return quantize_gelu(l, h, Tensor(), r, k, true, true); });
    y = empty(with_last(x.sizes(), t2.n_out()), BF16, l.dev);
    linear_fwd(l, in2.x_row, in2.gq, x.size(0), t2, y.data_ptr());
  }
  if (back || n1.bias || n2.bias) {
    auto n = make_node<TlokrMlpNode>(x, t1.w1.t, t1.a.t, t1.b.t, t2.w1.t, t2.a.t, t2.b.t);
    if (back) {
      n->save(h);
      save_input(*n, l, in1, rows, K, keep);
      save_input(*n, l, in2, rows, hid, keep);
    }
    n->need_x = n1.x;
    n->back = back;
    n->t1 = std::move(t1);
    n->t2 = std::move(t2);
    set_history(y, n);
  }
  return y;
}

Tensor tlokr_forward_only(const Op& x_row, const Op& gq, at::IntArrayRef lead, const TLinear& t) {
  check_bias(t.bias, t.n_out());
  const Launch l(x_row.store);
  std::vector<int64_t> shape(lead.begin(), lead.end());
  shape.push_back(t.n_out());
  Tensor y = empty(shape, BF16, l.dev);
  linear_fwd(l, x_row, gq, lead[0], t, y.data_ptr());
  return y;
}

std::vector<Tensor> tlokr_backward_only(const Op& gbq, const Op& gbq_col, const Op& gq, const Op& gq_col,
                                        at::IntArrayRef lead, const TLinear& t) {
  const Launch l(gbq.store);
  LinearGrads g = linear_bwd(l, gbq, gbq_col, gq, gq_col, lead, t, true);
  return {g.x, g.w1, g.a, g.b};
}

}  // namespace anima_host
