#include "tlokr.h"

namespace anima_host {

using torch::autograd::Function;

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

// Operands of the mixed tensor viewed as [rows * 8, rank]. At [8, 4096, 8, 128] the quantising mix beats mix +
// quantiser for the row form (38.4 against 28.7 + 18.9 us); its column forms do not (46.6 against 28.7 + 16.9).
std::pair<Op, Op> mix_operands(const Launch& l, const Tensor& hidden, const TLinear& t, int64_t batch, bool transpose,
                               bool row, bool col) {
  const int64_t r = t.rank(), R = hidden.size(0), items = R / 8;
  if (!col && can_quantise_mix(items, r)) {
    Op o = empty_op(R, r, l.dev);
    check(anima_tlokr_rank_mix_quant(hidden.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, items / batch, r,
                                     transpose ? 1 : 0, nullptr, ptr8(o.codes), ptr8(o.scales), nullptr, nullptr,
                                     l.stream));
    return {o, Op{}};
  }
  return quantize(l, as_matrix(mix(l, hidden, t, batch, transpose), r), row, col);
}

Tensor gemm_bf16(const Launch& l, const Op& a, const Op& b, double alpha = 1.0) {
  Tensor c = empty({a.rows(), b.rows()}, BF16, l.dev);
  gemm(l, a, b, {c.data_ptr(), b.rows(), false}, nullptr, nullptr, 0, alpha);
  return c;
}

// y = x W^T + bias + alpha * delta(x) into `y` [rows, n_out]. x_row and gq are the same codes as [rows, K] and as the
// grouped [rows * 8, K / 8]. Foldable shapes take two kernels: hidden = grouped . B^T with the 8x8 mix, the mask and
// the quantisation in its epilogue (hidden never leaves the SM), then ONE GEMM in which those planes times alpha * A
// are extra K-blocks of the base projection. Other shapes add alpha * delta in the last GEMM's stores.
void linear_fwd(const Launch& l, const Op& x_row, const Op& gq, int64_t batch, const TLinear& t, void* y) {
  const int64_t rows = x_row.rows(), n = t.n_out(), vp = t.vp(), r = t.rank();
  const Tensor b = t.bias && t.bias->defined() ? bf16_contiguous(*t.bias) : Tensor();
  if (t.can_fold(rows, n, batch) && n == 8 * vp) {
    Op planes = empty_op(rows * 8, r, l.dev);
    if (t.fuse_mix) {
      check(anima_tlokr_hidden_mix_planes(ptr8(gq.codes), ptr8(gq.scales), ptr8(t.bq.codes), ptr8(t.bq.scales),
                                          t.c.data_ptr(), mask_ptr(t.mask), batch, rows / batch, gq.k(), 0, nullptr,
                                          ptr8(planes.codes), ptr8(planes.scales), status_word(l.dev), l.stream));
    } else {
      const Tensor hidden = gemm_bf16(l, gq, t.bq);
      check(anima_tlokr_rank_mix_quant_planes(hidden.data_ptr(), t.c.data_ptr(), mask_ptr(t.mask), batch, rows / batch, r,
                                              0, ptr8(planes.codes), ptr8(planes.scales), nullptr, nullptr, l.stream));
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
  const int64_t batch = lead[0], rows = gbq.rows() / 8, K = t.k_in(), vp = t.vp(), r = t.rank(), vq = K / 8;
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
                                            ptr8(planes.codes), ptr8(planes.scales), ptr8(col.codes), ptr8(col.scales),
                                            l.stream));
    gb = gemm_f32(l, col, gq_col);                                     // grad_hidden^T @ grouped [r, vq]
    gemm_delta(l, regroup(l, gbq, rows, 8 * vp), t.w_col, planes, t.bq_col, g.x.data_ptr(), nullptr);
  } else {
    auto [ghq, ghq_col] = mix_operands(l, g_mixed, t, batch, true, need_x, true);
    gb = gemm_f32(l, ghq_col, gq_col);
    if (need_x) gemm(l, ghq, t.bq_col, {g.x.data_ptr(), vq, false}, nullptr, g.x.data_ptr(), vq);
  }
  g.w1 = cast(gc, t.w1.scalar_type());
  g.a = cast(ga, t.a.scalar_type());
  g.b = cast(gb, t.b.scalar_type());
  return g;
}

struct Needs {
  bool x, factors, bias;
  bool any() const { return x || factors || bias; }
};
Needs needs_of(const Tensor& x, const TLinear& t) { return {wants(x), wants(t.w1) || wants(t.a) || wants(t.b), wants(t.bias)}; }

// Operands of a layer input. With `keep` the grouped view is quantised in both forms by one pass and its row codes
// serve the base GEMM too; otherwise only the row form exists (`x_row`) and a placeholder stands in.
struct Input {
  Op x_row, gq, gq_col;
};
template <class Quantise>
Input input_operands(const Launch& l, Op x_row, int64_t rows, int64_t K, bool keep, bool hold_place, Quantise&& q) {
  Input in;
  if (keep) {
    std::tie(in.gq, in.gq_col) = q(rows * 8, K / 8);
    in.x_row = regroup(l, in.gq, rows, K);
  } else {
    in.x_row = std::move(x_row);
    in.gq = regroup(l, in.x_row, rows * 8, K / 8);
    if (hold_place) in.gq_col = placeholder(K / 8, rows * 8, l.dev);
  }
  return in;
}

void keep_mask(variable_list& v, const TLinear& t) {
  if (t.mask && t.mask->defined()) v.push_back(*t.mask);
}
// The tensors autograd saves are read back through it; the forms and the frozen weight ride along.
void take_factors(TLinear& t, const variable_list& v, size_t at) {
  t.w1 = v[at];
  t.a = v[at + 1];
  t.b = v[at + 2];
}
void take_mask(TLinear& t, const variable_list& v, size_t& at) {
  if (t.mask && t.mask->defined()) t.mask = v[at++];
}
// What a node keeps outside its saved tensors: the parameters and the mask go through save_for_backward.
TLinear without_saved(TLinear t) {
  t.w1 = t.a = t.b = Tensor();
  if (t.mask && t.mask->defined()) t.mask = t.c;          // only marks that there is one
  return t;
}

std::vector<int64_t> lead_of(const Tensor& x) { return {x.sizes().begin(), x.sizes().end() - 1}; }

Tensor grad_bias(const Tensor& gy) { return gy.reshape({-1, gy.size(-1)}).sum(0); }

// ------------------------------------------------------------------------------------------------ one linear
// ``x W^T + bias + alpha * delta(x)`` as one node: x is quantised once (base GEMM and delta contract the same codes
// under two scale tilings), so is the incoming gradient; saved are the MXFP8 operands of x in its grouped view and the
// small factors, the rank-space intermediates are recomputed in backward.
struct LinearHeld {
  TLinear t;
  Needs need;
};
struct LinearCall {
  Op x_row;
  TLinear t;
  bool first;
  Needs need;
};

Tensor run_linear(const Launch& l, const Tensor& x, LinearCall& c, Input& in) {
  const int64_t K = c.t.k_in(), rows = x.numel() / K;
  in = input_operands(l, c.x_row, rows, K, c.need.any() && !c.first, c.need.any(), [&](int64_t r, int64_t k) {
    return quantize(l, as_matrix(x, k), true, true);
  });
  Tensor y = empty(with_last(x.sizes(), c.t.n_out()), BF16, l.dev);
  linear_fwd(l, in.x_row, in.gq, x.size(0), c.t, y.data_ptr());
  return y;
}

struct TlokrLinear : Function<TlokrLinear> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const OptTensor&, const Tensor& w1, const Tensor& a,
                        const Tensor& b, LinearCall* c) {
    const Launch l(x);
    Input in;
    Tensor y = run_linear(l, x, *c, in);
    variable_list keep{w1, a, b};
    push(keep, in.gq);
    push(keep, in.gq_col);
    keep_mask(keep, c->t);
    ctx->save_for_backward(std::move(keep));
    hold(ctx, LinearHeld{without_saved(c->t), c->need});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    LinearHeld h = held<LinearHeld>(ctx);
    const variable_list saved = ctx->get_saved_variables();   // once: activation checkpointing unpacks on access
    take_factors(h.t, saved, 0);
    size_t at = 3;
    const Op gq = pop(saved, at, true), gq_col = pop(saved, at, true);
    take_mask(h.t, saved, at);
    const Tensor& gy = grads[0];
    const Launch l(gy);
    auto [gbq, gbq_col] = quantize(l, as_matrix(gy, h.t.vp()), true, true);
    LinearGrads g = linear_bwd(l, gbq, gbq_col, gq, gq_col, lead_of(gy), h.t, h.need.x);
    variable_list out(6);
    out[0] = g.x;
    if (h.need.bias) out[1] = grad_bias(gy);
    out[2] = g.w1;
    out[3] = g.a;
    out[4] = g.b;
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ MLP
// ``layer2(gelu(layer1(x)))``: the activation and its derivative are evaluated inside the quantiser, so neither
// gelu(h) nor grad * gelu'(h) is written as a bf16 tensor.
struct MlpHeld {
  TLinear t1, t2;
  bool need_x;
};
struct MlpCall {
  Op x_row;
  TLinear t1, t2;
  bool first, need_x, back;
};

Tensor run_mlp(const Launch& l, const Tensor& x, MlpCall& c, Tensor& h, Input& in1, Input& in2) {
  const int64_t K = c.t1.k_in(), rows = x.numel() / K, hid = c.t1.n_out();
  const bool keep = c.back && !c.first;
  in1 = input_operands(l, c.x_row, rows, K, keep, c.back,
                       [&](int64_t r, int64_t k) { return quantize(l, as_matrix(x, k), true, true); });
  h = empty(with_last(x.sizes(), hid), BF16, l.dev);
  linear_fwd(l, in1.x_row, in1.gq, x.size(0), c.t1, h.data_ptr());
  Op act_row;
  if (!keep) act_row = quantize_gelu(l, h, Tensor(), rows, hid, true, false).first;
  in2 = input_operands(l, act_row, rows, hid, keep, c.back,
                       [&](int64_t r, int64_t k) { return quantize_gelu(l, h, Tensor(), r, k, true, true); });
  Tensor y = empty(with_last(x.sizes(), c.t2.n_out()), BF16, l.dev);
  linear_fwd(l, in2.x_row, in2.gq, x.size(0), c.t2, y.data_ptr());
  return y;
}

struct TlokrMlp : Function<TlokrMlp> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& w1_1, const Tensor& a_1, const Tensor& b_1,
                        const Tensor& w1_2, const Tensor& a_2, const Tensor& b_2, MlpCall* c) {
    const Launch l(x);
    Tensor h;
    Input in1, in2;
    Tensor y = run_mlp(l, x, *c, h, in1, in2);
    variable_list keep{h, w1_1, a_1, b_1, w1_2, a_2, b_2};
    for (const Op* o : {&in1.gq, &in1.gq_col, &in2.gq, &in2.gq_col}) push(keep, *o);
    keep_mask(keep, c->t1);
    keep_mask(keep, c->t2);
    ctx->save_for_backward(std::move(keep));
    hold(ctx, MlpHeld{without_saved(c->t1), without_saved(c->t2), c->need_x});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    MlpHeld m = held<MlpHeld>(ctx);
    const variable_list saved = ctx->get_saved_variables();
    const Tensor& h = saved[0];
    take_factors(m.t1, saved, 1);
    take_factors(m.t2, saved, 4);
    size_t at = 7;
    const Op gq1 = pop(saved, at, true), gq1_col = pop(saved, at, true), gq2 = pop(saved, at, true),
             gq2_col = pop(saved, at, true);
    take_mask(m.t1, saved, at);
    take_mask(m.t2, saved, at);
    const Tensor& gy = grads[0];
    const Launch l(gy);
    const auto lead = lead_of(gy);
    LinearGrads g2, g1;
    {
      auto [gbq, gbq_col] = quantize(l, as_matrix(gy, m.t2.vp()), true, true);
      g2 = linear_bwd(l, gbq, gbq_col, gq2, gq2_col, lead, m.t2, true);
    }
    {
      const int64_t vp = m.t1.vp();
      auto [gbq, gbq_col] = quantize_gelu(l, h, g2.x, h.numel() / vp, vp, true, true);
      g2.x.reset();
      g1 = linear_bwd(l, gbq, gbq_col, gq1, gq1_col, lead, m.t1, m.need_x);
    }
    return {g1.x, g1.w1, g1.a, g1.b, g2.w1, g2.a, g2.b, Tensor()};
  }
};

}  // namespace

Tensor tlokr_linear(const Tensor& x, Op x_row, TLinear t, bool first) {
  const Needs need = needs_of(x, t);
  LinearCall c{std::move(x_row), std::move(t), first, need};
  if (need.any()) return TlokrLinear::apply(x, c.t.bias, c.t.w1, c.t.a, c.t.b, &c);
  const Launch l(x);
  Input in;
  return run_linear(l, x, c, in);
}

Tensor tlokr_mlp(const Tensor& x, Op x_row, TLinear t1, TLinear t2, bool first) {
  const Needs n1 = needs_of(x, t1), n2 = needs_of(x, t2);
  MlpCall c{std::move(x_row), std::move(t1), std::move(t2), first, n1.x, n1.x || n1.factors || n2.factors};
  if (c.back) return TlokrMlp::apply(x, c.t1.w1, c.t1.a, c.t1.b, c.t2.w1, c.t2.a, c.t2.b, &c);
  const Launch l(x);
  Tensor h;
  Input in1, in2;
  return run_mlp(l, x, c, h, in1, in2);
}

Tensor tlokr_forward_only(const Op& x_row, const Op& gq, at::IntArrayRef lead, const TLinear& t) {
  const Launch l(x_row.codes);
  std::vector<int64_t> shape(lead.begin(), lead.end());
  shape.push_back(t.n_out());
  Tensor y = empty(shape, BF16, l.dev);
  linear_fwd(l, x_row, gq, lead[0], t, y.data_ptr());
  return y;
}

std::vector<Tensor> tlokr_backward_only(const Op& gbq, const Op& gbq_col, const Op& gq, const Op& gq_col,
                                        at::IntArrayRef lead, const TLinear& t) {
  const Launch l(gbq.codes);
  LinearGrads g = linear_bwd(l, gbq, gbq_col, gq, gq_col, lead, t, true);
  return {g.x, g.w1, g.a, g.b};
}

}  // namespace anima_host
