#include "norm.h"

namespace anima_host {

using torch::autograd::Function;

namespace {

struct Rows {            // a (B, T, H, W, D) activation as rows of its B * T samples
  int64_t n, hw, d, samples;
};
Rows rows_of(const Tensor& x) {
  const auto s = x.sizes();
  return {s[0] * s[1] * s[2] * s[3], s[2] * s[3], s[4], s[0] * s[1]};
}
Tensor like(const Tensor& x, const at::Device& dev, at::ScalarType dt = BF16) {
  return at::detail::empty_cuda(x.sizes(), dt, dev, std::nullopt);
}
Tensor back_to(const Tensor& t, at::ScalarType dt) { return t.defined() ? cast(t, dt) : t; }

// ------------------------------------------------------------------------------------------------ AdaLN
struct AdalnCall {
  float eps;
  bool quant;
  Op emitted;
  Tensor x, scale, mean, rstd;      // as the kernel read them; kept for backward
};
struct AdalnHeld {
  at::ScalarType x, scale, shift;
};

Tensor adaln_fwd(const Launch& l, const Tensor& x, const Tensor& scale, const Tensor& shift, AdalnCall& c) {
  const Rows r = rows_of(x);
  c.x = bf16_contiguous(x);
  c.scale = bf16_contiguous(scale);
  const Tensor sh = bf16_contiguous(shift);
  Tensor y = like(x, l.dev);
  c.mean = empty({r.n}, F32, l.dev);
  c.rstd = empty({r.n}, F32, l.dev);
  float *mean = c.mean.data_ptr<float>(), *rstd = c.rstd.data_ptr<float>();
  if (c.quant) {
    c.emitted = empty_op(r.n, r.d, l.dev);
    check(anima_adaln_fwd_quant(c.x.data_ptr(), c.scale.data_ptr(), sh.data_ptr(), c.eps, r.n, r.hw, r.d, y.data_ptr(), mean,
                                rstd, ptr8(c.emitted.codes), ptr8(c.emitted.scales), ANIMA_SCALES_TILED, l.stream));
  } else {
    check(anima_adaln_fwd(c.x.data_ptr(), c.scale.data_ptr(), sh.data_ptr(), c.eps, r.n, r.hw, r.d, y.data_ptr(), mean, rstd,
                          l.stream));
  }
  return y;
}

// dx, dscale, dshift
std::tuple<Tensor, Tensor, Tensor> adaln_bwd(const Launch& l, const Tensor& dy_, const Tensor& x, const Tensor& scale,
                                             const Tensor& mean, const Tensor& rstd) {
  const Rows r = rows_of(x);
  const Tensor dy = bf16_contiguous(dy_);
  const int64_t bytes = check(anima_adaln_bwd_workspace_bytes(r.n, r.hw, r.d));
  Tensor ws = empty({bytes}, U8, l.dev), dx = like(x, l.dev), ds = like(scale, l.dev), db = like(scale, l.dev);
  check(anima_adaln_bwd(dy.data_ptr(), x.data_ptr(), scale.data_ptr(), mean.data_ptr<float>(), rstd.data_ptr<float>(), r.n,
                        r.hw, r.d, dx.data_ptr(), ds.data_ptr(), db.data_ptr(), ws.data_ptr(), bytes, l.stream));
  return {dx, ds, db};
}

std::pair<Tensor, Tensor> gated_bwd(const Launch& l, const Tensor& dout_, const Tensor& y, const Tensor& gate) {
  const Rows r = rows_of(y);
  const Tensor dout = bf16_contiguous(dout_);
  const int64_t bytes = check(anima_gated_add_bwd_workspace_bytes(r.n, r.hw, r.d));
  Tensor ws = empty({bytes}, U8, l.dev), dy = like(y, l.dev), dg = like(gate, l.dev);
  check(anima_gated_add_bwd(dout.data_ptr(), y.data_ptr(), gate.data_ptr(), r.n, r.hw, r.d, dy.data_ptr(), dg.data_ptr(),
                            ws.data_ptr(), bytes, l.stream));
  return {dy, dg};
}

struct AdaLN : Function<AdaLN> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& scale, const Tensor& shift, AdalnCall* c) {
    const Launch l(x);
    Tensor y = adaln_fwd(l, x, scale, shift, *c);
    ctx->save_for_backward({c->x, c->scale, c->mean, c->rstd});
    hold(ctx, AdalnHeld{x.scalar_type(), scale.scalar_type(), shift.scalar_type()});
    return y;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const AdalnHeld h = held<AdalnHeld>(ctx);
    const Launch l(s[0]);
    auto [dx, ds, db] = adaln_bwd(l, grads[0], s[0], s[1], s[2], s[3]);
    return {back_to(dx, h.x), back_to(ds, h.scale), back_to(db, h.shift), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ gated residual
Tensor gated_fwd(const Launch& l, const Tensor& x_, const Tensor& y, const Tensor& gate) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_);
  Tensor out = like(x, l.dev);
  check(anima_gated_add_fwd(x.data_ptr(), gate.data_ptr(), y.data_ptr(), r.n, r.hw, r.d, out.data_ptr(), l.stream));
  return out;
}

struct GatedAdd : Function<GatedAdd> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& y) {
    const Launch l(x);
    const Tensor yc = bf16_contiguous(y), gc = bf16_contiguous(gate);
    ctx->save_for_backward({yc, gc});
    hold(ctx, AdalnHeld{x.scalar_type(), gate.scalar_type(), y.scalar_type()});
    return gated_fwd(l, x, yc, gc);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const AdalnHeld h = held<AdalnHeld>(ctx);
    const Launch l(s[0]);
    auto [dy, dg] = gated_bwd(l, grads[0], s[0], s[1]);
    return {grads[0], back_to(dg, h.scale), back_to(dy, h.shift)};
  }
};

// ------------------------------------------------------------------------------------------------ both at once
struct BothCall {
  float eps;
  bool quant;
  Op emitted;
  Tensor sub, gate, x_new, scale, mean, rstd;
};
struct BothHeld {
  at::ScalarType x, gate, sub, scale, shift;
};

Tensor both_fwd(const Launch& l, const Tensor& x_, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                const Tensor& shift, BothCall& c) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_), sh = bf16_contiguous(shift);
  c.sub = bf16_contiguous(sub);
  c.gate = bf16_contiguous(gate);
  c.scale = bf16_contiguous(scale);
  c.x_new = like(x, l.dev);
  Tensor y = like(x, l.dev);
  c.mean = empty({r.n}, F32, l.dev);
  c.rstd = empty({r.n}, F32, l.dev);
  float *mean = c.mean.data_ptr<float>(), *rstd = c.rstd.data_ptr<float>();
  if (c.quant) {
    c.emitted = empty_op(r.n, r.d, l.dev);
    check(anima_gated_add_adaln_fwd_quant(x.data_ptr(), c.gate.data_ptr(), c.sub.data_ptr(), c.scale.data_ptr(),
                                          sh.data_ptr(), c.eps, r.n, r.hw, r.d, c.x_new.data_ptr(), y.data_ptr(), mean, rstd,
                                          ptr8(c.emitted.codes), ptr8(c.emitted.scales), ANIMA_SCALES_TILED, l.stream));
  } else {
    check(anima_gated_add_adaln_fwd(x.data_ptr(), c.gate.data_ptr(), c.sub.data_ptr(), c.scale.data_ptr(), sh.data_ptr(),
                                    c.eps, r.n, r.hw, r.d, c.x_new.data_ptr(), y.data_ptr(), mean, rstd, l.stream));
  }
  return y;
}

struct GatedAddAdaLN : Function<GatedAddAdaLN> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& sub,
                               const Tensor& scale, const Tensor& shift, BothCall* c) {
    const Launch l(x);
    Tensor y = both_fwd(l, x, gate, sub, scale, shift, *c);
    ctx->save_for_backward({c->sub, c->gate, c->x_new, c->scale, c->mean, c->rstd});
    ctx->set_materialize_grads(false);
    hold(ctx, BothHeld{x.scalar_type(), gate.scalar_type(), sub.scalar_type(), scale.scalar_type(), shift.scalar_type()});
    return {c->x_new, y};
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const BothHeld h = held<BothHeld>(ctx);
    variable_list out(6);
    const Tensor &d_xnew = grads[0], &d_y = grads[1];
    if (!d_xnew.defined() && !d_y.defined()) return out;
    const variable_list s = ctx->get_saved_variables();
    const Tensor &sub = s[0], &gate = s[1], &x_new = s[2], &scale = s[3], &mean = s[4], &rstd = s[5];
    const Launch l(x_new);
    Tensor dx, dsub, dscale, dshift, dgate;
    if (d_xnew.defined() && d_y.defined()) {      // the usual case: one kernel for both backward ops
      const Rows r = rows_of(x_new);
      const Tensor dy = bf16_contiguous(d_y), dn = bf16_contiguous(d_xnew);
      const int64_t bytes = check(anima_gated_add_adaln_bwd_workspace_bytes(r.n, r.hw, r.d));
      Tensor ws = empty({bytes}, U8, l.dev);
      dx = like(x_new, l.dev);
      dsub = like(x_new, l.dev);
      dscale = like(scale, l.dev);
      dshift = like(scale, l.dev);
      dgate = like(gate, l.dev);
      if (r.n)
        check(anima_gated_add_adaln_bwd(dy.data_ptr(), dn.data_ptr(), x_new.data_ptr(), scale.data_ptr(),
                                        mean.data_ptr<float>(), rstd.data_ptr<float>(), sub.data_ptr(), gate.data_ptr(), r.n,
                                        r.hw, r.d, dx.data_ptr(), dsub.data_ptr(), dscale.data_ptr(), dshift.data_ptr(),
                                        dgate.data_ptr(), ws.data_ptr(), bytes, l.stream));
    } else {
      dx = d_xnew;
      if (d_y.defined()) std::tie(dx, dscale, dshift) = adaln_bwd(l, d_y, x_new, scale, mean, rstd);
      std::tie(dsub, dgate) = gated_bwd(l, dx, sub, gate);
    }
    out[0] = back_to(dx, h.x);
    out[1] = back_to(dgate, h.gate);
    out[2] = back_to(dsub, h.sub);
    out[3] = back_to(dscale, h.scale);
    out[4] = back_to(dshift, h.shift);
    return out;
  }
};

// ------------------------------------------------------------------------------------------------ RMSNorm + RoPE
struct RopeCall {
  Tensor x, w, cos, sin, rstd;
  float eps;
};

Tensor rope_fwd(const Launch& l, const Tensor& x, const Tensor& weight, RopeCall& c) {
  TORCH_CHECK_TYPE(x.scalar_type() == BF16, "RMSNorm + RoPE needs bfloat16, got ", x.scalar_type());
  c.x = x.is_contiguous() ? x : x.detach().contiguous();
  c.w = weight.detach().to(F32).contiguous();
  const int64_t heads = x.size(-2), d = x.size(-1), tokens = x.numel() ? x.numel() / (heads * d) : 0;
  Tensor out = like(x, l.dev);
  c.rstd = empty({tokens * heads}, F32, l.dev);
  if (tokens)
    check(anima_rmsnorm_rope_fwd(c.x.data_ptr(), c.w.data_ptr<float>(), static_cast<float*>(ptr(c.cos)),
                                 static_cast<float*>(ptr(c.sin)), c.eps, tokens, heads, d, c.cos.defined() ? c.cos.size(0) : 1,
                                 out.data_ptr(), c.rstd.data_ptr<float>(), l.stream));
  return out;
}

struct RopeHeld {
  Tensor cos, sin;
};
struct RmsNormRope : Function<RmsNormRope> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, RopeCall* c) {
    const Launch l(x);
    Tensor out = rope_fwd(l, x, weight, *c);
    ctx->save_for_backward({c->x, c->w, c->rstd});
    hold(ctx, RopeHeld{c->cos, c->sin});
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const RopeHeld& h = held<RopeHeld>(ctx);
    const Tensor &x = s[0], &w = s[1], &rstd = s[2];
    const Launch l(x);
    const Tensor dout = bf16_contiguous(grads[0]);
    Tensor dx = like(x, l.dev);
    const int64_t heads = x.size(-2), d = x.size(-1), tokens = x.numel() ? x.numel() / (heads * d) : 0;
    if (tokens)
      check(anima_rmsnorm_rope_bwd(dout.data_ptr(), x.data_ptr(), w.data_ptr<float>(), static_cast<float*>(ptr(h.cos)),
                                   static_cast<float*>(ptr(h.sin)), rstd.data_ptr<float>(), tokens, heads, d,
                                   h.cos.defined() ? h.cos.size(0) : 1, dx.data_ptr(), l.stream));
    return {dx, Tensor(), Tensor()};
  }
};

}  // namespace

std::tuple<Tensor, Op> adaln(const Tensor& x, const Tensor& scale, const Tensor& shift, double eps, bool quant) {
  AdalnCall c{static_cast<float>(eps), quant};
  if (wants(x) || wants(scale) || wants(shift)) {
    Tensor y = AdaLN::apply(x, scale, shift, &c);
    return {y, c.emitted};
  }
  const Launch l(x);
  Tensor y = adaln_fwd(l, x, scale, shift, c);
  return {y, c.emitted};
}

Tensor gated_add(const Tensor& x, const Tensor& gate, const Tensor& y) {
  if (wants(x) || wants(gate) || wants(y)) return GatedAdd::apply(x, gate, y);
  const Launch l(x);
  return gated_fwd(l, x, bf16_contiguous(y), bf16_contiguous(gate));
}

std::tuple<Tensor, Tensor, Op> gated_add_adaln(const Tensor& x, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                                               const Tensor& shift, double eps, bool quant) {
  BothCall c{static_cast<float>(eps), quant};
  if (wants(x) || wants(gate) || wants(sub) || wants(scale) || wants(shift)) {
    variable_list r = GatedAddAdaLN::apply(x, gate, sub, scale, shift, &c);
    return {r[0], r[1], c.emitted};
  }
  const Launch l(x);
  Tensor y = both_fwd(l, x, gate, sub, scale, shift, c);
  return {c.x_new, y, c.emitted};
}

Tensor rmsnorm_rope(const Tensor& x, const Tensor& weight, const OptTensor& cos, const OptTensor& sin, double eps) {
  RopeCall c{Tensor(), Tensor(), cos.value_or(Tensor()), sin.value_or(Tensor()), Tensor(), static_cast<float>(eps)};
  if (wants(x)) return RmsNormRope::apply(x, weight, &c);
  const Launch l(x);
  return rope_fwd(l, x, weight, c);
}

}  // namespace anima_host
