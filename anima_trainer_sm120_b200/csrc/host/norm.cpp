#include "norm.h"

#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>

#include <mutex>

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

// The (B, T, 1, 1, D) modulation tensors of one call as the kernels take them: bf16 rows with one pitch. Chunks of a
// wider tensor (what a modulation MLP returns) are used where they lie; anything else is copied dense.
struct Mods {
  std::vector<Tensor> t;
  int64_t ld;
};
// pitch of the samples' rows; 0 = any (one sample), -1 = not usable in place
int64_t pitch_of(const Tensor& m) {
  if (m.scalar_type() != BF16 || m.dim() != 5 || m.stride(4) != 1 || m.size(2) * m.size(3) != 1 ||
      (reinterpret_cast<uintptr_t>(m.data_ptr()) & 15))
    return -1;
  const int64_t B = m.size(0), T = m.size(1);
  if (B * T == 1) return 0;
  if (B > 1 && T > 1 && m.stride(0) != T * m.stride(1)) return -1;
  const int64_t ld = T > 1 ? m.stride(1) : m.stride(0);
  return ld >= m.size(4) && ld % 8 == 0 ? ld : -1;
}
Mods mods_of(std::initializer_list<const Tensor*> ts) {
  Mods m{{}, 0};
  bool in_place = true;
  for (const Tensor* t : ts) {
    const int64_t ld = pitch_of(*t);
    if (ld < 0 || (ld && m.ld && ld != m.ld)) in_place = false;
    if (ld > 0) m.ld = ld;
  }
  if (!in_place || !m.ld) m.ld = (*ts.begin())->size(-1);
  for (const Tensor* t : ts) m.t.push_back(in_place ? *t : bf16_contiguous(*t));
  return m;
}
Tensor dense_like(const Tensor& t, const at::Device& dev) { return at::detail::empty_cuda(t.sizes(), BF16, dev, std::nullopt); }
Tensor scratch(int64_t bytes, const at::Device& dev) { return bytes ? empty({bytes}, U8, dev) : Tensor(); }

// ------------------------------------------------------------------------------------------------ AdaLN
struct AdalnOut {
  Tensor y, x, mean, rstd;      // x as the kernel read it
  Mods mods;                    // scale, shift
  Op emitted;
};
AdalnOut adaln_fwd(const Launch& l, const Tensor& x, const Tensor& scale, const Tensor& shift, float eps, bool quant) {
  const Rows r = rows_of(x);
  AdalnOut o{like(x, l.dev), bf16_contiguous(x), empty({r.n}, F32, l.dev), empty({r.n}, F32, l.dev), mods_of({&scale, &shift}), {}};
  if (quant) o.emitted = empty_op(r.n, r.d, l.dev);
  check(anima_adaln_fwd_ex(o.x.data_ptr(), nullptr, nullptr, o.mods.t[0].data_ptr(), o.mods.t[1].data_ptr(), o.mods.ld, eps, r.n,
                           r.hw, r.d, nullptr, o.y.data_ptr(), o.mean.data_ptr<float>(), o.rstd.data_ptr<float>(),
                           ptr8(o.emitted.codes), ptr8(o.emitted.scales), ANIMA_SCALES_TILED, l.stream));
  return o;
}

// dx (+ d_res, another gradient of x), dscale, dshift (undefined unless `mod`)
std::tuple<Tensor, Tensor, Tensor> adaln_bwd(const Launch& l, const Tensor& dy_, const Tensor& d_res_, const Tensor& x,
                                             const Tensor& scale, int64_t ld, const Tensor& mean, const Tensor& rstd,
                                             bool mod) {
  const Rows r = rows_of(x);
  const Tensor dy = bf16_contiguous(dy_), d_res = d_res_.defined() ? bf16_contiguous(d_res_) : Tensor();
  Tensor dx = like(x, l.dev), ds, db;
  const int64_t bytes = mod ? check(anima_adaln_bwd_workspace_bytes(r.n, r.hw, r.d)) : 0;
  const Tensor ws = scratch(bytes, l.dev);
  if (mod) {
    ds = dense_like(scale, l.dev);
    db = dense_like(scale, l.dev);
  }
  check(anima_adaln_bwd_ex(dy.data_ptr(), ptr(d_res), x.data_ptr(), scale.data_ptr(), nullptr, nullptr, ld,
                           mean.data_ptr<float>(), rstd.data_ptr<float>(), r.n, r.hw, r.d, dx.data_ptr(), nullptr, ptr(ds),
                           ptr(db), nullptr, ptr(ws), bytes, l.stream));
  return {dx, ds, db};
}

std::pair<Tensor, Tensor> gated_bwd(const Launch& l, const Tensor& dout_, const Tensor& y, const Tensor& gate, int64_t ld,
                                    bool mod) {
  const Rows r = rows_of(y);
  const Tensor dout = bf16_contiguous(dout_);
  const int64_t bytes = mod ? check(anima_gated_add_bwd_workspace_bytes(r.n, r.hw, r.d)) : 0;
  const Tensor ws = scratch(bytes, l.dev);
  Tensor dy = like(y, l.dev), dg;
  if (mod) dg = dense_like(gate, l.dev);
  check(anima_gated_add_bwd_ex(dout.data_ptr(), y.data_ptr(), gate.data_ptr(), ld, r.n, r.hw, r.d, dy.data_ptr(), ptr(dg),
                               ptr(ws), bytes, l.stream));
  return {dy, dg};
}

// The node has a second output slot, an alias of x: the gated residual that reads the same x right after its
// modulation (every sublayer does) takes its x from there, so its gradient arrives here and dx = that + dx_ln is one
// kernel instead of two and an addition (3 passes over a gradient). Values are those of the separate addition.
struct AdalnNode : public torch::autograd::Node {
  torch::autograd::SavedVariable x, scale, mean, rstd;
  int64_t ld;
  at::ScalarType dt_x, dt_scale, dt_shift;
  bool used = false;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!g[0].defined()) {      // only the alias was used: nothing of this node's own
      out[0] = g[1];
      return out;
    }
    used = true;
    const auto self = getptr();
    const Tensor xs = x.unpack(self), sc = scale.unpack(self), mu = mean.unpack(self), rs = rstd.unpack(self);
    const Launch l(xs);
    const bool mod = task_should_compute_output(1) || task_should_compute_output(2);
    auto [dx, ds, db] = adaln_bwd(l, g[0], g[1], xs, sc, ld, mu, rs, mod);
    out[0] = back_to(dx, dt_x);
    out[1] = back_to(ds, dt_scale);
    out[2] = back_to(db, dt_shift);
    return out;
  }
  // A pass that only went through the alias leaves the saved tensors for the one that needs them.
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!used) return;
    for (auto* v : {&x, &scale, &mean, &rstd}) v->reset_data();
  }
  std::string name() const override { return "FusedAdaLNBackward"; }
};

// The x last modulated on this thread and its node (both weak).
struct Modulated {
  c10::weak_intrusive_ptr<c10::TensorImpl> x{c10::intrusive_ptr<c10::TensorImpl>()};
  uint32_t version = 0;
  std::weak_ptr<torch::autograd::Node> node;
};
thread_local Modulated modulated;

void remember(const Tensor& x, const std::shared_ptr<torch::autograd::Node>& node) {
  modulated.x = c10::weak_intrusive_ptr<c10::TensorImpl>(x.getIntrusivePtr());
  modulated.version = x.unsafeGetTensorImpl()->version_counter().current_version();
  modulated.node = node;
}
// x, or its alias whose gradient goes to the modulation's node
Tensor through_modulation(const Tensor& x) {
  if (!wants(x) || x.is_inference()) return x;
  const auto node = modulated.node.lock();
  const auto was = modulated.x.lock();
  if (!node || was.get() != x.unsafeGetTensorImpl() ||
      x.unsafeGetTensorImpl()->version_counter().current_version() != modulated.version)
    return x;
  modulated.node.reset();
  Tensor alias(x.unsafeGetTensorImpl()->shallow_copy_and_detach(x.unsafeGetTensorImpl()->version_counter(), true));
  torch::autograd::impl::set_gradient_edge(alias, torch::autograd::Edge(node, 1));
  return alias;
}

// ------------------------------------------------------------------------------------------------ gated residual
struct GatedHeld {
  at::ScalarType x, gate, y;
  int64_t ld;
  bool mod;
};
Tensor gated_fwd(const Launch& l, const Tensor& x_, const Tensor& y, const Mods& gate) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_);
  Tensor out = like(x, l.dev);
  check(anima_gated_add_fwd_ex(x.data_ptr(), gate.t[0].data_ptr(), gate.ld, y.data_ptr(), r.n, r.hw, r.d, out.data_ptr(),
                               l.stream));
  return out;
}

struct GatedAdd : Function<GatedAdd> {
  static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& y, bool mod) {
    const Launch l(x);
    const Tensor yc = bf16_contiguous(y);
    const Mods g = mods_of({&gate});
    ctx->save_for_backward({yc, g.t[0]});
    hold(ctx, GatedHeld{x.scalar_type(), gate.scalar_type(), y.scalar_type(), g.ld, mod});
    return gated_fwd(l, x, yc, g);
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const variable_list s = ctx->get_saved_variables();
    const GatedHeld h = held<GatedHeld>(ctx);
    const Launch l(s[0]);
    auto [dy, dg] = gated_bwd(l, grads[0], s[0], s[1], h.ld, h.mod);
    return {grads[0], back_to(dg, h.gate), back_to(dy, h.y), Tensor()};
  }
};

// ------------------------------------------------------------------------------------------------ both at once
struct BothCall {
  float eps;
  bool quant, mod;
  Op emitted;
  Tensor sub, x_new, mean, rstd;
  Mods mods;      // gate, scale, shift
};
struct BothHeld {
  at::ScalarType x, gate, sub, scale, shift;
  int64_t ld;
  bool mod;
};

Tensor both_fwd(const Launch& l, const Tensor& x_, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                const Tensor& shift, BothCall& c) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_);
  c.sub = bf16_contiguous(sub);
  c.mods = mods_of({&gate, &scale, &shift});
  c.x_new = like(x, l.dev);
  Tensor y = like(x, l.dev);
  c.mean = empty({r.n}, F32, l.dev);
  c.rstd = empty({r.n}, F32, l.dev);
  if (c.quant) c.emitted = empty_op(r.n, r.d, l.dev);
  check(anima_adaln_fwd_ex(x.data_ptr(), c.mods.t[0].data_ptr(), c.sub.data_ptr(), c.mods.t[1].data_ptr(),
                           c.mods.t[2].data_ptr(), c.mods.ld, c.eps, r.n, r.hw, r.d, c.x_new.data_ptr(), y.data_ptr(),
                           c.mean.data_ptr<float>(), c.rstd.data_ptr<float>(), ptr8(c.emitted.codes), ptr8(c.emitted.scales),
                           ANIMA_SCALES_TILED, l.stream));
  return y;
}

struct GatedAddAdaLN : Function<GatedAddAdaLN> {
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& sub,
                               const Tensor& scale, const Tensor& shift, BothCall* c) {
    const Launch l(x);
    Tensor y = both_fwd(l, x, gate, sub, scale, shift, *c);
    ctx->save_for_backward({c->sub, c->mods.t[0], c->x_new, c->mods.t[1], c->mean, c->rstd});
    ctx->set_materialize_grads(false);
    hold(ctx, BothHeld{x.scalar_type(), gate.scalar_type(), sub.scalar_type(), scale.scalar_type(), shift.scalar_type(),
                       c->mods.ld, c->mod});
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
      const int64_t bytes = h.mod ? check(anima_gated_add_adaln_bwd_workspace_bytes(r.n, r.hw, r.d)) : 0;
      const Tensor ws = scratch(bytes, l.dev);
      dx = like(x_new, l.dev);
      dsub = like(x_new, l.dev);
      if (h.mod) {
        dscale = dense_like(scale, l.dev);
        dshift = dense_like(scale, l.dev);
        dgate = dense_like(gate, l.dev);
      }
      check(anima_adaln_bwd_ex(dy.data_ptr(), dn.data_ptr(), x_new.data_ptr(), scale.data_ptr(), gate.data_ptr(),
                               sub.data_ptr(), h.ld, mean.data_ptr<float>(), rstd.data_ptr<float>(), r.n, r.hw, r.d,
                               dx.data_ptr(), dsub.data_ptr(), ptr(dscale), ptr(dshift), ptr(dgate), ptr(ws), bytes,
                               l.stream));
    } else {
      dx = d_xnew;
      if (d_y.defined())
        std::tie(dx, dscale, dshift) = adaln_bwd(l, d_y, Tensor(), x_new, scale, h.ld, mean, rstd, h.mod);
      std::tie(dsub, dgate) = gated_bwd(l, dx, sub, gate, h.ld, h.mod);
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
  const bool grad = wants(x) || wants(scale) || wants(shift);
  const Launch l(x);
  AdalnOut o;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    o = adaln_fwd(l, x, scale, shift, static_cast<float>(eps), quant);
  }
  if (grad) {
    auto node = std::shared_ptr<AdalnNode>(new AdalnNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x, scale, shift));
    node->x = {o.x, false};
    node->scale = {o.mods.t[0], false};
    node->mean = {o.mean, false};
    node->rstd = {o.rstd, false};
    node->ld = o.mods.ld;
    node->dt_x = x.scalar_type();
    node->dt_scale = scale.scalar_type();
    node->dt_shift = shift.scalar_type();
    torch::autograd::set_history(o.y, node);
    node->add_input_metadata(x);
    if (x.requires_grad() && !x.is_inference()) remember(x, node);
  }
  return {o.y, o.emitted};
}

Tensor gated_add(const Tensor& x, const Tensor& gate, const Tensor& y) {
  if (wants(x) || wants(gate) || wants(y)) return GatedAdd::apply(through_modulation(x), gate, y, wants(gate));
  const Launch l(x);
  return gated_fwd(l, x, bf16_contiguous(y), mods_of({&gate}));
}

std::tuple<Tensor, Tensor, Op> gated_add_adaln(const Tensor& x, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                                               const Tensor& shift, double eps, bool quant) {
  const bool mod = wants(gate) || wants(scale) || wants(shift);
  BothCall c{static_cast<float>(eps), quant, mod};
  if (mod || wants(x) || wants(sub)) {
    variable_list r = GatedAddAdaLN::apply(through_modulation(x), gate, sub, scale, shift, &c);
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
