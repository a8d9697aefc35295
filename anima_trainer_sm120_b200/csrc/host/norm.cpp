#include "norm.h"

namespace anima_host {

using torch::autograd::set_history;

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

// The modulation tensors of one call as the kernels take them: bf16 rows of d with one pitch. (B, T, 1, 1, d) tensors, also
// chunks of a wider tensor (what a modulation MLP returns), are used where they lie; any other shape with as many elements
// is read in order, as dense rows. Backward asks again for what it unpacks: a saved-tensor hook may hand a chunk back dense.
struct Mods {
  std::vector<Tensor> t;
  int64_t ld;
};
// pitch of the samples' rows; 0 = any (one sample), -1 = not usable in place
int64_t pitch_of(const Tensor& m, int64_t d) {
  if (m.scalar_type() != BF16 || m.dim() != 5 || m.size(4) != d || m.stride(4) != 1 || m.size(2) * m.size(3) != 1 ||
      (reinterpret_cast<uintptr_t>(m.data_ptr()) & 15))
    return -1;
  const int64_t B = m.size(0), T = m.size(1);
  if (B * T == 1) return 0;
  if (B > 1 && T > 1 && m.stride(0) != T * m.stride(1)) return -1;
  const int64_t ld = T > 1 ? m.stride(1) : m.stride(0);
  return ld >= d && ld % 8 == 0 ? ld : -1;
}
Mods mods_of(int64_t d, std::initializer_list<const Tensor*> ts) {
  Mods m{{}, 0};
  bool in_place = true;
  const int64_t n = (*ts.begin())->numel();
  for (const Tensor* t : ts) {
    TORCH_CHECK_VALUE(t->numel() == n, "modulation tensors of different sizes");
    const int64_t ld = pitch_of(*t, d);
    if (ld < 0 || (ld && m.ld && ld != m.ld)) in_place = false;
    if (ld > 0) m.ld = ld;
  }
  if (!in_place || !m.ld) m.ld = d;
  for (const Tensor* t : ts) m.t.push_back(in_place ? *t : bf16_contiguous(*t));
  return m;
}
Tensor dense_like(const Tensor& t, const at::Device& dev) { return at::detail::empty_cuda(t.sizes(), BF16, dev, std::nullopt); }
Tensor scratch(int64_t bytes, const at::Device& dev) { return bytes ? empty({bytes}, U8, dev) : Tensor(); }

// ------------------------------------------------------------------------------------------------ AdaLN
struct AdalnOut {
  Tensor y, x, stats;           // x as the kernel read it; mean and rstd of its rows
  Mods mods;                    // scale, shift
  Op emitted;
};
AdalnOut adaln_fwd(const Launch& l, const Tensor& x, const Tensor& scale, const Tensor& shift, float eps, bool quant) {
  const Rows r = rows_of(x);
  AdalnOut o{like(x, l.dev), bf16_contiguous(x), empty({2, r.n}, F32, l.dev), mods_of(r.d, {&scale, &shift}), {}};
  float* stats = o.stats.data_ptr<float>();
  if (quant) o.emitted = empty_op(r.n, r.d, l.dev);
  check(anima_adaln_fwd_ex(o.x.data_ptr(), nullptr, nullptr, o.mods.t[0].data_ptr(), o.mods.t[1].data_ptr(), o.mods.ld, eps, r.n,
                           r.hw, r.d, nullptr, o.y.data_ptr(), stats, stats + r.n, o.emitted.codes, o.emitted.scales, ANIMA_SCALES_TILED, l.stream));
  return o;
}

// dx (+ d_res, another gradient of x), dscale, dshift (undefined unless `mod`)
std::tuple<Tensor, Tensor, Tensor> adaln_bwd(const Launch& l, const Tensor& dy_, const Tensor& d_res_, const Tensor& x,
                                             const Tensor& scale, int64_t ld, const Tensor& stats_, bool mod) {
  const Rows r = rows_of(x);
  const Tensor dy = bf16_contiguous(dy_), d_res = d_res_.defined() ? bf16_contiguous(d_res_) : Tensor();
  const float* stats = stats_.data_ptr<float>();
  Tensor dx = like(x, l.dev), ds, db;
  const int64_t bytes = mod ? check(anima_adaln_bwd_ex_workspace_bytes(r.n, r.hw, r.d, 2)) : 0;
  const Tensor ws = scratch(bytes, l.dev);
  if (mod) {
    ds = dense_like(scale, l.dev);
    db = dense_like(scale, l.dev);
  }
  check(anima_adaln_bwd_ex(dy.data_ptr(), ptr(d_res), x.data_ptr(), scale.data_ptr(), nullptr, nullptr, ld,
                           stats, stats + r.n, r.n, r.hw, r.d, dx.data_ptr(), nullptr, ptr(ds), ptr(db), nullptr, ptr(ws), bytes, l.stream));
  return {dx, ds, db};
}

std::pair<Tensor, Tensor> gated_bwd(const Launch& l, const Tensor& dout_, const Tensor& y, const Tensor& gate, int64_t ld,
                                    bool mod) {
  const Rows r = rows_of(y);
  const Tensor dout = bf16_contiguous(dout_);
  const int64_t bytes = mod ? check(anima_adaln_bwd_ex_workspace_bytes(r.n, r.hw, r.d, 1)) : 0;
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
struct AdalnNode : public HostNode {      // saves x, scale, statistics
  at::ScalarType dt_x, dt_scale, dt_shift;
  bool used = false;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(3);
    if (!g[0].defined() && g[1].defined()) {      // only the alias was used: nothing of this node's own
      out[0] = g[1];
      return out;
    }
    used = true;
    const Tensor x = get(0), scale = get(1), stats = get(2);
    const Launch l(x);
    const Mods m = mods_of(x.size(-1), {&scale});
    const bool mod = task_should_compute_output(1) || task_should_compute_output(2);
    auto [dx, ds, db] = adaln_bwd(l, grad_of(g, 0), g[1], x, m.t[0], m.ld, stats, mod);
    out[0] = back_to(dx, dt_x);
    out[1] = back_to(ds, dt_scale);
    out[2] = back_to(db, dt_shift);
    return out;
  }
  // A pass that only went through the alias leaves the saved tensors for the one that needs them.
  void release_variables() override {
    if (used) HostNode::release_variables();
  }
  std::string name() const override { return "FusedAdaLNBackward"; }
};

thread_local LastNode<torch::autograd::Node> modulated;

// x, or its alias whose gradient goes to the modulation's node
Tensor through_modulation(const Tensor& x) {
  if (!wants(x) || x.is_inference()) return x;
  const auto node = modulated.get(x);
  if (!node) return x;
  modulated.node.reset();
  Tensor alias(x.unsafeGetTensorImpl()->shallow_copy_and_detach(x.unsafeGetTensorImpl()->version_counter(), true));
  torch::autograd::impl::set_gradient_edge(alias, torch::autograd::Edge(node, 1));
  return alias;
}

// ------------------------------------------------------------------------------------------------ gated residual
Tensor gated_fwd(const Launch& l, const Tensor& x_, const Tensor& y, const Mods& gate) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_);
  Tensor out = like(x, l.dev);
  check(anima_gated_add_fwd_ex(x.data_ptr(), gate.t[0].data_ptr(), gate.ld, y.data_ptr(), r.n, r.hw, r.d, out.data_ptr(),
                               l.stream));
  return out;
}

struct GatedNode : public HostNode {      // saves y, gate
  at::ScalarType dt_gate, dt_y;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    const Tensor dout = grad_of(g, 0), y = get(0), gate = get(1);
    const Launch l(y);
    const Mods m = mods_of(y.size(-1), {&gate});
    auto [dy, dg] = gated_bwd(l, dout, y, m.t[0], m.ld, task_should_compute_output(1));
    return {dout, back_to(dg, dt_gate), back_to(dy, dt_y)};
  }
  std::string name() const override { return "FusedGatedAddBackward"; }
};

// ------------------------------------------------------------------------------------------------ both at once
struct Both {
  Tensor x_new, y, sub, stats;
  Mods mods;      // gate, scale, shift
  Op emitted;
};

Both both_fwd(const Launch& l, const Tensor& x_, const Tensor& gate, const Tensor& sub, const Tensor& scale,
              const Tensor& shift, float eps, bool quant) {
  const Rows r = rows_of(x_);
  const Tensor x = bf16_contiguous(x_);
  Both c{like(x, l.dev), like(x, l.dev), bf16_contiguous(sub), empty({2, r.n}, F32, l.dev), mods_of(r.d, {&gate, &scale, &shift}), {}};
  float* stats = c.stats.data_ptr<float>();
  if (quant) c.emitted = empty_op(r.n, r.d, l.dev);
  check(anima_adaln_fwd_ex(x.data_ptr(), c.mods.t[0].data_ptr(), c.sub.data_ptr(), c.mods.t[1].data_ptr(),
                           c.mods.t[2].data_ptr(), c.mods.ld, eps, r.n, r.hw, r.d, c.x_new.data_ptr(), c.y.data_ptr(), stats,
                           stats + r.n, c.emitted.codes, c.emitted.scales, ANIMA_SCALES_TILED, l.stream));
  return c;
}

struct BothNode : public HostNode {      // saves sub, gate, x_new, scale, statistics
  at::ScalarType dt_gate, dt_sub, dt_scale, dt_shift;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(5);
    const Tensor &d_y = grads[1], d_xnew = grads[0].defined() || d_y.defined() ? grads[0] : grad_of(grads, 0);
    const Tensor sub = get(0), x_new = get(2), stats = get(4), saved_gate = get(1), saved_scale = get(3);
    const Launch l(x_new);
    const Mods m = mods_of(x_new.size(-1), {&saved_gate, &saved_scale});
    const Tensor &gate = m.t[0], &scale = m.t[1];
    const int64_t ld = m.ld;
    const bool mod = task_should_compute_output(1) || task_should_compute_output(3) || task_should_compute_output(4);
    Tensor dx, dsub, dscale, dshift, dgate;
    if (d_xnew.defined() && d_y.defined()) {      // the usual case: one kernel for both backward ops
      const Rows r = rows_of(x_new);
      const Tensor dy = bf16_contiguous(d_y), dn = bf16_contiguous(d_xnew);
      const int64_t bytes = mod ? check(anima_adaln_bwd_ex_workspace_bytes(r.n, r.hw, r.d, 3)) : 0;
      const Tensor ws = scratch(bytes, l.dev);
      const float* st = stats.data_ptr<float>();
      dx = like(x_new, l.dev);
      dsub = like(x_new, l.dev);
      if (mod) {
        dscale = dense_like(scale, l.dev);
        dshift = dense_like(scale, l.dev);
        dgate = dense_like(gate, l.dev);
      }
      check(anima_adaln_bwd_ex(dy.data_ptr(), dn.data_ptr(), x_new.data_ptr(), scale.data_ptr(), gate.data_ptr(),
                               sub.data_ptr(), ld, st, st + r.n, r.n, r.hw, r.d, dx.data_ptr(), dsub.data_ptr(), ptr(dscale),
                               ptr(dshift), ptr(dgate), ptr(ws), bytes, l.stream));
    } else {
      dx = d_xnew;
      if (d_y.defined()) {
        std::tie(dx, dscale, dshift) = adaln_bwd(l, d_y, Tensor(), x_new, scale, ld, stats, mod);
      } else if (mod) {          // no gradient reached y: zeros, as for any output of a node that runs
        dscale = at::zeros_like(scale, at::MemoryFormat::Contiguous);
        dshift = at::zeros_like(scale, at::MemoryFormat::Contiguous);
      }
      std::tie(dsub, dgate) = gated_bwd(l, dx, sub, gate, ld, mod);
    }
    out[0] = dx;
    out[1] = back_to(dgate, dt_gate);
    out[2] = back_to(dsub, dt_sub);
    out[3] = back_to(dscale, dt_scale);
    out[4] = back_to(dshift, dt_shift);
    return out;
  }
  std::string name() const override { return "FusedGatedAddAdaLNBackward"; }
};

// ------------------------------------------------------------------------------------------------ RMSNorm + RoPE
// Saves x and rstd. A bf16 norm weight is copied by the forward kernel, behind rstd: it may change before backward (as when
// the node converted it). An fp32 one is read in place and may not.
struct RopeNode : public HostNode {
  Kept weight;
  int64_t copy_at = -1;         // place of that copy in rstd
  Tensor cos, sin;

  variable_list apply(variable_list&& g) override {
    std::lock_guard<std::mutex> lock(mutex_);
    if (!task_should_compute_output(0)) return variable_list(1);
    const Tensor dout = bf16_contiguous(grad_of(g, 0)), x = get(0), rstd = get(1);
    const bool copied = copy_at >= 0;
    const void* w = copied ? rstd.data_ptr<float>() + copy_at : weight.get().data_ptr();
    const Launch l(x);
    Tensor dx = like(x, l.dev);
    const int64_t heads = x.size(-2), d = x.size(-1), tokens = x.numel() ? x.numel() / (heads * d) : 0;
    if (tokens)
      check(anima_rmsnorm_rope_bwd_ex(dout.data_ptr(), x.data_ptr(), w, copied,
                                      static_cast<float*>(ptr(cos)), static_cast<float*>(ptr(sin)), rstd.data_ptr<float>(),
                                      tokens, heads, d, cos.defined() ? cos.size(0) : 1, dx.data_ptr(), l.stream));
    return {dx};
  }
  std::string name() const override { return "FusedRMSNormRoPEBackward"; }
};

}  // namespace

std::tuple<Tensor, Op> adaln(const Tensor& x, const Tensor& scale, const Tensor& shift, double eps, bool quant) {
  const bool grad = wants(x) || wants(scale) || wants(shift);
  const Launch l(x);
  admit(l, x, scale, shift);
  AdalnOut o;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    o = adaln_fwd(l, x, scale, shift, static_cast<float>(eps), quant);
  }
  if (grad) {
    auto node = make_node<AdalnNode>(x, scale, shift);
    node->save(o.x);
    node->save(o.mods.t[0]);
    node->save(o.stats);
    node->dt_x = x.scalar_type();
    node->dt_scale = scale.scalar_type();
    node->dt_shift = shift.scalar_type();
    set_history(o.y, node);
    node->add_input_metadata(x);
    if (x.requires_grad() && !x.is_inference()) modulated.set(x, node);
  }
  return {o.y, o.emitted};
}

Tensor gated_add(const Tensor& x_, const Tensor& gate, const Tensor& y) {
  const bool grad = wants(x_) || wants(gate) || wants(y);
  const Launch l(x_);
  admit(l, x_, gate, y);
  const Tensor x = grad ? through_modulation(x_) : x_;
  Tensor out, yc;
  Mods g;
  {
    Below below;
    yc = bf16_contiguous(y);
    g = mods_of(x.size(-1), {&gate});
    out = gated_fwd(l, x, yc, g);
  }
  if (grad) {
    auto node = make_node<GatedNode>(x, gate, y);
    node->save(yc);
    node->save(g.t[0]);
    node->dt_gate = gate.scalar_type();
    node->dt_y = y.scalar_type();
    set_history(out, node);
  }
  return out;
}

std::tuple<Tensor, Tensor, Op> gated_add_adaln(const Tensor& x_, const Tensor& gate, const Tensor& sub, const Tensor& scale,
                                               const Tensor& shift, double eps, bool quant) {
  const bool grad = wants(x_) || wants(sub) || wants(gate) || wants(scale) || wants(shift);
  const Launch l(x_);
  admit(l, x_, gate, sub, scale, shift);
  const Tensor x = grad ? through_modulation(x_) : x_;
  Both c;
  {
    Below below;
    c = both_fwd(l, x, gate, sub, scale, shift, static_cast<float>(eps), quant);
  }
  if (grad) {
    auto node = make_node<BothNode>(x, gate, sub, scale, shift);
    set_history(c.x_new, node);
    set_history(c.y, node);
    node->save(c.sub);
    node->save(c.mods.t[0]);
    node->save(c.x_new, true);
    node->save(c.mods.t[1]);
    node->save(c.stats);
    node->dt_gate = gate.scalar_type();
    node->dt_sub = sub.scalar_type();
    node->dt_scale = scale.scalar_type();
    node->dt_shift = shift.scalar_type();
  }
  return {c.x_new, c.y, c.emitted};
}

Tensor rmsnorm_rope(const Tensor& x, const Tensor& weight, const OptTensor& cos, const OptTensor& sin, double eps) {
  TORCH_CHECK_TYPE(x.scalar_type() == BF16, "RMSNorm + RoPE needs bfloat16, got ", x.scalar_type());
  const Launch l(x);
  admit(l, x, weight, cos, sin);
  const int64_t heads = x.size(-2), d = x.size(-1), tokens = x.numel() ? x.numel() / (heads * d) : 0;
  const bool grad = any_wants(x, weight, cos, sin), copied = grad && weight.scalar_type() == BF16;
  TORCH_CHECK_VALUE(weight.numel() >= d, "norm weight of ", weight.numel(), " elements for heads of ", d);
  const int64_t copy_at = (tokens * heads + 3) / 4 * 4;
  Tensor out, xc, w, rstd;
  {
    Below below;
    xc = x.is_contiguous() ? x : x.detach().contiguous();
    w = weight.scalar_type() == BF16 || weight.scalar_type() == F32 ? weight : weight.detach().to(F32);
    if (!w.is_contiguous() || (reinterpret_cast<uintptr_t>(w.data_ptr()) & 15)) w = w.detach().clone(at::MemoryFormat::Contiguous);
    out = like(x, l.dev);
    rstd = empty({copied ? copy_at + d / 2 : tokens * heads}, F32, l.dev);
    if (tokens)
      check(anima_rmsnorm_rope_fwd_keep(xc.data_ptr(), w.data_ptr(), w.scalar_type() == BF16, static_cast<float*>(ptr(cos)),
                                        static_cast<float*>(ptr(sin)), static_cast<float>(eps), tokens, heads, d,
                                        cos ? cos->size(0) : 1, out.data_ptr(), rstd.data_ptr<float>(),
                                        copied ? rstd.data_ptr<float>() + copy_at : nullptr, l.stream));
  }
  if (grad) {
    auto node = make_node<RopeNode>(x);
    node->save(xc);
    node->save(rstd);
    if (copied) node->copy_at = copy_at;
    else node->weight = Kept(w);
    node->cos = cos.value_or(Tensor());
    node->sin = sin.value_or(Tensor());
    set_history(out, node);
  }
  return out;
}

}  // namespace anima_host
