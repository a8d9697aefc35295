// Python binding of the native host path (anima_trainer_sm120_b200._host). MXFP8 operands cross the boundary as
// (codes, scales) tensor pairs; every call runs without the interpreter lock.
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/utils/pybind.h>

#include "linear.h"
#include "norm.h"
#include "tlokr.h"

namespace py = pybind11;
using namespace anima_host;

namespace {

using O = const OptTensor&;
// an operand as Python holds it: codes, scales and the allocation both lie in (or nothing)
using Triple = std::tuple<OptTensor, OptTensor, OptTensor>;
Triple triple_of(const Op& o, int layout = ANIMA_SCALES_TILED) {
  if (!o.defined()) return {};
  auto [codes, scales] = tensors_of(o, layout);
  return {codes, scales, o.other.defined() ? OptTensor() : OptTensor(o.store)};
}

std::pair<Triple, Triple> py_quantize(const Tensor& x, bool row, bool col, int layout) {
  TORCH_CHECK_TYPE(x.scalar_type() == BF16, "x must be bfloat16, got ", x.scalar_type());
  TORCH_CHECK_VALUE(x.dim() == 2, "x must be 2-D, got shape ", x.sizes());
  const Launch l(x);
  auto [r, c] = quantize(l, as_matrix(x, x.size(1)), row, col, layout);
  return {triple_of(r, layout), triple_of(c, layout)};
}

Tensor py_gemm(const Tensor& ac, const Tensor& as, const Tensor& bc, const Tensor& bs, const OptTensor& bias) {
  const Launch l(ac);
  TORCH_CHECK(bc.device() == l.dev && as.device() == l.dev && bs.device() == l.dev, "tensors on different devices");
  TORCH_CHECK(!bias || bias->device() == l.dev, "tensors on different devices");
  const Op a = op_of(ac, as), b = op_of(bc, bs);
  TORCH_CHECK_VALUE(!bias || (bias->scalar_type() == BF16 && bias->numel() == b.rows && bias->is_contiguous()),
                    "bias must be contiguous bfloat16 of length N");
  Tensor c = empty({a.rows, b.rows}, BF16, l.dev);
  gemm(l, a, b, {c.data_ptr(), b.rows, false}, ptr(bias));
  return c;
}

Tensor py_retile(const Tensor& scales, int64_t rows, int64_t k) {
  const Launch l(scales);
  const Tensor s = scales.is_contiguous() ? scales : scales.contiguous();
  Tensor t = empty({tiled_bytes(rows, k)}, U8, l.dev);
  check(anima_mx_scales_retile(ptr8(s), rows, k, ptr8(t), l.stream));
  return t;
}

Tensor py_lokr(const Tensor& x, O xrc, O xrs, O xr, O xcc, O xcs, O xc, const Tensor& W, O bias, const Tensor& w1,
               const Tensor& w2, double alpha, bool first) {
  return lokr_linear(x, op_of(xrc, xrs, xr), op_of(xcc, xcs, xc), W, bias, w1, w2, alpha, first);
}
Tensor py_merged(const Tensor& x, O xrc, O xrs, O xr, O xcc, O xcs, O xc, const Tensor& merged, O bias, bool first) {
  return merged_linear(x, op_of(xrc, xrs, xr), op_of(xcc, xcs, xc), merged, bias, first);
}
Tensor py_frozen(const Tensor& x, O xrc, O xrs, O xr, O wrc, O wrs, O wr, O wcc, O wcs, O wc, O w_bf16, O bias,
                 bool save_weight) {
  return frozen_linear(x, op_of(xrc, xrs, xr), op_of(wrc, wrs, wr), op_of(wcc, wcs, wc), w_bf16, bias, save_weight);
}
Tensor py_lokr_mlp(const Tensor& x, O xrc, O xrs, O xr, O xcc, O xcs, O xc, const Tensor& W1, O b1, const Tensor& w1a,
                   const Tensor& w2a, double alpha1, const Tensor& W2, O b2, const Tensor& w1b, const Tensor& w2b,
                   double alpha2, bool first) {
  return lokr_mlp(x, op_of(xrc, xrs, xr), op_of(xcc, xcs, xc), W1, b1, w1a, w2a, alpha1, W2, b2, w1b, w2b, alpha2, first);
}

TLinear py_tlinear(const Tensor& wrc, const Tensor& wrs, O wcc, O wcs, O bias, const Tensor& w1,
                   const Tensor& a, const Tensor& b, O mask, double alpha, const Tensor& c, const std::vector<Tensor>& forms,
                   bool fold, bool fuse_mix) {
  TORCH_CHECK_VALUE(forms.size() == 8 || forms.size() == 10, "T-LoKr factor forms: 8 or 10 tensors");
  OptTensor m = mask;
  if (m) m = bf16_contiguous(*m);
  TLinear t{op_of(wrc, wrs), op_of(wcc, wcs, std::nullopt), bias, w1, a, b, m, mask ? Kept(*mask) : Kept(), alpha, c, op_of(forms[0], forms[1]),
            op_of(forms[2], forms[3]), op_of(forms[4], forms[5]), op_of(forms[6], forms[7]), {}, fold, fuse_mix};
  if (forms.size() == 10) t.a_scaled = op_of(forms[8], forms[9]);
  return t;
}
Tensor py_tlokr(const Tensor& x, O xrc, O xrs, O xr, const TLinear& t, bool first) {
  return tlokr_linear(x, op_of(xrc, xrs, xr), t, first);
}
Tensor py_tlokr_mlp(const Tensor& x, O xrc, O xrs, O xr, const TLinear& t1, const TLinear& t2, bool first) {
  return tlokr_mlp(x, op_of(xrc, xrs, xr), t1, t2, first);
}
Tensor py_tlokr_fwd(const Tensor& xc, const Tensor& xs, const Tensor& gc, const Tensor& gs, const std::vector<int64_t>& lead,
                    const TLinear& t) {
  return tlokr_forward_only(op_of(xc, xs), op_of(gc, gs), lead, t);
}
std::vector<Tensor> py_tlokr_bwd(const std::vector<Tensor>& g, const std::vector<Tensor>& x, const std::vector<int64_t>& lead,
                                 const TLinear& t) {
  return tlokr_backward_only(op_of(g.at(0), g.at(1)), op_of(g.at(2), g.at(3)), op_of(x.at(0), x.at(1)),
                             op_of(x.at(2), x.at(3)), lead, t);
}

std::tuple<Tensor, Triple> py_adaln(const Tensor& x, const Tensor& scale, const Tensor& shift, double eps, bool quant) {
  auto [y, op] = adaln(x, scale, shift, eps, quant);
  return {y, triple_of(op)};
}
std::tuple<Tensor, Tensor, Triple> py_gated_add_adaln(const Tensor& x, const Tensor& gate, const Tensor& sub,
                                                      const Tensor& scale, const Tensor& shift, double eps, bool quant) {
  auto [n, y, op] = gated_add_adaln(x, gate, sub, scale, shift, eps, quant);
  return {n, y, triple_of(op)};
}

}  // namespace

#define ANIMA_DEF(name, fn) m.def(name, torch::wrap_pybind_function_no_gil(fn))

PYBIND11_MODULE(_host, m) {
  m.doc() = "native autograd nodes and launch sequences above libanima_b200.so";
  py::class_<TLinear>(m, "TLinear");
  ANIMA_DEF("status_word", status_word_tensor);
  ANIMA_DEF("time_gemms", time_gemms);
  ANIMA_DEF("gemm_times", gemm_times);
  ANIMA_DEF("mx_quantize", py_quantize);
  ANIMA_DEF("mx_gemm", py_gemm);
  ANIMA_DEF("scales_retile", py_retile);
  ANIMA_DEF("lokr_linear", py_lokr);
  ANIMA_DEF("merged_linear", py_merged);
  ANIMA_DEF("frozen_linear", py_frozen);
  ANIMA_DEF("lokr_mlp", py_lokr_mlp);
  ANIMA_DEF("tlinear", py_tlinear);
  ANIMA_DEF("tlokr_linear", py_tlokr);
  ANIMA_DEF("tlokr_mlp", py_tlokr_mlp);
  ANIMA_DEF("tlokr_forward_only", py_tlokr_fwd);
  ANIMA_DEF("tlokr_backward_only", py_tlokr_bwd);
  ANIMA_DEF("adaln", py_adaln);
  ANIMA_DEF("gated_add", gated_add);
  ANIMA_DEF("gated_add_adaln", py_gated_add_adaln);
  ANIMA_DEF("rmsnorm_rope", rmsnorm_rope);
}
