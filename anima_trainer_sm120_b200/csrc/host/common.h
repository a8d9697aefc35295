// Native host path: the autograd nodes of this package and the allocation / launch sequence of each, above the C ABI
// of libanima_b200.so. A pass over one linear is 8 - 17 launches; driven from Python (ctypes, one wrapper and several
// torch calls per launch) each launch cost 25 - 40 us of host time, which bounded every call below about 4096 rows.
// Here a launch costs its allocation and the driver call.
//
// Scratch comes from the caching allocator on every call: it is stream-ordered, goes back when the call ends, and is
// private to the caller's graph pool during a capture.
#pragma once

#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/custom_function.h>

#include <optional>
#include <tuple>
#include <utility>
#include <vector>

#include "../../../include/anima_b200.h"

namespace anima_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

constexpr auto BF16 = at::kBFloat16;
constexpr auto F32 = at::kFloat;
constexpr auto U8 = at::kByte;

// One K-major MXFP8 operand: e4m3 codes [rows, k] and e8m0 scales (TILED unless said otherwise).
struct Op {
  Tensor codes, scales;
  bool defined() const { return codes.defined(); }
  int64_t rows() const { return codes.size(0); }
  int64_t k() const { return codes.size(1); }
};
inline Op make_op(const OptTensor& codes, const OptTensor& scales) {
  return codes && codes->defined() ? Op{*codes, *scales} : Op{};
}

// A bf16 matrix as the kernels take it: pointer, rows, columns, row pitch; `keep` owns the memory.
struct Mat {
  Tensor keep;
  int64_t rows, cols, ld;
  const void* ptr() const { return keep.data_ptr(); }
};

[[noreturn]] void raise_status(int64_t status);
inline int64_t check(int64_t status) {
  if (status < 0) raise_status(status);
  return status;
}

inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline uint8_t* ptr8(const Tensor& t) { return static_cast<uint8_t*>(ptr(t)); }
inline void* ptr(const OptTensor& t) { return t ? ptr(*t) : nullptr; }

inline Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const at::Device& dev) {
  return at::detail::empty_cuda(size, dtype, dev, std::nullopt);
}
inline int64_t tiled_bytes(int64_t rows, int64_t k) { return ((rows + 127) / 128) * ((k + 127) / 128) * 512; }

// Current device and stream for the duration of one call.
struct Launch {
  explicit Launch(const Tensor& t);
  at::Device dev;
  c10::cuda::CUDAGuard guard;
  void* stream;
};

int32_t* status_word(const at::Device& dev);      // the GEMM's bounded-wait flag of a device
Tensor status_word_tensor(int64_t device_index);

Op empty_op(int64_t rows, int64_t k, const at::Device& dev);
// Stands in for an operand only backward would read, in a pass whose saved tensors a checkpoint drops: its shape and
// type without its memory.
Op placeholder(int64_t rows, int64_t k, const at::Device& dev);

Mat as_matrix(const Tensor& x, int64_t cols);     // any shape whose elements in order are [-1, cols]; cast to bf16
Tensor bf16_contiguous(const Tensor& t);          // detached

std::pair<Op, Op> quantize(const Launch& l, const Mat& x, bool row, bool col, int layout = ANIMA_SCALES_TILED);
// gelu(h) or grad * gelu'(h); h and grad viewed as [rows, cols]
std::pair<Op, Op> quantize_gelu(const Launch& l, const Tensor& h, const Tensor& grad, int64_t rows, int64_t cols, bool row,
                                bool col);
Op regroup(const Launch& l, const Op& a, int64_t rows, int64_t k);
std::pair<Op, Op> merge_quantize(const Launch& l, const Tensor& W, const Tensor& w1, const Tensor& w2, double alpha,
                                 bool row, bool col);

struct GemmOut {
  void* c;
  int64_t ldc;
  bool fp32;
};
void gemm(const Launch& l, const Op& a, const Op& b, const GemmOut& out, const void* bias = nullptr,
          const void* residual = nullptr, int64_t ldr = 0, double alpha = 1.0);
void gemm_delta(const Launch& l, const Op& a, const Op& b, const Op& planes, const Op& d, void* c, const void* bias);
Tensor gemm_f32(const Launch& l, const Op& a, const Op& b, double alpha = 1.0);        // [M, N] fp32
// (dw1, dw2) of dW = [N, K] fp32, in the factors' dtype
std::pair<Tensor, Tensor> kron_backward(const Launch& l, const Tensor& dw, const Tensor& w1, const Tensor& w2,
                                        double alpha);

inline std::vector<int64_t> with_last(at::IntArrayRef shape, int64_t last) {
  std::vector<int64_t> s(shape.begin(), shape.end());
  s.back() = last;
  return s;
}
inline bool wants(const Tensor& t) { return at::GradMode::is_enabled() && t.defined() && t.requires_grad(); }
inline bool wants(const OptTensor& t) { return t && wants(*t); }
inline Tensor cast(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }

// Plain values of a node, kept beside its saved tensors.
template <class T>
struct Held : torch::CustomClassHolder {
  T v;
};
template <class T>
void hold(AutogradContext* ctx, T v) {
  auto h = c10::make_intrusive<Held<T>>();
  h->v = std::move(v);
  ctx->saved_data["held"] = c10::IValue::make_capsule(std::move(h));
}
template <class T>
T& held(AutogradContext* ctx) {
  return static_cast<Held<T>*>(ctx->saved_data["held"].toCapsule().get())->v;
}

inline void push(variable_list& v, const Op& a) {
  if (a.defined()) {
    v.push_back(a.codes);
    v.push_back(a.scales);
  }
}
inline Op pop(const variable_list& v, size_t& at, bool there) {
  if (!there) return {};
  Op a{v[at], v[at + 1]};
  at += 2;
  return a;
}

}  // namespace anima_host
