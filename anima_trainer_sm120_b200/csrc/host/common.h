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
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>

#include <mutex>
#include <optional>
#include <tuple>
#include <utility>
#include <vector>

#include "../../../include/anima_b200.h"

namespace anima_host {

using at::Tensor;
using OptTensor = std::optional<Tensor>;
using torch::autograd::variable_list;

constexpr auto BF16 = at::kBFloat16;
constexpr auto F32 = at::kFloat;
constexpr auto U8 = at::kByte;

// One K-major MXFP8 operand: e4m3 codes [rows, k] and e8m0 scales (TILED unless said otherwise). Both lie in one
// allocation (`store`, bytes) when they were made here: one tensor to allocate and one for autograd to save.
struct Op {
  Tensor store, other;      // the memory; `other` only for operands that came as two tensors
  uint8_t *codes = nullptr, *scales = nullptr;
  int64_t rows = 0, k = 0;
  bool defined() const { return store.defined(); }
};
constexpr int64_t pad256(int64_t n) { return (n + 255) / 256 * 256; }
inline int64_t tiled_bytes(int64_t rows, int64_t k) { return ((rows + 127) / 128) * ((k + 127) / 128) * 512; }
inline int64_t store_bytes(int64_t rows, int64_t k) { return pad256(rows * k) + tiled_bytes(rows, k); }
Op op_in(const Tensor& store, int64_t rows, int64_t k);       // the operand laid out in `store`
Op op_of(const Tensor& codes, const Tensor& scales);          // [rows, k] codes and their scales
// what Python passes for an operand: nothing, (codes, scales, None) or (codes, scales, store)
Op op_of(const OptTensor& codes, const OptTensor& scales, const OptTensor& store);
// the tensors of an operand, as views of its store
std::pair<Tensor, Tensor> tensors_of(const Op& o, int layout = ANIMA_SCALES_TILED);

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

// Current device and stream for the duration of one call.
struct Launch {
  explicit Launch(const Tensor& t);
  at::Device dev;
  c10::cuda::CUDAGuard guard;
  void* stream;
};

// What these nodes cannot take: tensors of another device, and forward-mode tangents (an autograd function without a
// rule for them refuses; a node made by hand would drop them without notice).
void admit(const Launch& l, const Tensor& t);
inline void admit(const Launch& l, const OptTensor& t) {
  if (t) admit(l, *t);
}
template <class First, class... Rest>
void admit(const Launch& l, const First& first, const Rest&... rest) {
  admit(l, first);
  (admit(l, rest), ...);
}

int32_t* status_word(const at::Device& dev);      // the GEMM's bounded-wait flag of a device
Tensor status_word_tensor(int64_t device_index);

Op empty_op(int64_t rows, int64_t k, const at::Device& dev);
// Stands in for the store of an operand only backward would read, in a pass whose saved tensors a checkpoint drops:
// its shape and type without its memory.
Op placeholder(int64_t rows, int64_t k, const at::Device& dev);

Mat as_matrix(const Tensor& x, int64_t cols);     // any shape whose elements in order are [-1, cols]; cast to bf16
Tensor bf16_contiguous(const Tensor& t);          // detached
// A bias of n outputs as the GEMM's epilogue reads it (undefined: none). The kernels index it by n: check_bias, before
// anything is launched, refuses any other length.
void check_bias(const OptTensor& bias, int64_t n);
inline Tensor bias_rows(const OptTensor& bias) { return bias && bias->defined() ? bf16_contiguous(*bias) : Tensor(); }

std::pair<Op, Op> quantize(const Launch& l, const Mat& x, bool row, bool col, int layout = ANIMA_SCALES_TILED);
// gelu(h) or grad * gelu'(h); h and grad viewed as [rows, cols]
std::pair<Op, Op> quantize_gelu(const Launch& l, const Tensor& h, const Tensor& grad, int64_t rows, int64_t cols, bool row,
                                bool col);
Op regroup(const Launch& l, const Op& a, int64_t rows, int64_t k);
std::pair<Op, Op> merge_quantize(const Launch& l, const Tensor& W, const Tensor& w1, const Tensor& w2, double alpha,
                                 bool row, bool col);

// Measurement aid: while on, every GEMM of this path is bracketed by timed events on its stream (which also keeps it from
// overlapping its neighbours; not for captures). gemm_times: (ms, flops) of each since it was switched on, oldest first, which
// are then forgotten.
void time_gemms(bool on);
std::vector<std::pair<double, double>> gemm_times();

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
// An output belongs to the graph as soon as any tensor of the call wants a gradient, also one these nodes have no rule for
// (a frozen weight left trainable, the bias of a fused MLP, a norm weight): that tensor's gradient is then none.
template <class... T>
bool any_wants(const T&... t) {
  return (wants(t) || ...);
}
inline Tensor cast(const Tensor& t, at::ScalarType dt) { return t.scalar_type() == dt ? t : t.to(dt); }

// ------------------------------------------------------------------------------------------------ autograd nodes
// A parameter or another small tensor a node reads in backward without handing it to saved-tensor hooks (a
// checkpointed pass would call them for every tensor); like a saved tensor it may not change in place meanwhile.
struct Kept {
  Tensor t;
  uint32_t version = 0;
  Kept() = default;
  Kept(const Tensor& v) : t(v), version(now()) {}
  const Tensor& get() const;

 private:
  uint32_t now() const { return t.defined() && !t.is_inference() ? t.unsafeGetTensorImpl()->version_counter().current_version() : 0; }
};

// Base of the nodes: saved tensors go through torch's saved-tensor hooks (checkpointing), one output gradient by default.
struct HostNode : public torch::autograd::Node {
  std::vector<torch::autograd::SavedVariable> saved;

  void save(const Tensor& t, bool is_output = false) { saved.emplace_back(t, is_output); }
  void save(const Op& o) {       // an undefined operand saves nothing
    if (!o.defined()) return;
    save(o.store);
    if (o.other.defined()) save(o.other);
  }
  Tensor get(size_t i) { return saved.at(i).unpack(getptr()); }
  // the operand saved at position `at` (advanced), of a known shape
  Op get_op(size_t& at, const Op& shape);
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (auto& v : saved) v.reset_data();
  }
  // the gradient of output i; zeros where the graph has none
  Tensor grad_of(variable_list& g, size_t i) { return g[i].defined() ? g[i] : input_metadata(i).zeros_like(); }
};

inline torch::autograd::Edge edge_of(const Tensor& t) {
  return wants(t) ? torch::autograd::impl::gradient_edge(t) : torch::autograd::Edge();
}
inline torch::autograd::Edge edge_of(const OptTensor& t) { return t ? edge_of(*t) : torch::autograd::Edge(); }
template <class N, class... Inputs>
std::shared_ptr<N> make_node(const Inputs&... inputs) {
  auto node = std::shared_ptr<N>(new N(), torch::autograd::deleteNode);
  torch::autograd::edge_list edges;
  edges.reserve(sizeof...(inputs));
  (edges.push_back(edge_of(inputs)), ...);
  node->set_next_edges(std::move(edges));
  return node;
}
// The node last made for an input on this thread (both weak), for a later call on the same tensor whose gradient is to
// pass through it. `get` gives the node while t still is what it saw: same tensor, version, shape and graph edge.
template <class N>
struct LastNode {
  c10::weak_intrusive_ptr<c10::TensorImpl> x{c10::intrusive_ptr<c10::TensorImpl>()};
  uint32_t version = 0;
  at::DimVector sizes;
  std::weak_ptr<N> node;

  void set(const Tensor& t, const std::shared_ptr<N>& n) {      // n's first edge is t's
    x = c10::weak_intrusive_ptr<c10::TensorImpl>(t.getIntrusivePtr());
    version = t.unsafeGetTensorImpl()->version_counter().current_version();
    sizes = t.sizes();
    node = n;
  }
  std::shared_ptr<N> get(const Tensor& t) const {
    auto n = node.lock();
    const auto was = x.lock();
    if (!n || was.get() != t.unsafeGetTensorImpl() ||
        t.unsafeGetTensorImpl()->version_counter().current_version() != version || t.sizes() != at::IntArrayRef(sizes) ||
        edge_of(t) != n->next_edge(0))
      return nullptr;
    return n;
  }
};

// Kernels and allocations of a node run below autograd.
using Below = at::AutoDispatchBelowADInplaceOrView;

}  // namespace anima_host
