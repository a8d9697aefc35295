// Allocation and launch helpers of the native host path (see common.h).
#include "common.h"

#include <ATen/cuda/CUDAEvent.h>

#include <atomic>
#include <mutex>

namespace anima_host {

void raise_status(int64_t status) {
  const char* text = anima_last_error();
  const std::string msg =
      std::string("libanima_b200: ") + (text ? text : "") + " (status " + std::to_string(status) + ")";
  switch (status) {
    case ANIMA_E_UNSUPPORTED: TORCH_CHECK_NOT_IMPLEMENTED(false, msg); break;
    case ANIMA_E_CUDA: TORCH_CHECK(false, msg); break;
    default: TORCH_CHECK_VALUE(false, msg);
  }
  TORCH_CHECK(false, msg);
}

namespace {
std::mutex word_mu;
Tensor words[64];
std::atomic<int32_t*> word_ptr[64];
}  // namespace

Tensor status_word_tensor(int64_t i) {
  TORCH_CHECK(i >= 0 && i < 64, "device index ", i, " out of range");
  std::lock_guard<std::mutex> lock(word_mu);
  if (!words[i].defined()) {
    words[i] = at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(at::Device(at::kCUDA, static_cast<int8_t>(i))));
    word_ptr[i].store(words[i].data_ptr<int32_t>());
  }
  return words[i];
}

int32_t* status_word(const at::Device& dev) {
  const int i = dev.index();
  if (i >= 0 && i < 64)
    if (int32_t* p = word_ptr[i].load()) return p;
  return status_word_tensor(i).data_ptr<int32_t>();
}

static const Tensor& on_cuda(const Tensor& t) {
  TORCH_CHECK(t.is_cuda(), "anima_trainer_sm120_b200 kernels need CUDA tensors (no CPU path)");
  return t;
}
Launch::Launch(const Tensor& t)
    : dev(on_cuda(t).device()), guard(dev), stream(c10::cuda::getCurrentCUDAStream(dev.index()).stream()) {}

void admit(const Launch& l, const Tensor& t) {
  if (!t.defined()) return;
  TORCH_CHECK(t.device() == l.dev, "tensors on different devices: ", l.dev, " and ", t.device());
  TORCH_CHECK_NOT_IMPLEMENTED(!t._fw_grad(/*level=*/0).defined(), "forward-mode AD is not implemented for these kernels");
}

Op op_in(const Tensor& store, int64_t rows, int64_t k) {
  uint8_t* p = static_cast<uint8_t*>(store.data_ptr());
  return {store, Tensor(), p, p + pad256(rows * k), rows, k};
}
Op op_of(const Tensor& codes, const Tensor& scales) {
  TORCH_CHECK_VALUE(codes.dim() == 2 && codes.is_contiguous() && scales.is_contiguous(),
                    "mx_gemm operands must be contiguous (K-major)");
  return {codes, scales, static_cast<uint8_t*>(codes.data_ptr()), static_cast<uint8_t*>(scales.data_ptr()), codes.size(0),
          codes.size(1)};
}
Op op_of(const OptTensor& codes, const OptTensor& scales, const OptTensor& store) {
  if (!codes || !codes->defined()) return {};
  if (store && store->defined()) return op_in(*store, codes->size(0), codes->size(1));
  return op_of(*codes, *scales);
}
// A contiguous view of `size` bytes-typed elements at byte `offset`, without the dispatcher's view machinery.
static Tensor bytes_at(const Tensor& store, int64_t offset, at::IntArrayRef size) {
  auto impl = store.unsafeGetTensorImpl()->shallow_copy_and_detach(c10::VariableVersion(0), true);
  impl->set_storage_offset(store.storage_offset() + offset);
  impl->set_sizes_contiguous(size);
  return Tensor(std::move(impl));
}
std::pair<Tensor, Tensor> tensors_of(const Op& o, int layout) {
  if (o.other.defined()) return {o.store, o.other};
  const int64_t at = o.scales - o.codes;
  return {bytes_at(o.store, 0, {o.rows, o.k}), layout == ANIMA_SCALES_PLAIN ? bytes_at(o.store, at, {o.rows, o.k / 32})
                                                                            : bytes_at(o.store, at, {tiled_bytes(o.rows, o.k)})};
}

Op empty_op(int64_t rows, int64_t k, const at::Device& dev) { return op_in(empty({store_bytes(rows, k)}, U8, dev), rows, k); }

Op placeholder(int64_t rows, int64_t k, const at::Device& dev) {
  Op o;
  o.store = at::detail::empty_strided_cuda({store_bytes(rows, k)}, {0}, U8, dev);
  o.rows = rows;
  o.k = k;
  return o;
}

const Tensor& Kept::get() const {
  TORCH_CHECK(version == now(),
              "one of the variables needed for gradient computation has been modified by an inplace operation: a tensor of "
              "shape ", t.sizes(), " is at version ", now(), "; expected version ", version);
  return t;
}

Op HostNode::get_op(size_t& at, const Op& shape) {
  if (!shape.rows) return {};
  const Tensor first = get(at++);
  if (shape.other.defined()) return op_of(first, get(at++));
  TORCH_CHECK(first.is_contiguous() && first.numel() >= store_bytes(shape.rows, shape.k),
              "a saved operand [", shape.rows, ", ", shape.k, "] has no memory behind it: backward through a pass made under "
              "first_pass(), whose saved tensors only a checkpoint's recomputation fills in");
  return op_in(first, shape.rows, shape.k);
}

Mat as_matrix(const Tensor& x, int64_t cols) {
  const int64_t n = x.numel();
  if (x.scalar_type() == BF16 && x.is_contiguous()) return {x, cols ? n / cols : 0, cols, cols};
  Tensor t = x.detach().reshape({-1, cols});
  if (t.scalar_type() != BF16) t = t.to(BF16);
  if (t.stride(1) != 1 && cols > 1) t = t.contiguous();
  return {t, t.size(0), cols, t.size(0) > 1 ? t.stride(0) : cols};
}

Tensor bf16_contiguous(const Tensor& t) {
  Tensor d = t.scalar_type() == BF16 ? t : t.detach().to(BF16);
  return d.is_contiguous() ? d : d.detach().contiguous();
}

void check_bias(const OptTensor& bias, int64_t n) {
  TORCH_CHECK_VALUE(!bias || !bias->defined() || bias->numel() == n, "bias must be of length N = ", n, ", got ", bias->numel(),
                    " elements");
}

static void need_blocks(int64_t rows, int64_t cols, bool row, bool col) {
  TORCH_CHECK_VALUE(!row || cols % 32 == 0, "rowwise quantisation needs cols % 32 == 0, got ", cols);
  TORCH_CHECK_VALUE(!col || rows % 32 == 0, "columnwise quantisation needs rows % 32 == 0, got ", rows);
}

static Op alloc_form(int64_t rows, int64_t k, int layout, const at::Device& dev) {
  if (layout == ANIMA_SCALES_PLAIN) return op_in(empty({pad256(rows * k) + rows * (k / 32)}, U8, dev), rows, k);
  return empty_op(rows, k, dev);
}

std::pair<Op, Op> quantize(const Launch& l, const Mat& x, bool row, bool col, int layout) {
  need_blocks(x.rows, x.cols, row, col);
  Op r, c;
  if (row) r = alloc_form(x.rows, x.cols, layout, l.dev);
  if (col) c = alloc_form(x.cols, x.rows, layout, l.dev);
  if (x.rows && x.cols)
    check(anima_mx_quantize(x.ptr(), x.rows, x.cols, x.ld, r.codes, r.scales, c.codes, c.scales, layout, l.stream));
  return {r, c};
}

std::pair<Op, Op> quantize_gelu(const Launch& l, const Tensor& h, const Tensor& grad, int64_t rows, int64_t cols, bool row,
                                bool col) {
  need_blocks(rows, cols, row, col);
  Op r, c;
  if (row) r = empty_op(rows, cols, l.dev);
  if (col) c = empty_op(cols, rows, l.dev);
  if (rows && cols)
    check(anima_mx_quantize_gelu(h.data_ptr(), ptr(grad), rows, cols, cols, nullptr, r.codes, r.scales, c.codes, c.scales,
                                 ANIMA_SCALES_TILED, l.stream));
  return {r, c};
}

Op regroup(const Launch& l, const Op& a, int64_t rows, int64_t k) {
  TORCH_CHECK_VALUE(rows * k == a.rows * a.k && k % 32 == 0, "cannot view [", a.rows, ", ", a.k, "] as [", rows, ", ", k, "]");
  Op o = a;
  o.rows = rows;
  o.k = k;
  o.other = empty({tiled_bytes(rows, k)}, U8, l.dev);
  o.scales = static_cast<uint8_t*>(o.other.data_ptr());
  if (rows) check(anima_mx_scales_regroup(a.scales, a.rows, a.k, o.scales, rows, k, l.stream));
  return o;
}

static int factor_flag(const Tensor& w1, const Tensor& w2) {
  TORCH_CHECK_TYPE(w1.scalar_type() == w2.scalar_type() && (w1.scalar_type() == BF16 || w1.scalar_type() == F32),
                   "LoKr factors must both be bfloat16 or both float32");
  return w1.scalar_type() == F32 ? 1 : 0;
}
static Tensor dense(const Tensor& t) { return t.is_contiguous() ? t : t.detach().contiguous(); }

std::pair<Op, Op> merge_quantize(const Launch& l, const Tensor& W, const Tensor& w1_, const Tensor& w2_, double alpha,
                                 bool row, bool col) {
  TORCH_CHECK_TYPE(W.scalar_type() == BF16, "W must be bfloat16, got ", W.scalar_type());
  TORCH_CHECK_VALUE(W.dim() == 2, "W must be 2-D");
  TORCH_CHECK(w1_.device() == l.dev && w2_.device() == l.dev && W.device() == l.dev, "tensors on different devices");
  const Tensor w = dense(W), w1 = dense(w1_), w2 = dense(w2_);
  const int64_t N = w.size(0), K = w.size(1), up = w1.size(0), uq = w1.size(1);
  TORCH_CHECK_VALUE(N % up == 0 && K % uq == 0 && w2.size(0) == N / up && w2.size(1) == K / uq, "kron(", w1.sizes(), ", ",
                    w2.sizes(), ") does not match W ", w.sizes());
  Op r, c;
  if (row) r = empty_op(N, K, l.dev);
  if (col) c = empty_op(K, N, l.dev);
  check(anima_lokr_merge_quantize(w.data_ptr(), w1.data_ptr(), w2.data_ptr(), factor_flag(w1, w2),
                                  static_cast<float>(alpha), N, K, up, uq, nullptr, r.codes, r.scales, c.codes, c.scales,
                                  ANIMA_SCALES_TILED, l.stream));
  return {r, c};
}

namespace {
std::atomic<bool> timing{false};
std::mutex timed_mu;
struct Timed {
  at::cuda::CUDAEvent begin{cudaEventDefault}, end{cudaEventDefault};
  double flops;
};
std::vector<std::unique_ptr<Timed>> timed;

class GemmTimer {      // brackets the launches of its scope
 public:
  explicit GemmTimer(double flops) {
    if (!timing.load(std::memory_order_relaxed)) return;
    t_ = std::make_unique<Timed>();
    t_->flops = flops;
    t_->begin.record();
  }
  ~GemmTimer() {
    if (!t_) return;
    t_->end.record();
    std::lock_guard<std::mutex> lock(timed_mu);
    timed.push_back(std::move(t_));
  }

 private:
  std::unique_ptr<Timed> t_;
};
}  // namespace

void time_gemms(bool on) {
  std::lock_guard<std::mutex> lock(timed_mu);
  if (on) timed.clear();
  timing.store(on);
}
std::vector<std::pair<double, double>> gemm_times() {
  std::lock_guard<std::mutex> lock(timed_mu);
  std::vector<std::pair<double, double>> out;
  for (auto& t : timed) {
    t->end.synchronize();
    out.emplace_back(t->begin.elapsed_time(t->end), t->flops);
  }
  timed.clear();
  return out;
}

static void need_same_k(const Op& a, const Op& b) {
  TORCH_CHECK_VALUE(a.k == b.k, "contraction sizes differ: A has K=", a.k, ", B has K=", b.k);
}

void gemm(const Launch& l, const Op& a, const Op& b, const GemmOut& out, const void* bias, const void* residual,
          int64_t ldr, double alpha) {
  need_same_k(a, b);
  const int64_t M = a.rows, N = b.rows, K = a.k;
  const int64_t bytes = check(anima_mx_gemm_workspace_bytes(M, N, K));
  Tensor ws;
  if (bytes) ws = empty({bytes}, U8, l.dev);
  const GemmTimer timer(2.0 * M * N * K);
  check(anima_mx_gemm_ex(a.codes, a.scales, b.codes, b.scales, out.c, M, N, K, out.ldc, bias,
                         residual, ldr, static_cast<float>(alpha), out.fp32 ? 1 : 0, ptr(ws), bytes,
                         status_word(l.dev), l.stream));
}

void gemm_delta(const Launch& l, const Op& a, const Op& b, const Op& planes, const Op& d, void* c, const void* bias) {
  need_same_k(a, b);
  const int64_t M = a.rows, N = b.rows, K = a.k;
  const int64_t bytes = check(anima_mx_gemm_workspace_bytes(M, N, K));
  Tensor ws;
  if (bytes) ws = empty({bytes}, U8, l.dev);
  const GemmTimer timer(2.0 * M * N * K + 256.0 * M * N);
  check(anima_mx_gemm_delta(a.codes, a.scales, b.codes, b.scales, c, M, N, K, N, bias, 0,
                            planes.codes, planes.scales, d.codes, d.scales, ptr(ws), bytes,
                            status_word(l.dev), l.stream));
}

Tensor gemm_f32(const Launch& l, const Op& a, const Op& b, double alpha) {
  Tensor c = empty({a.rows, b.rows}, F32, l.dev);
  gemm(l, a, b, {c.data_ptr(), b.rows, true}, nullptr, nullptr, 0, alpha);
  return c;
}

std::pair<Tensor, Tensor> kron_backward(const Launch& l, const Tensor& dw, const Tensor& w1_, const Tensor& w2_,
                                        double alpha) {
  const Tensor w1 = dense(w1_), w2 = dense(w2_);
  const int64_t N = dw.size(0), K = dw.size(1), up = w1.size(0), uq = w1.size(1);
  const int64_t bytes = check(anima_lokr_kron_backward_workspace_bytes(N, K, up, uq));
  Tensor ws = empty({bytes}, U8, l.dev);
  Tensor d1 = empty({up, uq}, F32, l.dev), d2 = empty({N / up, K / uq}, F32, l.dev);
  check(anima_lokr_kron_backward(dw.data_ptr(), dw.scalar_type() == F32 ? 1 : 0, w1.data_ptr(), w2.data_ptr(),
                                 factor_flag(w1, w2), static_cast<float>(alpha), N, K, up, uq, d1.data_ptr<float>(),
                                 d2.data_ptr<float>(), ws.data_ptr(), bytes, l.stream));
  return {cast(d1, w1.scalar_type()), cast(d2, w2.scalar_type())};
}

}  // namespace anima_host
