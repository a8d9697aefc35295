// Per-head RMSNorm with optional rotary embedding, forward and backward, for the q / k
// projections of the attention layers (head width 128, bf16).
//
// In anima-trainer these two steps are third-party kernels (Liger RMSNorm, liger_patch.py:31-47, and
// Transformer Engine's fused RoPE, rope_patch.py:28-56); the stand-in DiT of this package would
// otherwise run them as ~10 eager elementwise launches per call. HBM-bound: 4 B/elem forward
// (+ 4 B per vector for rstd), 6 B/elem backward.
//   n   = x * rsqrt(mean(x^2) + eps) * w
//   out = n * cos + rotate_half(n) * sin   (cos / sin: fp32 tables [seq_len, 128], L2-resident)
//           rotate_half(n)[i] = -n[i+64] (i < 64), n[i-64] (i >= 64)
// The norm weight is treated as frozen (no weight gradient), which is the LoKr training setting.
#include "common.cuh"
#include "f32x2.cuh"

namespace anima {
namespace {

constexpr int kHeadDim = 128;
constexpr int kThreads = 256;
constexpr int kLanesPerToken = 8;                        // 8 lanes x (8 + 8) elements = one 128-wide head vector
constexpr int kTokensPerCta = kThreads / kLanesPerToken;

// Eight lanes own one token and walk its heads. Lane l holds elements 8l..8l+7 and 64+8l..64+8l+7 (two 16-byte
// accesses), so an element and its rotate-half partner are in the same lane: a vector costs three shuffles (its sum)
// instead of four plus one per element, which bound the half-warp form that held 8 consecutive elements per lane.
// With the norm weight folded into the token's rotation, held in registers and reused by every head,
//   a1 = w1 c1, b1 = w2 s1, a2 = w2 c2, b2 = w1 s2   (1 / 2: the halves; s, c: the tables)
//   out1 = rstd (x1 a1 - x2 b1),  out2 = rstd (x2 a2 + x1 b2)
//   gw1  = g1 a1 + g2 b2,         gw2  = g2 a2 - g1 b1                (the gradient of x / rms, backward)
// fp32 in pairs. [8, 4096, 16, 128]: forward 57.6 -> 46.2 us (5810 GB/s), backward 80.6 -> 64.4 (6250 GB/s).
struct Rotation {
  f2 a1[4], b1[4], a2[4], b2[4];   // without rotary: a1 = w1, a2 = w2
};

template <bool WBF16>
__device__ __forceinline__ void load8(const void* p, int at, f2 (&v)[4]) {
  if (WBF16) {
    const uint4 r = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p) + at);
    v[0] = f2_of_bf16(r.x); v[1] = f2_of_bf16(r.y); v[2] = f2_of_bf16(r.z); v[3] = f2_of_bf16(r.w);
  } else {
    const float4* q = reinterpret_cast<const float4*>(static_cast<const float*>(p) + at);
    const float4 lo = q[0], hi = q[1];
    v[0] = f2_make(lo.x, lo.y); v[1] = f2_make(lo.z, lo.w); v[2] = f2_make(hi.x, hi.y); v[3] = f2_make(hi.z, hi.w);
  }
}

template <bool ROPE, bool WBF16>
__device__ __forceinline__ void load_rotation(Rotation& r, const void* w, const float* cos_tab, const float* sin_tab,
                                              int64_t pos, int l) {
  f2 w1[4], w2[4];
  load8<WBF16>(w, l * 8, w1);
  load8<WBF16>(w, 64 + l * 8, w2);
  if (ROPE) {
    load8<false>(cos_tab + pos * kHeadDim, l * 8, r.a1);
    load8<false>(cos_tab + pos * kHeadDim, 64 + l * 8, r.a2);
    load8<false>(sin_tab + pos * kHeadDim, l * 8, r.b1);
    load8<false>(sin_tab + pos * kHeadDim, 64 + l * 8, r.b2);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (ROPE) {
      r.a1[e] = f2_mul(w1[e], r.a1[e]);
      r.a2[e] = f2_mul(w2[e], r.a2[e]);
      r.b1[e] = f2_mul(w2[e], f2_mul(r.b1[e], f2_dup(-1.f)));   // enters with its sign
      r.b2[e] = f2_mul(w1[e], r.b2[e]);
    } else {
      r.a1[e] = w1[e];
      r.a2[e] = w2[e];
    }
  }
}

// The loads run ahead of the arithmetic through a ring in shared memory filled with cp.async: each thread copies
// exactly the 16-byte chunks it reads itself (no barrier, no registers), kAhead heads ahead. With loads unrolled into
// registers the 128 registers a thread leave 16 warps and about 32 KB in flight a SM: 5.0 TB/s.
template <int CHUNKS, int STAGES>   // 16-byte chunks of one head, ring slots
struct Ring {
  uint32_t base;
  __device__ __forceinline__ Ring(void* smem) : base(static_cast<uint32_t>(__cvta_generic_to_shared(smem)) + threadIdx.x * 16) {}
  __device__ __forceinline__ uint32_t at(int slot, int c) const { return base + (slot * CHUNKS + c) * kThreads * 16; }
  __device__ __forceinline__ void copy(int slot, int c, const void* src) const {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(at(slot, c)), "l"(src) : "memory");
  }
  __device__ __forceinline__ static void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
  __device__ __forceinline__ static void wait() { asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory"); }
  __device__ __forceinline__ uint4 read(int slot, int c) const {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at(slot, c)));
    return v;
  }
};
constexpr int kFwdStages = 6, kBwdStages = 4;

__device__ __forceinline__ void widen(const uint4& v, f2 (&f)[4]) {
  f[0] = f2_of_bf16(v.x); f[1] = f2_of_bf16(v.y); f[2] = f2_of_bf16(v.z); f[3] = f2_of_bf16(v.w);
}
__device__ __forceinline__ uint4 narrow(const f2 (&f)[4]) {
  return make_uint4(bf16_of_f2(f[0]), bf16_of_f2(f[1]), bf16_of_f2(f[2]), bf16_of_f2(f[3]));
}
__device__ __forceinline__ float sum8(float v, unsigned mask) {   // over the token's eight lanes
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// blockIdx.y = group of heads (a grid of token blocks alone would leave SMs idle on short sequences)
template <bool ROPE, bool WBF16>
__global__ void __launch_bounds__(kThreads, 2)
rmsnorm_rope_fwd_kernel(const __nv_bfloat16* __restrict__ x, const void* __restrict__ w, const float* __restrict__ cos_tab,
                        const float* __restrict__ sin_tab, float eps, int64_t tokens, int heads, int heads_per_group,
                        int64_t seq_len, __nv_bfloat16* __restrict__ out, float* __restrict__ rstd_out,
                        uint4* __restrict__ w_copy) {
  after_previous();
  w = after_previous(w);
  if (w_copy != nullptr && blockIdx.x + blockIdx.y == 0 && threadIdx.x < kHeadDim * (WBF16 ? 2 : 4) / 16)
    w_copy[threadIdx.x] = static_cast<const uint4*>(w)[threadIdx.x];
  cos_tab = after_previous(cos_tab);
  sin_tab = after_previous(sin_tab);
  const int l = threadIdx.x & (kLanesPerToken - 1);
  const int64_t token = static_cast<int64_t>(blockIdx.x) * kTokensPerCta + threadIdx.x / kLanesPerToken;
  if (token >= tokens) return;   // the eight lanes of a token leave together; shuffles below stay inside them
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  const int h0 = blockIdx.y * heads_per_group, h1 = min(heads, h0 + heads_per_group);
  Rotation r;
  load_rotation<ROPE, WBF16>(r, w, cos_tab, sin_tab, ROPE ? token % seq_len : 0, l);
  const int64_t base = token * heads * kHeadDim + l * 8;
  extern __shared__ uint4 ring_smem[];
  const Ring<2, kFwdStages> ring(ring_smem);
  auto start = [&](int h, int slot) {
    if (h < h1) {
      ring.copy(slot, 0, x + base + h * kHeadDim);
      ring.copy(slot, 1, x + base + h * kHeadDim + 64);
    }
    ring.commit();
  };
#pragma unroll
  for (int i = 0; i < kFwdStages - 1; ++i) start(h0 + i, i);
  int slot = 0;
#pragma unroll 1
  for (int h = h0; h < h1; ++h) {
    ring.wait();
    f2 v1[4], v2[4];
    widen(ring.read(slot, 0), v1);
    widen(ring.read(slot, 1), v2);
    start(h + kFwdStages - 1, slot == 0 ? kFwdStages - 1 : slot - 1);   // the slot used one head ago
    slot = slot + 1 == kFwdStages ? 0 : slot + 1;
    f2 q0 = f2_mul(v1[0], v1[0]), q1 = f2_mul(v2[0], v2[0]);
#pragma unroll
    for (int e = 1; e < 4; ++e) {
      q0 = f2_fma(v1[e], v1[e], q0);
      q1 = f2_fma(v2[e], v2[e], q1);
    }
    const float rstd = rsqrtf(sum8(f2_sum(f2_add(q0, q1)), mask) / kHeadDim + eps);
    const f2 rs = f2_dup(rstd);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f2 o1 = f2_mul(v1[e], r.a1[e]), o2 = f2_mul(v2[e], r.a2[e]);
      if (ROPE) {
        o1 = f2_fma(v2[e], r.b1[e], o1);
        o2 = f2_fma(v1[e], r.b2[e], o2);
      }
      v1[e] = f2_mul(o1, rs);
      v2[e] = f2_mul(o2, rs);
    }
    stg_stream16(out + base + h * kHeadDim, narrow(v1));
    stg_stream16(out + base + h * kHeadDim + 64, narrow(v2));
    if (l == 0) rstd_out[token * heads + h] = rstd;
  }
}

template <bool ROPE, bool WBF16>
__global__ void __launch_bounds__(kThreads, 2)
rmsnorm_rope_bwd_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ x,
                        const void* __restrict__ w, const float* __restrict__ cos_tab, const float* __restrict__ sin_tab,
                        const float* __restrict__ rstd_in, int64_t tokens, int heads, int heads_per_group, int64_t seq_len,
                        __nv_bfloat16* __restrict__ dx) {
  after_previous();
  w = after_previous(w);
  cos_tab = after_previous(cos_tab);
  sin_tab = after_previous(sin_tab);
  const int l = threadIdx.x & (kLanesPerToken - 1);
  const int64_t token = static_cast<int64_t>(blockIdx.x) * kTokensPerCta + threadIdx.x / kLanesPerToken;
  if (token >= tokens) return;
  const unsigned mask = 0xffu << (threadIdx.x & 24);
  const int h0 = blockIdx.y * heads_per_group, h1 = min(heads, h0 + heads_per_group);
  Rotation r;
  load_rotation<ROPE, WBF16>(r, w, cos_tab, sin_tab, ROPE ? token % seq_len : 0, l);
  const int64_t base = token * heads * kHeadDim + l * 8;
  extern __shared__ uint4 ring_smem[];
  const Ring<4, kBwdStages> ring(ring_smem);
  auto start = [&](int h, int slot) {
    if (h < h1) {
      const int64_t at = base + h * kHeadDim;
      ring.copy(slot, 0, dout + at);
      ring.copy(slot, 1, dout + at + 64);
      ring.copy(slot, 2, x + at);
      ring.copy(slot, 3, x + at + 64);
    }
    ring.commit();
  };
#pragma unroll
  for (int i = 0; i < kBwdStages - 1; ++i) start(h0 + i, i);
  rstd_in = after_previous(rstd_in);
  float rstd_next = rstd_in[token * heads + h0];
  int slot = 0;
#pragma unroll 1
  for (int h = h0; h < h1; ++h) {
    const int64_t at = base + h * kHeadDim;
    const float rstd = rstd_next;
    if (h + 1 < h1) rstd_next = rstd_in[token * heads + h + 1];
    ring.wait();
    f2 g1[4], g2[4], v1[4], v2[4];
    widen(ring.read(slot, 0), g1);
    widen(ring.read(slot, 1), g2);
    widen(ring.read(slot, 2), v1);
    widen(ring.read(slot, 3), v2);
    start(h + kBwdStages - 1, slot == 0 ? kBwdStages - 1 : slot - 1);
    slot = slot + 1 == kBwdStages ? 0 : slot + 1;
    // dx = rstd * (gw - xhat * mean(gw * xhat)), xhat = x * rstd
    f2 d0 = f2_dup(0.f), d1 = d0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      f2 w1 = f2_mul(g1[e], r.a1[e]), w2 = f2_mul(g2[e], r.a2[e]);
      if (ROPE) {
        w1 = f2_fma(g2[e], r.b2[e], w1);
        w2 = f2_fma(g1[e], r.b1[e], w2);
      }
      d0 = f2_fma(w1, v1[e], d0);
      d1 = f2_fma(w2, v2[e], d1);
      g1[e] = w1;
      g2[e] = w2;
    }
    const float dot = sum8(f2_sum(f2_add(d0, d1)), mask) * rstd / kHeadDim;   // mean(gw * xhat)
    const f2 nm = f2_dup(-dot * rstd), rs = f2_dup(rstd);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      g1[e] = f2_mul(rs, f2_fma(v1[e], nm, g1[e]));
      g2[e] = f2_mul(rs, f2_fma(v2[e], nm, g2[e]));
    }
    stg_stream16(dx + at, narrow(g1));
    stg_stream16(dx + at + 64, narrow(g2));
  }
}

// Heads one CTA walks: all of them once the token blocks alone fill the GPU, fewer (down to 2) below that.
int heads_per_group(int64_t token_blocks, int64_t heads) {
  int64_t groups = std::max<int64_t>(1, 4LL * sm_count() / std::max<int64_t>(1, token_blocks));
  groups = std::min<int64_t>(groups, std::max<int64_t>(1, heads / 2));
  return static_cast<int>(ceil_div(heads, groups));
}

int check(const char* who, int64_t tokens, int64_t heads, int64_t head_dim, int64_t seq_len, const void* cos_tab, const void* sin_tab) {
  ANIMA_REQUIRE(tokens >= 0 && heads > 0, ANIMA_E_ARG, "%s: bad sizes", who);
  ANIMA_REQUIRE(head_dim == kHeadDim, ANIMA_E_UNSUPPORTED, "%s: head_dim=%lld is not supported (only %d)", who,
                (long long)head_dim, kHeadDim);
  ANIMA_REQUIRE(heads < (1ll << 31) && tokens * heads < (1ll << 40), ANIMA_E_TOO_LARGE, "%s: too many vectors", who);
  ANIMA_REQUIRE((cos_tab == nullptr) == (sin_tab == nullptr), ANIMA_E_ARG, "%s: give both tables or neither", who);
  ANIMA_REQUIRE(!cos_tab || (seq_len > 0 && tokens % seq_len == 0), ANIMA_E_SHAPE,
                "%s: tokens=%lld is not a multiple of seq_len=%lld", who, (long long)tokens, (long long)seq_len);
  return ANIMA_OK;
}

}  // namespace
}  // namespace anima

using namespace anima;

extern "C" int anima_rmsnorm_rope_fwd_keep(const void* x, const void* weight, int weight_is_bf16, const float* cos_tab,
                                           const float* sin_tab, float eps, int64_t tokens, int64_t heads, int64_t head_dim,
                                           int64_t seq_len, void* out, float* rstd, void* weight_copy, void* stream) {
  ANIMA_REQUIRE(x && weight && out && rstd, ANIMA_E_ARG, "rmsnorm_rope_fwd: null pointer");
  if (int rc = check("rmsnorm_rope_fwd", tokens, heads, head_dim, seq_len, cos_tab, sin_tab)) return rc;
  ANIMA_REQUIRE(aligned16(x) && aligned16(out) && aligned16(weight) && aligned16(weight_copy) && (!cos_tab || (aligned16(cos_tab) && aligned16(sin_tab))), ANIMA_E_ALIGN,
                "rmsnorm_rope_fwd: tensors must be 16-byte aligned");
  if (tokens * heads == 0) return ANIMA_OK;
  const int64_t blocks = ceil_div(tokens, kTokensPerCta);
  const int hpg = heads_per_group(blocks, heads);
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(ceil_div(heads, hpg)));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  auto* op = static_cast<__nv_bfloat16*>(out);
  constexpr int kSmem = kFwdStages * 2 * kThreads * 16;
  auto go = [&](auto kernel) { launch_after(kernel, grid, kThreads, kSmem, s, xp, weight, cos_tab, sin_tab, eps, tokens, (int)heads, hpg, seq_len, op, rstd, static_cast<uint4*>(weight_copy)); };
  if (cos_tab) weight_is_bf16 ? go(rmsnorm_rope_fwd_kernel<true, true>) : go(rmsnorm_rope_fwd_kernel<true, false>);
  else weight_is_bf16 ? go(rmsnorm_rope_fwd_kernel<false, true>) : go(rmsnorm_rope_fwd_kernel<false, false>);
  ANIMA_CHECK_LAUNCH("rmsnorm_rope_fwd");
  return ANIMA_OK;
}

extern "C" int anima_rmsnorm_rope_fwd_ex(const void* x, const void* weight, int weight_is_bf16, const float* cos_tab,
                                         const float* sin_tab, float eps, int64_t tokens, int64_t heads, int64_t head_dim,
                                         int64_t seq_len, void* out, float* rstd, void* stream) {
  return anima_rmsnorm_rope_fwd_keep(x, weight, weight_is_bf16, cos_tab, sin_tab, eps, tokens, heads, head_dim, seq_len, out,
                                     rstd, nullptr, stream);
}

extern "C" int anima_rmsnorm_rope_bwd_ex(const void* dout, const void* x, const void* weight, int weight_is_bf16,
                                         const float* cos_tab, const float* sin_tab, const float* rstd, int64_t tokens,
                                         int64_t heads, int64_t head_dim, int64_t seq_len, void* dx, void* stream) {
  ANIMA_REQUIRE(dout && x && weight && rstd && dx, ANIMA_E_ARG, "rmsnorm_rope_bwd: null pointer");
  if (int rc = check("rmsnorm_rope_bwd", tokens, heads, head_dim, seq_len, cos_tab, sin_tab)) return rc;
  ANIMA_REQUIRE(aligned16(dout) && aligned16(x) && aligned16(dx) && aligned16(weight) && (!cos_tab || (aligned16(cos_tab) && aligned16(sin_tab))),
                ANIMA_E_ALIGN, "rmsnorm_rope_bwd: tensors must be 16-byte aligned");
  if (tokens * heads == 0) return ANIMA_OK;
  const int64_t blocks = ceil_div(tokens, kTokensPerCta);
  const int hpg = heads_per_group(blocks, heads);
  const dim3 grid(static_cast<unsigned>(blocks), static_cast<unsigned>(ceil_div(heads, hpg)));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const auto* gp = static_cast<const __nv_bfloat16*>(dout);
  const auto* xp = static_cast<const __nv_bfloat16*>(x);
  auto* dp = static_cast<__nv_bfloat16*>(dx);
  constexpr int kSmem = kBwdStages * 4 * kThreads * 16;
  static PerDeviceOnce once;
  const cudaError_t rc = per_device_once(once, [] {
    for (auto k : {rmsnorm_rope_bwd_kernel<true, true>, rmsnorm_rope_bwd_kernel<true, false>, rmsnorm_rope_bwd_kernel<false, true>,
                   rmsnorm_rope_bwd_kernel<false, false>})
      if (cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem)) return e;
    return cudaSuccess;
  });
  ANIMA_REQUIRE(rc == cudaSuccess, ANIMA_E_CUDA, "rmsnorm_rope_bwd: cannot reserve %d bytes of shared memory: %s", kSmem,
                cudaGetErrorString(rc));
  auto go = [&](auto kernel) { launch_after(kernel, grid, kThreads, kSmem, s, gp, xp, weight, cos_tab, sin_tab, rstd, tokens, (int)heads, hpg, seq_len, dp); };
  if (cos_tab) weight_is_bf16 ? go(rmsnorm_rope_bwd_kernel<true, true>) : go(rmsnorm_rope_bwd_kernel<true, false>);
  else weight_is_bf16 ? go(rmsnorm_rope_bwd_kernel<false, true>) : go(rmsnorm_rope_bwd_kernel<false, false>);
  ANIMA_CHECK_LAUNCH("rmsnorm_rope_bwd");
  return ANIMA_OK;
}

extern "C" int anima_rmsnorm_rope_fwd(const void* x, const float* weight, const float* cos_tab, const float* sin_tab, float eps,
                                      int64_t tokens, int64_t heads, int64_t head_dim, int64_t seq_len,
                                      void* out, float* rstd, void* stream) {
  return anima_rmsnorm_rope_fwd_ex(x, weight, 0, cos_tab, sin_tab, eps, tokens, heads, head_dim, seq_len, out, rstd, stream);
}

extern "C" int anima_rmsnorm_rope_bwd(const void* dout, const void* x, const float* weight, const float* cos_tab,
                                      const float* sin_tab, const float* rstd, int64_t tokens, int64_t heads, int64_t head_dim,
                                      int64_t seq_len, void* dx, void* stream) {
  return anima_rmsnorm_rope_bwd_ex(dout, x, weight, 0, cos_tab, sin_tab, rstd, tokens, heads, head_dim, seq_len, dx, stream);
}
