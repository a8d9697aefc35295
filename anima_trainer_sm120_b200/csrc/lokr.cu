// LoKr weight kernels.
//
// (1) lokr_merge_quantize: builds merged = W + alpha * kron(w1, w2) for a wrapped
//     Linear and emits, from one read of W, the bf16 merged weight and/or its
//     row-wise and column-wise MXFP8 forms. Replaces the eager
//     get_weight -> cast -> add of lokr_patch.py:76-84 (which materialises the
//     [N,K] Kronecker product in HBM every forward and every checkpoint recompute)
//     plus the two weight quantisations of fp8_quant.py:234-235 / :501.
// (2) lokr_kron_backward: the adapter gradients from dW = dy^T x, i.e. the autograd
//     of torch.kron that lokr_patch.py:19-21 relies on, as one pass over dW.
//
// Rounding of the merged weight follows the eager bf16 path: the Kronecker product
// is rounded to bf16 (torch.kron of bf16 factors; an fp32 product cast to the
// weight dtype rounds the same way), then W + alpha * diff is evaluated in fp32 and
// rounded to bf16 once (torch.add(W, diff, alpha=alpha); alpha == 1 is W + diff).
#include "f32x2.cuh"
#include "mx_quantize_tile.cuh"

namespace anima {
namespace {

using namespace mxq;

template <class F>
__device__ __forceinline__ float to_f32(F v);
template <>
__device__ __forceinline__ float to_f32<float>(float v) { return v; }
template <>
__device__ __forceinline__ float to_f32<__nv_bfloat16>(__nv_bfloat16 v) { return __bfloat162float(v); }

// W + alpha * kron(w1, w2). A thread keeps its place in the Kronecker grid: column block j and offset q are those of
// its columns for the whole tile, row block and offset advance by 16 rows without a division.
template <class F>
struct MergeLoader {
  const __nv_bfloat16* w;
  const F* w1;  // [up, uq]
  const F* w2;  // [vp, vq]
  __nv_bfloat16* merged;  // optional [N, K]
  float alpha;
  int64_t K;
  int vp, vq, uq;
  using Raw = uint4;
  static constexpr bool kZeroSafe = false;   // finish reads the factors
  static constexpr int kSmemBytes = 0;
  struct Cursor {
    int64_t off;     // of the chunk in W (and merged)
    int i, p;        // row block, row inside it
    int j, q;        // column block, column inside it
  };
  __device__ __forceinline__ void prepare(void*) {}
  __device__ __forceinline__ Cursor begin(int64_t r, int64_t c) const {
    const int ri = static_cast<int>(r), ci = static_cast<int>(c);   // N, K < 2^31 is checked on the host
    const int i = ri / vp, j = ci / vq;                             // vq % 8 == 0: the 8 columns share j
    return {r * K + c, i, ri - i * vp, j, ci - j * vq};
  }
  __device__ __forceinline__ void next(Cursor& at) const {
    at.off += 16 * K;
    at.p += 16;
    while (at.p >= vp) {
      at.p -= vp;
      ++at.i;
    }
  }
  __device__ __forceinline__ Raw fetch(const Cursor& at) const { return ldg_stream16(w + at.off); }
  // W comes from HBM (fetch); the factors are small and cache-resident and are read here. The Kronecker product is
  // rounded to bf16 before it is scaled and added, as the eager path does; with alpha == 1 the sum of two bf16 rounded
  // once is one packed bf16 addition.
  __device__ __forceinline__ uint4 finish(const Raw& raw, const Cursor& at) const {
    const f2 a = f2_dup(to_f32(w1[at.i * uq + at.j]));
    const F* src = w2 + static_cast<int64_t>(at.p) * vq + at.q;  // 8 consecutive factors: vq % 8 == 0 keeps them 16/32-byte aligned
    f2 b[4];
    if constexpr (sizeof(F) == 4) {
      const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
      b[0] = f2_make(lo.x, lo.y); b[1] = f2_make(lo.z, lo.w); b[2] = f2_make(hi.x, hi.y); b[3] = f2_make(hi.z, hi.w);
    } else {
      const uint4 v = *reinterpret_cast<const uint4*>(src);
      b[0] = f2_of_bf16(v.x); b[1] = f2_of_bf16(v.y); b[2] = f2_of_bf16(v.z); b[3] = f2_of_bf16(v.w);
    }
    const uint32_t wv[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t o[4];
    if (alpha == 1.0f) {
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = bf16x2_add(wv[e], bf16_of_f2(f2_mul(a, b[e])));
    } else {
      const f2 al = f2_dup(alpha);
#pragma unroll
      for (int e = 0; e < 4; ++e)
        o[e] = bf16_of_f2(f2_fma(al, f2_of_bf16(bf16_of_f2(f2_mul(a, b[e]))), f2_of_bf16(wv[e])));
    }
    const uint4 packed = make_uint4(o[0], o[1], o[2], o[3]);
    if (merged) stg_stream16(merged + at.off, packed);
    return packed;
  }
};

// Writes only the merged bf16 weight (no quantised output requested).
template <class F>
__global__ void __launch_bounds__(256) lokr_merge_only_kernel(const MergeLoader<F> load, int64_t N, int64_t K) {
  const int64_t total = N * (K / 8);
  for (int64_t idx = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = idx / (K / 8);
    const typename MergeLoader<F>::Cursor at = load.begin(r, (idx - r * (K / 8)) * 8);
    (void)load.finish(load.fetch(at), at);
  }
}

// ---- Kronecker backward ------------------------------------------------------
// An item is 8 consecutive elements of one row of w2: (p, q .. q + 7). A CTA takes 32 items at a time: warp i walks the
// uq blocks of block row i of dW for them (lane = item), so one pass over dW has up * vp * vq / 8 threads at work. Its
// dw2 terms meet in shared memory (summed over i in ascending order), its dw1[i][:] sums stay in registers until the
// CTA's last item and are then reduced over the lanes. One thread per item walking all 64 blocks left a 2048 x 1024
// weight with 32 CTAs: 9.0 us; now 5.7, 2048 x 2048 8.8 -> 6.2 (finalize included); 8192 x 2048 fills the GPU either way.
constexpr int kMaxFactor = 8;
constexpr int kKronThreads = 32 * kMaxFactor;
constexpr int kKronCtasPerSm = 4;
// A cluster of four CTAs sums its dw1 terms over distributed shared memory and writes one partial of 64 floats: at most
// one per 128 items, which is what the workspace holds.
constexpr int kKronCluster = 4;

int64_t kron_partials(int64_t vp, int64_t vq) { return ceil_div(vp * (vq / 8), 32 * kKronCluster); }
int64_t kron_clusters(int64_t vp, int64_t vq) {
  return std::min<int64_t>(kron_partials(vp, vq),
                           ceil_div(static_cast<int64_t>(kKronCtasPerSm) * sm_count(), static_cast<int64_t>(kKronCluster)));
}

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float cluster_peer(const float* own, uint32_t rank) {   // the same variable in CTA `rank`
  uint32_t addr = static_cast<uint32_t>(__cvta_generic_to_shared(own));
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(addr) : "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

template <class T>
__device__ __forceinline__ void load8_f2(const T* src, f2 (&v)[4]) {
  if constexpr (sizeof(T) == 2) {
    const uint4 r = *reinterpret_cast<const uint4*>(src);
    v[0] = f2_of_bf16(r.x); v[1] = f2_of_bf16(r.y); v[2] = f2_of_bf16(r.z); v[3] = f2_of_bf16(r.w);
  } else {
    const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
    v[0] = f2_make(lo.x, lo.y); v[1] = f2_make(lo.z, lo.w); v[2] = f2_make(hi.x, hi.y); v[3] = f2_make(hi.z, hi.w);
  }
}

template <class G, class F>
__global__ void __cluster_dims__(kKronCluster, 1, 1) __launch_bounds__(kKronThreads, kKronCtasPerSm)
kron_backward_kernel(const G* __restrict__ dw, const F* __restrict__ w1, const F* __restrict__ w2,
                     float alpha, int64_t K, int vp, int vq, int up, int uq, float* __restrict__ dw2,
                     float* __restrict__ partial) {
  __shared__ __align__(16) float acc_s[kMaxFactor][32 * 8];
  after_previous();
  dw = after_previous(dw);
  w1 = after_previous(w1);
  w2 = after_previous(w2);
  const int t = threadIdx.x, lane = t & 31, i = t >> 5;
  const int vq8 = vq / 8, items = vp * vq8;
  float w1r[kMaxFactor], t1[kMaxFactor];
#pragma unroll
  for (int j = 0; j < kMaxFactor; ++j) {
    w1r[j] = (i < up && j < uq) ? to_f32(w1[i * uq + j]) : 0.f;
    t1[j] = 0.f;
  }
  for (int g0 = blockIdx.x * 32; g0 < items; g0 += gridDim.x * 32) {
    const int item = g0 + lane;
    f2 acc[4] = {0ull, 0ull, 0ull, 0ull};
    if (i < up && item < items) {
      const int p = item / vq8, q = (item - p * vq8) * 8;
      f2 w2v[4];
      const F* f = w2 + static_cast<int64_t>(p) * vq + q;
      if ((reinterpret_cast<uintptr_t>(w2) & 15) == 0) {
        load8_f2(f, w2v);
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) w2v[e] = f2_make(to_f32(f[2 * e]), to_f32(f[2 * e + 1]));
      }
      const G* src = dw + (static_cast<int64_t>(i) * vp + p) * K + q;
#pragma unroll
      for (int j = 0; j < kMaxFactor; ++j) {
        if (j < uq) {
          f2 d[4];
          load8_f2(src + static_cast<int64_t>(j) * vq, d);
          const f2 a1 = f2_dup(w1r[j]);
          f2 s = f2_mul(d[0], w2v[0]);
          acc[0] = f2_fma(d[0], a1, acc[0]);
#pragma unroll
          for (int e = 1; e < 4; ++e) {
            s = f2_fma(d[e], w2v[e], s);
            acc[e] = f2_fma(d[e], a1, acc[e]);
          }
          t1[j] += f2_sum(s);
        }
      }
    }
    f2* dst = reinterpret_cast<f2*>(acc_s[i] + lane * 8);
#pragma unroll
    for (int e = 0; e < 4; ++e) dst[e] = acc[e];
    __syncthreads();
    const int64_t at = static_cast<int64_t>(g0) * 8 + t;   // dw2 [vp, vq] is the items in order
    float sum = 0.f;
#pragma unroll
    for (int k = 0; k < kMaxFactor; ++k) sum += acc_s[k][t];
    if (at < static_cast<int64_t>(items) * 8) dw2[at] = alpha * sum;
    __syncthreads();
  }
  __shared__ float sums[kMaxFactor * kMaxFactor];
#pragma unroll
  for (int j = 0; j < kMaxFactor; ++j) {
    const float s = warp_sum(t1[j]);
    if (lane == 0) sums[i * kMaxFactor + j] = s;
  }
  __syncthreads();
  cluster_sync();
  if (blockIdx.x % kKronCluster == 0 && t < kMaxFactor * kMaxFactor) {
    float s = sums[t];
#pragma unroll
    for (uint32_t r = 1; r < kKronCluster; ++r) s += cluster_peer(sums + t, r);
    partial[blockIdx.x / kKronCluster * (kMaxFactor * kMaxFactor) + t] = s;
  }
  cluster_sync();   // no CTA leaves while its sums may be read
}

__global__ void kron_backward_finalize_kernel(const float* __restrict__ partial, int blocks, float alpha,
                                              int up, int uq, float* __restrict__ dw1) {
  after_previous();
  partial = after_previous(partial);
  const float s = sum_partials_64(partial, blocks);
  const int i = threadIdx.x / kMaxFactor, j = threadIdx.x % kMaxFactor;
  if (threadIdx.x < kMaxFactor * kMaxFactor && i < up && j < uq) dw1[i * uq + j] = alpha * s;
}

int check_factors(const char* who, int64_t N, int64_t K, int64_t up, int64_t uq) {
  ANIMA_REQUIRE(N > 0 && K > 0 && up > 0 && uq > 0, ANIMA_E_ARG, "%s: bad sizes", who);
  ANIMA_REQUIRE(N % up == 0 && K % uq == 0, ANIMA_E_SHAPE,
                "%s: N=%lld, K=%lld not divisible by the w1 shape [%lld,%lld]", who, (long long)N,
                (long long)K, (long long)up, (long long)uq);
  ANIMA_REQUIRE((K / uq) % 8 == 0, ANIMA_E_SHAPE, "%s: K/uq=%lld must be a multiple of 8", who,
                (long long)(K / uq));
  return ANIMA_OK;
}

template <class F>
int launch_merge(const void* w, const void* w1, const void* w2, float alpha, int64_t N, int64_t K,
                 int64_t up, int64_t uq, void* merged, uint8_t* codes_row, uint8_t* scales_row,
                 uint8_t* codes_colT, uint8_t* scales_col, int scale_layout, cudaStream_t s) {
  const MergeLoader<F> load{static_cast<const __nv_bfloat16*>(w), static_cast<const F*>(w1),
                            static_cast<const F*>(w2), static_cast<__nv_bfloat16*>(merged), alpha,
                            K, static_cast<int>(N / up), static_cast<int>(K / uq), static_cast<int>(uq)};
  const bool row = codes_row != nullptr, col = codes_colT != nullptr;
  if (!row && !col) {
    const int64_t total = N * (K / 8);
    lokr_merge_only_kernel<F><<<static_cast<unsigned>(std::min<int64_t>(ceil_div(total, 256), 16LL * sm_count())),
                                256, 0, s>>>(load, N, K);
    return ANIMA_OK;
  }
  QuantParams p{N, K, codes_row, scales_row, codes_colT, scales_col, scale_layout == ANIMA_SCALES_TILED};
  const dim3 grid(static_cast<unsigned>(ceil_div(K, kTile)), static_cast<unsigned>(ceil_div(N, kTile)));
  if (row && col)
    launch_after(mx_quantize_kernel<true, true, MergeLoader<F>>, grid, kThreads, 0, s, p, load);
  else if (row)
    launch_after(mx_quantize_kernel<true, false, MergeLoader<F>>, grid, kThreads, 0, s, p, load);
  else
    launch_after(mx_quantize_kernel<false, true, MergeLoader<F>>, grid, kThreads, 0, s, p, load);
  return ANIMA_OK;
}

}  // namespace
}  // namespace anima

using namespace anima;

extern "C" int anima_lokr_merge_quantize(const void* w, const void* w1, const void* w2,
                                         int factors_are_fp32, float alpha, int64_t N, int64_t K,
                                         int64_t up, int64_t uq, void* merged, uint8_t* codes_row,
                                         uint8_t* scales_row, uint8_t* codes_colT, uint8_t* scales_col,
                                         int scale_layout, void* stream) {
  ANIMA_REQUIRE(w && w1 && w2, ANIMA_E_ARG, "lokr_merge_quantize: null pointer");
  if (int rc = check_factors("lokr_merge_quantize", N, K, up, uq)) return rc;
  const bool row = codes_row != nullptr, col = codes_colT != nullptr;
  ANIMA_REQUIRE(merged || row || col, ANIMA_E_ARG, "lokr_merge_quantize: no output requested");
  ANIMA_REQUIRE((codes_row == nullptr) == (scales_row == nullptr) &&
                    (codes_colT == nullptr) == (scales_col == nullptr),
                ANIMA_E_ARG, "lokr_merge_quantize: codes and scales must be given in pairs");
  ANIMA_REQUIRE(scale_layout == ANIMA_SCALES_PLAIN || scale_layout == ANIMA_SCALES_TILED, ANIMA_E_ARG,
                "lokr_merge_quantize: bad scale_layout %d", scale_layout);
  ANIMA_REQUIRE(!row || K % 32 == 0, ANIMA_E_SHAPE, "lokr_merge_quantize: rowwise needs K %% 32 == 0");
  ANIMA_REQUIRE(!col || N % 32 == 0, ANIMA_E_SHAPE, "lokr_merge_quantize: columnwise needs N %% 32 == 0");
  ANIMA_REQUIRE(ceil_div(N, kTile) <= 65535 && K < (1ll << 31), ANIMA_E_TOO_LARGE, "lokr_merge_quantize: N or K too large");
  ANIMA_REQUIRE(aligned16(w) && aligned16(w2) && (!merged || aligned16(merged)) && (!row || aligned16(codes_row)) &&
                    (!col || aligned16(codes_colT)),
                ANIMA_E_ALIGN, "lokr_merge_quantize: W, w2, merged and code buffers must be 16-byte aligned");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (factors_are_fp32)
    launch_merge<float>(w, w1, w2, alpha, N, K, up, uq, merged, codes_row, scales_row, codes_colT,
                        scales_col, scale_layout, s);
  else
    launch_merge<__nv_bfloat16>(w, w1, w2, alpha, N, K, up, uq, merged, codes_row, scales_row,
                                codes_colT, scales_col, scale_layout, s);
  ANIMA_CHECK_LAUNCH("lokr_merge_quantize");
  return ANIMA_OK;
}

extern "C" int64_t anima_lokr_kron_backward_workspace_bytes(int64_t N, int64_t K, int64_t up,
                                                            int64_t uq) {
  if (N <= 0 || K <= 0 || up <= 0 || uq <= 0 || N % up || K % uq || (K / uq) % 8) return ANIMA_E_SHAPE;
  return kron_partials(N / up, K / uq) * kMaxFactor * kMaxFactor * static_cast<int64_t>(sizeof(float));
}

extern "C" int anima_lokr_kron_backward(const void* dw, int dw_is_fp32, const void* w1, const void* w2,
                                        int factors_are_fp32, float alpha, int64_t N, int64_t K,
                                        int64_t up, int64_t uq, float* dw1, float* dw2, void* workspace,
                                        int64_t workspace_bytes, void* stream) {
  ANIMA_REQUIRE(dw && w1 && w2 && dw1 && dw2, ANIMA_E_ARG, "lokr_kron_backward: null pointer");
  if (int rc = check_factors("lokr_kron_backward", N, K, up, uq)) return rc;
  ANIMA_REQUIRE(up <= kMaxFactor && uq <= kMaxFactor, ANIMA_E_UNSUPPORTED,
                "lokr_kron_backward: w1 larger than %dx%d is not supported", kMaxFactor, kMaxFactor);
  ANIMA_REQUIRE((N / up) * (K / uq) < (1ll << 31), ANIMA_E_TOO_LARGE, "lokr_kron_backward: w2 too large");
  ANIMA_REQUIRE(aligned16(dw) && aligned16(dw2) && (K * (dw_is_fp32 ? 4 : 2)) % 16 == 0, ANIMA_E_ALIGN,
                "lokr_kron_backward: dW and dw2 must be 16-byte aligned");
  const int64_t need = anima_lokr_kron_backward_workspace_bytes(N, K, up, uq);
  ANIMA_REQUIRE(workspace && workspace_bytes >= need, ANIMA_E_WORKSPACE,
                "lokr_kron_backward: workspace of %lld bytes required, got %lld", (long long)need,
                (long long)workspace_bytes);
  const int vp = static_cast<int>(N / up), vq = static_cast<int>(K / uq);
  const int partials = static_cast<int>(kron_clusters(vp, vq)), blocks = partials * kKronCluster;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float* ws = static_cast<float*>(workspace);
#define ANIMA_KRON(G, F)                                                                            \
  launch_after(kron_backward_kernel<G, F>, blocks, kKronThreads, 0, s,                              \
      static_cast<const G*>(dw), static_cast<const F*>(w1), static_cast<const F*>(w2), alpha, K, vp, \
      vq, (int)up, (int)uq, dw2, ws)
  if (dw_is_fp32) {
    if (factors_are_fp32) ANIMA_KRON(float, float); else ANIMA_KRON(float, __nv_bfloat16);
  } else {
    if (factors_are_fp32) ANIMA_KRON(__nv_bfloat16, float); else ANIMA_KRON(__nv_bfloat16, __nv_bfloat16);
  }
#undef ANIMA_KRON
  ANIMA_CHECK_LAUNCH("lokr_kron_backward");
  launch_after(kron_backward_finalize_kernel, 1, kFinalizeThreads, 0, s, ws, partials, alpha, (int)up, (int)uq, dw1);
  ANIMA_CHECK_LAUNCH("lokr_kron_backward finalize");
  return ANIMA_OK;
}
