// Fused AdaLN (LayerNorm without affine, then *(1+scale)+shift) and the gated
// residual x + gate*y, forward and backward, for bf16 activations.
//
// Replaces anima-trainer's five Triton kernels in adaln_kernel.py:
//   _fwd_kernel (:34-68), _bwd_dx_kernel (:71-103), _bwd_dsdb_kernel (:106-154),
//   _gated_add_fwd_kernel (:272-295), _gated_add_bwd_dgate_kernel (:298-329).
// All kernels here are HBM-bound; each tensor is read or written once with
// 16-byte streaming accesses:
//   adaln_fwd      4 B/elem (+ 8 B/row of saved statistics)
//   adaln_bwd      6 B/elem: dx AND the dscale/dshift partial sums come from one
//                  pass over dy and x (the reference makes two passes)
//   gated_add_fwd  6 B/elem
//   gated_add_bwd  6 B/elem: dy and the dgate partial sums from one pass
// The reductions over the hw rows of a sample are two-stage (per-block partials in
// caller-provided scratch, then a fixed-order sum), so results are bit-reproducible;
// the reference uses fp32 atomics. A caller that wants none of them passes null outputs:
// nothing is accumulated, written or summed then.
// Modulation rows (scale, shift, gate) may have a pitch of their own (chunks of one tensor).
#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "f32x2.cuh"
#include "mx_quantize_tile.cuh"

namespace anima {
namespace {

constexpr int kThreads = 256;
constexpr int kRowsPerIter = 4;
constexpr int kMaxBwdThreads = 512;   // one 16-byte chunk per thread and row: d <= 4096

using bf16_t = __nv_bfloat16;

// ------------------------------------------------------------------ forward
// One warp per row; lane l owns the 16-byte chunks l, l+32, ... of the row. The row stays packed (bf16)
// in registers through the three passes (sum, centred squares, output): that keeps the kernel at 64 registers, so
// 4 CTAs (32 warps, 128 KB of loads in flight) fit on an SM. The bound was half instruction issue, half memory
// latency, so the passes take bf16 operands unwidened (add / sub.f32.bf16) and fp32 in pairs (f32x2): 9.5 -> 5
// instructions per element. At [8, 4096, 2048]: plain 54.5 -> 42.4 us (6330 GB/s, the rate of a plain copy), plain +
// operand 86.4 -> 62.5, residual 103.4 -> 84.7, residual + operand 125.6 -> 105.7.
//
// GATED: the row normalised is x_new = x + gate * sub (the gated residual of the PREVIOUS sublayer, same
// arithmetic as gated_add_fwd_kernel: one fp32 fma, rounded once to bf16), which is also written out; the
// two kernels of "residual update, then modulation of the next sublayer" become one pass that reads x and sub
// and writes x_new and y (8 B/elem instead of 6 + 4).
//
// QUANT: the row-wise MXFP8 operand of y (e4m3 codes + one scale byte per 32 columns, the arithmetic of
// mx_quantize on the bf16-rounded y) leaves the same pass: the four lanes that hold 32 consecutive columns
// share their amax with two shuffles, and the scale bytes of 128 columns are gathered into one 32-bit store.
// The linears that consume y then need no quantiser launch of their own (+1.03 B/elem written here against
// 2 B read + 1.03 B written there); y itself may be left unwritten (y == nullptr).
//
// STAGED (hw % 8 == 0: the 8 rows of a CTA belong to one sample): the CTA converts the sample's modulation row
// once, (1 + scale) and shift as fp32 in shared memory, instead of every warp unpacking and adding them for
// its own row; the output pass then reads two 16-byte pieces per operand (split so that consecutive lanes read
// consecutive 16 bytes). Same arithmetic, same bits.
struct FwdArgs {
  const bf16_t *x, *gate, *sub, *scale, *shift;
  float eps;
  int64_t rows, hw, ld_mod;
  int d;
  bf16_t *x_new, *y;
  float *mean, *rstd;
  uint8_t *codes, *scales;   // QUANT: [rows, d], plain [rows, d/32] or tiled (128 x 4 chunks)
  int tiled;
};

template <int NCH, bool GATED, bool QUANT, bool STAGED>
__global__ void __launch_bounds__(kThreads, NCH > 8 ? 2 : 4) adaln_fwd_kernel(const FwdArgs a) {
  extern __shared__ float4 mod_smem[];   // STAGED: [4][d / 8]: (1 + scale) low / high halves, shift low / high
  const int lane = threadIdx.x & 31, d = a.d;
  const int64_t row = static_cast<int64_t>(blockIdx.x) * (kThreads / 32) + (threadIdx.x >> 5);
  if (!STAGED && row >= a.rows) return;    // STAGED: rows % 8 == 0, every warp of every CTA has a row
  const int64_t bt = row / a.hw;
  const bf16_t* xr = a.x + row * d;
  const bf16_t *scale = a.scale + bt * a.ld_mod, *shift = a.shift + bt * a.ld_mod;

  uint4 raw[NCH];
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    const int col = (i * 32 + lane) * 8;
    raw[i] = make_uint4(0u, 0u, 0u, 0u);
    if (col < d) raw[i] = ldg_stream16(xr + col);
  }
  if (STAGED) {
    const int chunks = d >> 3;
    for (int ch = threadIdx.x; ch < chunks; ch += kThreads) {
      float s[8], b[8];
      unpack8(*reinterpret_cast<const uint4*>(scale + ch * 8), s);
      unpack8(*reinterpret_cast<const uint4*>(shift + ch * 8), b);
      mod_smem[ch] = make_float4(1.0f + s[0], 1.0f + s[1], 1.0f + s[2], 1.0f + s[3]);
      mod_smem[chunks + ch] = make_float4(1.0f + s[4], 1.0f + s[5], 1.0f + s[6], 1.0f + s[7]);
      mod_smem[2 * chunks + ch] = make_float4(b[0], b[1], b[2], b[3]);
      mod_smem[3 * chunks + ch] = make_float4(b[4], b[5], b[6], b[7]);
    }
    __syncthreads();   // far ahead of the first read: two reductions over the row come first
  }
  if (GATED) {
    const bf16_t *sub = a.sub + row * d, *gate = a.gate + bt * a.ld_mod;
    // the sublayer output is fetched two chunks ahead of its use (the row of x already fills half the registers);
    // one ahead: 94.4 us at [8, 4096, 2048], two 84.7, three 85.2, four 86.6; 3 CTAs/SM with four 89.8
    constexpr int kAhead = NCH < 2 ? NCH : 2;
    uint4 ring[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; ++i)
      if ((i * 32 + lane) * 8 < d) ring[i] = ldg_stream16(sub + (i * 32 + lane) * 8);
#pragma unroll
    for (int i = 0; i < NCH; ++i) {
      const int col = (i * 32 + lane) * 8;
      const uint4 s = ring[i % kAhead];
      if (i + kAhead < NCH && col + 256 * kAhead < d) ring[i % kAhead] = ldg_stream16(sub + col + 256 * kAhead);
      if (col < d) {
        const uint4 g = *reinterpret_cast<const uint4*>(gate + col);
        raw[i].x = bf16_of_f2(f2_fma_bf16(g.x, s.x, f2_of_bf16(raw[i].x)));
        raw[i].y = bf16_of_f2(f2_fma_bf16(g.y, s.y, f2_of_bf16(raw[i].y)));
        raw[i].z = bf16_of_f2(f2_fma_bf16(g.z, s.z, f2_of_bf16(raw[i].z)));
        raw[i].w = bf16_of_f2(f2_fma_bf16(g.w, s.w, f2_of_bf16(raw[i].w)));
        stg_stream16(a.x_new + row * d + col, raw[i]);   // the normalisation below sees the rounded values
      }
    }
  }
  float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    add_bf16(s0, s1, raw[i].x);
    add_bf16(s2, s3, raw[i].y);
    add_bf16(s0, s1, raw[i].z);
    add_bf16(s2, s3, raw[i].w);
  }
  const float mean = warp_sum((s0 + s1) + (s2 + s3)) / static_cast<float>(d);
  f2 q0 = f2_dup(0.f), q1 = q0;
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    if ((i * 32 + lane) * 8 < d) {  // padded tail must not add mean^2 (adaln_kernel.py:55-57)
      const f2 c0 = f2_bf16_minus(raw[i].x, mean), c1 = f2_bf16_minus(raw[i].y, mean);
      const f2 c2 = f2_bf16_minus(raw[i].z, mean), c3 = f2_bf16_minus(raw[i].w, mean);
      q0 = f2_fma(c0, c0, q0);
      q1 = f2_fma(c1, c1, q1);
      q0 = f2_fma(c2, c2, q0);
      q1 = f2_fma(c3, c3, q1);
    }
  }
  const float var = warp_sum(f2_sum(f2_add(q0, q1))) / static_cast<float>(d);
  const float rstd = 1.0f / sqrtf(var + a.eps);
  const f2 rstd2 = f2_dup(rstd);
#pragma unroll
  for (int i = 0; i < NCH; ++i) {
    const int col = (i * 32 + lane) * 8;
    const bool ok = col < d;
    uint4 out = make_uint4(0u, 0u, 0u, 0u);
    if (ok) {
      f2 s[4], b[4];
      if (STAGED) {
        const int chunks = d >> 3, ch = i * 32 + lane;
        const float4 sl = mod_smem[ch], sh = mod_smem[chunks + ch];
        const float4 bl = mod_smem[2 * chunks + ch], bh = mod_smem[3 * chunks + ch];
        s[0] = f2_make(sl.x, sl.y); s[1] = f2_make(sl.z, sl.w); s[2] = f2_make(sh.x, sh.y); s[3] = f2_make(sh.z, sh.w);
        b[0] = f2_make(bl.x, bl.y); b[1] = f2_make(bl.z, bl.w); b[2] = f2_make(bh.x, bh.y); b[3] = f2_make(bh.z, bh.w);
      } else {
        const uint4 sr = *reinterpret_cast<const uint4*>(scale + col), br = *reinterpret_cast<const uint4*>(shift + col);
        const f2 one = f2_dup(1.0f);
        s[0] = f2_add(one, f2_of_bf16(sr.x)); s[1] = f2_add(one, f2_of_bf16(sr.y));
        s[2] = f2_add(one, f2_of_bf16(sr.z)); s[3] = f2_add(one, f2_of_bf16(sr.w));
        b[0] = f2_of_bf16(br.x); b[1] = f2_of_bf16(br.y); b[2] = f2_of_bf16(br.z); b[3] = f2_of_bf16(br.w);
      }
      out.x = bf16_of_f2(f2_fma(f2_mul(f2_bf16_minus(raw[i].x, mean), rstd2), s[0], b[0]));
      out.y = bf16_of_f2(f2_fma(f2_mul(f2_bf16_minus(raw[i].y, mean), rstd2), s[1], b[1]));
      out.z = bf16_of_f2(f2_fma(f2_mul(f2_bf16_minus(raw[i].z, mean), rstd2), s[2], b[2]));
      out.w = bf16_of_f2(f2_fma(f2_mul(f2_bf16_minus(raw[i].w, mean), rstd2), s[3], b[3]));
      if (!QUANT || a.y != nullptr) stg_stream16(a.y + row * d + col, out);
    }
    if (QUANT) {   // reached by all 32 lanes (d % 32 == 0: the four lanes of a block are in or out together)
      uint2 codes;
      uint32_t sb = mxq::mx_row_block(out, codes);
      if (ok) *reinterpret_cast<uint2*>(a.codes + row * d + col) = codes;
      // scale bytes of blocks 8i + lane/4; lanes 0 and 16 collect the four bytes of their 128 columns
      sb |= __shfl_down_sync(0xffffffffu, sb, 4) << 8;
      sb |= __shfl_down_sync(0xffffffffu, sb, 8) << 16;
      if ((lane & 15) == 0 && ok) {
        const int64_t kb4 = d / 128;   // d % 128 == 0 (checked by the host)
        const int64_t c4 = i * 2 + (lane >> 4);
        uint8_t* dst = a.tiled ? a.scales + ((row >> 7) * kb4 + c4) * 512 + mxq::tiled_offset(static_cast<int>(row & 127), 0)
                               : a.scales + (row * kb4 + c4) * 4;
        *reinterpret_cast<uint32_t*>(dst) = sb;
      }
    }
  }
  if (lane == 0) {
    a.mean[row] = mean;
    a.rstd[row] = rstd;
  }
}

// ------------------------------------------------------------------ backward
// Work split shared by adaln_bwd and gated_add_bwd: the hw rows of every sample are cut into `chunks` contiguous
// pieces, one CTA each; thread t owns the 16-byte column chunk t of every row and carries its partial sums in
// registers. A CTA has as many threads as a row has chunks (rounded up to a warp), so a short row does not leave
// threads idle; the grid then holds proportionally more CTAs.
struct RowSplit {
  int threads;
  int chunks;          // CTAs per sample
  int rows_per_chunk;  // multiple of kRowsPerIter
};

// `sums` = column sums carried (2 dscale, dshift; 3 with dgate; 1 dgate alone). Two splits: the least one, two CTAs a SM,
// and the full one, which keeps 512 threads a SM (1024 for dgate alone: fewer registers) also where rows are narrow. Every
// CTA writes partial sums, so the full split needs up to eight times the workspace. The entries of a fixed workspace contract
// use the least split; the _ex entries the full one where the caller's workspace holds it.
constexpr int kGatedThreadsPerSm = 1024;   // gated_add_bwd: 64 registers, two groups of rows in flight per scheduler
RowSplit make_split(int64_t bt, int64_t hw, int64_t d, int sums, bool full) {
  const int threads = static_cast<int>(std::min<int64_t>(kMaxBwdThreads, ceil_div(ceil_div(d, 8), 32) * 32));
  const int per_sm = full ? std::max(2, (sums == 1 ? kGatedThreadsPerSm : 512) / threads) : 2;
  const int64_t target = static_cast<int64_t>(sm_count()) * per_sm;
  int64_t chunks = std::max<int64_t>(1, ceil_div(target, std::max<int64_t>(bt, 1)));
  int64_t rpc = ceil_div(ceil_div(hw, chunks), kRowsPerIter) * kRowsPerIter;
  chunks = ceil_div(hw, rpc);
  return {threads, static_cast<int>(chunks), static_cast<int>(rpc)};
}

__device__ __forceinline__ uint32_t smem_u32_of(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp_async16(uint32_t smem_addr, const void* gptr) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr), "l"(gptr) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ uint4 lds16(uint32_t smem_addr) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(smem_addr));
  return v;
}

// What reaches x besides the LayerNorm gradient.
//  kPlain   nothing: dx = dx_ln
//  kResid   another gradient of the same tensor: dx = d_res + bf16(dx_ln)   (instead of a separate add)
//  kGated   x is the x_new = x_prev + gate * sub of the one-pass forward: dout = d_res + bf16(dx_ln) is written (it is
//           also the gradient of x_prev), then dsub = gate * dout and the dgate partial sums in the same thread.
// Every rounding point is that of the separate kernels, so all outputs are bit-identical to running them.
enum BwdMode { kPlain, kResid, kGated };

struct BwdArgs {
  const bf16_t *dy, *x, *scale, *d_res, *sub, *gate;
  const float *mean, *rstd;
  int64_t hw, ld_mod;
  int d, rows_per_chunk;
  bf16_t *dx, *dsub;
  float* partial;
};

// MOD: accumulate dscale / dshift (/ dgate) partial sums.
// PF: the next group of rows is copied global -> shared with cp.async while the current one is worked on, each
// thread fetching exactly the 16-byte chunks it will read itself, so no barrier is involved and no register is
// spent on the prefetch. Without it the kernel alternates between waiting for its loads and computing at 16
// resident warps: DRAM half busy, 2.6 long-scoreboard stalls per issue.
// Shared layout: [stage 2][tensor (dy, x[, d_res])][row R][thread] x 16 bytes, then for kGated [row R][thread] of sub,
// which is needed last: its copy starts with the group and is waited for after the row sums.
// The two row sums of a group's R rows are reduced by halving exchanges (9 shuffles for 8 values instead of 40),
// crossed between the warps through shared memory and broadcast by shuffles, not by 64 shared loads per thread.
// At [8, 4096, 2048] with all sums: plain 84.4 -> 74.1 us (5430 GB/s), gated 166.8 -> 140.5 (5730 GB/s); at
// [1, 1200, 2048] 21.3 -> 9.3 and 23.9 -> 11.0, most of it the finalize pass.
constexpr int bwd_prefetch_bytes(BwdMode mode, int threads) {
  return (2 * (mode == kPlain ? 2 : 3) + (mode == kGated ? 1 : 0)) * kRowsPerIter * threads * 16;
}

template <BwdMode MODE, bool MOD, bool PF>
__global__ void __launch_bounds__(kMaxBwdThreads, 1) adaln_bwd_kernel(const BwdArgs a) {
  constexpr int R = kRowsPerIter;
  static_assert(R == 4, "the reduction below is written for four rows (eight sums)");
  constexpr int NOUT = MODE == kGated ? 3 : 2;
  constexpr bool RES = MODE != kPlain, GATED = MODE == kGated;
  constexpr int kMaxWarps = kMaxBwdThreads / 32;
  __shared__ float2 red[2][kMaxWarps][R];

  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, nthreads = blockDim.x, warps = nthreads >> 5;
  const int d = a.d, col = t * 8;
  const bool in = col < d;
  const int64_t bt = blockIdx.y;
  const int64_t row_begin = bt * a.hw + static_cast<int64_t>(blockIdx.x) * a.rows_per_chunk;
  const int64_t row_end = min(bt * a.hw + a.hw, row_begin + a.rows_per_chunk);
  const float inv_d = 1.0f / static_cast<float>(d);

  f2 ops[4], ds[4], db[4], dg[4];
  uint4 gt = make_uint4(0u, 0u, 0u, 0u);
  {
    uint4 s = make_uint4(0u, 0u, 0u, 0u);
    if (in) s = *reinterpret_cast<const uint4*>(a.scale + bt * a.ld_mod + col);
    const f2 one = f2_dup(1.0f);
    ops[0] = f2_add(one, f2_of_bf16(s.x)); ops[1] = f2_add(one, f2_of_bf16(s.y));
    ops[2] = f2_add(one, f2_of_bf16(s.z)); ops[3] = f2_add(one, f2_of_bf16(s.w));
    if (GATED && in) gt = *reinterpret_cast<const uint4*>(a.gate + bt * a.ld_mod + col);
  }
#pragma unroll
  for (int e = 0; e < 4; ++e) ds[e] = db[e] = dg[e] = f2_dup(0.f);

  extern __shared__ uint4 pf_smem[];
  constexpr int kPfTensors = RES ? 3 : 2;
  const uint32_t pf_base = PF ? smem_u32_of(pf_smem) + t * 16 : 0;
  auto pf_addr = [&](int stage, int tensor, int k) {
    return pf_base + static_cast<uint32_t>(((stage * kPfTensors + tensor) * R + k) * nthreads * 16);
  };
  auto prefetch = [&](int64_t r0n, int stage) {   // this thread's chunks of rows r0n .. r0n + R - 1
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int64_t row = r0n + k;
      if (row < row_end && in) {
        cp_async16(pf_addr(stage, 0, k), a.dy + row * d + col);
        cp_async16(pf_addr(stage, 1, k), a.x + row * d + col);
        if (RES) cp_async16(pf_addr(stage, 2, k), a.d_res + row * d + col);
      }
    }
    cp_async_commit();
  };
  if (PF && row_begin < row_end) prefetch(row_begin, 0);

  int buf = 0;
  for (int64_t r0 = row_begin; r0 < row_end; r0 += R) {
    f2 g[R][4], xh[R][4];  // dxhat, xhat
    float mu[R], rs[R];
    if (PF) {
      // start this group's sub and the next group, then wait for this one (a slot is rewritten only after its values
      // were used); two copy groups follow every time, the second one empty at the end
      if (GATED && MOD) {
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (r0 + k < row_end && in) cp_async16(pf_addr(2, 0, k), a.sub + (r0 + k) * d + col);
        cp_async_commit();
      }
      prefetch(r0 + R, buf ^ 1);
      cp_async_wait<GATED && MOD ? 2 : 1>();
    }
    float v[2 * R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const int64_t row = r0 + k;
      const bool row_ok = row < row_end;
      mu[k] = row_ok ? a.mean[row] : 0.f;
      rs[k] = row_ok ? a.rstd[row] : 0.f;
      uint4 gy = make_uint4(0u, 0u, 0u, 0u), xv = gy;
      if (row_ok && in) {
        gy = PF ? lds16(pf_addr(buf, 0, k)) : ldg_stream16(a.dy + row * d + col);
        xv = PF ? lds16(pf_addr(buf, 1, k)) : ldg_stream16(a.x + row * d + col);
      }
      const uint32_t gw[4] = {gy.x, gy.y, gy.z, gy.w}, xw[4] = {xv.x, xv.y, xv.z, xv.w};
      const f2 rs2 = f2_dup(rs[k]);
      f2 p1 = f2_dup(0.f), p2 = p1;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        // a chunk outside the row has dy = 0: whatever its xhat is, it adds nothing below
        const f2 xhat = f2_mul(f2_bf16_minus(xw[e], mu[k]), rs2);
        const f2 dyv = f2_of_bf16(gw[e]);
        if (MOD) {
          ds[e] = f2_fma(dyv, xhat, ds[e]);
          db[e] = f2_add(db[e], dyv);
        }
        const f2 dxhat = f2_mul(dyv, ops[e]);
        xh[k][e] = xhat;
        g[k][e] = dxhat;
        p1 = f2_add(p1, dxhat);
        p2 = f2_fma(dxhat, xhat, p2);
      }
      v[2 * k] = f2_sum(p1);
      v[2 * k + 1] = f2_sum(p2);
    }
    {
      // after the exchanges lane l holds the warp's total of sum (l >> 2): 8 -> 4 -> 2 -> 1 values, then two adds
      const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
      float w4[4], w2[2], w1;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float keep = b4 ? v[4 + i] : v[i], send = b4 ? v[i] : v[4 + i];
        w4[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float keep = b3 ? w4[2 + i] : w4[i], send = b3 ? w4[i] : w4[2 + i];
        w2[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
      }
      {
        const float keep = b2 ? w2[1] : w2[0], send = b2 ? w2[0] : w2[1];
        w1 = keep + __shfl_xor_sync(0xffffffffu, send, 4);
      }
      w1 += __shfl_xor_sync(0xffffffffu, w1, 2);
      w1 += __shfl_xor_sync(0xffffffffu, w1, 1);
      if ((lane & 3) == 0) reinterpret_cast<float*>(red[buf][warp])[lane >> 2] = w1;
    }
    __syncthreads();
    // lane l adds row (l & 3)'s two sums over warps (l >> 2), + 8; then over the lanes of the same row
    float2 c = make_float2(0.f, 0.f);
    if ((lane >> 2) < warps) c = red[buf][lane >> 2][lane & 3];
    if ((lane >> 2) + 8 < warps) {
      const float2 c8 = red[buf][(lane >> 2) + 8][lane & 3];
      c.x += c8.x;
      c.y += c8.y;
    }
#pragma unroll
    for (int o = 4; o < 32; o <<= 1) {
      c.x += __shfl_xor_sync(0xffffffffu, c.x, o);
      c.y += __shfl_xor_sync(0xffffffffu, c.y, o);
    }
    c.x *= -inv_d;
    c.y *= -inv_d;
    if (PF && GATED && MOD) cp_async_wait<1>();   // sub has landed
#pragma unroll
    for (int k = 0; k < R; ++k) {
      const f2 nc1 = f2_dup(__shfl_sync(0xffffffffu, c.x, k)), nc2 = f2_dup(__shfl_sync(0xffffffffu, c.y, k));
      const int64_t row = r0 + k;
      if (row < row_end && in) {
        const f2 rs2 = f2_dup(rs[k]);
        uint4 o;   // rs * ((dxhat - c1) - xhat * c2)
        o.x = bf16_of_f2(f2_mul(rs2, f2_fma(xh[k][0], nc2, f2_add(g[k][0], nc1))));
        o.y = bf16_of_f2(f2_mul(rs2, f2_fma(xh[k][1], nc2, f2_add(g[k][1], nc1))));
        o.z = bf16_of_f2(f2_mul(rs2, f2_fma(xh[k][2], nc2, f2_add(g[k][2], nc1))));
        o.w = bf16_of_f2(f2_mul(rs2, f2_fma(xh[k][3], nc2, f2_add(g[k][3], nc1))));
        if (RES) {   // bf16 sum of the two gradients, as the separate add would store it
          const uint4 res = PF ? lds16(pf_addr(buf, 2, k)) : ldg_stream16(a.d_res + row * d + col);
          o.x = bf16x2_add(res.x, o.x);
          o.y = bf16x2_add(res.y, o.y);
          o.z = bf16x2_add(res.z, o.z);
          o.w = bf16x2_add(res.w, o.w);
        }
        stg_stream16(a.dx + row * d + col, o);
        if (GATED) {
          if (MOD) {
            const uint4 sub = PF ? lds16(pf_addr(2, 0, k)) : ldg_stream16(a.sub + row * d + col);
            dg[0] = f2_fma_bf16(o.x, sub.x, dg[0]);
            dg[1] = f2_fma_bf16(o.y, sub.y, dg[1]);
            dg[2] = f2_fma_bf16(o.z, sub.z, dg[2]);
            dg[3] = f2_fma_bf16(o.w, sub.w, dg[3]);
          }
          // the fp32 product of two bf16 is exact, so the packed bf16 product rounds to the same value
          o.x = mxq::bf16x2_mul(gt.x, o.x);
          o.y = mxq::bf16x2_mul(gt.y, o.y);
          o.z = mxq::bf16x2_mul(gt.z, o.z);
          o.w = mxq::bf16x2_mul(gt.w, o.w);
          stg_stream16(a.dsub + row * d + col, o);
        }
      }
    }
    buf ^= 1;
  }

  // partial[bt][chunk][0] = dscale sums, [1] = dshift sums, ([2] = dgate sums); fp32 [d] each.
  if (MOD && in) {
    float* out = a.partial + ((bt * gridDim.x + blockIdx.x) * NOUT) * static_cast<int64_t>(d) + col;
    auto put = [](float* dst, const f2 (&s)[4]) {
      *reinterpret_cast<float4*>(dst) = make_float4(f2_lo(s[0]), f2_hi(s[0]), f2_lo(s[1]), f2_hi(s[1]));
      *reinterpret_cast<float4*>(dst + 4) = make_float4(f2_lo(s[2]), f2_hi(s[2]), f2_lo(s[3]), f2_hi(s[3]));
    };
    put(out, ds);
    put(out + d, db);
    if (GATED) put(out + 2 * d, dg);
  }
}

// out_k[bt][c] = bf16( sum over chunks of partial[bt][chunk][k][c] ), k < nout. A CTA owns 64 columns of one sum:
// 16 threads of four columns times 16 groups, group q adding its contiguous slice of the chunks in ascending order,
// then the group sums in ascending order: fixed association, and no thread walks more than chunks / 16 loads (one
// thread per column walked all of them: 13 us for the 150 chunks of one 1200-row sample, now 3 us).
__global__ void __launch_bounds__(256)
finalize_partials_kernel(const float* __restrict__ partial, int chunks, int nout, int d, bf16_t* __restrict__ out0,
                         bf16_t* __restrict__ out1, bf16_t* __restrict__ out2) {
  __shared__ float4 sums[16][16];
  const int cx = threadIdx.x & 15, q = threadIdx.x >> 4;
  const int64_t bt = blockIdx.y;
  const int k = blockIdx.z;
  const int col = blockIdx.x * 64 + cx * 4;
  bf16_t* out = k == 0 ? out0 : k == 1 ? out1 : out2;
  if (out == nullptr) return;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (col < d) {
    const int per = (chunks + 15) / 16, c0 = q * per, c1 = min(chunks, c0 + per);
    const float* src = partial + ((bt * chunks + c0) * nout + k) * static_cast<int64_t>(d) + col;
    const int64_t step = static_cast<int64_t>(nout) * d;
#pragma unroll 4
    for (int c = c0; c < c1; ++c, src += step) {
      const float4 v = *reinterpret_cast<const float4*>(src);
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
  }
  sums[q][cx] = s;
  __syncthreads();
  if (threadIdx.x < 64 && blockIdx.x * 64 + threadIdx.x < d) {
    float t = 0.f;
#pragma unroll
    for (int g = 0; g < 16; ++g) t += reinterpret_cast<const float*>(sums[g])[threadIdx.x];
    out[bt * d + blockIdx.x * 64 + threadIdx.x] = __float2bfloat16_rn(t);
  }
}

void launch_finalize(const float* partial, int64_t bt, int chunks, int nout, int64_t d, void* o0, void* o1, void* o2,
                     cudaStream_t s) {
  const dim3 grid(static_cast<unsigned>(ceil_div(d, 64)), static_cast<unsigned>(bt), static_cast<unsigned>(nout));
  finalize_partials_kernel<<<grid, 256, 0, s>>>(partial, chunks, nout, static_cast<int>(d), static_cast<bf16_t*>(o0),
                                                static_cast<bf16_t*>(o1), static_cast<bf16_t*>(o2));
}

// ------------------------------------------------------------------ gated residual
// A thread owns one 16-byte column chunk and walks rows: the gate is read once, and no index is divided per chunk.
// cw = chunks of a row a CTA covers side by side, threads / cw rows at a time; rows wider than a CTA have `tiles` column
// tiles, the inner part of blockIdx.x. blockIdx.y = sample, in steps of gridDim.y where there are more than a grid has.
template <int U>
__global__ void __launch_bounds__(kThreads)
gated_add_fwd_kernel(const bf16_t* __restrict__ x, const bf16_t* __restrict__ gate, const bf16_t* __restrict__ y, int64_t hw,
                     int64_t ld_mod, int64_t d, int cw, int64_t rows_per_cta, int64_t samples, unsigned tiles,
                     bf16_t* __restrict__ out) {
  const int ty = threadIdx.x / cw, tx = threadIdx.x - ty * cw, ny = kThreads / cw;
  const unsigned part = blockIdx.x / tiles, tile = blockIdx.x - part * tiles;
  const int64_t c = (static_cast<int64_t>(tile) * cw + tx) * 8;
  if (ty >= ny || c >= d) return;
  const int64_t begin = part * rows_per_cta, end = min(hw, begin + rows_per_cta);
  for (int64_t bt = blockIdx.y; bt < samples; bt += gridDim.y) {
    const uint4 g = *reinterpret_cast<const uint4*>(gate + bt * ld_mod + c);
    const int64_t base = bt * hw * d + c;
    for (int64_t r = begin + ty; r < end; r += static_cast<int64_t>(ny) * U) {
      uint4 xa[U], ya[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t row = r + static_cast<int64_t>(u) * ny;
        if (row < end) {
          xa[u] = ldg_stream16(x + base + row * d);
          ya[u] = ldg_stream16(y + base + row * d);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int64_t row = r + static_cast<int64_t>(u) * ny;
        if (row < end) {
          uint4 o;
          o.x = bf16_of_f2(f2_fma_bf16(g.x, ya[u].x, f2_of_bf16(xa[u].x)));
          o.y = bf16_of_f2(f2_fma_bf16(g.y, ya[u].y, f2_of_bf16(xa[u].y)));
          o.z = bf16_of_f2(f2_fma_bf16(g.z, ya[u].z, f2_of_bf16(xa[u].z)));
          o.w = bf16_of_f2(f2_fma_bf16(g.w, ya[u].w, f2_of_bf16(xa[u].w)));
          stg_stream16(out + base + row * d, o);
        }
      }
    }
  }
}

template <bool MOD>
__global__ void __launch_bounds__(kMaxBwdThreads, kGatedThreadsPerSm / kMaxBwdThreads)
gated_add_bwd_kernel(const bf16_t* __restrict__ dout, const bf16_t* __restrict__ y, const bf16_t* __restrict__ gate,
                     int64_t hw, int64_t ld_mod, int d, int rows_per_chunk, bf16_t* __restrict__ dy,
                     float* __restrict__ partial) {
  constexpr int R = kRowsPerIter;
  const int col = threadIdx.x * 8;
  const int64_t bt = blockIdx.y;
  const int64_t row_begin = bt * hw + static_cast<int64_t>(blockIdx.x) * rows_per_chunk;
  const int64_t row_end = min(bt * hw + hw, row_begin + rows_per_chunk);
  if (col >= d) return;
  const uint4 g = *reinterpret_cast<const uint4*>(gate + bt * ld_mod + col);
  f2 dg[4];
#pragma unroll
  for (int e = 0; e < 4; ++e) dg[e] = f2_dup(0.f);
  for (int64_t r0 = row_begin; r0 < row_end; r0 += R) {
    uint4 a[R], b[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      a[k] = b[k] = make_uint4(0u, 0u, 0u, 0u);
      if (r0 + k < row_end) {
        a[k] = ldg_stream16(dout + (r0 + k) * d + col);
        if (MOD) b[k] = ldg_stream16(y + (r0 + k) * d + col);
      }
    }
#pragma unroll
    for (int k = 0; k < R; ++k) {
      if (MOD) {
        dg[0] = f2_fma_bf16(a[k].x, b[k].x, dg[0]);
        dg[1] = f2_fma_bf16(a[k].y, b[k].y, dg[1]);
        dg[2] = f2_fma_bf16(a[k].z, b[k].z, dg[2]);
        dg[3] = f2_fma_bf16(a[k].w, b[k].w, dg[3]);
      }
      const uint4 o = make_uint4(mxq::bf16x2_mul(g.x, a[k].x), mxq::bf16x2_mul(g.y, a[k].y), mxq::bf16x2_mul(g.z, a[k].z),
                                 mxq::bf16x2_mul(g.w, a[k].w));
      if (r0 + k < row_end) stg_stream16(dy + (r0 + k) * d + col, o);
    }
  }
  if (MOD) {
    float* out = partial + (bt * gridDim.x + blockIdx.x) * static_cast<int64_t>(d) + col;
    *reinterpret_cast<float4*>(out) = make_float4(f2_lo(dg[0]), f2_hi(dg[0]), f2_lo(dg[1]), f2_hi(dg[1]));
    *reinterpret_cast<float4*>(out + 4) = make_float4(f2_lo(dg[2]), f2_hi(dg[2]), f2_lo(dg[3]), f2_hi(dg[3]));
  }
}

int check_rows(const char* who, int64_t rows, int64_t hw, int64_t d, int64_t max_d) {
  ANIMA_REQUIRE(rows >= 0 && hw > 0 && d > 0, ANIMA_E_ARG, "%s: bad sizes rows=%lld hw=%lld d=%lld", who,
                (long long)rows, (long long)hw, (long long)d);
  ANIMA_REQUIRE(rows % hw == 0, ANIMA_E_SHAPE, "%s: rows=%lld is not a multiple of hw=%lld", who,
                (long long)rows, (long long)hw);
  ANIMA_REQUIRE(d % 8 == 0, ANIMA_E_SHAPE, "%s: d=%lld must be a multiple of 8", who, (long long)d);
  ANIMA_REQUIRE(d <= max_d, ANIMA_E_TOO_LARGE, "%s: d=%lld exceeds the supported maximum %lld", who,
                (long long)d, (long long)max_d);
  return ANIMA_OK;
}
int check_mod(const char* who, int64_t ld_mod, int64_t d) {
  ANIMA_REQUIRE(ld_mod >= d && ld_mod % 8 == 0, ANIMA_E_ALIGN,
                "%s: modulation row pitch %lld must be a multiple of 8 and at least d=%lld", who, (long long)ld_mod,
                (long long)d);
  return ANIMA_OK;
}
int check_batch(const char* who, int64_t bt) {
  ANIMA_REQUIRE(bt <= 65535, ANIMA_E_TOO_LARGE, "%s: rows/hw=%lld exceeds 65535", who, (long long)bt);
  return ANIMA_OK;
}
// common rule of the tensors: present and 16-byte aligned
bool all_aligned(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if (!aligned16(p)) return false;
  return true;
}
bool all_there(std::initializer_list<const void*> ps) {
  for (const void* p : ps)
    if (!p) return false;
  return true;
}
const bf16_t* in(const void* p) { return static_cast<const bf16_t*>(p); }
bf16_t* out(void* p) { return static_cast<bf16_t*>(p); }

// ANIMA_ADALN_FWD_STAGING=0 keeps the modulation in global memory (read per call; for tests and comparison).
bool adaln_fwd_staging_enabled() {
  const char* v = getenv("ANIMA_ADALN_FWD_STAGING");
  return !(v && v[0] == '0');
}

// One launcher for the four forward forms; the kernel is picked by the row length (256 columns per chunk).
template <bool GATED, bool QUANT>
void launch_adaln_fwd(const FwdArgs& a, cudaStream_t s) {
  const unsigned grid = static_cast<unsigned>(ceil_div(a.rows, kThreads / 32));
  // one sample per CTA (8 rows) lets the CTA convert the modulation row once; 8 * d bytes of shared memory
  const bool staged = a.hw % (kThreads / 32) == 0 && adaln_fwd_staging_enabled();
  const size_t smem = staged ? static_cast<size_t>(a.d) * 8 : 0;
#define ANIMA_LAUNCH_FWD(N)                                                                  \
  do {                                                                                       \
    if (staged) adaln_fwd_kernel<N, GATED, QUANT, true><<<grid, kThreads, smem, s>>>(a);     \
    else adaln_fwd_kernel<N, GATED, QUANT, false><<<grid, kThreads, 0, s>>>(a);              \
  } while (0)
  const int chunks = static_cast<int>(ceil_div(a.d, 256));
  if (chunks <= 1) ANIMA_LAUNCH_FWD(1);
  else if (chunks <= 2) ANIMA_LAUNCH_FWD(2);
  else if (chunks <= 4) ANIMA_LAUNCH_FWD(4);
  else if (chunks <= 6) ANIMA_LAUNCH_FWD(6);
  else if (chunks <= 8) ANIMA_LAUNCH_FWD(8);
  else if (chunks <= 12) ANIMA_LAUNCH_FWD(12);
  else ANIMA_LAUNCH_FWD(16);
#undef ANIMA_LAUNCH_FWD
}

int check_row_codes(const char* who, int64_t rows, int64_t d, const uint8_t* codes_row, const uint8_t* scales_row,
                    int scale_layout) {
  ANIMA_REQUIRE(codes_row && scales_row, ANIMA_E_ARG, "%s: null code or scale buffer", who);
  ANIMA_REQUIRE(scale_layout == ANIMA_SCALES_PLAIN || scale_layout == ANIMA_SCALES_TILED, ANIMA_E_ARG,
                "%s: bad scale_layout %d", who, scale_layout);
  ANIMA_REQUIRE(d % 128 == 0, ANIMA_E_SHAPE, "%s: d=%lld must be a multiple of 128", who, (long long)d);
  ANIMA_REQUIRE(scale_layout == ANIMA_SCALES_PLAIN || rows % 128 == 0, ANIMA_E_SHAPE,
                "%s: tiled scales need rows %% 128 == 0 (rows=%lld)", who, (long long)rows);
  ANIMA_REQUIRE((reinterpret_cast<uintptr_t>(codes_row) & 7) == 0 && (reinterpret_cast<uintptr_t>(scales_row) & 3) == 0,
                ANIMA_E_ALIGN, "%s: codes must be 8-byte and scales 4-byte aligned", who);
  return ANIMA_OK;
}

// All forward forms. gated: x_new = x + gate * sub first; quant: the operand of y too (y may then be null).
int forward(const char* who, bool gated, bool quant, const FwdArgs& a, int scale_layout, void* stream) {
  ANIMA_REQUIRE(all_there({a.x, a.scale, a.shift, a.mean, a.rstd}) && (quant || a.y) &&
                    (!gated || all_there({a.gate, a.sub, a.x_new})),
                ANIMA_E_ARG, "%s: null pointer", who);
  if (int rc = check_rows(who, a.rows, a.hw, a.d, 4096)) return rc;
  if (int rc = check_mod(who, a.ld_mod, a.d)) return rc;
  if (quant)
    if (int rc = check_row_codes(who, a.rows, a.d, a.codes, a.scales, scale_layout)) return rc;
  ANIMA_REQUIRE(all_aligned({a.x, a.gate, a.sub, a.scale, a.shift, a.x_new, a.y}), ANIMA_E_ALIGN,
                "%s: tensors must be 16-byte aligned", who);
  if (a.rows == 0) return ANIMA_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (gated && quant) launch_adaln_fwd<true, true>(a, s);
  else if (gated) launch_adaln_fwd<true, false>(a, s);
  else if (quant) launch_adaln_fwd<false, true>(a, s);
  else launch_adaln_fwd<false, false>(a, s);
  ANIMA_CHECK_LAUNCH(who);
  return ANIMA_OK;
}

template <BwdMode MODE, bool MOD>
int launch_adaln_bwd(dim3 grid, int threads, const BwdArgs& a, cudaStream_t s) {
  const char* env = getenv("ANIMA_ADALN_BWD_PREFETCH");   // 0 keeps the plain loads, for comparison; same bits
  if (env && env[0] == '0') {
    adaln_bwd_kernel<MODE, MOD, false><<<grid, threads, 0, s>>>(a);
    return ANIMA_OK;
  }
  constexpr int kMost = bwd_prefetch_bytes(MODE, kMaxBwdThreads);
  static PerDeviceOnce once;
  const cudaError_t rc = per_device_once(once, [] {
    return cudaFuncSetAttribute(adaln_bwd_kernel<MODE, MOD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMost);
  });
  ANIMA_REQUIRE(rc == cudaSuccess, ANIMA_E_CUDA, "adaln_bwd: cannot reserve %d bytes of shared memory: %s", kMost,
                cudaGetErrorString(rc));
  adaln_bwd_kernel<MODE, MOD, true><<<grid, threads, bwd_prefetch_bytes(MODE, threads), s>>>(a);
  return ANIMA_OK;
}

int64_t partial_bytes(int64_t rows, int64_t hw, int64_t d, int sums, bool full) {
  if (rows < 0 || hw <= 0 || d <= 0 || rows % hw) return ANIMA_E_SHAPE;
  const int64_t chunks = make_split(rows / hw, hw, d, sums, full).chunks;
  return (rows / hw) * chunks * sums * d * static_cast<int64_t>(sizeof(float));
}

// All AdaLN backward forms (see BwdMode); null dscale, dshift and dgate: no partial sums, no workspace.
int backward(const char* who, BwdMode mode, BwdArgs a, int64_t rows, void* dscale, void* dshift, void* dgate, void* workspace,
             int64_t workspace_bytes, void* stream) {
  ANIMA_REQUIRE(all_there({a.dy, a.x, a.scale, a.mean, a.rstd, a.dx}) && (mode == kPlain || a.d_res) &&
                    (mode != kGated || all_there({a.sub, a.gate, a.dsub})),
                ANIMA_E_ARG, "%s: null pointer", who);
  if (int rc = check_rows(who, rows, a.hw, a.d, 4096)) return rc;
  if (int rc = check_mod(who, a.ld_mod, a.d)) return rc;
  ANIMA_REQUIRE(all_aligned({a.dy, a.x, a.scale, a.d_res, a.sub, a.gate, a.dx, a.dsub}), ANIMA_E_ALIGN,
                "%s: tensors must be 16-byte aligned", who);
  if (rows == 0) return ANIMA_OK;
  const int64_t bt = rows / a.hw;
  if (int rc = check_batch(who, bt)) return rc;
  const bool mod = dscale || dshift || dgate;
  const int nout = mode == kGated ? 3 : 2;
  const RowSplit sp = make_split(bt, a.hw, a.d, nout, !mod || workspace_bytes >= partial_bytes(rows, a.hw, a.d, nout, true));
  if (mod) {
    const int64_t need = partial_bytes(rows, a.hw, a.d, nout, false);
    ANIMA_REQUIRE(workspace && aligned16(workspace) && workspace_bytes >= need, ANIMA_E_WORKSPACE,
                  "%s: workspace of %lld bytes (16-byte aligned) required, got %lld", who, (long long)need,
                  (long long)workspace_bytes);
  }
  a.rows_per_chunk = sp.rows_per_chunk;
  a.partial = static_cast<float*>(workspace);
  const dim3 grid(sp.chunks, static_cast<unsigned>(bt));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int rc;
  if (mode == kGated) rc = mod ? launch_adaln_bwd<kGated, true>(grid, sp.threads, a, s) : launch_adaln_bwd<kGated, false>(grid, sp.threads, a, s);
  else if (mode == kResid) rc = mod ? launch_adaln_bwd<kResid, true>(grid, sp.threads, a, s) : launch_adaln_bwd<kResid, false>(grid, sp.threads, a, s);
  else rc = mod ? launch_adaln_bwd<kPlain, true>(grid, sp.threads, a, s) : launch_adaln_bwd<kPlain, false>(grid, sp.threads, a, s);
  if (rc) return rc;
  ANIMA_CHECK_LAUNCH(who);
  if (mod) {
    launch_finalize(a.partial, bt, sp.chunks, nout, a.d, dscale, dshift, dgate, s);
    ANIMA_CHECK_LAUNCH("adaln_bwd finalize");
  }
  return ANIMA_OK;
}

// What an entry of a fixed workspace contract may use of its workspace: the least split's bytes, however large it is, so
// that its sums do not depend on the size.
int64_t at_most_least(int64_t workspace_bytes, int64_t rows, int64_t hw, int64_t d, int sums) {
  const int64_t least = partial_bytes(rows, hw, d, sums, false);
  return least >= 0 ? std::min(workspace_bytes, least) : workspace_bytes;
}

int gated_forward(const void* x, const void* gate, int64_t ld_gate, const void* y, int64_t rows, int64_t hw, int64_t d,
                  void* o, void* stream) {
  ANIMA_REQUIRE(all_there({x, gate, y, o}), ANIMA_E_ARG, "gated_add_fwd: null pointer");
  if (int rc = check_rows("gated_add_fwd", rows, hw, d, INT32_MAX / 2)) return rc;
  if (int rc = check_mod("gated_add_fwd", ld_gate, d)) return rc;
  ANIMA_REQUIRE(all_aligned({x, gate, y, o}), ANIMA_E_ALIGN, "gated_add_fwd: tensors must be 16-byte aligned");
  if (rows == 0) return ANIMA_OK;
  const int64_t bt = rows / hw, d8 = d / 8;
  constexpr int U = 4;
  const int cw = static_cast<int>(std::min<int64_t>(d8, kThreads)), ny = kThreads / cw;
  const int64_t tiles = ceil_div(d8, cw);
  // about eight CTAs a SM; a CTA takes at least one unrolled step of rows
  const int64_t want = std::max<int64_t>(1, 8LL * sm_count() / std::max<int64_t>(1, bt * tiles));
  const int64_t rpc = ceil_div(ceil_div(hw, want), static_cast<int64_t>(ny) * U) * ny * U;
  const dim3 grid(static_cast<unsigned>(ceil_div(hw, rpc) * tiles), static_cast<unsigned>(std::min<int64_t>(bt, 65535)));
  gated_add_fwd_kernel<U><<<grid, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(
      in(x), in(gate), in(y), hw, ld_gate, d, cw, rpc, bt, static_cast<unsigned>(tiles), out(o));
  ANIMA_CHECK_LAUNCH("gated_add_fwd");
  return ANIMA_OK;
}

int gated_backward(const void* dout, const void* y, const void* gate, int64_t ld_gate, int64_t rows, int64_t hw, int64_t d,
                   void* dy, void* dgate, void* workspace, int64_t workspace_bytes, void* stream) {
  ANIMA_REQUIRE(all_there({dout, gate, dy}) && (y || !dgate), ANIMA_E_ARG, "gated_add_bwd: null pointer");
  if (int rc = check_rows("gated_add_bwd", rows, hw, d, 4096)) return rc;
  if (int rc = check_mod("gated_add_bwd", ld_gate, d)) return rc;
  ANIMA_REQUIRE(all_aligned({dout, y, gate, dy}), ANIMA_E_ALIGN, "gated_add_bwd: tensors must be 16-byte aligned");
  if (rows == 0) return ANIMA_OK;
  const int64_t bt = rows / hw;
  if (int rc = check_batch("gated_add_bwd", bt)) return rc;
  const RowSplit sp = make_split(bt, hw, d, 1, !dgate || workspace_bytes >= partial_bytes(rows, hw, d, 1, true));
  const dim3 grid(sp.chunks, static_cast<unsigned>(bt));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  float* ws = static_cast<float*>(workspace);
  if (!dgate) {
    gated_add_bwd_kernel<false><<<grid, sp.threads, 0, s>>>(in(dout), in(y), in(gate), hw, ld_gate, (int)d, sp.rows_per_chunk, out(dy), nullptr);
    ANIMA_CHECK_LAUNCH("gated_add_bwd");
    return ANIMA_OK;
  }
  const int64_t need = partial_bytes(rows, hw, d, 1, false);
  ANIMA_REQUIRE(workspace && aligned16(workspace) && workspace_bytes >= need, ANIMA_E_WORKSPACE,
                "gated_add_bwd: workspace of %lld bytes (16-byte aligned) required, got %lld",
                (long long)need, (long long)workspace_bytes);
  gated_add_bwd_kernel<true><<<grid, sp.threads, 0, s>>>(in(dout), in(y), in(gate), hw, ld_gate, (int)d, sp.rows_per_chunk, out(dy), ws);
  ANIMA_CHECK_LAUNCH("gated_add_bwd");
  launch_finalize(ws, bt, sp.chunks, 1, d, dgate, nullptr, nullptr, s);
  ANIMA_CHECK_LAUNCH("gated_add_bwd finalize");
  return ANIMA_OK;
}

}  // namespace
}  // namespace anima

using namespace anima;

// The entries with every option: pitch of the modulation rows, null outputs for gradients nobody wants, full row split.
extern "C" int64_t anima_adaln_bwd_ex_workspace_bytes(int64_t rows, int64_t hw, int64_t d, int sums) {
  if (sums < 1 || sums > 3) return ANIMA_E_ARG;
  return partial_bytes(rows, hw, d, sums, true);
}

extern "C" int anima_adaln_fwd_ex(const void* x, const void* gate, const void* sub, const void* scale, const void* shift,
                                  int64_t ld_mod, float eps, int64_t rows, int64_t hw, int64_t d, void* x_new, void* y,
                                  float* mean, float* rstd, uint8_t* codes_row, uint8_t* scales_row, int scale_layout,
                                  void* stream) {
  const FwdArgs a{in(x), in(gate), in(sub), in(scale), in(shift), eps, rows, hw, ld_mod, static_cast<int>(std::min<int64_t>(d, INT32_MAX)),
                  out(x_new), out(y), mean, rstd, codes_row, scales_row, scale_layout == ANIMA_SCALES_TILED};
  return forward("adaln_fwd_ex", sub != nullptr, codes_row != nullptr, a, scale_layout, stream);
}

extern "C" int anima_adaln_bwd_ex(const void* dy, const void* d_res, const void* x, const void* scale, const void* gate,
                                  const void* sub, int64_t ld_mod, const float* mean, const float* rstd, int64_t rows,
                                  int64_t hw, int64_t d, void* dx, void* dsub, void* dscale, void* dshift, void* dgate,
                                  void* workspace, int64_t workspace_bytes, void* stream) {
  const BwdArgs a{in(dy), in(x), in(scale), in(d_res), in(sub), in(gate), mean, rstd, hw, ld_mod,
                  static_cast<int>(std::min<int64_t>(d, INT32_MAX)), 0, out(dx), out(dsub), nullptr};
  return backward("adaln_bwd_ex", sub ? kGated : d_res ? kResid : kPlain, a, rows, dscale, dshift, dgate, workspace,
                  workspace_bytes, stream);
}

extern "C" int anima_gated_add_fwd_ex(const void* x, const void* gate, int64_t ld_gate, const void* y, int64_t rows,
                                      int64_t hw, int64_t d, void* o, void* stream) {
  return gated_forward(x, gate, ld_gate, y, rows, hw, d, o, stream);
}
extern "C" int anima_gated_add_bwd_ex(const void* dout, const void* y, const void* gate, int64_t ld_gate, int64_t rows,
                                      int64_t hw, int64_t d, void* dy, void* dgate, void* workspace,
                                      int64_t workspace_bytes, void* stream) {
  return gated_backward(dout, y, gate, ld_gate, rows, hw, d, dy, dgate, workspace, workspace_bytes, stream);
}

extern "C" int anima_adaln_fwd(const void* x, const void* scale, const void* shift, float eps,
                               int64_t rows, int64_t hw, int64_t d, void* y, float* mean, float* rstd,
                               void* stream) {
  const FwdArgs a{in(x), nullptr, nullptr, in(scale), in(shift), eps, rows, hw, d, static_cast<int>(std::min<int64_t>(d, INT32_MAX)),
                  nullptr, out(y), mean, rstd, nullptr, nullptr, 0};
  return forward("adaln_fwd", false, false, a, 0, stream);
}

extern "C" int anima_adaln_fwd_quant(const void* x, const void* scale, const void* shift, float eps, int64_t rows,
                                     int64_t hw, int64_t d, void* y, float* mean, float* rstd, uint8_t* codes_row,
                                     uint8_t* scales_row, int scale_layout, void* stream) {
  const FwdArgs a{in(x), nullptr, nullptr, in(scale), in(shift), eps, rows, hw, d, static_cast<int>(std::min<int64_t>(d, INT32_MAX)),
                  nullptr, out(y), mean, rstd, codes_row, scales_row, scale_layout == ANIMA_SCALES_TILED};
  return forward("adaln_fwd_quant", false, true, a, scale_layout, stream);
}

extern "C" int anima_gated_add_adaln_fwd(const void* x, const void* gate, const void* sub, const void* scale,
                                         const void* shift, float eps, int64_t rows, int64_t hw, int64_t d,
                                         void* x_new, void* y, float* mean, float* rstd, void* stream) {
  const FwdArgs a{in(x), in(gate), in(sub), in(scale), in(shift), eps, rows, hw, d, static_cast<int>(std::min<int64_t>(d, INT32_MAX)),
                  out(x_new), out(y), mean, rstd, nullptr, nullptr, 0};
  return forward("gated_add_adaln_fwd", true, false, a, 0, stream);
}

extern "C" int anima_gated_add_adaln_fwd_quant(const void* x, const void* gate, const void* sub, const void* scale,
                                               const void* shift, float eps, int64_t rows, int64_t hw, int64_t d,
                                               void* x_new, void* y, float* mean, float* rstd, uint8_t* codes_row,
                                               uint8_t* scales_row, int scale_layout, void* stream) {
  const FwdArgs a{in(x), in(gate), in(sub), in(scale), in(shift), eps, rows, hw, d, static_cast<int>(std::min<int64_t>(d, INT32_MAX)),
                  out(x_new), out(y), mean, rstd, codes_row, scales_row, scale_layout == ANIMA_SCALES_TILED};
  return forward("gated_add_adaln_fwd_quant", true, true, a, scale_layout, stream);
}

extern "C" int64_t anima_adaln_bwd_workspace_bytes(int64_t rows, int64_t hw, int64_t d) {
  return partial_bytes(rows, hw, d, 2, false);
}

extern "C" int anima_adaln_bwd(const void* dy, const void* x, const void* scale, const float* mean,
                               const float* rstd, int64_t rows, int64_t hw, int64_t d, void* dx,
                               void* dscale, void* dshift, void* workspace, int64_t workspace_bytes,
                               void* stream) {
  ANIMA_REQUIRE(dscale && dshift, ANIMA_E_ARG, "adaln_bwd: null pointer");
  return anima_adaln_bwd_ex(dy, nullptr, x, scale, nullptr, nullptr, d, mean, rstd, rows, hw, d, dx, nullptr, dscale, dshift,
                            nullptr, workspace, at_most_least(workspace_bytes, rows, hw, d, 2), stream);
}

extern "C" int64_t anima_gated_add_adaln_bwd_workspace_bytes(int64_t rows, int64_t hw, int64_t d) {
  return partial_bytes(rows, hw, d, 3, false);
}

extern "C" int anima_gated_add_adaln_bwd(const void* d_y, const void* d_xnew, const void* x_new, const void* scale,
                                         const float* mean, const float* rstd, const void* sub, const void* gate,
                                         int64_t rows, int64_t hw, int64_t d, void* dx, void* dsub, void* dscale,
                                         void* dshift, void* dgate, void* workspace, int64_t workspace_bytes,
                                         void* stream) {
  ANIMA_REQUIRE(sub && dscale && dshift && dgate, ANIMA_E_ARG, "gated_add_adaln_bwd: null pointer");
  return anima_adaln_bwd_ex(d_y, d_xnew, x_new, scale, gate, sub, d, mean, rstd, rows, hw, d, dx, dsub, dscale, dshift,
                            dgate, workspace, at_most_least(workspace_bytes, rows, hw, d, 3), stream);
}

extern "C" int anima_gated_add_fwd(const void* x, const void* gate, const void* y, int64_t rows,
                                   int64_t hw, int64_t d, void* o, void* stream) {
  return gated_forward(x, gate, d, y, rows, hw, d, o, stream);
}

extern "C" int64_t anima_gated_add_bwd_workspace_bytes(int64_t rows, int64_t hw, int64_t d) {
  return partial_bytes(rows, hw, d, 1, false);
}

extern "C" int anima_gated_add_bwd(const void* dout, const void* y, const void* gate, int64_t rows,
                                   int64_t hw, int64_t d, void* dy, void* dgate, void* workspace,
                                   int64_t workspace_bytes, void* stream) {
  ANIMA_REQUIRE(y && dgate, ANIMA_E_ARG, "gated_add_bwd: null pointer");
  return gated_backward(dout, y, gate, d, rows, hw, d, dy, dgate, workspace, at_most_least(workspace_bytes, rows, hw, d, 1),
                        stream);
}

// ------------------------------------------------------------------ adaln_bwd without caller scratch
// Some hosts of this library may not allocate device memory at the point where they call it: a plugin that
// is handed only its input and output buffers by a framework that owns every other byte of the GPU, or a
// service whose memory plan is frozen after start-up so that a late cudaMalloc could fail or stall. For them
// the partial sums of adaln_bwd live in this fixed array inside the library image instead of a workspace.
namespace {
constexpr int64_t kStaticScratchBytes = ANIMA_ADALN_BWD_NOALLOC_MAX_BYTES;  // resident on every GPU that loads the library
__device__ __align__(256) float g_adaln_bwd_scratch[kStaticScratchBytes / sizeof(float)];

// Device address of the array for the current device. The symbol name is only a host-side handle; the
// address has to be asked for once per device, with that device current.
int static_scratch(float** out) {
  static std::mutex mu;
  static float* cached[64];
  int dev = 0;
  ANIMA_REQUIRE(cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64, ANIMA_E_CUDA,
                "adaln_bwd_noalloc: cannot identify the current device");
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == nullptr) {
    float* p = nullptr;
    const cudaError_t rc = cudaGetSymbolAddress(reinterpret_cast<void**>(&p), g_adaln_bwd_scratch);
    ANIMA_REQUIRE(rc == cudaSuccess && p != nullptr, ANIMA_E_CUDA,
                  "adaln_bwd_noalloc: cudaGetSymbolAddress failed on device %d: %s", dev, cudaGetErrorString(rc));
    cached[dev] = p;
  }
  *out = cached[dev];
  return ANIMA_OK;
}
}  // namespace

extern "C" int anima_adaln_bwd_noalloc(const void* dy, const void* x, const void* scale, const float* mean,
                                       const float* rstd, int64_t rows, int64_t hw, int64_t d, void* dx,
                                       void* dscale, void* dshift, void* stream) {
  const int64_t need = anima_adaln_bwd_workspace_bytes(rows, hw, d);
  ANIMA_REQUIRE(need >= 0, ANIMA_E_SHAPE, "adaln_bwd_noalloc: rows=%lld is not a multiple of hw=%lld (or a size is not positive)",
                (long long)rows, (long long)hw);
  ANIMA_REQUIRE(need <= kStaticScratchBytes, ANIMA_E_TOO_LARGE,
                "adaln_bwd_noalloc: this shape needs %lld bytes of scratch but the built-in array holds %lld; "
                "use anima_adaln_bwd with a caller workspace",
                (long long)need, (long long)kStaticScratchBytes);
  float* scratch = nullptr;
  if (int rc = static_scratch(&scratch)) return rc;
  // Every partial-sum slot that the final pass reads is written earlier in this same call, so nothing in the
  // array has to start at zero and what an earlier call left behind is never read.
  return anima_adaln_bwd(dy, x, scale, mean, rstd, rows, hw, d, dx, dscale, dshift, scratch, kStaticScratchBytes,
                         stream);
}
