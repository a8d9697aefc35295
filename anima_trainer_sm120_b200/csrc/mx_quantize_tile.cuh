// Tile kernel shared by the MXFP8 quantiser and the fused LoKr merge + quantise:
// one CTA owns a 128 x 128 tile whose bf16 values come from a Loader functor
// (plain global loads, or W + alpha * kron(w1, w2) built on the fly).
#pragma once

#include <cuda_fp8.h>

#include "common.cuh"

namespace anima {
namespace mxq {

constexpr int kTile = 128;      // tile edge in elements
constexpr int kThreads = 256;
constexpr float kAmaxFloor = 1e-30f;  // mxfp8_gemm.py:114

struct QuantParams {
  int64_t rows, cols;
  uint8_t* codes_row;
  uint8_t* scales_row;
  uint8_t* codes_colT;
  uint8_t* scales_col;
  int tiled;  // scale layout
};

// e = ceil(log2(amax / 448)) clamped to [-127, 127], for amax >= 1e-30 (normal fp32).
__device__ __forceinline__ int mx_exponent(float amax) {
  const uint32_t u = __float_as_uint(amax);
  const int E = static_cast<int>(u >> 23) - 127;
  const uint32_t mant = u & 0x7fffffu;
  if (E == 128) return 127;  // inf / nan: log2 -> inf, clamped
  int e = E - 8 + (mant > 0x600000u ? 1 : 0);
  return max(-127, min(127, e));
}

// 2^-e as fp32 for e in [-127, 127]; 2^-127 is the subnormal 0x00400000.
__device__ __forceinline__ float mx_inv_scale(int e) {
  return e >= 127 ? __uint_as_float(0x00400000u) : __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
}

__device__ __forceinline__ uint32_t e4m3x2(float lo, float hi) {
  return static_cast<uint32_t>(
      __nv_cvt_float2_to_fp8x2(make_float2(lo, hi), __NV_SATFINITE, __NV_E4M3));
}

// packed bf16 pair helpers (operands and results as raw 32-bit words)
__device__ __forceinline__ uint32_t bf16x2_max(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmax2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint32_t bf16x2_mul(uint32_t a, uint32_t b) {
  const __nv_bfloat162 r = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
  return *reinterpret_cast<const uint32_t*>(&r);
}

// Exponent and conversion of one row block from its packed bf16 bits. `am` is the block's largest |x| in each half
// of a word (sign bits clear). On the 15 magnitude bits a of a bf16 the rule of mx_exponent is a shift: e + 127 =
// ((a + 31) >> 7) - 8, because mantissa > 1.75 is exactly what carries; amax below 1e-30 gives 19, inf / nan 254.
__device__ __forceinline__ uint32_t mx_scale_byte(uint32_t am) {
  const uint32_t a = max(am & 0xffffu, am >> 16);
  const int sb = max(19, static_cast<int>((a + 31u) >> 7) - 8);
  return a >= 0x7f80u ? 254u : static_cast<uint32_t>(sb);
}
// 2^-e as a bf16 in both halves
__device__ __forceinline__ uint32_t mx_inv_bf16x2(uint32_t sb) {
  const uint32_t one = sb >= 254u ? 0x0040u : (254u - sb) << 7;
  return one | (one << 16);
}
// four values (two words) times 2^-e -> four e4m3 codes; the packed bf16 product is exact for a power of two
__device__ __forceinline__ uint32_t mx_codes4(uint32_t w0, uint32_t w1, uint32_t inv2) {
  const uint32_t a = bf16x2_mul(w0, inv2), b = bf16x2_mul(w1, inv2);
  return e4m3x2(__uint_as_float(a << 16), __uint_as_float(a & 0xffff0000u)) |
         (e4m3x2(__uint_as_float(b << 16), __uint_as_float(b & 0xffff0000u)) << 16);
}
// Scale byte and codes of the 8 values a thread holds of a 32-value row block spread over four adjacent lanes (all
// lanes of the warp call it). The running maximum starts at 0 and ignores NaN, as fmaxf does.
__device__ __forceinline__ uint32_t mx_row_block(const uint4& v, uint2& codes) {
  uint32_t am = bf16x2_max(0u, v.x & 0x7fff7fffu);
  am = bf16x2_max(am, v.y & 0x7fff7fffu);
  am = bf16x2_max(am, v.z & 0x7fff7fffu);
  am = bf16x2_max(am, v.w & 0x7fff7fffu);
  am = bf16x2_max(am, __shfl_xor_sync(0xffffffffu, am, 1));
  am = bf16x2_max(am, __shfl_xor_sync(0xffffffffu, am, 2));
  const uint32_t sb = mx_scale_byte(am), inv2 = mx_inv_bf16x2(sb);
  codes.x = mx_codes4(v.x, v.y, inv2);
  codes.y = mx_codes4(v.z, v.w, inv2);
  return sb;
}

__device__ __forceinline__ int tiled_offset(int r, int j) {
  return (r & 31) * 16 + (r >> 5) * 4 + j;
}

// ---- what both quantiser kernels do with a 128 x 128 tile ---------------------------------------------------------
// Thread t works on the 8 chunks (8 values, 16 bytes) at tile column 8 * (t & 15), tile rows (t >> 4) + 16 i in the row
// pass, and on column pair t & 63 of the 32-row group t >> 6 in the column pass. Both passes stay on packed bf16 words
// (amax, exponent and scaling), addresses advance by constant strides; see mx_row_block for the arithmetic.
struct RowPass {
  uint8_t* dst;        // code address of chunk 0
  int64_t step;        // 16 rows
  int rows_left;       // rows of the tile inside the matrix, minus this thread's first row; 0 when its columns are outside
  int sc0;             // scale staging index of chunk 0
  bool tiled;
  __device__ __forceinline__ RowPass(const QuantParams& p, int64_t tile_r, int64_t col, int t)
      : dst(p.codes_row + (tile_r + (t >> 4)) * p.cols + col), step(16 * p.cols), tiled(p.tiled) {
    const int64_t left = p.rows - tile_r;
    rows_left = col < p.cols ? static_cast<int>(left < kTile ? left : kTile) - (t >> 4) : 0;
    sc0 = (t >> 4) * (tiled ? 16 : 4) + ((t & 15) >> 2);
  }
  __device__ __forceinline__ bool in(int i) const { return 16 * i < rows_left; }
  // all lanes of the warp call it; v is zero outside the matrix
  __device__ __forceinline__ void put(int i, const uint4& v, uint8_t* sc, int t) {
    uint2 codes;
    const uint32_t sb = mx_row_block(v, codes);
    if (in(i)) {
      *reinterpret_cast<uint2*>(dst) = codes;
      if ((t & 3) == 0) sc[sc0 + (tiled ? 256 * (i & 1) + 4 * (i >> 1) : 64 * i)] = static_cast<uint8_t>(sb);
    }
    dst += step;
  }
};

// Column pass: codes of the column pair in w0 / w1 (32 rows each), scale bytes staged. `tile32`: the tile as words.
__device__ __forceinline__ void col_codes(const QuantParams& p, const uint32_t* tile32, int64_t tile_r, int64_t tile_c, int t,
                                          uint8_t* sc, uint32_t (&w0)[8], uint32_t (&w1)[8]) {
  const int cp = t & 63, g = t >> 6;
  uint32_t cw[32], am = 0u;   // the running maximum starts at 0 and ignores NaN
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    cw[i] = tile32[(32 * g + i) * 64 + cp];
    am = bf16x2_max(am, cw[i] & 0x7fff7fffu);
  }
  const uint32_t sb0 = mx_scale_byte(am & 0xffffu), sb1 = mx_scale_byte(am >> 16);
  const uint32_t inv2 = (mx_inv_bf16x2(sb0) & 0xffffu) | (mx_inv_bf16x2(sb1) & 0xffff0000u);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    float a[4], b[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t v = bf16x2_mul(cw[4 * q + k], inv2);
      a[k] = __uint_as_float(v << 16);
      b[k] = __uint_as_float(v & 0xffff0000u);
    }
    w0[q] = e4m3x2(a[0], a[1]) | (e4m3x2(a[2], a[3]) << 16);
    w1[q] = e4m3x2(b[0], b[1]) | (e4m3x2(b[2], b[3]) << 16);
  }
  if (tile_c + 2 * cp < p.cols && tile_r + 32 * g < p.rows) {
    sc[p.tiled ? tiled_offset(2 * cp, g) : 8 * cp + g] = static_cast<uint8_t>(sb0);
    if (tile_c + 2 * cp + 1 < p.cols) sc[p.tiled ? tiled_offset(2 * cp + 1, g) : 8 * cp + 4 + g] = static_cast<uint8_t>(sb1);
  }
}
// Transposed codes go through shared memory (the input tile is dead once every thread holds its column pair) so that
// the global writes are full 128-byte lines: column c of the tile owns 128 bytes = 8 pieces of 16; piece q is stored at
// q ^ ((c >> 1) & 7) to keep both the per-thread writes and the cooperative reads free of bank conflicts.
__device__ __forceinline__ void stage_cols(uint4* tile, int t, const uint32_t (&w0)[8], const uint32_t (&w1)[8]) {
  const int cp = t & 63, g = t >> 6, sw = cp & 7;
  uint4* c = tile + cp * 16;
  c[(2 * g) ^ sw] = make_uint4(w0[0], w0[1], w0[2], w0[3]);
  c[(2 * g + 1) ^ sw] = make_uint4(w0[4], w0[5], w0[6], w0[7]);
  c[8 + ((2 * g) ^ sw)] = make_uint4(w1[0], w1[1], w1[2], w1[3]);
  c[8 + ((2 * g + 1) ^ sw)] = make_uint4(w1[4], w1[5], w1[6], w1[7]);
}
__device__ __forceinline__ void store_cols(const QuantParams& p, const uint4* tile, int64_t tile_r, int64_t tile_c, int t) {
  const int c = t >> 3, q = t & 7;      // column c + 32 h, piece q; rows % 32 == 0: a piece is all in or all out
  uint8_t* dst = p.codes_colT + (tile_c + c) * p.rows + tile_r + q * 16;
  const uint4* src = tile + c * 8 + (q ^ ((c >> 1) & 7));
  const int64_t cols_left = p.cols - tile_c - c;
  if (tile_r + q * 16 < p.rows) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
      if (32 * h < cols_left) stg_stream16(dst + 32 * h * p.rows, src[256 * h]);
  }
}
// Scale bytes of the tile, staged in shared memory: 128 "rows" x 4 blocks of a matrix with `rows` rows and `kb` blocks.
template <bool CLEAR>
__device__ __forceinline__ void store_scales(uint8_t* out, uint8_t* sc, bool tiled, int64_t rows, int64_t kb, int64_t tile_row,
                                             int64_t tile_blk, int t) {
  if (tiled) {
    if (t < 128) {
      uint32_t* src = reinterpret_cast<uint32_t*>(sc) + t;
      reinterpret_cast<uint32_t*>(out + (tile_row * ceil_div(kb, static_cast<int64_t>(4)) + tile_blk) * 512)[t] = *src;
      if (CLEAR) *src = 0u;     // each entry is zeroed again by the thread that stored it
    }
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int idx = t + h * kThreads;
      const int64_t r = tile_row * kTile + (idx >> 2), k = tile_blk * 4 + (idx & 3);
      if (r < rows && k < kb) out[r * kb + k] = sc[idx];
      if (CLEAR) sc[idx] = 0;
    }
  }
}

// Loader interface (device side):
//   using Raw = ...;                            what one chunk needs from HBM
//   struct Cursor; Cursor begin(r, c) const;    this thread's chunk at row r, columns c .. c + 7
//   void next(Cursor&) const;                   16 rows on
//   Raw   fetch(const Cursor&) const;           issues the long-latency loads only
//   uint4 finish(const Raw&, const Cursor&) const;   the 8 bf16 values
//   static constexpr bool kZeroSafe;            finish(Raw{}, ...) == 0 and reads no memory
//   static constexpr int kSmemBytes; void prepare(void* smem);  per-CTA shared-memory state (a lookup table)
// All eight fetches of a thread are issued before the first finish, so a loader that computes
// (merge, GELU) does not serialise its chunks on memory latency.
template <bool ROW, bool COL, class Loader>
__global__ void __launch_bounds__(kThreads, COL ? 3 : 4) mx_quantize_kernel(const QuantParams p, const Loader load_arg) {
  __shared__ uint4 tile[COL ? kTile * 16 : 1];  // 128 rows x 256 B
  __shared__ __align__(16) uint8_t loader_smem[Loader::kSmemBytes > 0 ? Loader::kSmemBytes : 16];
  Loader load = load_arg;
  __shared__ __align__(16) uint8_t sc_row[ROW ? 512 : 16];
  __shared__ __align__(16) uint8_t sc_col[COL ? 512 : 16];

  after_previous();
  const int t = threadIdx.x;
  const int64_t tile_r = static_cast<int64_t>(blockIdx.y) * kTile;
  const int64_t tile_c = static_cast<int64_t>(blockIdx.x) * kTile;
  const int64_t col = tile_c + (t & 15) * 8;  // cols % 32 == 0 or % 8 == 0: a chunk is all in or all out
  RowPass row(p, tile_r, col, t);

  // Padding entries of a partial tile must be 0 in the tiled layout.
  if (ROW) reinterpret_cast<uint16_t*>(sc_row)[t] = 0;
  if (COL) reinterpret_cast<uint16_t*>(sc_col)[t] = 0;

  typename Loader::Raw fetched[8];
  const typename Loader::Cursor first = load.begin(tile_r + (t >> 4), row.rows_left > 0 ? col : 0);
  {
    typename Loader::Cursor at = first;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      fetched[i] = typename Loader::Raw{};
      if (row.in(i)) fetched[i] = load.fetch(at);
      load.next(at);
    }
  }
  load.prepare(loader_smem);   // after the tile's loads are in flight; visible to all threads after the barrier
  __syncthreads();             // also: zero fill of sc_* visible before the byte stores

  typename Loader::Cursor at = first;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    // kZeroSafe loaders map an all-zero Raw to zeros without touching memory, so out-of-range chunks need no branch
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (Loader::kZeroSafe || row.in(i)) v = load.finish(fetched[i], at);
    load.next(at);
    if (COL) tile[((t >> 4) + 16 * i) * 16 + (t & 15)] = v;
    if (ROW) row.put(i, v, sc_row, t);
  }
  if (COL) {
    __syncthreads();
    uint32_t w0[8], w1[8];
    col_codes(p, reinterpret_cast<const uint32_t*>(tile), tile_r, tile_c, t, sc_col, w0, w1);
    __syncthreads();
    stage_cols(tile, t, w0, w1);
    __syncthreads();
    store_cols(p, tile, tile_r, tile_c, t);
  } else {
    __syncthreads();
  }
  if (ROW) store_scales<false>(p.scales_row, sc_row, p.tiled, p.rows, p.cols / 32, blockIdx.y, blockIdx.x, t);
  if (COL) store_scales<false>(p.scales_col, sc_col, p.tiled, p.cols, p.rows / 32, blockIdx.x, blockIdx.y, t);
}

}  // namespace mxq
}  // namespace anima
