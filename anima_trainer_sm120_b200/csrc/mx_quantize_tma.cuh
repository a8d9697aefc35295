// TMA-fed, persistent form of the MXFP8 quantiser (same arithmetic and outputs as
// mx_quantize_kernel<ROW, COL, Loader>; see mx_quantize_tile.cuh for the tile algorithm).
//
// A CTA walks tiles b, b + gridDim.x, ... of 128 x 128 bf16 values. Two shared-memory stages hold input
// tiles; one elected thread keeps a `cp.async.bulk.tensor.2d` load of the NEXT tile in flight while the CTA
// works on the current one, so HBM reads overlap the arithmetic inside a CTA (the non-persistent kernel
// overlaps only across the CTAs of an SM) at no register cost, and the row pass reads its 16-byte chunks from
// shared memory instead of issuing global loads and shared stores itself. Tiles past the edge of the tensor
// are zero-filled by the copy engine; stores are predicated as in the tile kernel.
// Stage s, once its tile is in registers, doubles as the staging buffer for the transposed codes.
// Every mbarrier wait is bounded; a CTA that gives up raises g_quantize_timeout and leaves the loop.
//
// A loader that computes (GELU, GELU gradient) transforms the raw tile in place during the row pass: each
// thread rewrites the chunks it reads, a barrier follows, and the column pass sees the transformed tile. Its
// lookup table is copied to shared memory once per CTA instead of once per tile, and a second input (the
// incoming gradient) is fetched into registers one tile ahead, right after the row pass has consumed the
// current one. What the loader adds to the interface of mx_quantize_tile.cuh:
//   static constexpr bool kIdentity;        finish() returns the raw chunk (no rewrite, no extra barrier)
//   static constexpr bool kSecond;          there is a second input
//   static constexpr int kTmaCtasPerSm;     resident CTAs the kernel is compiled for (shared memory: two 32 KB
//                                           stages plus the table)
//   uint4 second(const Cursor&) const;                       the second input's chunk (a load)
//   uint4 transform(const uint4& raw, const uint4& second) const;
//   bool emits() const; void emit(const uint4&, const Cursor&) const;    the transformed values are also wanted in HBM
#pragma once

#include "mx_quantize_tile.cuh"
#include "tma_util.cuh"

namespace anima {
namespace mxq {

constexpr int kTmaStageBytes = kTile * kTile * 2;                      // 32 KB
constexpr int kTmaSmemBytes = 2 * kTmaStageBytes + 128 /*alignment*/;  // + the loader's table; barriers and scale staging are static

__device__ int g_quantize_timeout;  // sticky; read by anima_mx_quantize_status()

template <bool ROW, bool COL, class Loader>
__global__ void __launch_bounds__(kThreads, Loader::kTmaCtasPerSm)
mx_quantize_tma_kernel(const __grid_constant__ CUtensorMap map_x, const QuantParams p, const Loader load_arg) {
  extern __shared__ uint8_t smem_raw[];
  Loader load = load_arg;
  __shared__ __align__(8) uint64_t full_bar[2];
  __shared__ volatile int abort_flag;
  __shared__ __align__(16) uint8_t sc_row[ROW ? 512 : 16];
  __shared__ __align__(16) uint8_t sc_col[COL ? 512 : 16];

  after_previous();
  const int t = threadIdx.x;
  // dynamic shared memory: the loader's table first (its lookups pack two addresses into 16-bit halves, so it
  // must sit low), then the two stages
  constexpr uint32_t kTableBytes = (Loader::kSmemBytes + 127u) & ~127u;
  const uint32_t table0 = (smem_u32(smem_raw) + 127u) & ~127u;
  uint8_t* const table_ptr = smem_raw + (table0 - smem_u32(smem_raw));
  const uint32_t stage0 = table0 + kTableBytes;
  uint8_t* const stage_ptr0 = table_ptr + kTableBytes;
  // tile counts fit 32 bits (checked by the host): the index divisions stay cheap
  const uint32_t tiles_x = static_cast<uint32_t>(ceil_div(p.cols, static_cast<int64_t>(kTile)));
  const uint32_t n_tiles = tiles_x * static_cast<uint32_t>(ceil_div(p.rows, static_cast<int64_t>(kTile)));
  const uint32_t first = blockIdx.x, step = gridDim.x;
  auto coords = [&](uint32_t id, uint32_t& ty, uint32_t& tx) {
    ty = id / tiles_x;
    tx = id - ty * tiles_x;
  };

  if (ROW) reinterpret_cast<uint16_t*>(sc_row)[t] = 0;  // padding entries of a partial tile must be 0
  if (COL) reinterpret_cast<uint16_t*>(sc_col)[t] = 0;
  auto issue = [&](uint32_t tile_id, int s) {  // one thread: arm the stage's barrier and start the copy
    uint32_t ty, tx;
    coords(tile_id, ty, tx);
    mbar_expect_tx(smem_u32(&full_bar[s]), kTmaStageBytes);
    tma_load_2d(stage0 + s * kTmaStageBytes, &map_x, smem_u32(&full_bar[s]), static_cast<int>(tx * kTile),
                static_cast<int>(ty * kTile));
  };
  if (t == 0) {
    abort_flag = 0;
    mbar_init(smem_u32(&full_bar[0]), 1);
    mbar_init(smem_u32(&full_bar[1]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(&map_x) : "memory");
    if (first < n_tiles) issue(first, 0);
    if (first + step < n_tiles) issue(first + step, 1);
  }
  load.prepare(table_ptr);  // the table, once per CTA, behind the first copies
  uint4 second[Loader::kSecond ? 8 : 1];
  auto fetch_second = [&](uint32_t tile_id) {
    uint32_t ty, tx;
    coords(tile_id, ty, tx);
    const int64_t tile_r = static_cast<int64_t>(ty) * kTile, col = static_cast<int64_t>(tx) * kTile + (t & 15) * 8;
    const RowPass row(p, tile_r, col, t);
    typename Loader::Cursor at = load.begin(tile_r + (t >> 4), row.rows_left > 0 ? col : 0);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      second[i] = make_uint4(0u, 0u, 0u, 0u);
      if (row.in(i)) second[i] = load.second(at);
      load.next(at);
    }
  };
  if (Loader::kSecond && first < n_tiles) fetch_second(first);
  __syncthreads();

  int it = 0;
  for (uint32_t tile_id = first; tile_id < n_tiles; tile_id += step, ++it) {
    const int s = it & 1;
    uint32_t tile_y, tile_x;
    coords(tile_id, tile_y, tile_x);
    const int64_t tile_r = static_cast<int64_t>(tile_y) * kTile, tile_c = static_cast<int64_t>(tile_x) * kTile;
    const int64_t col = tile_c + (t & 15) * 8;
    uint4* tile = reinterpret_cast<uint4*>(stage_ptr0 + s * kTmaStageBytes);
    RowPass row(p, tile_r, col, t);

    if (!mbar_wait(smem_u32(&full_bar[s]), (it >> 1) & 1u, &abort_flag)) break;

    if (ROW || !Loader::kIdentity) {
      uint4* chunk = tile + (t >> 4) * 16 + (t & 15);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        uint4 v = chunk[256 * i];
        if (!Loader::kIdentity) {
          v = row.in(i) ? load.transform(v, second[Loader::kSecond ? i : 0]) : make_uint4(0u, 0u, 0u, 0u);
          if (COL) chunk[256 * i] = v;
          if (load.emits() && row.in(i)) load.emit(v, load.begin(tile_r + (t >> 4) + 16 * i, col));
        }
        if (ROW) row.put(i, v, sc_row, t);
      }
    }

    if (Loader::kSecond && tile_id + step < n_tiles) fetch_second(tile_id + step);  // lands under the column pass

    if (COL) {
      if (!Loader::kIdentity) __syncthreads();  // the transformed tile is complete
      uint32_t w0[8], w1[8];
      col_codes(p, reinterpret_cast<const uint32_t*>(tile), tile_r, tile_c, t, sc_col, w0, w1);
      __syncthreads();  // every thread holds its part of the input tile: the stage becomes the staging buffer
      stage_cols(tile, t, w0, w1);
      __syncthreads();
      store_cols(p, tile, tile_r, tile_c, t);
    } else {
      __syncthreads();  // scale bytes of the row pass visible
    }
    if (ROW) store_scales<true>(p.scales_row, sc_row, p.tiled, p.rows, p.cols / 32, tile_y, tile_x, t);
    if (COL) store_scales<true>(p.scales_col, sc_col, p.tiled, p.cols, p.rows / 32, tile_x, tile_y, t);
    // this thread's generic-proxy accesses to the stage are ordered before the copy engine's next write to it
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();  // the stage and the scale staging are free
    if (t == 0 && n_tiles - tile_id > 2 * step) issue(tile_id + 2 * step, s);
  }
  if (abort_flag) {
    // copies may still be in flight into this CTA's shared memory: give them time to land before it is released
    for (int i = 0; i < 200; ++i) __nanosleep(1000);
    if (t == 0) atomicExch(&g_quantize_timeout, 1);
  }
}

}  // namespace mxq
}  // namespace anima
