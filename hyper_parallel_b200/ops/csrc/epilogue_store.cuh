// Epilogue of the tcgen05 GEMMs: one warp moves its 32 accumulator rows from tensor memory to C with
// TMA stores.
//
// A thread owns one row, so plain stores put 16 bytes into each of 32 rows per instruction: half a
// sector each, and 32 lines per instruction in the load/store unit.  That held products with a short
// contraction (weight gradients of a few hundred tokens), which are bound by writing C, at 1.2-1.4 TB/s.
// Here the rows of a 128-byte wide column block go through a 4 KB shared tile in the 128-byte swizzle
// (conflict-free 16-byte writes) and leave as one bulk store; two tiles per warp alternate, and the
// tensor-memory load of the next block is in flight while this one is converted.  Measured (B200,
// forward + backward): 32 experts of 7168 x 2048 on 77 tokens 3.69 -> 2.22 ms, a Llama-3-8B block on
// 2 x 4096 tokens 11.26 -> 10.84 ms, the 128256-wide output layer on 8192 tokens 25.7 -> 25.1 ms.
#pragma once
#include "sm100_common.cuh"

namespace hpb {

constexpr int EPI_TILE_BYTES = 32 * 128;               // 32 rows x 128 bytes
constexpr int EPI_WARP_BYTES = 2 * EPI_TILE_BYTES;
constexpr int EPI_BYTES = 4 * EPI_WARP_BYTES;          // four epilogue warps

__device__ __forceinline__ void tma_store_3d(const CUtensorMap* m, const void* smem_src, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
                   reinterpret_cast<uint64_t>(m)),
               "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
               : "memory");
}

// `taddr` addresses the warp's 32 lanes of a COLS-wide fp32 accumulator; the block goes to rows
// [row0, row0 + 32), columns [col0, col0 + COLS) of slice z, clipped by the tensor map.  `live` (warp
// uniform) false: nothing is stored; `zero`: zeros are.  `release()` runs once the accumulator has been
// read.  `flip` is the warp's running tile index.  All 32 lanes call it.
template <int COLS, bool OUT_F32, typename Release>
__device__ __forceinline__ void epilogue_tma(const CUtensorMap* map, uint8_t* tiles, uint32_t taddr, int row0,
                                             int col0, int z, int n_cols, bool live, bool zero, int lane, int& flip,
                                             Release&& release) {
  constexpr int CH = OUT_F32 ? 32 : 64;                // columns per 128-byte row of a tile
  constexpr int NCH = COLS / CH;
  uint32_t r[2][CH];
#pragma unroll
  for (int h = 0; h < CH / 32; ++h) tmem_ld_32x32b_x32(taddr + h * 32, *reinterpret_cast<uint32_t(*)[32]>(r[0] + h * 32));
#pragma unroll
  for (int c = 0; c < NCH; ++c) {
    uint32_t* v = r[c & 1];
    tmem_ld_wait();
    if (c + 1 < NCH) {
#pragma unroll
      for (int h = 0; h < CH / 32; ++h)
        tmem_ld_32x32b_x32(taddr + (c + 1) * CH + h * 32, *reinterpret_cast<uint32_t(*)[32]>(r[(c + 1) & 1] + h * 32));
    } else {
      release();
    }
    const int col = col0 + c * CH;
    if (live && col < n_cols) {
      uint8_t* tile = tiles + (flip & 1) * EPI_TILE_BYTES;
      ++flip;
      if (lane == 0) tma_store_wait_read<1>();         // the store before last has left this tile
      __syncwarp();
      uint8_t* row = tile + lane * 128;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        uint4 u;
        if constexpr (OUT_F32) {
          u = make_uint4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        } else {
          __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
          for (int e = 0; e < 4; ++e)
            b[e] = __floats2bfloat162_rn(__uint_as_float(v[8 * j + 2 * e]), __uint_as_float(v[8 * j + 2 * e + 1]));
        }
        if (zero) u = make_uint4(0, 0, 0, 0);
        *reinterpret_cast<uint4*>(row + ((j ^ (lane & 7)) << 4)) = u;
      }
      fence_proxy_async();
      __syncwarp();
      if (lane == 0) {
        tma_store_3d(map, tile, col, row0, z);
        tma_store_commit();
      }
    }
  }
}

// The first `n` of 32 columns of one row, element by element (rows of C that do not start on 16-byte
// boundaries, the last columns of a row).  Static indices keep `r` in registers, and with ACCUM all loads
// come before the first store: as one loop over the live columns the 32 values went through local memory
// and every element waited for its own load.  1000 x 1003 x 512 to bf16 57.6 -> 40.4 us, to fp32 51.7 ->
// 25.7, accumulating 112 -> 52; with C on vectors, accumulating, 8192 x 8192 x 128 142 -> 126.
template <bool ACCUM, typename T>
__device__ __forceinline__ void store_row32_elements(T* dst, const uint32_t (&r)[32], int n) {
  float old[32];
  if constexpr (ACCUM) {
#pragma unroll
    for (int j = 0; j < 32; ++j) old[j] = j < n ? static_cast<float>(dst[j]) : 0.f;
  }
#pragma unroll
  for (int j = 0; j < 32; ++j)
    if (j < n) dst[j] = static_cast<T>(ACCUM ? __uint_as_float(r[j]) + old[j] : __uint_as_float(r[j]));
}

// Tensor map of C as [slices][rows][cols] for epilogue_tma (box: 32 rows x 128 bytes); false when the pointer,
// the row stride or the width is not a multiple of 16 bytes.  The kernels then take plain stores: of 16 bytes as
// far as whole vectors go where the rows start on 16-byte boundaries, else element by element.
bool make_tmap_c(CUtensorMap* map, void* c, bool f32, uint64_t cols, uint64_t rows, uint64_t slices, int64_t ldc);

}  // namespace hpb
