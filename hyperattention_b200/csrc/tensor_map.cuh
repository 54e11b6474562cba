// Tensor maps of the TMA loads: a 4-D map of 128-row tiles (contiguous rows of one head) and a 2-D map of single rows
// (tile::gather4, rows named by index).  Encoded on the host per launch and passed to the kernel by value.
#pragma once
#include <cuda.h>

#include "common.cuh"

namespace ha {

// rows x width elements (2 bytes each) of every (batch, head); 64-element boxes of `box_rows` rows, 128-byte swizzle.
// false: strides or alignment the map cannot express (the caller then loads with cp.async).
bool encode_tile_map(CUtensorMap* map, int dtype, const void* base, int width, long long rows, int H, int B, int64_t sn, int64_t sh, int64_t sb,
                     int box_rows);

// The same tensor as one list of rows: row (b, h, i) has number (b sb + h sh + i sn) / pitch, pitch = the strides' common divisor.
bool encode_row_map(CUtensorMap* map, int dtype, const void* base, int width, long long rows, int H, int B, int64_t sn, int64_t sh, int64_t sb,
                    int64_t* pitch);

// fp32 accumulators [heads][rows][width], contiguous: boxes of 32 columns x 128 rows, 128-byte swizzle
bool encode_acc_map(CUtensorMap* map, float* base, int width, long long rows, long long heads);

// 128-row box at (column, row, head, batch) -> swizzled slab; the bytes are counted on `bar`
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap* map, int x, int row, int h, int b, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst), "l"(map), "r"(x),
      "r"(row), "r"(h), "r"(b), "r"(bar)
      : "memory");
}
// four rows by number -> 4 x 128 bytes of a swizzled slab
__device__ __forceinline__ void tma_gather4(uint32_t dst, const CUtensorMap* map, int x, int r0, int r1, int r2, int r3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(dst),
      "l"(map), "r"(x), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar)
      : "memory");
}
// swizzled 32 x 128 fp32 tile -> added to (stored at) the accumulator rows
__device__ __forceinline__ void tma_add_tile(const CUtensorMap* map, int x, int row, int head, uint32_t src) {
  asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map), "r"(x), "r"(row), "r"(head),
               "r"(src)
               : "memory");
}
__device__ __forceinline__ void tma_store_tile(const CUtensorMap* map, int x, int row, int head, uint32_t src) {
  asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(map), "r"(x), "r"(row), "r"(head), "r"(src)
               : "memory");
}
// bytes to come on the barrier's current phase, without an arrival
__device__ __forceinline__ void mbar_add_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

}  // namespace ha
