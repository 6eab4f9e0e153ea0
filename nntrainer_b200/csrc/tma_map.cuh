// SPDX-License-Identifier: Apache-2.0
/**
 * @file  tma_map.cuh
 * @brief Tensor maps of two-dimensional arrays for tiled copies, and the copy itself.
 */
#ifndef NNTR_TMA_MAP_CUH_
#define NNTR_TMA_MAP_CUH_

#include <cuda.h>

#include "common.cuh"

namespace nntr {

/** Map over rows of `width` elements (1 or 2 bytes each) `stride` bytes apart; a copy takes a box of box_rows x box_width.
 *  swizzle: rows of the box, of 128 or 64 bytes, are stored swizzled. base 16-byte aligned, stride and box_width * size multiples of
 *  16. Maps depend on the arguments alone; every thread keeps the last ones it made, because a model's calls come back. */
int encode_map_2d(CUtensorMap *map, const void *base, unsigned elem_bytes, uint64_t width, uint64_t rows, uint64_t stride,
                  unsigned box_width, unsigned box_rows, bool swizzle);

/** Copies the box at element x, row y of the map into shared memory; its bytes are counted on the mbarrier. x * element size
 *  must be a multiple of 16 bytes. */
__device__ __forceinline__ void tma_tile(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
               "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
               : "memory");
}

} // namespace nntr
#endif
