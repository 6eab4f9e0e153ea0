// SPDX-License-Identifier: Apache-2.0
/**
 * @file  act_tiles.cuh
 * @brief Quantized activations in the order in which the warp MMAs of gemm_mma.cu read them: the layout and the stores
 *        of a warp that has just quantized one row's 256 elements.
 */
#ifndef NNTR_ACT_TILES_CUH_
#define NNTR_ACT_TILES_CUH_

#include "common.cuh"

namespace nntr {

/* Activations: tiles of 8 rows in the order the B fragments are read: lane 4g + t of a warp holds row g of
 * the tile. Per tile and unit of 256 of K, act_row_bytes(QT) per row (rows of a tile beyond the problem's are never written;
 * they only reach output columns that are never stored):
 *   [4 pairs of 32][32 lanes][16 bytes]  the lane's 8 values of the even and the 8 of the odd 32-block
 *   Q4_K: [8] float d, [32 lanes] words (lo, hi of the 32-block t, lo, hi of t + 4): the block's sum is lo + 32 * (hi - 128)
 *   Q4_0: [4 pairs][8 rows][even, odd 32-block] half d
 * A tile of th < 8 rows is laid out with th in the place of 8 and 4 th in the place of 32 lanes. */
__host__ __device__ constexpr int act_row_bytes(int qtype) { return qtype == NNTR_Q4_0 ? 272 : 288; }

/** Unit b of tile k of a block of n_tiles tiles (all the rows of a dense problem, or those of one expert) that starts with tile
 *  `first` of the buffer. Units are outermost, so that neighbouring tiles of a unit are one piece of memory. */
template <int QT, typename Byte>
__device__ __forceinline__ Byte *act_unit(Byte *act, int first, int n_tiles, int k, int th, int nb, int b) {
  return act + ((size_t)first * nb + (size_t)b * n_tiles + k) * (size_t)(th * act_row_bytes(QT));
}

/** The values of a warp that has quantized 256 elements (lane: 8 of them from element 8 * lane) into row i of a tile. */
__device__ __forceinline__ void put_q8K(uint8_t *unit, int th, int i, const Q8KLane &q, int lane) {
  const int j = lane >> 2, t = lane & 3;
  *reinterpret_cast<uint2 *>(unit + (j >> 1) * (64 * th) + (4 * i + t) * 16 + (j & 1) * 8) = make_uint2(q.w0, q.w1);
  int s = q.sum8 + __shfl_xor_sync(FULL, q.sum8, 1);
  s += __shfl_xor_sync(FULL, s, 2);
  if (t == 0)
    *reinterpret_cast<uint16_t *>(unit + 260 * th + (4 * i + (j & 3)) * 4 + 2 * (j >> 2)) =
      (uint16_t)((s & 31) | (((s >> 5) + 128) << 8)); // |s| <= 32 * 127
  if (lane == 0)
    *reinterpret_cast<float *>(unit + 256 * th + 4 * i) = q.d;
}
__device__ __forceinline__ void put_q80(uint8_t *unit, int th, int i, const Q80Lane &q, int lane) {
  // 4-byte groups of the 32-block: group w = 2 * (lane % 4) (+ 1) belongs to lane w % 4, first word for w < 4
  const int j = lane >> 2, w = 2 * (lane & 3);
  uint8_t *dst = unit + (j >> 1) * (64 * th) + (4 * i + (w & 3)) * 16 + (j & 1) * 8 + (w >> 2) * 4;
  *reinterpret_cast<uint32_t *>(dst) = q.w0;
  *reinterpret_cast<uint32_t *>(dst + 16) = q.w1;
  if ((lane & 3) == 0)
    *reinterpret_cast<uint16_t *>(unit + 256 * th + 32 * (j >> 1) + 4 * i + 2 * (j & 1)) = q.d_bits; // th is 8
}

} // namespace nntr
#endif
