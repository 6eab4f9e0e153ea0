// SPDX-License-Identifier: Apache-2.0
/**
 * @file  tma_map.cu
 * @brief Tensor maps for tiled copies (host side). The driver's encoder is looked up through the runtime: the library does not
 *        link against the driver.
 */
#include <atomic>
#include <cstring>

#include "tma_map.cuh"

namespace nntr {

int encode_map_2d(CUtensorMap *map, const void *base, unsigned elem_bytes, uint64_t width, uint64_t rows, uint64_t stride,
                  unsigned box_width, unsigned box_rows, bool swizzle) {
  typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
  static std::atomic<EncodeTiled> encode{nullptr};
  EncodeTiled enc = encode.load(std::memory_order_acquire);
  if (!enc) {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    NNTR_CHECK_CUDA(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found));
    if (!fn || found != cudaDriverEntryPointSuccess)
      return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "the driver has no cuTensorMapEncodeTiled");
    enc = reinterpret_cast<EncodeTiled>(fn);
    encode.store(enc, std::memory_order_release);
  }
  struct Key { // compared as bytes: no padding
    const void *base;
    uint64_t width, rows, stride;
    unsigned box_width, box_rows, elem_bytes, swizzle; // never all zero: an empty entry matches nothing
  };
  struct Entry {
    Key key;
    CUtensorMap map;
  };
  constexpr unsigned SLOTS = 256; // 45 KB per thread
  static thread_local Entry slots[SLOTS] = {};
  const Key key = {base, width, rows, stride, box_width, box_rows, elem_bytes, swizzle};
  Entry &slot = slots[((uint32_t)(reinterpret_cast<uintptr_t>(base) >> 8) * 2654435761u >> 24) ^ (swizzle ? 1u : 0u)];
  if (memcmp(&slot.key, &key, sizeof key) == 0) {
    *map = slot.map;
    return NNTR_CUDA_OK;
  }
  const cuuint64_t dims[2] = {width, rows}, strides[1] = {stride};
  const cuuint32_t box[2] = {box_width, box_rows}, estr[2] = {1, 1};
  const CUresult r = enc(&slot.map, elem_bytes == 1 ? CU_TENSOR_MAP_DATA_TYPE_UINT8 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2,
                         const_cast<void *>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         !swizzle                        ? CU_TENSOR_MAP_SWIZZLE_NONE
                         : box_width * elem_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B
                                                        : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    slot.key = Key{};
    return set_error(NNTR_CUDA_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  }
  slot.key = key;
  *map = slot.map;
  return NNTR_CUDA_OK;
}

} // namespace nntr
