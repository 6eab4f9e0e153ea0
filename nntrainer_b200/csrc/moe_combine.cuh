// SPDX-License-Identifier: Apache-2.0
/**
 * @file  moe_combine.cuh
 * @brief The weighted sum of a token's expert outputs in ASCENDING expert index (qwen_moe_layer.cpp:493-498), as the
 *        combine kernel of moe.cu computes it.
 */
#ifndef NNTR_MOE_COMBINE_CUH_
#define NNTR_MOE_COMBINE_CUH_

#include "common.cuh"

namespace nntr {

/** y[t][h] = sum over the token's experts, ascending expert index, of (dn[pair][h] (+ bias)) * w[pair]. ord[t][k] is
 *  the slot of the token's k-th smallest expert index (the router writes it), so AT values are in flight at a time
 *  and added in that order without sorting here. The loads of a round hang on chains of up to four (slot, expert, table,
 *  bias): they are issued level by level, without a branch per expert, so that a round costs one chain and not AT of them
 *  (a last round that is not full reads its last expert again). Four neighbouring outputs at a time (h % 4 == 0, rows of dn
 *  16-byte aligned). */
template <int AT>
__device__ __forceinline__ float4 moe_combine_elem4(const float *__restrict__ dn, const int *__restrict__ idx,
                                                    const int *__restrict__ ord, const float *__restrict__ w,
                                                    const float *const *__restrict__ down_b, long t, int h, int H,
                                                    int topk) {
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int k0 = 0; k0 < topk; k0 += AT) {
    const int n = topk - k0 < AT ? topk - k0 : AT;
    long pair[AT];
    float4 v[AT];
    float ww[AT];
#pragma unroll
    for (int k = 0; k < AT; ++k)
      pair[k] = t * topk + ord[t * topk + k0 + (k < n ? k : n - 1)];
#pragma unroll
    for (int k = 0; k < AT; ++k) {
      v[k] = __ldcg(reinterpret_cast<const float4 *>(dn + pair[k] * H + h));
      ww[k] = w[pair[k]];
    }
    if (down_b) {
      const float *b[AT];
      float4 bv[AT];
#pragma unroll
      for (int k = 0; k < AT; ++k)
        b[k] = down_b[idx[pair[k]]] + h;
#pragma unroll
      for (int k = 0; k < AT; ++k)
        bv[k] = make_float4(b[k][0], b[k][1], b[k][2], b[k][3]);
#pragma unroll
      for (int k = 0; k < AT; ++k)
        v[k] = make_float4(__fadd_rn(v[k].x, bv[k].x), __fadd_rn(v[k].y, bv[k].y), __fadd_rn(v[k].z, bv[k].z),
                           __fadd_rn(v[k].w, bv[k].w));
    }
#pragma unroll
    for (int k = 0; k < AT; ++k)
      if (k < n)
        acc = make_float4(__fadd_rn(acc.x, __fmul_rn(v[k].x, ww[k])), __fadd_rn(acc.y, __fmul_rn(v[k].y, ww[k])),
                          __fadd_rn(acc.z, __fmul_rn(v[k].z, ww[k])), __fadd_rn(acc.w, __fmul_rn(v[k].w, ww[k])));
  }
  return acc;
}

} // namespace nntr
#endif
