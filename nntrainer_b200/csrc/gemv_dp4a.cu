// SPDX-License-Identifier: Apache-2.0
/**
 * @file  gemv_dp4a.cu
 * @brief Decode GEMVs on CUDA cores (dp4a) of Q4_0 and Q6_K, for the shapes that the streaming kernels do not take.
 *
 * They reproduce the reference's per-output float chains exactly:
 *   Q4_0  one fused multiply-add per 32-block (nntr_ggml_impl.cpp:9751-9753).
 *   Q6_K  eight partial sums per row (elements 4l..4l+3 of every 32-chunk go to
 *         lane l), fused multiply-add per super-block, fixed pairwise final sum
 *         (nntr_vec_dot_q6_K_q8_K, :8600-8696; nntr_ggml_impl_utils.h:59-65).
 *
 * Work split: one warp per group of 8 output rows; it walks K in units of 256 weights and runs the chains in the lanes
 * 0-7 (one per output row). Lane (r = lane%8, c = lane/8) computes the integer sums of quarter c of the unit for row r.
 * The CTA quantizes the activation into shared memory first.
 */
#include <cstdlib>

#include "common.cuh"

namespace nntr {

constexpr int DP_WARPS = 8; // warps per CTA

__device__ __forceinline__ uint32_t ld_u32_a2(const uint8_t *p) { // 2-byte aligned 32-bit load
  const uint16_t *h = reinterpret_cast<const uint16_t *>(p);
  return (uint32_t)h[0] | ((uint32_t)h[1] << 16);
}
__device__ __forceinline__ int dp4a_us_(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

/* ------------------------------------------------------------------ Q4_0 */
/* The CTA first quantizes x into shared memory (plain block_q8_0 layout). */
__global__ void __launch_bounds__(DP_WARPS * 32)
gemv_q4_0_dp4a_kernel(const float *__restrict__ x, const BlockQ40x8 *__restrict__ W, float *__restrict__ y, int n_groups,
                      int nb32) {
  extern __shared__ __align__(16) uint8_t dp_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int K = nb32 * 32;
  for (int u = warp; u < (K + 255) / 256; u += DP_WARPS) {
    const int e0 = u * 256 + lane * 8;
    const bool valid = e0 < K;
    float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b4 = a;
    if (valid) {
      a = *reinterpret_cast<const float4 *>(x + e0);
      b4 = *reinterpret_cast<const float4 *>(x + e0 + 4);
    }
    const Q80Lane q = q80_quantize_warp(a, b4);
    if (valid) {
      uint8_t *out = dp_smem + (size_t)(e0 / 32) * sizeof(BlockQ80);
      uint16_t *qs = reinterpret_cast<uint16_t *>(out + 2) + (lane & 3) * 4;
      qs[0] = (uint16_t)(q.w0 & 0xffff);
      qs[1] = (uint16_t)(q.w0 >> 16);
      qs[2] = (uint16_t)(q.w1 & 0xffff);
      qs[3] = (uint16_t)(q.w1 >> 16);
      if ((lane & 3) == 0)
        *reinterpret_cast<uint16_t *>(out) = q.d_bits;
    }
  }
  __syncthreads();
  const int r = lane & 7, c = lane >> 3;
  const int g = (int)blockIdx.x * DP_WARPS + warp;
  if (g >= n_groups)
    return;
  float acc = 0.f;
  const int nu = (nb32 + 7) / 8; // units of 8 blocks = 256 weights
  for (int u = 0; u < nu; ++u) {
    // the lane's two 32-blocks of this unit: s = 2c, 2c+1
    uint2 q0[2], q1[2];
    float dw[2];
    bool have[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int b = u * 8 + 2 * c + s;
      have[s] = b < nb32;
      const BlockQ40x8 *blk = W + (size_t)g * nb32 + (have[s] ? b : 0);
      q0[s] = *reinterpret_cast<const uint2 *>(blk->qs + r * 8);      // elements 0-7 (low), 16-23 (high)
      q1[s] = *reinterpret_cast<const uint2 *>(blk->qs + 64 + r * 8); // elements 8-15 (low), 24-31 (high)
      dw[s] = half_bits_to_float(blk->d[r]);
    }
    int Is[2];
    float sd[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int b = u * 8 + 2 * c + s;
      const uint8_t *a = dp_smem + (size_t)(have[s] ? b : 0) * sizeof(BlockQ80);
      uint32_t aw[8];
#pragma unroll
      for (int k = 0; k < 8; ++k)
        aw[k] = ld_u32_a2(a + 2 + 4 * k);
      // the interleave stores nibble ^ 8: undone here, the - 8 goes into the sum of the activations
      const uint32_t w0 = q0[s].x ^ 0x88888888u, w1 = q0[s].y ^ 0x88888888u, w2 = q1[s].x ^ 0x88888888u,
                     w3 = q1[s].y ^ 0x88888888u;
      int dot = 0, asum = 0;
      dot = __dp4a((int)(w0 & 0x0f0f0f0fu), (int)aw[0], dot);
      dot = __dp4a((int)(w1 & 0x0f0f0f0fu), (int)aw[1], dot);
      dot = __dp4a((int)(w2 & 0x0f0f0f0fu), (int)aw[2], dot);
      dot = __dp4a((int)(w3 & 0x0f0f0f0fu), (int)aw[3], dot);
      dot = __dp4a((int)((w0 >> 4) & 0x0f0f0f0fu), (int)aw[4], dot);
      dot = __dp4a((int)((w1 >> 4) & 0x0f0f0f0fu), (int)aw[5], dot);
      dot = __dp4a((int)((w2 >> 4) & 0x0f0f0f0fu), (int)aw[6], dot);
      dot = __dp4a((int)((w3 >> 4) & 0x0f0f0f0fu), (int)aw[7], dot);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        asum = __dp4a(0x01010101, (int)aw[k], asum);
      Is[s] = dot - 8 * asum; // sum of (nibble - 8) * activation
      sd[s] = __fmul_rn(dw[s], half_bits_to_float(*reinterpret_cast<const uint16_t *>(a)));
    }
    // gather the unit's eight (I, scale) pairs of a row into its lane c == 0, in block order
    int Iall[8];
    float sall[8];
#pragma unroll
    for (int cc = 0; cc < 4; ++cc) {
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        Iall[2 * cc + s] = __shfl_sync(FULL, Is[s], r + 8 * cc);
        sall[2 * cc + s] = __shfl_sync(FULL, sd[s], r + 8 * cc);
      }
    }
    if (lane < 8) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (u * 8 + k < nb32)
          acc = __fmaf_rn((float)Iall[k], sall[k], acc);
    }
  }
  if (lane < 8)
    y[g * 8 + r] = acc;
}

/* ------------------------------------------------------------------ Q6_K */
/* The CTA first quantizes x into shared memory (plain block_q8_K layout). Rows of W are plain block_q6_K rows
 * (210-byte blocks, 2-byte aligned). */
__global__ void __launch_bounds__(DP_WARPS * 32)
gemv_q6_K_dp4a_kernel(const float *__restrict__ x, const uint8_t *__restrict__ W, float *__restrict__ y, int N, int nb) {
  extern __shared__ __align__(16) uint8_t dp_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int b = warp; b < nb; b += DP_WARPS) {
    const float *src = x + b * QK_K + lane * 8;
    const Q8KLane q = q8K_quantize_warp(*reinterpret_cast<const float4 *>(src), *reinterpret_cast<const float4 *>(src + 4),
                                        lane, 0);
    BlockQ8K *out = reinterpret_cast<BlockQ8K *>(dp_smem) + b;
    uint32_t *qs = reinterpret_cast<uint32_t *>(out->qs);
    qs[lane * 2] = q.w0;
    qs[lane * 2 + 1] = q.w1;
    if (lane == 0)
      out->d = q.d;
  }
  __syncthreads();
  const int r = lane & 7, c = lane >> 3;
  const int g = (int)blockIdx.x * DP_WARPS + warp;
  if (g * 8 >= N)
    return;
  const int n = g * 8 + r;
  const bool row_ok = n < N;
  float acc[8];
#pragma unroll
  for (int l = 0; l < 8; ++l)
    acc[l] = 0.f;
  for (int b = 0; b < nb; ++b) {
    const uint8_t *blk = W + ((size_t)(row_ok ? n : 0) * nb + b) * sizeof(BlockQ6K);
    // the lane's two 32-element chunks: ch = 2c, 2c+1; chunk ch = (half h = ch/4, quarter w = ch%4)
    uint32_t v[2][8]; // 6-bit values, one byte each, 4 per word; word l = elements 4l..4l+3 of the chunk
    int sc[2][2];     // scale of elements 0-15 / 16-31 of the chunk
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int ch = 2 * c + s, h = ch >> 2, w = ch & 3;
      const uint8_t *ql = blk + 64 * h + 32 * (w & 1), *qh = blk + 128 + 32 * h;
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        const uint32_t lw = ld_u32_a2(ql + 4 * l), hw = ld_u32_a2(qh + 4 * l);
        const uint32_t nib = (w & 2) ? ((lw >> 4) & 0x0f0f0f0fu) : (lw & 0x0f0f0f0fu);
        v[s][l] = nib | (((hw >> (2 * w)) & 0x03030303u) << 4);
      }
      const int8_t *scp = reinterpret_cast<const int8_t *>(blk + 192) + 8 * h + 2 * w;
      sc[s][0] = scp[0];
      sc[s][1] = scp[1];
    }
    const float dw = half_bits_to_float(*reinterpret_cast<const uint16_t *>(blk + 208));
    const uint8_t *a = dp_smem + (size_t)b * sizeof(BlockQ8K);
    int part[8];
#pragma unroll
    for (int l = 0; l < 8; ++l)
      part[l] = 0;
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const uint32_t *aw = reinterpret_cast<const uint32_t *>(a + 4 + 32 * (2 * c + s));
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        const uint32_t av = aw[l];
        const int dot = dp4a_us_(v[s][l], av, 0) - 32 * __dp4a(0x01010101, (int)av, 0);
        part[l] += sc[s][l >> 2] * dot;
      }
    }
#pragma unroll
    for (int l = 0; l < 8; ++l) { // sum over the four quarters of the super-block
      part[l] += __shfl_xor_sync(FULL, part[l], 8);
      part[l] += __shfl_xor_sync(FULL, part[l], 16);
    }
    if (lane < 8) {
      const float d = __fmul_rn(*reinterpret_cast<const float *>(a), dw);
#pragma unroll
      for (int l = 0; l < 8; ++l)
        acc[l] = __fmaf_rn(d, (float)part[l], acc[l]);
    }
  }
  if (lane < 8 && row_ok)
    y[n] = __fadd_rn(__fadd_rn(__fadd_rn(acc[4], acc[0]), __fadd_rn(acc[6], acc[2])),
                     __fadd_rn(__fadd_rn(acc[5], acc[1]), __fadd_rn(acc[7], acc[3])));
}

/* ---------------------------------------------------------------- launchers */
static unsigned grid_for(long tasks) { return (unsigned)((tasks + DP_WARPS - 1) / DP_WARPS); }

static int set_smem_attr(const void *fn, size_t bytes) {
  if (bytes > 48 * 1024)
    NNTR_CHECK_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
  return NNTR_CUDA_OK;
}

int launch_gemv_q4_0(unsigned N, unsigned K, const float *x, const void *B, float *y, unsigned flags, cudaStream_t st) {
  static const bool stream_off = [] {
    const char *e = getenv("NNTR_CUDA_Q40_STREAM");
    return e && e[0] == '0';
  }();
  if (!stream_off && x && B && y && N && !(reinterpret_cast<uintptr_t>(B) & 15) && gemv_q4_0_stream_supported(N, K))
    return launch_gemv_q4_0_stream(N, K, x, B, y, flags, st);
  if (!x || !B || !y || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(B) & 7))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemv_q4_0: null or misaligned pointer");
  if (N == 0)
    return NNTR_CUDA_OK;
  const size_t smem = (size_t)(K / 32) * sizeof(BlockQ80) + 16;
  if (smem > 200 * 1024)
    return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "gemv_q4_0: K=%u too large", K);
  int rc = set_smem_attr(reinterpret_cast<const void *>(gemv_q4_0_dp4a_kernel), smem);
  if (rc)
    return rc;
  gemv_q4_0_dp4a_kernel<<<grid_for(N / 8), DP_WARPS * 32, smem, st>>>(x, static_cast<const BlockQ40x8 *>(B), y, (int)(N / 8),
                                                                      (int)(K / 32));
  count_launch();
  return check_cuda(cudaGetLastError(), "gemv_q4_0 launch");
}

int launch_gemv_q6_K(unsigned N, unsigned K, const float *x, const void *B, float *y, unsigned flags, cudaStream_t st) {
  // the streaming kernel takes every shape whose rows group into 16-byte aligned stages; the rest stays here
  static const bool stream_off = [] {
    const char *e = getenv("NNTR_CUDA_Q6K_STREAM");
    return e && e[0] == '0';
  }();
  if (!stream_off && x && B && y && N && !(reinterpret_cast<uintptr_t>(B) & 15) && gemv_q6_K_stream_supported(N, K)) {
    unsigned done = 0;
    const int rc = launch_gemv_q6_K_stream(N, K, x, B, y, flags, st, &done);
    if (rc || done == N)
      return rc;
    // the last rows (less than one stage of the ring) go through the kernel below
    B = static_cast<const uint8_t *>(B) + (size_t)done * (K / QK_K) * sizeof(BlockQ6K);
    y += done;
    N -= done;
  }
  if (!x || !B || !y || (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(B) & 1))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemv_q6_K: null or misaligned pointer");
  if (N == 0)
    return NNTR_CUDA_OK;
  const size_t smem = (size_t)(K / QK_K) * sizeof(BlockQ8K) + 16;
  if (smem > 200 * 1024)
    return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "gemv_q6_K: K=%u too large", K);
  int rc = set_smem_attr(reinterpret_cast<const void *>(gemv_q6_K_dp4a_kernel), smem);
  if (rc)
    return rc;
  gemv_q6_K_dp4a_kernel<<<grid_for((N + 7) / 8), DP_WARPS * 32, smem, st>>>(x, static_cast<const uint8_t *>(B), y, (int)N,
                                                                           (int)(K / QK_K));
  count_launch();
  return check_cuda(cudaGetLastError(), "gemv_q6_K launch");
}

} // namespace nntr
