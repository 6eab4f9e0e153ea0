// SPDX-License-Identifier: Apache-2.0
/**
 * @file  attention.cu
 * @brief Single-token attention over an fp16 key/value cache with grouped-query heads, rotary embedding, a sliding
 *        window and attention sinks: what MHACoreLayer::one_batch_incremental_forwarding does for one decode step
 *        (Applications/CausalLM/layers/mha_core.cpp:459-533 and :535-613 with sinks).
 *
 * The reference's CPU code fixes the order of every floating-point sum, and the kernels keep it, so the attention
 * output equals the reference's bit for bit:
 *   rotary        nntrainer/tensor/cpu_backend/x86/avx2_impl.cpp:1652-1738 -- out0 = a*cos - b*sin, out1 = a*sin + b*cos
 *                 with separately rounded products; keys and values go to the cache as fp16 (round to nearest even);
 *   scores        avx2_impl.cpp:1595-1650 -- per (cache row, head): eight partial sums (element i goes to lane i % 8,
 *                 fused multiply-adds in ascending i), summed as ((l0+l4)+(l1+l5)) + ((l2+l6)+(l3+l7)), divided by
 *                 sqrt(head_dim) in double precision;
 *   softmax       avx2_impl.cpp:1181-1307 -- per head over the cache rows: maximum (with the sink logit), the 10th-order
 *                 polynomial exponential (:1085-1179), the sum accumulated row by row in ascending order starting from
 *                 the sink's term, one division per element;
 *   values        avx2_impl.cpp:1512-1593 -- per (head, d): one fused multiply-add per cache row in ascending order.
 * The row-ordered sums make the softmax denominator and the value product serial chains as long as the context per
 * output; with a few thousand outputs in flight they cost a few microseconds per layer. That is the price of
 * reproducing the reference's bits; the cache (rows x kv heads x head_dim fp16, read once for keys and once for values)
 * is the only traffic that matters.
 *
 * Cache layout as the reference's: [row][kv head][head_dim] fp16, one row per position.
 */
#include <algorithm>
#include <atomic>

#include "cluster.cuh"
#include "common.cuh"
#include "pipeline.cuh"
#include "tma_map.cuh"

namespace nntr {

/* ------------------------------------------------------------------ rotary */

/* One head by one warp: optional RMS norm over the head (sums in the order of rms_norm_wrt_width_fp32_intrinsic, as in
 * glue.cu) times gamma, then the rotary embedding of the pairs (k, k + head_dim/2) with the position's cos / sin rows;
 * the result is left in st[head_dim] (shared memory, this warp's). A lane owns both elements of its pairs, so the
 * rotation is done in place. */
__device__ __forceinline__ void rope_head(const float *__restrict__ src, const float *__restrict__ gamma, float eps,
                                          const float *__restrict__ ct, const float *__restrict__ sn, int hd, int lane,
                                          float *st) {
  if (gamma) {
    float acc = 0.f;
    int i = 0;
    for (; i + 32 <= hd; i += 32) {
      const float x = src[i + lane];
      acc = __fmaf_rn(x, x, acc);
    }
    for (; i + 8 <= hd; i += 8)
      if (lane < 8) {
        const float x = src[i + lane];
        acc = __fmaf_rn(x, x, acc);
      }
    float t = __fadd_rn(acc, __shfl_down_sync(FULL, acc, 4));
    t = __fadd_rn(t, __shfl_down_sync(FULL, t, 1));
    t = __fadd_rn(t, __shfl_down_sync(FULL, t, 2));
    const float h0 = __shfl_sync(FULL, t, 0), h1 = __shfl_sync(FULL, t, 8), h2 = __shfl_sync(FULL, t, 16),
                h3 = __shfl_sync(FULL, t, 24);
    const float sumsq = __fadd_rn(__fadd_rn(__fadd_rn(h0, h1), h2), h3);
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sumsq, (float)hd), eps)));
    for (int e = lane; e < hd; e += 32)
      st[e] = __fmul_rn(__fmul_rn(src[e], scale), gamma[e]);
  } else {
    for (int e = lane; e < hd; e += 32)
      st[e] = src[e];
  }
  __syncwarp();
  const int half = hd / 2;
  for (int kk = lane; kk < half; kk += 32) {
    const float a0 = st[kk], a1 = st[kk + half], c = ct[kk], s = sn[kk];
    st[kk] = __fsub_rn(__fmul_rn(a0, c), __fmul_rn(a1, s));
    st[kk + half] = __fadd_rn(__fmul_rn(a0, s), __fmul_rn(a1, c));
  }
  __syncwarp();
}

/* The same for heads of 32 * NE dimensions (64, 128): a lane's NE elements lane + 32 k are both what it adds up for the norm
 * and whole rotary pairs, so everything stays in registers and all loads are issued at once. */
template <int NE>
__device__ __forceinline__ void rope_head_regs(const float *__restrict__ src, const float *__restrict__ gamma, float eps,
                                               const float *__restrict__ ct, const float *__restrict__ sn, int lane, float *st) {
  float x[NE], gm[NE], c[NE / 2], sv[NE / 2];
#pragma unroll
  for (int k = 0; k < NE; ++k)
    x[k] = src[lane + 32 * k];
#pragma unroll
  for (int k = 0; k < NE / 2; ++k) {
    c[k] = ct[lane + 32 * k];
    sv[k] = sn[lane + 32 * k];
  }
  if (gamma) {
#pragma unroll
    for (int k = 0; k < NE; ++k)
      gm[k] = gamma[lane + 32 * k];
    float acc = 0.f;
#pragma unroll
    for (int k = 0; k < NE; ++k)
      acc = __fmaf_rn(x[k], x[k], acc);
    float t = __fadd_rn(acc, __shfl_down_sync(FULL, acc, 4));
    t = __fadd_rn(t, __shfl_down_sync(FULL, t, 1));
    t = __fadd_rn(t, __shfl_down_sync(FULL, t, 2));
    const float h0 = __shfl_sync(FULL, t, 0), h1 = __shfl_sync(FULL, t, 8), h2 = __shfl_sync(FULL, t, 16),
                h3 = __shfl_sync(FULL, t, 24);
    const float sumsq = __fadd_rn(__fadd_rn(__fadd_rn(h0, h1), h2), h3);
    const float scale = __fdiv_rn(1.0f, __fsqrt_rn(__fadd_rn(__fdiv_rn(sumsq, (float)(32 * NE)), eps)));
#pragma unroll
    for (int k = 0; k < NE; ++k)
      x[k] = __fmul_rn(__fmul_rn(x[k], scale), gm[k]);
  }
#pragma unroll
  for (int k = 0; k < NE / 2; ++k) {
    const float a0 = x[k], a1 = x[k + NE / 2];
    st[lane + 32 * k] = __fsub_rn(__fmul_rn(a0, c[k]), __fmul_rn(a1, sv[k]));
    st[lane + 32 * (k + NE / 2)] = __fadd_rn(__fmul_rn(a0, sv[k]), __fmul_rn(a1, c[k]));
  }
}

/* One warp per head (query heads, then key heads, then value heads). Optional per-head RMS norm first
 * (ReshapedRMSNormLayer on q and k: Applications/CausalLM/qwen3_causallm.cpp:60-93, sums in the order of
 * rms_norm_wrt_width_fp32_intrinsic as in glue.cu), then the rotary embedding: q in place, k into cache row `pos` as
 * fp16, v converted into cache row `pos`. The normalised head goes through shared memory so that a lane finds both
 * elements of its (k, k + head_dim/2) pairs whatever the head size. */
constexpr int ROPE_WARPS = 4;
__global__ void rope_cache_append_kernel(float *__restrict__ q, const float *__restrict__ k, const float *__restrict__ v,
                                         const float *__restrict__ q_gamma, const float *__restrict__ k_gamma, float eps,
                                         uint16_t *__restrict__ kcache, uint16_t *__restrict__ vcache,
                                         const float *__restrict__ cos_tab, const float *__restrict__ sin_tab,
                                         const unsigned *__restrict__ pos_dev, unsigned pos, int hq, int hkv, int hd,
                                         long long ld) {
  extern __shared__ __align__(16) float rsm[]; // [ROPE_WARPS][hd]
  pdl_launch_dependents(); // the next kernel may start its own prologue (weight prefetch); it waits before it reads
  pdl_wait();
  const unsigned p = (pos_dev ? *pos_dev : pos) + blockIdx.y; // consecutive tokens, ld elements apart
  q += blockIdx.y * ld;
  k += blockIdx.y * ld;
  v += blockIdx.y * ld;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int head = blockIdx.x * ROPE_WARPS + warp;
  if (head >= hq + 2 * hkv)
    return;
  if (head >= hq + hkv) { // value head: conversion only
    const int h = head - hq - hkv;
    const float *b = v + (size_t)h * hd;
    uint16_t *dst = vcache + ((size_t)p * hkv + h) * hd;
    for (int e = lane; e < hd; e += 32)
      dst[e] = float_to_half_bits_rn(b[e]);
    return;
  }
  const bool is_q = head < hq;
  const float *src = is_q ? q + (size_t)head * hd : k + (size_t)(head - hq) * hd;
  float *st = rsm + (size_t)warp * hd;
  rope_head(src, is_q ? q_gamma : k_gamma, eps, cos_tab + (size_t)p * hd, sin_tab + (size_t)p * hd, hd, lane, st);
  if (is_q) {
    float *dst = q + (size_t)head * hd;
    for (int e = lane; e < hd; e += 32)
      dst[e] = st[e];
  } else {
    uint16_t *dst = kcache + ((size_t)p * hkv + (head - hq)) * hd;
    for (int e = lane; e < hd; e += 32)
      dst[e] = float_to_half_bits_rn(st[e]);
  }
}

/* ------------------------------------------------------------------ scores */

/* A CTA takes 16 cache rows of one kv head (4 warps x 4 rows); lane = (row j = lane / 8, vector lane l = lane % 8).
 * The group's query heads and the key rows are staged in shared memory with 16-byte loads; every query head of the
 * group is then dotted against the rows. */
constexpr int SCORE_WARPS = 4;
__global__ void attn_scores_kernel(const float *__restrict__ q, const uint16_t *__restrict__ kcache,
                                   float *__restrict__ scores, const unsigned *__restrict__ pos_dev, unsigned pos,
                                   int hq, int hkv, int hd, unsigned window) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  pdl_launch_dependents(); // the next kernel may start its own prologue; it waits before it reads
  pdl_wait();
  const unsigned num_rows = (pos_dev ? *pos_dev : pos) + 1;
  const unsigned start_row = num_rows < window ? 0u : num_rows - window;
  const unsigned row_cnt = num_rows < window ? num_rows : window;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n = blockIdx.y;
  const int gqa = hq / hkv;
  if (blockIdx.x * SCORE_WARPS * 4 >= row_cnt)
    return;
  float *qs = reinterpret_cast<float *>(smem_raw);                           // [gqa][hd]
  uint16_t *kall = reinterpret_cast<uint16_t *>(smem_raw + (size_t)gqa * hd * 4); // [16][hd]
  for (int c = threadIdx.x; c < gqa * hd / 4; c += blockDim.x)
    reinterpret_cast<float4 *>(qs)[c] = reinterpret_cast<const float4 *>(q + (size_t)n * gqa * hd)[c];
  const unsigned t0 = (blockIdx.x * SCORE_WARPS + warp) * 4;
  uint16_t *ks = kall + (size_t)warp * 4 * hd;
  const int chunks_per_row = hd / 8;
  for (int c = lane; c < 4 * chunks_per_row; c += 32) {
    const int r = c / chunks_per_row, cc = c - r * chunks_per_row;
    uint4 vv = make_uint4(0, 0, 0, 0);
    if (t0 + r < row_cnt)
      vv = *reinterpret_cast<const uint4 *>(kcache + ((size_t)(start_row + t0 + r) * hkv + n) * hd + cc * 8);
    *reinterpret_cast<uint4 *>(ks + (size_t)r * hd + cc * 8) = vv;
  }
  __syncthreads();
  if (t0 >= row_cnt)
    return;
  const int j = lane >> 3, l = lane & 7;
  const uint16_t *kr = ks + (size_t)j * hd;
  const double norm = sqrt((double)(float)hd);
  for (int g = 0; g < gqa; ++g) {
    const float *qh = qs + (size_t)g * hd;
    float acc = 0.f;
#pragma unroll 8
    for (int i = 0; i < hd; i += 8)
      acc = __fmaf_rn(qh[i + l], half_bits_to_float(kr[i + l]), acc);
    float s = __fadd_rn(acc, __shfl_down_sync(FULL, acc, 4));
    s = __fadd_rn(s, __shfl_down_sync(FULL, s, 1));
    s = __fadd_rn(s, __shfl_down_sync(FULL, s, 2));
    if (l == 0 && t0 + j < row_cnt) {
      const float sum = __fadd_rn(0.0f, s);
      scores[(size_t)(t0 + j) * hq + n * gqa + g] = (float)((double)sum / norm);
    }
  }
}

/* ----------------------------------------------------------------- softmax */

/** exp256_ps, avx2_impl.cpp:1085-1179 ("low-precision version III"), one lane */
__device__ __forceinline__ float exp256_lane(float x) {
  const float LOG2EF = 1.44269504088896341f, LN2 = 0.6931471805599453f;
  const float max_x = 88.3762626647949f, min_x = -88.3762626647949f;
  const float t = max_x < x ? max_x : x;
  x = min_x > t ? min_x : t;
  float fx = __fmul_rn(x, LOG2EF);
  fx = floorf(__fadd_rn(fx, 0.5f));
  const float r = __fsub_rn(x, __fmul_rn(fx, LN2));
  float y = 1.0f / 3628800.0f;
  y = __fmaf_rn(y, r, 1.0f / 362880.0f);
  y = __fmaf_rn(y, r, 1.0f / 40320.0f);
  y = __fmaf_rn(y, r, 1.0f / 5040.0f);
  y = __fmaf_rn(y, r, 1.0f / 720.0f);
  y = __fmaf_rn(y, r, 1.0f / 120.0f);
  y = __fmaf_rn(y, r, 1.0f / 24.0f);
  y = __fmaf_rn(y, r, 1.0f / 6.0f);
  y = __fmaf_rn(y, r, 0.5f);
  y = __fmaf_rn(y, r, 1.0f);
  y = __fmaf_rn(y, r, 1.0f);
  const int nn = __float2int_rn(fx);
  return __fmul_rn(y, __uint_as_float((uint32_t)(nn + 127) << 23));
}

/* One CTA per head. Phase 1: maximum over the rows (any order: exact). Phase 2: e = exp(x - max) for every row, in
 * parallel, kept in shared memory (cap_rows of them; rows beyond that stay in global memory). Phase 3: thread 0 adds
 * the e's in ascending row order (the reference's order), starting from the sink's term. Phase 4: every element
 * divided by the sum and written back. */
constexpr int SOFTMAX_THREADS = 256;
__global__ void attn_softmax_kernel(float *__restrict__ scores, const float *__restrict__ sink,
                                    const unsigned *__restrict__ pos_dev, unsigned pos, int hq, unsigned window,
                                    unsigned cap_rows) {
  extern __shared__ __align__(16) float es[];
  __shared__ float red[SOFTMAX_THREADS / 32];
  __shared__ float s_bcast;
  pdl_launch_dependents();
  pdl_wait();
  const unsigned num_rows = (pos_dev ? *pos_dev : pos) + 1;
  const unsigned row_cnt = num_rows < window ? num_rows : window;
  const unsigned in_smem = row_cnt < cap_rows ? row_cnt : cap_rows;
  const int c = blockIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float mx = -INFINITY;
  for (unsigned r = threadIdx.x; r < row_cnt; r += SOFTMAX_THREADS) {
    const float v = scores[(size_t)r * hq + c];
    if (r < in_smem)
      es[r] = v;
    mx = fmaxf(mx, v);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
  if (lane == 0)
    red[warp] = mx;
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = red[0];
    for (int w = 1; w < SOFTMAX_THREADS / 32; ++w)
      m = fmaxf(m, red[w]);
    if (sink)
      m = fmaxf(m, sink[c]);
    s_bcast = m;
  }
  __syncthreads();
  mx = s_bcast;
  for (unsigned r = threadIdx.x; r < row_cnt; r += SOFTMAX_THREADS) {
    if (r < in_smem) {
      es[r] = exp256_lane(__fsub_rn(es[r], mx));
    } else {
      float *p = scores + (size_t)r * hq + c;
      *p = exp256_lane(__fsub_rn(*p, mx));
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float sum = sink ? exp256_lane(__fsub_rn(sink[c], mx)) : 0.0f;
    unsigned r = 0;
    for (; r + 16 <= in_smem; r += 16) { // loads issued together, adds in order
      float e[16];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        e[u] = es[r + u];
#pragma unroll
      for (int u = 0; u < 16; ++u)
        sum = __fadd_rn(sum, e[u]);
    }
    for (; r < in_smem; ++r)
      sum = __fadd_rn(sum, es[r]);
    for (; r + 8 <= row_cnt; r += 8) {
      float e[8];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        e[u] = scores[(size_t)(r + u) * hq + c];
#pragma unroll
      for (int u = 0; u < 8; ++u)
        sum = __fadd_rn(sum, e[u]);
    }
    for (; r < row_cnt; ++r)
      sum = __fadd_rn(sum, scores[(size_t)r * hq + c]);
    s_bcast = sum;
  }
  __syncthreads();
  const float sum = s_bcast;
  for (unsigned r = threadIdx.x; r < row_cnt; r += SOFTMAX_THREADS) {
    float *p = scores + (size_t)r * hq + c;
    *p = __fdiv_rn(r < in_smem ? es[r] : *p, sum);
  }
}

/* ------------------------------------------------------------------ values */

__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_4(uint32_t dst, const void *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

/* One thread per (head, d): out = chain over the window's rows of fma(p[row][head], v[row][kv head][d], out), rows
 * ascending. CTA = (kv head, 32 consecutive d) x all heads of the group: warp h = head h of the group, lane = d. Tiles
 * of VT rows (values as fp16 and the group's probabilities) are copied asynchronously into a ring of VBUF shared-memory
 * buffers, several tiles ahead of the one being consumed, so the chain runs at the latency of its own fused
 * multiply-adds. */
constexpr int VT = 64;   // rows per tile
constexpr int VBUF = 6; // buffers in the ring
__global__ void attn_values_kernel(const float *__restrict__ probs, const uint16_t *__restrict__ vcache,
                                   float *__restrict__ out, const unsigned *__restrict__ pos_dev, unsigned pos, int hq,
                                   int hkv, int hd, unsigned window) {
  extern __shared__ __align__(16) uint8_t vsm[];
  pdl_launch_dependents();
  pdl_wait();
  const unsigned row_num = pos_dev ? *pos_dev : pos;
  const unsigned first = row_num < window ? 0u : row_num + 1 - window;
  const unsigned cnt = row_num + 1 - first;
  const int gqa = hq / hkv;
  const int n = blockIdx.y;
  const int d0 = blockIdx.x * 32;
  const int lane = threadIdx.x & 31, h = threadIdx.x >> 5;
  // buffers: V tile [VT][32] fp16 (64 B per row), P tile [VT][gqa] fp32
  const size_t vbytes = (size_t)VT * 64, pbytes = (size_t)VT * gqa * 4;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(vsm);
  auto issue = [&](unsigned tile, int buf) {
    const unsigned j0 = tile * VT;
    const unsigned rows = cnt - j0 < (unsigned)VT ? cnt - j0 : (unsigned)VT;
    const uint32_t vdst = sbase + buf * (uint32_t)(vbytes + pbytes), pdst = vdst + (uint32_t)vbytes;
    for (unsigned c = threadIdx.x; c < rows * 4; c += blockDim.x) { // up to 4 chunks of 16 B (8 values) per row
      const unsigned r = c >> 2, cc = c & 3;
      if (d0 + (int)cc * 8 < hd)
        cp_async_16(vdst + r * 64 + cc * 16, vcache + ((size_t)(first + j0 + r) * hkv + n) * hd + d0 + cc * 8);
    }
    for (unsigned c = threadIdx.x; c < rows * gqa; c += blockDim.x) {
      const unsigned r = c / gqa, g = c - r * gqa;
      cp_async_4(pdst + c * 4, probs + (size_t)(j0 + r) * hq + n * gqa + g);
    }
    cp_async_commit();
  };
  // ring of VBUF buffers, VBUF - 1 tiles in flight ahead of the one being consumed; one commit group per iteration
  // (an empty one past the last tile) so that "all but the newest VBUF - 1 groups have landed" means "tile t is here"
  const unsigned n_tiles = (cnt + VT - 1) / VT;
  for (int t = 0; t < VBUF - 1; ++t) {
    if ((unsigned)t < n_tiles)
      issue(t, t);
    else
      cp_async_commit();
  }
  float acc = 0.f;
  for (unsigned t = 0; t < n_tiles; ++t) {
    const int buf = t % VBUF;
    if (t + VBUF - 1 < n_tiles)
      issue(t + VBUF - 1, (t + VBUF - 1) % VBUF); // the buffer tile t - 1 used: everyone left it at the barrier below
    else
      cp_async_commit();
    asm volatile("cp.async.wait_group %0;" ::"n"(VBUF - 1) : "memory");
    __syncthreads();
    const uint16_t *vt = reinterpret_cast<const uint16_t *>(vsm + buf * (vbytes + pbytes));
    const float *pt = reinterpret_cast<const float *>(vsm + buf * (vbytes + pbytes) + vbytes);
    const unsigned rows = cnt - t * VT < (unsigned)VT ? cnt - t * VT : (unsigned)VT;
    unsigned j = 0;
    for (; j + 8 <= rows; j += 8) {
      float a[8], b[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        a[u] = pt[(j + u) * gqa + h];
        b[u] = half_bits_to_float(vt[(j + u) * 32 + lane]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        acc = __fmaf_rn(a[u], b[u], acc);
    }
    for (; j < rows; ++j)
      acc = __fmaf_rn(pt[j * gqa + h], half_bits_to_float(vt[j * 32 + lane]), acc);
    __syncthreads(); // done with this buffer before a later tile is copied into it
  }
  if (d0 + lane < hd)
    out[(size_t)(n * gqa + h) * hd + d0 + lane] = acc;
}

/* ------------------------------------------------- the whole step in one launch */

/* One cluster of CTAs per kv head (and up to eight of its query heads); everything a token's attention does for those heads
 * stays inside it.
 *   scores   every CTA normalises and rotates the group's query heads for itself (a few hundred operations per head) and
 *            dots them against its share of the cache rows: key tiles by tiled TMA copies (128-byte swizzle, so that
 *            thread = row reads its 16-byte pieces without bank conflicts), eight partial sums per (row, head) in the
 *            thread. A score goes straight into the shared memory of the CTA(s) that own the head. The token's own row
 *            comes from the inputs, rounded to fp16 as the cache holds it: the CTA that scores it patches it into its
 *            tile and appends it to the caches.
 *   softmax  a CTA owns one head (or 64 of its dimensions): maximum, exponentials and division by all threads, the sum in
 *            ascending row order by one warp (ordered_sum).
 *   values   a thread per dimension runs the row-ordered chain over value tiles that a producer warp keeps ahead of it
 *            (tiled TMA copies, started before the scores). CTAs of 32 dimensions (long windows): six warps turn the tiles round, and
 *            the chain loads eight rows of its dimension at once: at 4096 rows 27700 clocks instead of 33300, the launch 33.5 us
 *            instead of 36.5.
 * Clock stamps of one CTA, 64 / 8 heads of 64, at 512 rows (CTAs of 64 dimensions) / at 4096 (of 32), in clocks: up to the grid dependency
 * 1800 / 2500, first copies and heads rotated 1350 / 1600, wait for the cluster 400 / 60, score tiles 1600 / 5850, barrier behind them
 * 2050 / 1450, maximum and exponentials 1500 / 3900, ordered sum 2500 / 12050, division 450 / 1450, value chain 5400 / 28000. The value
 * chain is half of a long context at 6.8 clocks per row, where a dependent multiply-add alone takes four (CTAs of 64 dimensions: about 8,
 * six inside a tile, the rest where it waits for one). In a decode step, whose launches find neither code nor caches at hand, the phases
 * up to 512 rows take half as long again (32 / 8 heads of 128 at 100 rows 14300 clocks behind the dependency, alone 8900). 32 / 8 heads
 * of 128 at 512 rows 11.2 us (with generic accesses to the tiles, and value tiles of 128 rows, 12.3), at 128 rows of a window
 * 8.0 us with the copy of q (8.4). Measured with CTAs of 64 dimensions at 4096 rows, 36.5 us, and not kept: eight rows at a time with
 * twenty-four more on their way (40.7 us, sixteen and sixteen 36.6: a warp waits for its loads by few counters), half of the ring waited for
 * at a time (44), four blocks of the ordered sum at once (16900 clocks instead of 11500), the integers of all blocks of 32 rows by all warps
 * beforehand (2 us more), two rows and two heads per thread in the scores (heads of 64: 1800 a tile instead of 1900; of 128: 2660 instead of
 * 2200).
 * Ring positions are counted, not divided: an integer division in a loop that one thread runs costs more than a tile's copy. */
constexpr int AC_THREADS = 256;
constexpr int AC_WARPS = AC_THREADS / 32;
/** cache rows per tile of keys: 32 rows and one or two heads for each warp */
template <int DIMS> constexpr int AC_KROWS = DIMS == 32 ? 256 : 128;
constexpr uint32_t AC_SMEM_ALONE = 200u * 1024u; // beside which an SM has room for launches of up to about 26 KB only
constexpr int AC_KBUF_MAX = 4;
constexpr int AC_VBUF_MAX = 6;
/** cache rows per tile of values: a wait for a tile costs 350 clocks of the chain */
template <int DIMS> constexpr int AC_VROWS = DIMS <= 64 ? 256 : 128;
constexpr unsigned AC_MAX_ROWS = 16384; // rows of one head kept as floats in shared memory
/* CTAs of 32 dimensions: the warps between the first, which runs the value chain, and the last, which starts copies, turn the value tiles
 * round, so that the chain loads eight rows of its dimension at once. */
constexpr int AC_TURNERS = AC_WARPS - 2;
constexpr unsigned AC_SLICED_ROWS = 1400;
constexpr int AC_TBUF_MAX = 4;
constexpr int AC_TPITCH = 2 * 256 + 16; // bytes of a dimension's rows in a turned tile: 16-byte pieces of neighbours in different banks
constexpr uint32_t AC_TBYTES = 32 * AC_TPITCH;
constexpr uint32_t AC_POLLS = 1u << 22;
__device__ int g_attn_status = 0; // raised when a bounded wait for a tile runs out

/** Out of line: inlined, it costs the loops around it registers (16 tokens over four layers of 32 / 8 heads of 128 at 512 rows,
 *  attention in 64 of 368 launches: 3373 us, out of line 3346). */
__device__ __noinline__ void raise_attn(uint32_t flag) { raise_in_cluster(flag); }

struct AttnStep {
  const float *q, *k, *v, *q_gamma, *k_gamma;
  float eps;
  uint16_t *kcache, *vcache;
  const float *cos_tab, *sin_tab;
  float *q_rot, *q_inplace, *out;
  const float *sink;
  const unsigned *pos_dev;
  unsigned pos, window, cap_rows;
  int hq, hkv, hd;
  int groups; // clusters per kv head: more than eight query heads per kv head are split over several
  int rope;   // 0: q is rotated already and the token's rows are in the caches
  int k_bufs, v_bufs, t_bufs; // tiles of keys, of values, turned ones of values
  unsigned tokens;   // consecutive tokens (blockIdx.y), q_ld and out_ld elements apart; their rows are in the caches
  long long q_ld, out_ld;
  int k_box, v_box; // rows a copy brings: a tile, fewer where one short tile is all there is
};

/** store to the same shared-memory address of another CTA of the cluster */
__device__ __forceinline__ void st_cluster(uint32_t addr, uint32_t rank, float v) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote), "f"(v) : "memory");
}

struct AcLayout {
  uint32_t ktile, vtile, e, q, total; // offsets; the tiles are 1024-byte aligned; turned values take the keys' place
};
__host__ __device__ inline AcLayout ac_layout(int gqa, int hd, int dims, int k_rows, int k_bufs, int v_bufs, int t_bufs, int v_box, unsigned cap_rows) {
  AcLayout L;
  uint32_t o = 0;
  L.ktile = o;
  o += (uint32_t)k_bufs * (uint32_t)((hd + 63) / 64) * k_rows * 128;
  if (o < (uint32_t)t_bufs * AC_TBYTES)
    o = ((uint32_t)t_bufs * AC_TBYTES + 1023u) & ~1023u;
  L.vtile = o;
  o += (uint32_t)v_bufs * v_box * dims * 2; // one tile, or whole ones
  L.e = o; // scores, exponentials, probabilities of whole tiles; a spare block so that the sum may read ahead
  o += (cap_rows + 255) / 256 * 256 * 4 + 1024;
  L.q = o; // rotated query heads, then the new key head
  o += (uint32_t)(gqa + 1) * hd * 4;
  L.total = o + 1024;
  return L;
}

/** Scores (not yet divided) of one thread's key row against the H query heads at qs: ascending groups of eight elements. */
template <int H, int HD, int ROWS>
__device__ __forceinline__ void dot_rows(const uint8_t *tile, int row, const float *qs, int hd, float (&sum)[H]) {
  float acc[H][8];
#pragma unroll
  for (int h = 0; h < H; ++h)
#pragma unroll
    for (int l = 0; l < 8; ++l)
      acc[h][l] = 0.f;
#pragma unroll 8
  for (int c = 0; c < (HD ? HD : hd) / 8; ++c) {
    const uint4 w = *reinterpret_cast<const uint4 *>(tile + (c >> 3) * (ROWS * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4));
    const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
    float2 kv[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      kv[i] = __half22float2(*reinterpret_cast<const __half2 *>(&ws[i]));
#pragma unroll
    for (int h = 0; h < H; ++h) {
      const float4 a = *reinterpret_cast<const float4 *>(qs + h * hd + 8 * c),
                   b = *reinterpret_cast<const float4 *>(qs + h * hd + 8 * c + 4);
      fma2(acc[h][0], acc[h][1], a.x, a.y, kv[0].x, kv[0].y);
      fma2(acc[h][2], acc[h][3], a.z, a.w, kv[1].x, kv[1].y);
      fma2(acc[h][4], acc[h][5], b.x, b.y, kv[2].x, kv[2].y);
      fma2(acc[h][6], acc[h][7], b.z, b.w, kv[3].x, kv[3].y);
    }
  }
#pragma unroll
  for (int h = 0; h < H; ++h)
    sum[h] = __fadd_rn(__fadd_rn(__fadd_rn(acc[h][0], acc[h][4]), __fadd_rn(acc[h][1], acc[h][5])),
                       __fadd_rn(__fadd_rn(acc[h][2], acc[h][6]), __fadd_rn(acc[h][3], acc[h][7])));
}

/** s + e[lo] + e[lo + 1] + ... + e[hi - 1], one rounded addition after the other; lo and hi multiples of 8, e may be read up
 *  to hi + 63. */
__device__ __forceinline__ float serial_sum(const float *e, unsigned lo, unsigned hi, float s) {
  const float4 *e4 = reinterpret_cast<const float4 *>(e);
  // thirty-two rows are added while the next thirty-two are on their way
  float4 ev[2][8];
#pragma unroll
  for (int u = 0; u < 8; ++u)
    ev[0][u] = e4[lo / 4 + u];
  unsigned r = lo;
  auto add32 = [&](float4(&cur)[8], float4(&nxt)[8]) {
#pragma unroll
    for (int u = 0; u < 8; ++u)
      nxt[u] = e4[r / 4 + 8 + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      s = __fadd_rn(s, cur[u].x);
      s = __fadd_rn(s, cur[u].y);
      s = __fadd_rn(s, cur[u].z);
      s = __fadd_rn(s, cur[u].w);
    }
    r += 32;
  };
  for (; r + 64 <= hi;) {
    add32(ev[0], ev[1]);
    add32(ev[1], ev[0]);
  }
  if (r + 32 <= hi)
    add32(ev[0], ev[1]);
  for (; r < hi; r += 4) {
    const float4 v = e4[r / 4];
    s = __fadd_rn(s, v.x);
    s = __fadd_rn(s, v.y);
    s = __fadd_rn(s, v.z);
    s = __fadd_rn(s, v.w);
  }
  return s;
}

/* The ordered sum of cnt values e >= 0 (cnt a multiple of 8) by one warp, with the bits of the serial chain. While the running sum s stays inside one
 * power of two [2^k, 2^(k+1)) it is an integer multiple S of u = 2^(k-23), and adding e rounds e / u to an integer: to the
 * nearest, and only for an exact half does the choice depend on S. So the integers of 256 rows are added in any order, eight rows
 * per lane, and S + their sum is the serial result as long as it stays below 2^24 and no half occurred. Where one of the two
 * happens, the lanes in front of the first such lane are taken, that lane's eight rows are added serially, and the next 256
 * rows start behind them. That takes 700 (4096 rows) to 1000 (2048) clocks per 256 rows, interruptions among them, against 1250 for the
 * serial chain (4.9 clocks a row). A power of two is passed log2(rows) times; a half has probability e / s per row, so the first rows
 * are added serially. After AC_SUM_STOPS interruptions the rest is added serially. */
constexpr unsigned AC_SUM_SERIAL = 64;    // rows at the start
/* Below this many rows the serial chain. The two forms cross later, between 1400 rows (64 / 8 heads of 64: 19.6 us, with the serial chain
 * 18.2; 800 rows 15.2 and 13.6; 32 / 8 heads of 128 within 0.6 of these) and 2048 (8300 clocks, serial about 10000). */
constexpr unsigned AC_SUM_PARALLEL = 768;
constexpr int AC_SUM_STOPS = 40;
__device__ __forceinline__ float ordered_sum(const float *e, unsigned cnt, float s, int lane) {
  if (cnt < AC_SUM_PARALLEL)
    return serial_sum(e, 0, cnt, s);
  s = serial_sum(e, 0, AC_SUM_SERIAL, s);
  unsigned r = AC_SUM_SERIAL;
  int stops = 0;
  while (r + 256 <= cnt && stops < AC_SUM_STOPS) {
    const uint32_t ex = __float_as_uint(s) >> 23;
    if (ex < 32 || ex >= 255) // too small for u to be a normal number, or no number: the serial chain keeps it
      break;
    const float inv_u = __uint_as_float((277u - ex) << 23), u = __uint_as_float((ex - 23u) << 23); // u = 2^(k - 23), k = ex - 127
    const int S = (int)(s * inv_u);                         // in [2^23, 2^24)
    const float4 a = *reinterpret_cast<const float4 *>(e + r + 8 * lane), b = *reinterpret_cast<const float4 *>(e + r + 8 * lane + 4);
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    int sum = 0;
    bool half = false;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float x = fminf(v[i] * inv_u, 16777216.f); // exact, or far below one half
      const int n = __float2int_rn(x);
      half |= fabsf(x - (float)n) == 0.5f;
      sum += n;
    }
    sum = min(sum, 1 << 24);
    const int total = (int)__reduce_add_sync(FULL, (unsigned)sum);
    if (S + total < (1 << 24) && !__any_sync(FULL, half)) {
      s = (float)(S + total) * u;
      r += 256;
      continue;
    }
    int incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(FULL, incl, d);
      if (lane >= d)
        incl += o;
    }
    const int stop = __ffs(__ballot_sync(FULL, half || S + incl >= (1 << 24))) - 1;
    const int before = __shfl_sync(FULL, incl - sum, stop);
    s = (float)(S + before) * u;
    r += 8 * stop;
#pragma unroll
    for (int i = 0; i < 8; ++i)
      s = __fadd_rn(s, e[r + i]);
    r += 8;
    ++stops;
  }
  return serial_sum(e, r, cnt, s);
}

template <int HD, int DIMS> // head_dim (0: a.hd), dimensions a CTA owns
__global__ void __launch_bounds__(AC_THREADS, 1)
attn_cluster_kernel(const __grid_constant__ CUtensorMap kmap, const __grid_constant__ CUtensorMap vmap,
                    const __grid_constant__ AttnStep a) {
  extern __shared__ uint8_t ac_raw[];
  __shared__ __align__(8) unsigned long long kbar[AC_KBUF_MAX], vfull[AC_VBUF_MAX], vempty[AC_VBUF_MAX],
    tfull[AC_TBUF_MAX], tempty[AC_TBUF_MAX];
  __shared__ float red[AC_WARPS];
  __shared__ float s_bcast;
  __shared__ int abort_word;
  volatile int *abort_flag = &abort_word;
  constexpr int KROWS = AC_KROWS<DIMS>, VROWS = AC_VROWS<DIMS>;
  constexpr bool TURN = DIMS == 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gqa = a.hq / a.hkv / a.groups, hd = HD ? HD : a.hd, per_head = (hd + DIMS - 1) / DIMS, items = gqa * per_head;
  const uint32_t rank = (uint32_t)cluster_rank(), csize = (uint32_t)cluster_size();
  const int cluster = (int)(blockIdx.x / csize), n = cluster / a.groups, h0 = cluster * gqa; // kv head, first query head
  uint8_t *base = ac_raw + (-smem_u32(ac_raw) & 1023u); // an offset: rounding the pointer itself up makes every access a generic one
  const AcLayout L = ac_layout(gqa, hd, DIMS, KROWS, a.k_bufs, a.v_bufs, a.t_bufs, a.v_box, a.cap_rows);
  uint8_t *ktile = base + L.ktile, *vtile = base + L.vtile;
  float *e = reinterpret_cast<float *>(base + L.e), *qs = reinterpret_cast<float *>(base + L.q), *kown = qs + gqa * hd;
  const int k_halves = (hd + 63) / 64;
  const uint32_t kbytes = (uint32_t)k_halves * KROWS * 128, vbytes = (uint32_t)a.v_box * DIMS * 2; // of a buffer
  const uint32_t ksm = smem_u32(ktile), vsm = smem_u32(vtile), esm = smem_u32(e);
  const uint32_t kbar0 = smem_u32(kbar), vfull0 = smem_u32(vfull), vempty0 = smem_u32(vempty),
                 tfull0 = smem_u32(tfull), tempty0 = smem_u32(tempty);
  if (tid == 0) {
    abort_word = 0;
    for (int i = 0; i < a.k_bufs; ++i)
      mbar_init(kbar0 + 8 * i, 1);
    for (int i = 0; i < a.v_bufs; ++i) {
      mbar_init(vfull0 + 8 * i, 1);
      mbar_init(vempty0 + 8 * i, TURN ? AC_TURNERS : DIMS / 32);
    }
    for (int i = 0; TURN && i < a.t_bufs; ++i) {
      mbar_init(tfull0 + 8 * i, AC_TURNERS);
      mbar_init(tempty0 + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  cluster_arrive(); // "this CTA has started": waited for before the first store into another one
  pdl_launch_dependents();
  pdl_wait();
  const unsigned p = (a.pos_dev ? *a.pos_dev : a.pos) + blockIdx.y;
  const float *q_in = a.q + (long long)blockIdx.y * a.q_ld;
  float *out = a.out + (long long)blockIdx.y * a.out_ld;
  const unsigned first = p + 1 < a.window ? 0u : p + 1 - a.window;
  unsigned cnt = p + 1 - first;
  if (cnt > a.cap_rows)
    cnt = a.cap_rows; // the launch was sized for cap_rows
  const unsigned cached = a.rope ? cnt - 1 : cnt; // rows whose values are read from the cache
  const unsigned share = (cnt + csize - 1) / csize, r_lo = min(rank * share, cnt), r_hi = min((rank + 1) * share, cnt);
  const int item_head = (int)rank / per_head, item_d0 = ((int)rank % per_head) * DIMS;
  const bool has_item = (int)rank < items, has_own = a.rope && r_lo < cnt && r_hi == cnt;
  const bool append = has_own && cluster % a.groups == 0; // one cluster per kv head appends the token's rows
  const unsigned k_tiles = (r_hi - r_lo + KROWS - 1) / KROWS, v_tiles = (cached + VROWS - 1) / VROWS;
  auto issue_k = [&](unsigned t, int buf) {
    const uint32_t bar = kbar0 + 8 * buf;
    mbar_expect_tx(bar, (uint32_t)(k_halves * a.k_box) * 128);
    for (int h = 0; h < k_halves; ++h)
      tma_tile(ksm + buf * kbytes + h * (KROWS * 128), &kmap, n * hd + 64 * h, (int)(first + r_lo + t * KROWS), bar);
  };
  auto issue_v = [&](unsigned t, int buf) {
    const uint32_t bar = vfull0 + 8 * buf;
    mbar_expect_tx(bar, (uint32_t)a.v_box * DIMS * 2);
    tma_tile(vsm + buf * vbytes, &vmap, n * hd + item_d0, (int)(first + t * VROWS), bar);
  };
  if (tid == 0)
    for (unsigned t = 0; t < (unsigned)a.k_bufs && t < k_tiles; ++t)
      issue_k(t, (int)t);
  if (tid == AC_THREADS - 32 && has_item)
    for (unsigned t = 0; t < (unsigned)a.v_bufs && t < v_tiles; ++t)
      issue_v(t, (int)t);
  /* ---- query heads; the CTA that scores the token's own row also makes its key */
  const float *ct = a.cos_tab + (size_t)p * hd, *sn = a.sin_tab + (size_t)p * hd;
  for (int g = warp; g < gqa + has_own; g += AC_WARPS) {
    const float *src = g < gqa ? q_in + (size_t)(h0 + g) * hd : a.k + (size_t)n * hd;
    const float *gamma = g < gqa ? a.q_gamma : a.k_gamma;
    if (!a.rope)
      for (int i = lane; i < hd; i += 32)
        qs[g * hd + i] = src[i];
    else if constexpr (HD != 0)
      rope_head_regs<HD / 32>(src, gamma, a.eps, ct, sn, lane, qs + g * hd);
    else
      rope_head(src, gamma, a.eps, ct, sn, hd, lane, qs + g * hd);
  }
  if (append && warp == AC_WARPS - 1)
    for (int i = lane; i < hd; i += 32)
      a.vcache[((size_t)p * a.hkv + n) * hd + i] = float_to_half_bits_rn(a.v[(size_t)n * hd + i]);
  __syncthreads();
  if (a.q_rot && rank == 0)
    for (int i = tid; i < gqa * hd; i += AC_THREADS)
      a.q_rot[(size_t)h0 * hd + i] = qs[i];
  cluster_wait();
  /* ---- scores */
  const double norm = sqrt((double)(float)hd);
  auto put = [&](unsigned t, int g, float sum) {
    const float v = HD == 64 ? __fmul_rn(__fadd_rn(0.0f, sum), 0.125f) // sqrt(64): the same quotient
                             : (float)((double)__fadd_rn(0.0f, sum) / norm);
#pragma unroll 2
    for (int i = 0; i < per_head; ++i)
      st_cluster(esm + 4 * t, (uint32_t)(g * per_head + i), v);
  };
  bool ok = true;
  int kbuf = 0;
  uint32_t kpar = 0;
  for (unsigned t = 0; t < k_tiles; ++t) {
    ok = ok && mbar_wait_bounded(kbar0 + 8 * kbuf, kpar, abort_flag, &g_attn_status, AC_POLLS, 1024);
    uint8_t *tile = ktile + kbuf * kbytes;
    const unsigned t0 = r_lo + t * KROWS, rows = min(r_hi - t0, (unsigned)KROWS);
    if (has_own && t + 1 == k_tiles) { // the token's own row, as the cache will hold it, over what the copy found there
      const int row = (int)rows - 1;
      for (int c = tid; c < hd / 8; c += AC_THREADS) {
        const float *src = kown + 8 * c;
        uint32_t w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          w[i] = (uint32_t)float_to_half_bits_rn(src[2 * i]) | ((uint32_t)float_to_half_bits_rn(src[2 * i + 1]) << 16);
        const uint4 v = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4 *>(tile + (c >> 3) * (KROWS * 128) + row * 128 + (((c & 7) ^ (row & 7)) << 4)) = v;
        if (append)
          *reinterpret_cast<uint4 *>(a.kcache + ((size_t)p * a.hkv + n) * hd + 8 * c) = v;
      }
      __syncthreads();
    }
    if (ok) { // a unit of work: 32 rows and one or two heads
      const int lg = rows <= 32 ? 0 : rows <= 64 ? 1 : KROWS == 128 || rows <= 128 ? 2 : 3, mask = (1 << lg) - 1;
      if (gqa % 2 == 0 && ((gqa / 2) << lg) >= AC_WARPS) { // two heads at a time: a key row is converted once for both
        for (int u = warp; u < (gqa / 2) << lg; u += AC_WARPS) {
          const int row = (u & mask) * 32 + lane, g = 2 * (u >> lg);
          float s[2];
          dot_rows<2, HD, KROWS>(tile, row, qs + g * hd, hd, s);
          if (row < (int)rows) {
            put(t0 + row, g, s[0]);
            put(t0 + row, g + 1, s[1]);
          }
        }
      } else {
        for (int u = warp; u < gqa << lg; u += AC_WARPS) {
          const int row = (u & mask) * 32 + lane, g = u >> lg;
          float s[1];
          dot_rows<1, HD, KROWS>(tile, row, qs + g * hd, hd, s);
          if (row < (int)rows)
            put(t0 + row, g, s[0]);
        }
      }
    }
    if (t + a.k_bufs < k_tiles) {
      __syncthreads(); // the tile's readers are done
      if (tid == 0 && ok) // after a wait that ran out none is started: a CTA without a head may leave behind the next barrier
        issue_k(t + a.k_bufs, kbuf);
    }
    if (++kbuf == a.k_bufs) {
      kbuf = 0;
      kpar ^= 1;
    }
  }
  if (!ok)
    raise_attn(smem_u32(&abort_word)); // the heads' owners lack these scores
  __syncwarp();
  cluster_arrive();
  cluster_wait(); // every score of this CTA's head is here
  ok = !*abort_flag;
  if (a.q_inplace && rank == 0) // every CTA of the cluster has read the raw heads
    for (int i = tid; i < gqa * hd; i += AC_THREADS)
      a.q_inplace[(size_t)h0 * hd + i] = qs[i];
  if (!has_item)
    return;
  /* ---- softmax of head item_head (attn_softmax_kernel's steps) */
  const int head = h0 + item_head;
  float mx = -INFINITY;
  for (unsigned r = tid; r < cnt; r += AC_THREADS)
    mx = fmaxf(mx, e[r]);
#pragma unroll
  for (int o = 16; o; o >>= 1)
    mx = fmaxf(mx, __shfl_xor_sync(FULL, mx, o));
  if (lane == 0)
    red[warp] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int w = 1; w < AC_WARPS; ++w)
    mx = fmaxf(mx, red[w]);
  if (a.sink)
    mx = fmaxf(mx, a.sink[head]);
  const unsigned cnt32 = (cnt + 31) & ~31u; // zeros behind the last row: adding them changes nothing
  for (unsigned r = tid; r < cnt32; r += AC_THREADS)
    e[r] = r < cnt ? exp256_lane(__fsub_rn(e[r], mx)) : 0.f;
  __syncthreads();
  // A turner's share of value tile t (which lies in the ring's place vbuf) into turned tile tbuf: 32 rows of 8 dimensions at a time,
  // transposed by the load; a lane then holds pairs of rows of one dimension.
  int vbuf = 0, tbuf = 0;
  uint32_t vpar = 0, tpar = 1;
  auto turn = [&](unsigned t) {
    if (!mbar_wait_warp(vfull0 + 8 * vbuf, vpar, abort_flag, &g_attn_status, AC_POLLS, 1024))
      return false;
    const int units = (int)(min(cached - t * VROWS, (unsigned)VROWS) + 31) / 32 * 4;
    const uint32_t src = vsm + vbuf * vbytes, dst = ksm + tbuf * AC_TBYTES;
    for (int u = warp - 1; u < units; u += AC_TURNERS) {
      const int row = 32 * (u >> 2) + lane, c = u & 3; // rows of 64 bytes, their 16-byte pieces swizzled
      uint32_t w[4];
      asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                   : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3])
                   : "r"(src + row * 64 + ((c ^ ((row >> 1) & 3)) << 4))
                   : "memory");
#pragma unroll
      for (int m = 0; m < 4; ++m)
        sts32(dst + (8 * c + (lane >> 2)) * AC_TPITCH + (32 * (u >> 2) + 8 * m + 2 * (lane & 3)) * 2, w[m]);
    }
    __syncwarp();
    if (lane == 0) {
      mbar_arrive(tfull0 + 8 * tbuf);
      mbar_arrive(vempty0 + 8 * vbuf);
    }
    if (++vbuf == a.v_bufs)
      vbuf = 0, vpar ^= 1;
    if (++tbuf == a.t_bufs)
      tbuf = 0, tpar ^= 1;
    return true;
  };
  unsigned turned = 0;
  const bool turner = TURN && warp > 0 && warp <= AC_TURNERS;
  if (turner) // the tiles that are on their way already, while the sum is formed (the keys in their place have been read)
    while (ok && turned < (unsigned)min(a.t_bufs, a.v_bufs) && turned < v_tiles)
      ok = turn(turned++);
  if (warp == 0) {
    const float sum = ordered_sum(e, cnt32, a.sink ? exp256_lane(__fsub_rn(a.sink[head], mx)) : 0.0f, lane);
    if (lane == 0)
      s_bcast = sum;
  }
  __syncthreads();
  const float sum = s_bcast;
  for (unsigned r = tid; r < cnt; r += AC_THREADS)
    e[r] = __fdiv_rn(e[r], sum);
  __syncthreads();
  /* ---- values */
  if (warp == AC_WARPS - 1) { // keeps the ring of value tiles full
    if (lane == 0) {
      int buf = 0;
      uint32_t par = 0;
      for (unsigned t = a.v_bufs; t < v_tiles; ++t) {
        if (!mbar_wait_bounded(vempty0 + 8 * buf, par, abort_flag, &g_attn_status, AC_POLLS, 1024))
          break;
        issue_v(t, buf);
        if (++buf == a.v_bufs) {
          buf = 0;
          par ^= 1;
        }
      }
    }
    __syncwarp();
  } else if (turner) {
    while (ok && turned < v_tiles)
      ok = mbar_wait_warp(tempty0 + 8 * tbuf, tpar, abort_flag, &g_attn_status, AC_POLLS, 1024) && turn(turned++);
  } else if (TURN && warp == 0) {
    // Thirty-two rows in the chain while the next thirty-two are on their way: twelve loads, where row by row it would be forty, whose
    // latency the chain's four clocks a row do not hide.
    const int d = item_d0 + lane;
    float acc = 0.f;
    float pr[2][32];
    uint4 vq[2][4];
    auto load = [&](uint32_t vt, uint32_t pt, float(&pp)[32], uint4(&vv)[4]) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
        vv[u] = lds128(vt + 16 * u);
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const uint4 f = lds128(pt + 16 * u);
        pp[4 * u] = __uint_as_float(f.x), pp[4 * u + 1] = __uint_as_float(f.y), pp[4 * u + 2] = __uint_as_float(f.z),
               pp[4 * u + 3] = __uint_as_float(f.w);
      }
    };
    auto chain = [&](const float(&pp)[32], const uint4(&vv)[4], int n) { // the first n rows
#pragma unroll
      for (int u = 0; u < 32; ++u) {
        const uint32_t w[4] = {vv[u >> 3].x, vv[u >> 3].y, vv[u >> 3].z, vv[u >> 3].w};
        if (u < n)
          acc = __fmaf_rn(pp[u], half_bits_to_float((uint16_t)(w[(u >> 1) & 3] >> (16 * (u & 1)))), acc);
      }
    };
    int buf = 0;
    uint32_t par = 0, vt = ksm + lane * AC_TPITCH;
    if (v_tiles) {
      ok = mbar_wait_bounded(tfull0, 0, abort_flag, &g_attn_status, AC_POLLS, 1024) && ok;
      load(vt, esm, pr[0], vq[0]); // reads past the last row stay in the tile and are not used
    }
    for (unsigned t = 0; t < v_tiles; ++t) {
      const uint32_t pt = esm + 4 * t * VROWS;
      const int rows = (int)min(cached - t * VROWS, (unsigned)VROWS);
      const bool more = t + 1 < v_tiles; // then this tile is a whole one
      int nbuf = buf + 1;
      uint32_t npar = par;
      if (nbuf == a.t_bufs)
        nbuf = 0, npar ^= 1;
      // asked now, needed thirty-two rows before this tile's end: the answer takes about a hundred clocks
      const bool next_here = more && mbar_try_wait(tfull0 + 8 * nbuf, npar);
      int j = 0;
#pragma unroll 1
      for (; j + 64 <= rows; j += 64) {
        load(vt + 2 * (j + 32), pt + 4 * (j + 32), pr[1], vq[1]);
        chain(pr[0], vq[0], 32);
        uint32_t ahead = vt + 2 * (j + 64);
        if (j + 64 == VROWS) {
          if (more && !next_here)
            ok = mbar_wait_bounded(tfull0 + 8 * nbuf, npar, abort_flag, &g_attn_status, AC_POLLS, 1024) && ok;
          ahead = ksm + nbuf * AC_TBYTES + lane * AC_TPITCH; // behind the last tile: read and not used
        }
        load(ahead, pt + 4 * (j + 64), pr[0], vq[0]);
        chain(pr[1], vq[1], 32);
      }
      if (j < rows) { // the last tile: up to 63 rows, the first 32 of them in registers
        if (rows - j > 32) {
          load(vt + 2 * (j + 32), pt + 4 * (j + 32), pr[1], vq[1]);
          chain(pr[0], vq[0], 32);
          chain(pr[1], vq[1], rows - j - 32);
        } else {
          chain(pr[0], vq[0], rows - j);
        }
      }
      __syncwarp();
      if (lane == 0)
        mbar_arrive(tempty0 + 8 * buf);
      buf = nbuf;
      par = npar;
      vt = ksm + buf * AC_TBYTES + lane * AC_TPITCH;
    }
    if (ok) {
      if (a.rope)
        acc = __fmaf_rn(e[cnt - 1], half_bits_to_float(float_to_half_bits_rn(a.v[(size_t)n * hd + d])), acc);
      out[(size_t)head * hd + d] = acc;
    }
  } else if (!TURN && warp < DIMS / 32) {
    const int d = item_d0 + tid;
    float acc = 0.f;
    // Sixteen rows in the chain while the next sixteen -- of the next tile at a tile's end -- are on their way.
    float pr[2][16];
    uint16_t vb[2][16];
    auto load = [&](const uint16_t *vt, const float *pt, float(&pp)[16], uint16_t(&vv)[16]) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const float4 f = *reinterpret_cast<const float4 *>(pt + 4 * u);
        pp[4 * u] = f.x, pp[4 * u + 1] = f.y, pp[4 * u + 2] = f.z, pp[4 * u + 3] = f.w;
      }
#pragma unroll
      for (int u = 0; u < 16; ++u)
        vv[u] = vt[u * DIMS];
    };
    int buf = 0;
    uint32_t par = 0;
    const uint16_t *vt = reinterpret_cast<const uint16_t *>(vtile) + tid;
    if (v_tiles) {
      ok = mbar_wait_bounded(vfull0, 0, abort_flag, &g_attn_status, AC_POLLS, 1024) && ok;
      load(vt, e, pr[0], vb[0]); // reads past the last row stay in shared memory and are not used
    }
    for (unsigned t = 0; t < v_tiles; ++t) {
      const float *pt = e + t * VROWS;
      const unsigned rows = min(cached - t * VROWS, (unsigned)VROWS);
      int nbuf = buf + 1;
      uint32_t npar = par;
      if (nbuf == a.v_bufs) {
        nbuf = 0;
        npar ^= 1;
      }
      const uint16_t *nvt = reinterpret_cast<const uint16_t *>(vtile + nbuf * vbytes) + tid;
      // asked now, needed sixteen rows before this tile's end: the answer takes about a hundred clocks (a question that may not suspend
      // the thread, test_wait, measured the same: 37.2 us for 4096 rows, replay 3225 and 3231)
      const bool next_here = t + 1 < v_tiles && mbar_try_wait(vfull0 + 8 * nbuf, npar);
      if (rows == VROWS) {
        // Unrolled all the way, a tile of 256 rows is 14 KB of code: 1.6 us less for 4096 rows (36.8 and 35.2), but 4 % more for a decode
        // step at a context of 512 (16 tokens over four layers 3386 us, 3252 like this), where every launch fetches its code anew. Not
        // unrolled at all: 39.5 us.
#pragma unroll(DIMS == 64 ? 2 : 4)
        for (int j = 0; j < VROWS; j += 32) {
          load(vt + (j + 16) * DIMS, pt + j + 16, pr[1], vb[1]);
#pragma unroll
          for (int u = 0; u < 16; ++u)
            acc = __fmaf_rn(pr[0][u], half_bits_to_float(vb[0][u]), acc);
          const bool end = j + 32 == VROWS;
          if (end && t + 1 < v_tiles && !next_here)
            ok = mbar_wait_bounded(vfull0 + 8 * nbuf, npar, abort_flag, &g_attn_status, AC_POLLS, 1024) && ok;
          load(end ? nvt : vt + (j + 32) * DIMS, pt + j + 32, pr[0], vb[0]); // behind the last tile: read and not used
#pragma unroll
          for (int u = 0; u < 16; ++u)
            acc = __fmaf_rn(pr[1][u], half_bits_to_float(vb[1][u]), acc);
        }
      } else { // the last tile
        // The compiler unrolls these two loops further where it is let, and a short context's launch, which has just this tile, waits for
        // the code: 16 tokens over four layers at a context of 30 / 100 / 512 2976 / 3058 / 3241 us, like this 2922 / 2939 / 3219 (value
        // phase at 100 rows 5700 clocks, 3700; taken alone, with the code at hand, 2200 and 2000). Not unrolled at all 2911 / 2928 / 3225,
        // but 0.2 us more for a launch of 128 rows alone.
        unsigned j = 0;
#pragma unroll 2
        for (; j + 16 <= rows; j += 16) {
          load(vt + j * DIMS, pt + j, pr[0], vb[0]);
#pragma unroll
          for (int u = 0; u < 16; ++u)
            acc = __fmaf_rn(pr[0][u], half_bits_to_float(vb[0][u]), acc);
        }
#pragma unroll 2
        for (; j < rows; ++j)
          acc = __fmaf_rn(pt[j], half_bits_to_float(vt[j * DIMS]), acc);
      }
      __syncwarp();
      if (lane == 0) // the tile's last loads were issued sixteen multiply-adds ago
        mbar_arrive(vempty0 + 8 * buf);
      buf = nbuf;
      par = npar;
      vt = nvt;
    }
    if (d < hd && ok) {
      if (a.rope)
        acc = __fmaf_rn(e[cnt - 1], half_bits_to_float(float_to_half_bits_rn(a.v[(size_t)n * hd + d])), acc);
      out[(size_t)head * hd + d] = acc;
    }
  }
  if (*abort_flag) // give the copies in flight time to land in this CTA's shared memory
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
}

int read_attn_status(int *out) {
  int v = 0;
  NNTR_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_attn_status, sizeof(int)));
  *out = v;
  return NNTR_CUDA_OK;
}
int clear_attn_status() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_attn_status, &zero, sizeof(int)), "clear_attn_status");
}

/* ---------------------------------------------------------------- launchers */

static int check_attn(const nntr_attn_desc *a) {
  if (!a || a->n_heads_q == 0 || a->n_heads_kv == 0 || a->head_dim == 0)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention: null or empty description");
  if (a->n_heads_q % a->n_heads_kv)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention: %u query heads are not a multiple of %u key/value heads",
                     a->n_heads_q, a->n_heads_kv);
  // the reference's scalar tails (libm exp for head counts that are not multiples of 8) are not reproduced
  if (a->n_heads_q % 8 || a->head_dim % 8)
    return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "attention: head count and head_dim must be multiples of 8 (%u, %u)",
                     a->n_heads_q, a->head_dim);
  if (a->n_heads_q / a->n_heads_kv > 16)
    return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "attention: at most 16 query heads per key/value head");
  if (a->window == 0)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention: window of 0 rows");
  return NNTR_CUDA_OK;
}

static void pdl_cfg(cudaLaunchConfig_t &cfg, cudaLaunchAttribute *attr, unsigned flags, cudaStream_t st) {
  cfg.stream = st;
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (flags & NNTR_CUDA_GEMV_PDL) ? 1 : 0;
}

static int launch_rope_rows(const nntr_attn_desc *a, unsigned pos, const unsigned *pos_dev, unsigned tokens, size_t ld, float *q,
                            const float *k, const float *v, const float *q_gamma, const float *k_gamma, float eps,
                            uint16_t *kcache, uint16_t *vcache, const float *cos_tab, const float *sin_tab, unsigned flags,
                            cudaStream_t st) {
  int rc = check_attn(a);
  if (rc)
    return rc;
  if (!q || !k || !v || !kcache || !vcache || !cos_tab || !sin_tab)
    return set_error(NNTR_CUDA_ERR_INVALID, "rope_cache_append: null pointer");
  const int heads = (int)(a->n_heads_q + 2 * a->n_heads_kv);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  pdl_cfg(cfg, attr, flags, st);
  cfg.gridDim = dim3((unsigned)((heads + ROPE_WARPS - 1) / ROPE_WARPS), tokens);
  cfg.blockDim = dim3(32 * ROPE_WARPS);
  cfg.dynamicSmemBytes = (size_t)ROPE_WARPS * a->head_dim * sizeof(float);
  cudaError_t e = cudaLaunchKernelEx(&cfg, rope_cache_append_kernel, q, k, v, q_gamma, k_gamma, eps, kcache, vcache,
                                     cos_tab, sin_tab, pos_dev, pos, (int)a->n_heads_q, (int)a->n_heads_kv,
                                     (int)a->head_dim, (long long)ld);
  count_launch();
  return check_cuda(e, "rope_cache_append launch");
}

int launch_rope_cache_append(const nntr_attn_desc *a, unsigned pos, const unsigned *pos_dev, float *q, const float *k,
                             const float *v, const float *q_gamma, const float *k_gamma, float eps, uint16_t *kcache,
                             uint16_t *vcache, const float *cos_tab, const float *sin_tab, unsigned flags,
                             cudaStream_t st) {
  return launch_rope_rows(a, pos, pos_dev, 1, 0, q, k, v, q_gamma, k_gamma, eps, kcache, vcache, cos_tab, sin_tab, flags, st);
}

size_t attention_workspace_bytes(const nntr_attn_desc *a, unsigned max_rows) {
  if (!a)
    return 0;
  const size_t rows = max_rows < a->window ? max_rows : a->window;
  return ((rows + 3) & ~(size_t)3) * a->n_heads_q * sizeof(float); // head-major rows are padded to four elements
}

/* The cluster launch, or *taken = false where it does not apply: heads of more than 128 dimensions, more rows than shared
 * memory keeps, or NNTR_CUDA_ATTN_SEPARATE. bound, rows: rows of the caches and of a window that the launch must be able to take;
 * likely: rows of the window that it is expected to have, no more than rows. */
static int launch_attn_cluster(AttnStep a, unsigned bound, unsigned rows, unsigned likely, unsigned flags, cudaStream_t st, bool *taken) {
  const int hd = a.hd;
  *taken = false;
  if ((flags & NNTR_CUDA_ATTN_SEPARATE) || hd > 128 || rows > AC_MAX_ROWS)
    return NNTR_CUDA_OK;
  int gqa = a.hq / a.hkv;
  const bool many = a.tokens > 1;
  // Of one token with a long window, a CTA for 32 dimensions of a head where the chip has room for that, in clusters of four. Shorter
  // windows in a decode step are slower so (16 tokens over four layers, 32 / 8 heads of 128 at a context of 100 / 512: 2959 / 3197 us, with
  // slices 3094 / 3278), because every launch there fetches its code anew and this is more of it; 64 / 8 heads of 64 at 2000: 3906, with
  // slices 3803. Alone 64 / 8 heads of 64 at 2000 / 4096 / 6000 rows 23.2 / 36.6 / 50.4 us, with slices 21.6 / 33.5 / 45.0; 32 / 8 of 128 at
  // 1500 / 5000 20.3 / 44.7 and 18.7 / 40.8. Heads whose CTAs would own 128 dimensions each leave most of the chip idle without: 32 / 4 heads
  // of 128 at 512 / 3000 rows 12.2 / 34.1, with slices 10.5 / 28.1; decode steps at 100 / 512 3012 / 3325 and 3081 / 3253, three layers at
  // 1500 3146 and 2912. The rows that count are those that the window is likely to have: 16 tokens over three layers at a context of 100 with
  // caches of 8192 rows, 32 / 8 heads 2160 us, with slices 2234, 64 / 8 heads of 64 2146 and 2196; at 3000 3182 and 3260, 3065 and 3180.
  const int slices = hd / 32, slice_heads = hd == 64 ? 2 : 1;
  static std::atomic<uint32_t> attr_done[64];
  static ClusterFit fit64, fit128;
  int dev = 0;
  NNTR_CHECK_CUDA(cudaGetDevice(&dev));
  if (!attr_done[dev & 63].load(std::memory_order_acquire)) {
    for (const auto k : {attn_cluster_kernel<128, 32>, attn_cluster_kernel<128, 64>, attn_cluster_kernel<128, 128>, attn_cluster_kernel<64, 32>,
                         attn_cluster_kernel<64, 64>, attn_cluster_kernel<0, 64>, attn_cluster_kernel<0, 128>})
      NNTR_CHECK_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, AC_SMEM_ALONE));
    attr_done[dev & 63].store(1, std::memory_order_release);
  }
  const bool sliced = !many && likely > (hd > 64 && gqa > 4 ? 256u : AC_SLICED_ROWS) && (hd == 64 || hd == 128) && gqa % slice_heads == 0 &&
                      a.hq * slices / 4 <= (hd == 64 ? fit64(attn_cluster_kernel<64, 32>, 4, AC_THREADS, AC_SMEM_ALONE)
                                                     : fit128(attn_cluster_kernel<128, 32>, 4, AC_THREADS, AC_SMEM_ALONE));
  a.groups = sliced ? gqa / slice_heads : 1;
  while (gqa % a.groups || gqa / a.groups > 8) // at most 16 query heads in all (check_attn)
    ++a.groups;
  gqa /= a.groups;
  // else a CTA owns 64 dimensions of a head where eight CTAs are enough for that, or -- and for many tokens, which fill the
  // machine anyway -- the whole head
  const int dims = sliced ? 32 : hd <= 64 || (gqa * 2 <= 8 && !many) ? 64 : 128;
  const int items = gqa * ((hd + dims - 1) / dims);
  // eight CTAs per cluster while that leaves no cluster waiting for SMs -- 16 clusters of eight run in two waves (11.1 us for a
  // window of 50 rows, clusters of four 8), because a cluster lies inside one part of the chip --, at least as many as items
  const unsigned clusters = (unsigned)(a.hkv * a.groups);
  unsigned csize = sliced || (clusters > 12 && items <= 4) ? 4 : 8;
  while (csize > 1 && (many || clusters * csize > 144u) && (int)(csize / 2) >= items)
    csize /= 2;
  // buffers for what the launch can need, no more: a prompt's CTAs share an SM where they fit
  a.cap_rows = rows;
  const unsigned k_rows = sliced ? 256u : 128u, share = (rows + csize - 1) / csize;
  const unsigned k_tiles = (share + k_rows - 1) / k_rows, v_rows = dims <= 64 ? 256u : 128u, v_tiles = (rows + v_rows - 1) / v_rows;
  a.t_bufs = sliced ? (int)std::min(v_tiles, (unsigned)AC_TBUF_MAX) : 0;
  const unsigned k_max = hd > 64 ? 2u : sliced ? 3u : 4u;
  a.k_bufs = (int)(k_tiles < k_max ? k_tiles : k_max);
  const unsigned v_max = dims == 64 ? 3u : (unsigned)AC_VBUF_MAX;
  a.v_bufs = (int)(v_tiles < v_max ? v_tiles : v_max);
  const auto box = [&](unsigned n) { return n <= 32 ? 32 : n <= 64 ? 64 : n <= 128 ? 128 : k_rows; };
  a.k_box = (int)box(share);
  a.v_box = (int)((rows < v_rows ? rows : v_rows) + 31) / 32 * 32;
  const auto layout = [&] { return ac_layout(gqa, hd, dims, (int)k_rows, a.k_bufs, a.v_bufs, a.t_bufs, a.v_box, rows); };
  AcLayout L = layout();
  while (L.total > AC_SMEM_ALONE && (a.v_bufs > 2 || a.k_bufs > 1)) {
    a.v_bufs > 2 ? --a.v_bufs : --a.k_bufs;
    L = layout();
  }
  const auto kernel = hd == 128  ? (dims == 32   ? attn_cluster_kernel<128, 32>
                                    : dims == 64 ? attn_cluster_kernel<128, 64>
                                                 : attn_cluster_kernel<128, 128>)
                      : hd == 64 ? (dims == 32 ? attn_cluster_kernel<64, 32> : attn_cluster_kernel<64, 64>)
                                 : (dims == 64 ? attn_cluster_kernel<0, 64> : attn_cluster_kernel<0, 128>);
  CUtensorMap kmap, vmap;
  // maps over the caches, [bound rows][hkv * hd] fp16; keys swizzled: 64 values = 128 bytes
  const uint64_t width = (uint64_t)a.hkv * hd;
  int rc = encode_map_2d(&kmap, a.kcache, 2, width, bound, width * 2, 64, (unsigned)a.k_box, true);
  if (rc || (rc = encode_map_2d(&vmap, a.vcache, 2, width, bound, width * 2, (unsigned)dims, (unsigned)a.v_box, sliced)))
    return rc;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = csize;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = (flags & NNTR_CUDA_GEMV_PDL) ? 2 : 1;
  cfg.stream = st;
  cfg.gridDim = dim3(clusters * csize, a.tokens);
  cfg.blockDim = dim3(AC_THREADS);
  // A decode step's CTAs keep their SMs to themselves: a second one of them, or the next launch's, let in early, takes issue slots and
  // the way to memory from a kernel that is bound by latency. 16 tokens over four layers, 32 / 8 heads of 128 at a context of 30 / 100 /
  // 250 / 512: 3028 / 3059 / 3103 / 3252 us with what the buffers need, 2935 / 2949 / 3042 / 3217 with 200 KB; 64 / 8 heads of 64 at 100 /
  // 512 / 2000: 2977 / 3229 / 3880 and 2922 / 3140 / 3880.
  cfg.dynamicSmemBytes = a.tokens == 1 && L.total < AC_SMEM_ALONE ? AC_SMEM_ALONE : L.total;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, kmap, vmap, a);
  count_launch();
  *taken = true;
  return check_cuda(e, "attention launch");
}

/* Rows that the window is expected to have: with the position in device memory (a captured step) pos says where the positions start. The
 * bound of such a launch says nothing about it: caches are as long as the longest context. */
static unsigned likely_rows(const nntr_attn_desc *a, unsigned pos, unsigned bound) {
  return std::min(std::min(pos, bound - 1) + 1, a->window);
}

int launch_attention_decode(const nntr_attn_desc *a, unsigned pos, const unsigned *pos_dev, unsigned max_rows,
                            const float *q, const uint16_t *kcache, const uint16_t *vcache, float *out, void *ws,
                            size_t ws_bytes, unsigned flags, cudaStream_t st) {
  int rc = check_attn(a);
  if (rc)
    return rc;
  if (!q || !kcache || !vcache || !out || !ws)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_decode: null pointer");
  // grids are sized for the largest row count this call can see: pos + 1 when the position comes by value, else the
  // caller's bound
  const unsigned bound = pos_dev ? max_rows : pos + 1;
  if (bound == 0 || (!pos_dev && max_rows && pos + 1 > max_rows))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_decode: position %u beyond the %u rows allowed", pos, max_rows);
  const unsigned rows = bound < a->window ? bound : a->window;
  const size_t ws_need = (((size_t)rows + 3) & ~(size_t)3) * a->n_heads_q * sizeof(float);
  if (ws_bytes < ws_need)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_decode: workspace of %zu bytes needed, %zu given", ws_need, ws_bytes);
  if ((reinterpret_cast<uintptr_t>(kcache) & 15) || (reinterpret_cast<uintptr_t>(vcache) & 15) ||
      (reinterpret_cast<uintptr_t>(ws) & 15) || (reinterpret_cast<uintptr_t>(q) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_decode: q, caches and workspace must be 16-byte aligned");
  float *scores = static_cast<float *>(ws);
  const int hq = (int)a->n_heads_q, hkv = (int)a->n_heads_kv, hd = (int)a->head_dim;
  AttnStep s = {};
  s.q = q, s.kcache = const_cast<uint16_t *>(kcache), s.vcache = const_cast<uint16_t *>(vcache);
  s.out = out, s.sink = a->sink, s.pos_dev = pos_dev, s.pos = pos, s.window = a->window;
  s.hq = hq, s.hkv = hkv, s.hd = hd, s.tokens = 1;
  bool taken;
  if ((rc = launch_attn_cluster(s, bound, rows, likely_rows(a, pos, bound), flags, st, &taken)) || taken)
    return rc;
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  pdl_cfg(cfg, attr, flags, st);
  cfg.gridDim = dim3((rows + SCORE_WARPS * 4 - 1) / (SCORE_WARPS * 4), (unsigned)hkv);
  cfg.blockDim = dim3(32 * SCORE_WARPS);
  cfg.dynamicSmemBytes = (size_t)(hq / hkv) * hd * sizeof(float) + (size_t)SCORE_WARPS * 4 * hd * sizeof(uint16_t);
  cudaError_t e = cudaLaunchKernelEx(&cfg, attn_scores_kernel, q, kcache, scores, pos_dev, pos, hq, hkv, hd, a->window);
  count_launch();
  if ((rc = check_cuda(e, "attention scores launch")))
    return rc;
  cfg.gridDim = dim3((unsigned)hq);
  cfg.blockDim = dim3(SOFTMAX_THREADS);
  const unsigned cap_rows = rows < 11264u ? rows : 11264u; // 44 KB of shared memory at most; later rows stay in global
  cfg.dynamicSmemBytes = (size_t)cap_rows * sizeof(float);
  e = cudaLaunchKernelEx(&cfg, attn_softmax_kernel, scores, a->sink, pos_dev, pos, hq, a->window, cap_rows);
  count_launch();
  if ((rc = check_cuda(e, "attention softmax launch")))
    return rc;
  cfg.gridDim = dim3((unsigned)((hd + 31) / 32), (unsigned)hkv);
  cfg.blockDim = dim3(32 * (unsigned)(hq / hkv));
  cfg.dynamicSmemBytes = VBUF * ((size_t)VT * 64 + (size_t)VT * (hq / hkv) * sizeof(float));
  e = cudaLaunchKernelEx(&cfg, attn_values_kernel, static_cast<const float *>(scores), vcache, out, pos_dev, pos, hq, hkv,
                         hd, a->window);
  count_launch();
  return check_cuda(e, "attention values launch");
}

/* One token's whole attention step: per-head norms (gammas may be null) + rotary + cache append + scores + softmax +
 * values -- one launch where launch_attn_cluster applies, else the rotary launch followed by launch_attention_decode, which
 * rotates q in place. For windows beyond ATTN_INPLACE_ROWS q is rotated in place either way, as the interface says. */
constexpr unsigned ATTN_INPLACE_ROWS = 2048;
int launch_attention_step(const nntr_attn_desc *a, unsigned pos, const unsigned *pos_dev, unsigned max_rows, float *q,
                          const float *k, const float *v, const float *q_gamma, const float *k_gamma, float eps,
                          uint16_t *kcache, uint16_t *vcache, const float *cos_tab, const float *sin_tab, float *q_rot,
                          float *out, void *ws, size_t ws_bytes, unsigned flags, cudaStream_t st) {
  int rc = check_attn(a);
  if (rc)
    return rc;
  if (!q || !k || !v || !kcache || !vcache || !cos_tab || !sin_tab || !out || !ws)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_step: null pointer");
  if ((q_gamma == nullptr) != (k_gamma == nullptr))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_step: q_gamma and k_gamma come together or not at all");
  const unsigned bound = pos_dev ? max_rows : pos + 1;
  if (bound == 0 || (!pos_dev && max_rows && pos + 1 > max_rows))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_step: position %u beyond the %u rows allowed", pos, max_rows);
  const unsigned rows = bound < a->window ? bound : a->window;
  const int hq = (int)a->n_heads_q, hkv = (int)a->n_heads_kv, hd = (int)a->head_dim;
  if ((reinterpret_cast<uintptr_t>(kcache) & 15) || (reinterpret_cast<uintptr_t>(vcache) & 15) ||
      (reinterpret_cast<uintptr_t>(ws) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_step: caches and workspace must be 16-byte aligned");
  const size_t ws_need = (((size_t)rows + 3) & ~(size_t)3) * a->n_heads_q * sizeof(float);
  if (ws_bytes < ws_need)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_step: workspace of %zu bytes needed, %zu given", ws_need, ws_bytes);
  AttnStep s = {};
  s.q = q, s.k = k, s.v = v, s.q_gamma = q_gamma, s.k_gamma = k_gamma, s.eps = eps;
  s.kcache = kcache, s.vcache = vcache, s.cos_tab = cos_tab, s.sin_tab = sin_tab;
  s.q_rot = q_rot, s.q_inplace = rows > ATTN_INPLACE_ROWS ? q : nullptr, s.out = out, s.sink = a->sink;
  s.pos_dev = pos_dev, s.pos = pos, s.window = a->window;
  s.hq = hq, s.hkv = hkv, s.hd = hd, s.rope = 1, s.tokens = 1;
  bool taken;
  if ((rc = launch_attn_cluster(s, bound, rows, likely_rows(a, pos, bound), flags, st, &taken)) || taken)
    return rc;
  if ((rc = launch_rope_cache_append(a, pos, pos_dev, q, k, v, q_gamma, k_gamma, eps, kcache, vcache, cos_tab, sin_tab, flags,
                                     st)))
    return rc;
  if (q_rot)
    NNTR_CHECK_CUDA(cudaMemcpyAsync(q_rot, q, (size_t)hq * hd * sizeof(float), cudaMemcpyDeviceToDevice, st));
  return launch_attention_decode(a, pos, pos_dev, max_rows, q, kcache, vcache, out, ws, ws_bytes, flags, st);
}

/* Consecutive tokens of a prompt: every token's rotary work and cache rows in one launch, every token's attention -- over its own
 * row and the rows before it -- in a second one. The same kernels as a decode step's, so the same bits as that many steps. */
int launch_attention_rows(const nntr_attn_desc *a, unsigned pos, unsigned tokens, unsigned max_rows, float *q, const float *k,
                          const float *v, size_t ld, const float *q_gamma, const float *k_gamma, float eps, uint16_t *kcache, uint16_t *vcache,
                          const float *cos_tab, const float *sin_tab, float *out, size_t ld_out, unsigned flags,
                          cudaStream_t st) {
  int rc = check_attn(a);
  if (rc)
    return rc;
  if (!q || !k || !v || !kcache || !vcache || !cos_tab || !sin_tab || !out)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_rows: null pointer");
  if ((q_gamma == nullptr) != (k_gamma == nullptr))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_rows: q_gamma and k_gamma come together or not at all");
  if ((reinterpret_cast<uintptr_t>(kcache) & 15) || (reinterpret_cast<uintptr_t>(vcache) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_rows: caches must be 16-byte aligned");
  if (tokens == 0)
    return NNTR_CUDA_OK;
  if ((unsigned long long)pos + tokens > max_rows)
    return set_error(NNTR_CUDA_ERR_INVALID, "attention_rows: positions %u to %llu beyond the %u rows allowed", pos,
                     (unsigned long long)pos + tokens - 1, max_rows);
  const unsigned bound = pos + tokens, rows = bound < a->window ? bound : a->window;
  if (tokens > 65535 || a->head_dim > 128 || rows > AC_MAX_ROWS)
    return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "attention_rows: heads of at most 128 dimensions, windows of at most %u rows",
                     AC_MAX_ROWS);
  if ((rc = launch_rope_rows(a, pos, nullptr, tokens, ld, q, k, v, q_gamma, k_gamma, eps, kcache, vcache, cos_tab, sin_tab, flags,
                             st)))
    return rc;
  AttnStep s = {};
  s.q = q, s.kcache = kcache, s.vcache = vcache, s.out = out, s.sink = a->sink, s.pos = pos, s.window = a->window;
  s.hq = (int)a->n_heads_q, s.hkv = (int)a->n_heads_kv, s.hd = (int)a->head_dim;
  s.tokens = tokens, s.q_ld = (long long)ld, s.out_ld = (long long)ld_out;
  bool taken;
  return launch_attn_cluster(s, bound, rows, rows, flags & ~NNTR_CUDA_ATTN_SEPARATE, st, &taken);
}

} // namespace nntr
