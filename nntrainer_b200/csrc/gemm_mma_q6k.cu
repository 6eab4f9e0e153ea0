// SPDX-License-Identifier: Apache-2.0
/**
 * @file  gemm_mma_q6k.cu
 * @brief Bit-exact GEMM for Q6_K weights with more than one activation row (the lm_head of concurrent decode streams): fp16
 *        warp MMAs whose products and sums are all integers that fp32 holds.
 *
 * Reference chain reproduced (nntr_vec_dot_q6_K_q8_K, nntr_ggml_impl.cpp:8600-8696; nntr_ggml_impl_utils.h:59-65): per
 * super-block eight integers, number l summing sc * (q - 32) * a over the elements 4l .. 4l+3 of each of the eight
 * 32-element chunks; acc[l] = fma(d_a * d_w, (float)sum_l, acc[l]) block after block; result
 * ((a4+a0)+(a6+a2))+((a5+a1)+(a7+a3)).
 *
 * The sum number l is a contraction over 32 elements with eight different scales in it. With the scale folded into the
 * weight, sc * (q - 32) needs 13 bits; the scale split into 16 * sh + sl, both products fit fp16:
 *     |sh * (q - 32)| <= 256,   sl * (q - 32) <= 480
 * so two m16n8k16 MMAs for each part give sum_l exactly: every partial sum is at most 32 * 32 * 128 * 127 < 2^24 in
 * magnitude whatever the order. (Weights enter over 4 and activations times 4: (1024 + q) * 4 sh and the 1056 * 4 sh that
 * is subtracted in the same fused step then stay inside fp16, all exact.)
 *
 * Fragments: for sum l lane (g, t) of the warp holds, for the rows g and g + 8, word l of the 32 ql bytes that the quarters
 * t % 2 and t % 2 + 2 of half t / 2 share as low and high nibbles, and word l of that half's 32 qh bytes. The 210-byte
 * blocks are only 2-byte aligned: the 16-byte aligned 224 bytes around each of a warp's 16 blocks of a super-block come into
 * shared memory by bulk copies (which leave the L1 cache to the activations), and the words read there are funnel-shifted.
 *
 * A warp owns 16 weight rows and up to 16 activation rows (32 chain accumulators per 8 rows) over all of K and shares
 * nothing with other warps; with few rows eight warps share them along K (SPLIT below). Bound by the unpack (about 390 logic and 270
 * multiply instructions per 16 x 256 weights, at half rate both; issue slots 58 % full, the logic pipe 54 %): 8 x 151936 x 2560 124 us
 * (CUDA-core kernel before: 697; the weights' bytes alone take 49), 31 rows 339 us (2360). Bringing the rows in by 4- and 8-byte
 * asynchronous copies or through registers measured the same or slower.
 */
#include "cluster.cuh"
#include "common.cuh"
#include "pipeline.cuh"

namespace nntr {

namespace {

constexpr int Q6M_WARPS = 4;
constexpr int Q6M_COPY = 224;     // 16-byte aligned bytes around a block
constexpr int Q6M_ROW_WORDS = 60; // 4 more: neighbouring rows fall into different banks
constexpr uint32_t Q6M_POLLS = 1u << 22;
constexpr int Q6M_STAGE_WORDS = 16 * Q6M_ROW_WORDS; // 16 rows
/* Activations: per tile of 8 rows and super-block [8 sums l][lane 4g + t][16 bytes]: elements 4l + {0,2,1,3} of the quarters
 * t % 2 and t % 2 + 2 of half t / 2 of row g, as fp16(4 q8); then the 8 rows' scales. */
constexpr int Q6M_TILE = 8 * 512 + 32;

__device__ int g_q6m_status = 0;

__device__ __forceinline__ uint32_t h2u(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }
__device__ __forceinline__ __half2 u2h(uint32_t u) { return *reinterpret_cast<const __half2 *>(&u); }

__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma_f16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
/* Three-input logic written out: the compiler otherwise distributes masks and shifts over the two parts of a 6-bit value
 * (502 instead of about 250 logic instructions per 16 x 256 weights). */
template <int LUT> __device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
  uint32_t d;
  asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
  return d;
}
constexpr int LUT_SELECT = 0xE4;  // (a & c) | (b & ~c)
constexpr int LUT_AND_OR = 0xEA;  // (a & b) | c
constexpr int LUT_AND_XOR = 0x6A; // (a & b) ^ c

/* CTAS: CTAs per SM that registers and shared memory are held to. Four with 4 bytes of spills and two stages (which leave the L1
 * cache room for the activations; with three stages 137 us instead of 122 for 8 x 151936 x 2560, three CTAs of three stages 128), where
 * four per SM need fewer rounds. */
template <int CTAS> constexpr int Q6M_STAGES = CTAS == 3 ? 3 : 2;
/* SPLIT: the CTA has eight warps, all of them on the same 16 weight rows, and each takes every eighth super-block; the chains go from warp
 * to warp, one super-block further at each. For calls with too few rows to fill the chip, where the 3400 clocks that a warp on its own
 * takes for a super-block, one after the other, are the call's time: 5 x 4096 x 4096 30.0 -> 11.3 us, 8 x 2560 x 9728 65 -> 21. */
constexpr int Q6S_WARPS = 8;
constexpr int Q6S_SMEM = Q6S_WARPS * (2 * Q6M_STAGE_WORDS * 4 + 8 * 32 * 16);
template <int NT, int CTAS, bool SPLIT>
__global__ void __launch_bounds__((SPLIT ? Q6S_WARPS : Q6M_WARPS) * 32, CTAS)
gemm_q6_K_mma_kernel(const uint8_t *__restrict__ act, const uint8_t *__restrict__ W, float *__restrict__ C, int ldc, int M,
                     int N, int nb) {
  // High nibbles used where they lie, with their own factors: the same number of operations, 187 against 193 us for 16 x 151936 x
  // 2560 and 338 against 346 for 31 rows; with one tile of rows 130 against 128 and 32.4 against 30.3 for 5 x 4096 x 4096.
  constexpr bool IN_PLACE = NT == 2;
  constexpr int STAGES = Q6M_STAGES<CTAS>;
  // a shift less per word of high bits (1 % with four CTAs); with three, where a warp's own latency counts, 5 x 4096 x 4096 31.7 us instead of 30.0
  constexpr bool DENSE = NT == 1 && CTAS == 4;
  constexpr int WARPS = SPLIT ? Q6S_WARPS : Q6M_WARPS, EVERY = SPLIT ? WARPS : 1; // a warp's super-blocks
  static_assert(!SPLIT || NT == 1, "a hand-over per super-block and warp");
  extern __shared__ __align__(16) uint32_t split_smem[]; // SPLIT: the stages, then the chains on their way
  __shared__ alignas(16) uint32_t stage[SPLIT ? 1 : WARPS][SPLIT ? 1 : STAGES][SPLIT ? 1 : Q6M_STAGE_WORDS];
  __shared__ alignas(8) unsigned long long bars[WARPS][STAGES];
  __shared__ int aborted[SPLIT ? 1 : WARPS]; // one per warp that stores for itself: the warps of such a CTA do not meet
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3, run = t & 1, h = t >> 1;
  const int n0 = (SPLIT ? blockIdx.y : blockIdx.y * WARPS + warp) * 16, m0 = blockIdx.x * 8 * NT;
  if (n0 >= N) {
    pdl_wait();
    return;
  }
  const int nt = min(NT, (M - m0 + 7) >> 3);
  const size_t row_bytes = (size_t)nb * sizeof(BlockQ6K);
  const uint32_t bar = smem_u32(bars[warp]);
  auto stage_of = [&](int k) { // this warp's
    if constexpr (SPLIT)
      return split_smem + (warp * STAGES + k) * Q6M_STAGE_WORDS;
    else
      return stage[warp][k];
  };
  const uint32_t sm = smem_u32(stage_of(0));
  volatile int *abort_flag = &aborted[SPLIT ? 0 : warp];
  if (lane == 0) {
    for (int k = 0; k < STAGES; ++k)
      mbar_init(bar + 8 * k, 1);
    if (!SPLIT || warp == 0)
      *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  SPLIT ? __syncthreads() : __syncwarp();
  // Copies super-block b of the 16 rows, lane i the block of row i (rows past the end repeat the last one). A block starts 0
  // to 14 bytes into a 16-byte piece, so its 210 bytes always lie in 14 whole pieces, and the copy never leaves the piece
  // that holds the block's own first or last byte.
  const uint8_t *mine = W + (size_t)min(n0 + (lane & 15), N - 1) * row_bytes;
  auto fetch = [&](int u) { // the warp's u-th
    const int k = u % STAGES, b = SPLIT ? warp + u * EVERY : u;
    if (lane == 0)
      mbar_expect_tx(bar + 8 * k, 16 * Q6M_COPY);
    __syncwarp();
    if (lane < 16)
      bulk_g2s(sm + (k * Q6M_STAGE_WORDS + lane * Q6M_ROW_WORDS) * 4,
               reinterpret_cast<const void *>(reinterpret_cast<uintptr_t>(mine + (size_t)b * sizeof(BlockQ6K)) & ~(uintptr_t)15),
               Q6M_COPY, bar + 8 * k);
  };
  const int units = SPLIT ? (nb - warp + EVERY - 1) / EVERY : nb; // super-blocks of this warp
  for (int u = 0; u < STAGES - 1 && u < units; ++u) // the weights do not depend on the kernel before
    fetch(u);
  pdl_wait(); // the activation tiles do
  pdl_launch_dependents();
  float acc[NT][8][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int l = 0; l < 8; ++l)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[i][l][c] = 0.f;
  const uint8_t *tile = act + (size_t)(m0 / 8) * nb * Q6M_TILE;
  // where the rows' blocks start inside 16 bytes
  const uint32_t a0 = (uint32_t)(reinterpret_cast<uintptr_t>(W) + (size_t)min(n0 + g, N - 1) * row_bytes),
                 a1 = (uint32_t)(reinterpret_cast<uintptr_t>(W) + (size_t)min(n0 + g + 8, N - 1) * row_bytes);
  bool ok = true;
  for (int un = 0; un < units; ++un) {
    const int b = SPLIT ? warp + un * EVERY : un;
    const bool here = mbar_wait_bounded(bar + 8 * (un % STAGES), (un / STAGES) & 1, abort_flag, &g_q6m_status, Q6M_POLLS, 2048);
    if constexpr (SPLIT) {
      ok = __all_sync(FULL, here) && ok; // without the data the chains have to pass all the same
      if (ok && un + STAGES - 1 < units)
        fetch(un + STAGES - 1);
    } else {
      if (!(ok = __all_sync(FULL, here)))
        break;
      if (un + STAGES - 1 < units) // into the slot that was read in the previous round
        fetch(un + STAGES - 1);
    }
    const uint32_t *st = stage_of(un % STAGES);
    uint32_t sh[2];
    const uint32_t *row[2];
    float d[NT][4];
    {
      float dw[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t at = ((r ? a1 : a0) + (uint32_t)b * (uint32_t)sizeof(BlockQ6K)) & 15;
        sh[r] = (at & 2) * 8;
        row[r] = st + (g + 8 * r) * Q6M_ROW_WORDS + (at >> 2);
        dw[r] = half_bits_to_float((uint16_t)(row[r][52] >> sh[r]));
      }
#pragma unroll
      for (int i = 0; i < NT; ++i)
        if (i < nt) {
          const float2 da = *reinterpret_cast<const float2 *>(tile + ((size_t)i * nb + b) * Q6M_TILE + 4096 + 8 * t);
#pragma unroll
          for (int c = 0; c < 4; ++c)
            d[i][c] = __fmul_rn((c & 1) ? da.y : da.x, dw[c >> 1]);
        }
    }
    uint4 x[NT]; // activations of the sum that comes next
    const uint4 *xp = reinterpret_cast<const uint4 *>(tile + (size_t)b * Q6M_TILE) + lane;
#pragma unroll
    for (int i = 0; i < NT; ++i)
      if (i < nt)
        x[i] = __ldg(xp + (size_t)i * nb * (Q6M_TILE / 16));
    uint32_t ql[2], qh[2], scales[2][2]; // word l of the lane's ql run and of its half's qh bytes, before the shift
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      ql[r] = row[r][8 * t];
      qh[r] = row[r][32 + 8 * h];
      const uint32_t w0 = row[r][48 + 2 * h], w1 = row[r][49 + 2 * h], w2 = row[r][50 + 2 * h];
      scales[r][0] = __funnelshift_r(w0, w1, sh[r]) >> (16 * run); // scale of quarter run: elements 0-15, 16-31
      scales[r][1] = __funnelshift_r(w1, w2, sh[r]) >> (16 * run);
    }
#pragma unroll
    for (int e = 0; e < 2; ++e) { // sums 0-3 and 4-7: the first and the second scale of every quarter
      __half2 s_lo[2][2], s_hi[2][2], o_lo[2][2], o_hi[2][2]; // [row][quarter]: sl / 4, 4 sh and -1056 times them
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          // the byte in both halves; its low nibble over 1024, its high nibble + 8 (sign bit flipped) over 64
          const uint32_t sc = __byte_perm(scales[r][k], 0, e ? 0x4141 : 0x4040);
          const float over = IN_PLACE && k ? 0.0625f : 1.f, offset = IN_PLACE && k ? -1536.f : -1056.f; // in place: values times 16
          s_lo[r][k] = __hfma2(u2h(lop3<LUT_AND_OR>(sc, 0x000f000fu, 0x64006400u)), __float2half2_rn(0.25f * over), __float2half2_rn(-256.f * over));
          s_hi[r][k] = __hfma2(u2h(lop3<LUT_AND_XOR>(sc, 0x00f000f0u, 0x54805480u)), __float2half2_rn(4.f * over), __float2half2_rn(-288.f * over));
          o_lo[r][k] = __hmul2(s_lo[r][k], __float2half2_rn(offset));
          o_hi[r][k] = __hmul2(s_hi[r][k], __float2half2_rn(offset));
        }
#pragma unroll
      for (int l4 = 0; l4 < 4; ++l4) {
        const int l = 4 * e + l4;
        uint32_t al[2][4], ah[2][4]; // fragments of the two quarters: times sl / 4, times 4 sh
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const uint32_t ql1 = row[r][8 * t + l + 1], qh1 = row[r][32 + 8 * h + l + 1];
          const uint32_t lw = __funnelshift_r(ql[r], ql1, sh[r]);
          // DENSE: bits 2 run and up of the word, so that the low quarter's lie four places lower than they are put
          const uint32_t hw = __funnelshift_r(qh[r], qh1, DENSE ? sh[r] + 2 * run : sh[r]);
          ql[r] = ql1;
          qh[r] = qh1;
          __half2 q0[2], q1[2]; // of the two quarters: bytes 0, 2 and 1, 3 as halves 1024 + q
          if (IN_PLACE) {      // (high nibbles: 1024 + 16 q)
            const uint32_t l8 = lw >> 8, u = hw << (4 - 2 * run), u8 = hw >> (4 + 2 * run);
            q0[0] = u2h(lop3<LUT_AND_OR>(lw, 0x000f000fu, lop3<LUT_AND_OR>(u, 0x00300030u, 0x64006400u)));
            q0[1] = u2h(lop3<LUT_AND_OR>(lw, 0x00f000f0u, lop3<LUT_AND_OR>(u, 0x03000300u, 0x64006400u)));
            q1[0] = u2h(lop3<LUT_AND_OR>(l8, 0x000f000fu, lop3<LUT_AND_OR>(u8, 0x00300030u, 0x64006400u)));
            q1[1] = u2h(lop3<LUT_AND_OR>(l8, 0x00f000f0u, lop3<LUT_AND_OR>(u8, 0x03000300u, 0x64006400u)));
          } else {
#pragma unroll
            for (int k = 0; k < 2; ++k) {
              // low nibbles of one word, above them the bits of the other (bits 6 and 7 of the bytes are masked off below)
              const uint32_t n = k ? lw >> 4 : lw, up = DENSE ? (k ? hw : hw << 4) : k ? hw >> (2 * run) : hw << (4 - 2 * run);
              const uint32_t q = lop3<LUT_SELECT>(n, up, 0x0f0f0f0fu);
              q0[k] = u2h(lop3<LUT_AND_OR>(q, 0x003f003fu, 0x64006400u));
              q1[k] = u2h(lop3<LUT_AND_OR>(q >> 8, 0x003f003fu, 0x64006400u));
            }
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            al[k][r] = h2u(__hfma2(q0[k], s_lo[r][k], o_lo[r][k]));
            al[k][r + 2] = h2u(__hfma2(q1[k], s_lo[r][k], o_lo[r][k]));
            ah[k][r] = h2u(__hfma2(q0[k], s_hi[r][k], o_hi[r][k]));
            ah[k][r + 2] = h2u(__hfma2(q1[k], s_hi[r][k], o_hi[r][k]));
          }
        }
#pragma unroll
        for (int i = 0; i < NT; ++i)
          if (i < nt) {
            const uint4 v = x[i];
            if (l < 7)
              x[i] = __ldg(xp + (size_t)i * nb * (Q6M_TILE / 16) + 32 * (l + 1));
            float p[4], p2[4]; // two short chains of MMAs instead of one of four; their sum is exact
            mma_f16_first(p, ah[0], v.x, v.y);
            mma_f16_first(p2, ah[1], v.z, v.w);
            mma_f16(p, al[0], v.x, v.y);
            mma_f16(p2, al[1], v.z, v.w);
#pragma unroll
            for (int c = 0; c < 4; c += 2) {
              const float2 sum = add2(p[c], p[c + 1], p2[c], p2[c + 1]);
              if constexpr (SPLIT)
                acc[i][l][c] = sum.x, acc[i][l][c + 1] = sum.y;
              else
                fma2(acc[i][l][c], acc[i][l][c + 1], d[i][c], d[i][c + 1], sum.x, sum.y);
            }
          }
      }
    }
    if constexpr (SPLIT) { // take the chains over, add this super-block, pass them on
      float4 *const chains = reinterpret_cast<float4 *>(split_smem + WARPS * STAGES * Q6M_STAGE_WORDS) + lane;
      const int from = warp, to = warp + 1 < WARPS ? warp + 1 : 0;
      if (b > 0)
        pair_sync(1 + from);
#pragma unroll
      for (int l = 0; l < 8; ++l) {
        float4 f = b > 0 ? chains[(from * 8 + l) * 32] : make_float4(0.f, 0.f, 0.f, 0.f);
        fma2(f.x, f.y, d[0][0], d[0][1], acc[0][l][0], acc[0][l][1]);
        fma2(f.z, f.w, d[0][2], d[0][3], acc[0][l][2], acc[0][l][3]);
        if (b + 1 < nb)
          chains[(to * 8 + l) * 32] = f;
        acc[0][l][0] = f.x, acc[0][l][1] = f.y, acc[0][l][2] = f.z, acc[0][l][3] = f.w;
      }
      if (b + 1 < nb)
        pair_arrive(1 + to);
    }
    __syncwarp(); // the slot is refilled in the next round
  }
  if (!ok) { // a wait ran out: give the copies in flight time to land in this CTA's shared memory
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
    return;
  }
  if (SPLIT && (warp != (nb - 1) % WARPS || !nobody_gave_up(ok, abort_flag))) // the chains end in the last super-block's warp
    return;
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int m = m0 + 8 * i + 2 * t + (c & 1), n = n0 + g + 8 * (c >> 1);
      if (m < M && n < N) {
        const float(&a)[8][4] = acc[i];
        C[(size_t)m * ldc + n] =
          __fadd_rn(__fadd_rn(__fadd_rn(a[4][c], a[0][c]), __fadd_rn(a[6][c], a[2][c])),
                    __fadd_rn(__fadd_rn(a[5][c], a[1][c]), __fadd_rn(a[7][c], a[3][c])));
      }
    }
}

/** fp32 rows -> the activation tiles above; one warp per (row, super-block). */
__global__ void __launch_bounds__(256)
act_tiles_q6_kernel(const float *__restrict__ x, int64_t ldx, uint8_t *__restrict__ act, int M, int nb) {
  pdl_wait();
  pdl_launch_dependents(); // the GEMM behind fetches weights, which a kernel in front of this one may have written, and waits for the rest
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (w >= (int64_t)M * nb)
    return;
  const int m = (int)(w / nb), b = (int)(w - (int64_t)m * nb), g = m & 7;
  const float *src = x + (int64_t)m * ldx + (int64_t)b * QK_K + lane * 8;
  const Q8KLane q = q8K_quantize_warp(*reinterpret_cast<const float4 *>(src), *reinterpret_cast<const float4 *>(src + 4), lane,
                                      0); // ggml_interface_omp.cpp:545-551: the row quantizer for all rows
  uint8_t *tile = act + ((size_t)(m >> 3) * nb + b) * Q6M_TILE;
  // elements 8 lane .. +7: half lane / 16, quarter (lane / 4) % 4, sums 2 (lane % 4) and the next
  const int t = 2 * (lane >> 4) + ((lane >> 2) & 1), k = (lane >> 3) & 1, l = 2 * (lane & 3);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const uint32_t v = e ? q.w1 : q.w0;
    const __half2 p0 = __floats2half2_rn((float)(4 * (int)(int8_t)v), (float)(4 * (int)(int8_t)(v >> 16))),
                  p1 = __floats2half2_rn((float)(4 * (int)(int8_t)(v >> 8)), (float)(4 * (int)(int8_t)(v >> 24)));
    *reinterpret_cast<uint2 *>(tile + (l + e) * 512 + (4 * g + t) * 16 + k * 8) = make_uint2(h2u(p0), h2u(p1));
  }
  if (lane == 0)
    *reinterpret_cast<float *>(tile + 4096 + 4 * g) = q.d;
}

} // namespace

size_t gemm_mma_q6_K_workspace_bytes(unsigned M, unsigned K) { return (size_t)((M + 7) / 8) * (K / QK_K) * Q6M_TILE; }

int launch_gemm_mma_q6_K(unsigned M, unsigned N, unsigned K, const float *A, const void *B, float *C, unsigned ldc, void *ws,
                         cudaStream_t st) {
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(ws) & 15) || (reinterpret_cast<uintptr_t>(B) & 1))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm_q6_K: misaligned pointer");
  const int nb = (int)(K / QK_K);
  NNTR_CHECK_CUDA(launch_in_clusters(act_tiles_q6_kernel, dim3((unsigned)(((int64_t)M * nb + 7) / 8)), 1, 256, 0, st, A, (int64_t)K,
                                     static_cast<uint8_t *>(ws), (int)M, nb));
  count_launch();
  const unsigned row_tiles = (N + 15) / 16, sms = (unsigned)sm_count();
  // A wave of shared tiles (two CTAs per SM) takes about 3.5 us and 0.45 for each super-block of K; a warp on its own 2 us for each,
  // however few they are, 3.2 with two tiles of rows. One tile, shared / not: 8 x 4736 x 2560 (1 wave) 9.5 / 18.5 us, 9472 rows (2) 16.8 / 20.1,
  // 14208 (3) 23.8 / 20.1; 14208 x 8192 53.5 / 62.0, 18944 x 8192 (4) 71.6 / 74.9. More rows: 31 x 1024 x 2560 9.3 / 33.9, 31 x 4096 x 4096 (4)
  // 38.5 / 49.7, 24 x 6144 x 2560 (4) 30.1 / 32.7, 300 x 1000 x 2560 (9) 62 / 38.
  const uint64_t waves = ((uint64_t)row_tiles * ((M + 7) / 8) + 2 * sms - 1) / (2 * sms);
  const bool split = nb > 1 && waves * (8 + nb) <= (M <= 8 ? 4u : 7u) * nb;
  const unsigned nt = split || M <= 8 ? 1 : 2;
  const dim3 grid((M + 8 * nt - 1) / (8 * nt), split ? row_tiles : (row_tiles + Q6M_WARPS - 1) / Q6M_WARPS);
  // One tile of rows: four CTAs per SM where that saves a round, each of which takes them about a fifth longer. Three / four CTAs, 8 rows: 37072 x
  // 2560 (580 CTAs, two rounds / one) 41.4 / 30.7 us, 40912 x 2560 (640: two / two) 42.2 / 44.6, 56272 x 4096 (880: two / two) 76.3 / 91.8, x
  // 8192 150 / 195, 61392 x 2560 (960: three / two) 61.6 / 54.6, 83152 x 4096 (1300: three / three) 111.5 / 124.3, 151936 x 2560 (six / five) 128.2 /
  // 122.5; 64 CTAs, 5 x 4096 x 4096, 30.0 / 36.9.
  const unsigned ctas = grid.x * grid.y;
  const bool dense = nt == 1 && (ctas + 4 * sms - 1) / (4 * sms) < (ctas + 3 * sms - 1) / (3 * sms);
  const auto kernel = split     ? gemm_q6_K_mma_kernel<1, 2, true>
                      : dense   ? gemm_q6_K_mma_kernel<1, 4, false>
                      : nt == 1 ? gemm_q6_K_mma_kernel<1, 3, false>
                                : gemm_q6_K_mma_kernel<2, 3, false>;
  if (split) {
    static std::atomic<uint64_t> done{0}; // a bit per device
    int dev = 0;
    NNTR_CHECK_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !(done.load(std::memory_order_acquire) >> dev & 1)) {
      NNTR_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Q6S_SMEM));
      if (dev < 64)
        done.fetch_or(1ull << dev, std::memory_order_release);
    }
  }
  const cudaError_t e = launch_in_clusters(kernel, grid, 1, (split ? Q6S_WARPS : Q6M_WARPS) * 32, split ? Q6S_SMEM : 0, st,
                                           static_cast<const uint8_t *>(ws), static_cast<const uint8_t *>(B), C, (int)ldc,
                                           (int)M, (int)N, nb);
  count_launch();
  return check_cuda(e, "gemm_q6_K launch");
}

int read_q6m_status(int *out) {
  int v = 0;
  NNTR_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_q6m_status, sizeof(int)));
  *out = v;
  return NNTR_CUDA_OK;
}
int clear_q6m_status() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_q6m_status, &zero, sizeof(int)), "clear_q6m_status");
}

} // namespace nntr
