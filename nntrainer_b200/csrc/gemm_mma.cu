// SPDX-License-Identifier: Apache-2.0
/**
 * @file  gemm_mma.cu
 * @brief Bit-exact GEMM for Q4_K and Q4_0 weights with more than one activation row, dense and grouped by expert:
 *        integer warp MMAs on fragments that are unpacked in registers, the reference's float chains in registers.
 *
 * They reproduce the reference's per-output float chains exactly:
 *   Q4_K  rows below 4*floor(M/4): four fused multiply-adds per super-block, one per pair of sub-blocks
 *         (nntr_gemm_q4_K_8x8_q8_K, nntr_ggml_impl.cpp:6284-6984); the last M%4 rows and every row of a grouped call: one
 *         per super-block (nntr_gemv_q4_K_8x8_q8_K, :7405-7422).
 *   Q4_0  one fused multiply-add per 32-block (:9751-9753), same for both.
 * Those chains leave the integer domain once per 64, 256 or 32 of K, so an accumulator that lives in tensor memory would
 * be drained that often. The warp MMA m16n8k32 leaves its sums in registers instead, one sub-block per instruction, and
 * its A fragment is what one 8-byte (Q4_K) or 4-byte (Q4_0) piece of the interleaved weight block holds: the low and the
 * high nibbles of 4 bytes each, a mask and at most a shift per fragment register.
 *
 * A sub-block's sum and its 6-bit scale meet as integers (|I| <= 15 * 127 * 32, sc <= 63): a pair of sub-blocks stays below
 * 2^23, which fp32 holds, a super-block below 2^25, whose one conversion rounds as the reference's does. The sums of the mins
 * term come from one fp16 MMA of [min, 32 min] with the sums of 32 activations split into [sum & 31, sum >> 5], all of them
 * integers fp16 holds. Float steps go two at a time (fma.rn.f32x2), each rounded as by itself.
 *
 * Two splits of the work:
 *   gemm_mma_rows_kernel   a warp owns 16 weight rows and up to 32 activation rows over all of K; the CTA's four warps share
 *                          the unit's activation tiles and weights, which a fifth warp brings into a ring by bulk copies. CTAs
 *                          stay and go through items of 64 weight rows. Bound by instruction issue, shared memory and half-rate
 *                          operations alike: per 16 x 8 x 32 of Q4_0 about 20 instructions, 4 wavefronts of shared memory, 8 half-rate
 *                          operations, four to five clocks of an SM each, seven taken. Q4_0 1000 x 8000 x 4096 208 us (a
 *                          computing thread starting the copies, 25 instructions: 303), 509 x 2880 x 2880 36.9 us (51.6); Q4_K
 *                          255 x 9728 x 2560 77.8 us, on the one-step chain of gemv_rows 55.7 (87.8 and 75.5).
 *   gemm_mma_ksplit_kernel eight warps share the tile and take every eighth unit of 256 along K; the float chains go from warp
 *                          to warp, one unit further at each. For the others: bound by that hand-over (270 clocks a unit) when
 *                          K is long, by launch and round trips when it is short. With the quantizer's launch: Q4_K 8 x 2560 x 2560
 *                          5.9 us, 8 x 2560 x 9728 12.0 us (terms through shared memory to one thread per chain: 8.5 and 18.6).
 */
#include <type_traits>

#include "act_tiles.cuh"
#include "common.cuh"
#include "pipeline.cuh"

namespace nntr {

namespace {

struct MmaArgs {
  const uint8_t *act;
  const void *W;
  float *C;
  int ldc;
  int M, M4;    // activation rows; rows below M4 take the four-step chain of Q4_K
  int N, nb;    // weight rows, units of 256 (the last one of Q4_0 may be short)
  int nblk;     // Q4_0: 32-blocks of a row
  int th;       // rows per activation tile: 8, or the rows there are if the caller's scratch has no room for 8
  /* grouped (see launch_gemm_grouped) */
  const void *const *w_table[2];
  const int *off, *tile_off, *act_off, *perm;
  int n_experts, c_mul;
};

__device__ __forceinline__ void mma_u8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_s8s8(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
  asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void mma_f16_k8(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%7,%7};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(b0), "f"(0.f));
}
__device__ __forceinline__ void mma_f16_k16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
               : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}

__device__ __forceinline__ uint32_t h2_bits(__half2 h) { return *reinterpret_cast<const uint32_t *>(&h); }
__device__ __forceinline__ __half2 bits_h2(uint32_t u) { return *reinterpret_cast<const __half2 *>(&u); }
/** (v, 32 v) of byte K of four 6-bit values as half2; 0x64vv is 1024 + v */
template <int K> __device__ __forceinline__ uint32_t min_halves(uint32_t v) {
  return h2_bits(__hfma2(bits_h2(__byte_perm(v, 0x64646464u, 0x4040 | (K * 0x101))), __floats2half2_rn(1.f, 32.f),
                         __floats2half2_rn(-1024.f, -32768.f)));
}
/** (lo, hi - 128) of one 16-bit half K of an activation row's word as half2 */
template <int K> __device__ __forceinline__ uint32_t sum_halves(uint32_t w) {
  return h2_bits(__hsub2(bits_h2(__byte_perm(w, 0x64646464u, K ? 0x4342 : 0x4140)), __floats2half2_rn(1024.f, 1152.f)));
}

/* ------------------------------------------------------------------ Q4_K */
/** What the MMAs and chains need besides the nibbles. */
struct Q4KScales {
  uint32_t sc[4];  // gathered from the quad: word t' = scales of sub-blocks t' and t' + 4 of row g (bytes 0, 1), row g + 8 (2, 3)
  uint32_t mn[4];  // A fragment of the mins: [row g, t], [row g + 8, t], [row g, t + 4], [row g + 8, t + 4]
  float dw[2], dm[2];
};
__device__ __forceinline__ void q4k_scales(Q4KScales &s, const uint32_t (&head)[2][2][3], const uint32_t (&d)[2], int g, int lane) {
  // the bytes of this lane's rows out of the three words of a group, four (row, sub-block) at a time: word i -> x[i]
  uint32_t x[3];
  const uint32_t two = (g & 3) * 0x11 + 0x40; // byte g % 4 of either operand
#pragma unroll
  for (int i = 0; i < 3; ++i)
    x[i] = __byte_perm(__byte_perm(head[0][0][i], head[0][1][i], two), __byte_perm(head[1][0][i], head[1][1][i], two), 0x5410);
  // rows 0 - 3 of a group: the low six bits of words 0 (scale) and 1 (min); rows 4 - 7: a nibble of word 2 under their top bits
  const uint32_t low = g < 4 ? 0x3f3f3f3fu : 0u, nib = g < 4 ? 0u : 0x0f0f0f0fu, top = g < 4 ? 0u : 0x30303030u;
  const uint32_t own = (x[0] & low) | ((x[2] & nib) | ((x[0] >> 2) & top));
  const uint32_t mins = (x[1] & low) | (((x[2] >> 4) & nib) | ((x[1] >> 2) & top));
  s.mn[0] = min_halves<0>(mins);
  s.mn[1] = min_halves<2>(mins);
  s.mn[2] = min_halves<1>(mins);
  s.mn[3] = min_halves<3>(mins);
#pragma unroll
  for (int i = 0; i < 4; ++i)
    s.sc[i] = __shfl_sync(FULL, own, (lane & ~3) + i);
#pragma unroll
  for (int row = 0; row < 2; ++row) {
    s.dw[row] = half_bits_to_float((uint16_t)d[row]);
    s.dm[row] = half_bits_to_float((uint16_t)(d[row] >> 16));
  }
}
/** the same from blocks in shared memory */
__device__ __forceinline__ void q4k_scales(Q4KScales &s, const BlockQ4Kx8 *lo, const BlockQ4Kx8 *hi, int g, int t, int lane) {
  uint32_t head[2][2][3], d[2];
#pragma unroll
  for (int row = 0; row < 2; ++row) {
    const BlockQ4Kx8 *b = row ? hi : lo;
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        head[row][k][i] = *(reinterpret_cast<const uint32_t *>(b->scales + 12 * (t + 4 * k)) + i);
    d[row] = (uint32_t)b->d[g] | ((uint32_t)b->dmin[g] << 16);
  }
  q4k_scales(s, head, d, g, lane);
}
/** scale of sub-block J of row g + 8 * row */
template <int J> __device__ __forceinline__ int q4k_scale_int(const Q4KScales &s, int row) {
  return (int)__byte_perm(s.sc[J & 3], 0, 0x4440 | ((J >> 2) + 2 * row));
}

/** One lane's view of a tile's unit. TH8: the tile is laid out for 8 rows. */
struct ActQ4K {
  uint4 b[4];
  uint32_t sums;
  float2 d; // rows 2t, 2t + 1
};
template <bool TH8> __device__ __forceinline__ uint4 act_frag(const uint8_t *unit, int p, int th, int lane) {
  if (TH8)
    return *reinterpret_cast<const uint4 *>(unit + p * 512 + lane * 16);
  return lane < 4 * th ? *reinterpret_cast<const uint4 *>(unit + p * (64 * th) + lane * 16) : make_uint4(0, 0, 0, 0);
}
template <bool TH8> __device__ __forceinline__ uint32_t act_sums(const uint8_t *unit, int th, int lane) {
  if (TH8)
    return *reinterpret_cast<const uint32_t *>(unit + 260 * 8 + lane * 4);
  return lane < 4 * th ? *reinterpret_cast<const uint32_t *>(unit + 260 * th + lane * 4) : 0u;
}
template <bool TH8> __device__ __forceinline__ float2 act_d(const uint8_t *unit, int th, int t) {
  return *reinterpret_cast<const float2 *>(unit + 256 * (TH8 ? 8 : th) + 8 * t); // rows at or beyond th: other bytes of the unit
}
template <bool TH8> __device__ __forceinline__ void act_load(ActQ4K &a, const uint8_t *unit, int th, int lane) {
#pragma unroll
  for (int p = 0; p < 4; ++p)
    a.b[p] = act_frag<TH8>(unit, p, th, lane);
  a.sums = act_sums<TH8>(unit, th, lane);
  a.d = act_d<TH8>(unit, th, lane & 3);
}

/* ------------------------------------------------------------------ Q4_0 */
struct ActQ40 {
  uint4 b[4];
  uint2 d[4]; // scales of the 32-blocks 2p, 2p + 1 of the rows 2t and 2t + 1
};
__device__ __forceinline__ uint2 act_d2(const uint8_t *unit, int p, int t) {
  return *reinterpret_cast<const uint2 *>(unit + 256 * 8 + 32 * p + 8 * t);
}
template <bool TH8> __device__ __forceinline__ void act_load(ActQ40 &a, const uint8_t *unit, int, int lane) {
  static_assert(TH8, "only Q4_K has a call with short tiles");
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    a.b[p] = act_frag<true>(unit, p, 8, lane);
    a.d[p] = act_d2(unit, p, lane & 3);
  }
}
/** a * b of two halves, exact in fp32: the instruction that multiplies halves into a float adds -0 */
__device__ __forceinline__ float mul_halves(uint16_t a, uint16_t b) {
  float d;
  asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(a), "h"(b), "f"(-0.f));
  return d;
}
/* A block of a 16 x 8 tile. The stored nibble (q ^ 8) is q - 8 in two's complement, so in the upper half of a byte it is that
 * times 16, and everything that follows is taken times 16 too, down to the result, which is exact: the scales are halves, so a chain's
 * values are multiples of 2^-48 and stay below 2^60 wherever they are numbers. */
/** x: the sums times 16, s: the products of the scales; q: low nibbles of rows g, g + 8, high nibbles of them, in the upper halves of
 *  the bytes; dw0, dw1: scales of the two rows; da: act_d2 of the pair of blocks of which this is number J */
template <int J>
__device__ __forceinline__ void q40_terms(float (&x)[4], float (&s)[4], const uint32_t (&q)[4], uint32_t b0, uint32_t b1, uint16_t dw0,
                                          uint16_t dw1, uint2 da) {
  int v[4];
  mma_s8s8(v, q[0], q[1], q[2], q[3], b0, b1);
  const uint16_t d0 = (uint16_t)(da.x >> (16 * J)), d1 = (uint16_t)(da.y >> (16 * J));
  s[0] = mul_halves(dw0, d0), s[1] = mul_halves(dw0, d1), s[2] = mul_halves(dw1, d0), s[3] = mul_halves(dw1, d1);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    x[c] = (float)v[c];
}

/* ------------------------------------------------------- where a tile lies */
/** Activation rows of one CTA: `rows` of them, outputs from position `pos`, tiles from act_k on of the act_tiles that start at
 *  act_first; weights W. */
struct Tile {
  const void *W;
  int pos, rows, act_first, act_tiles, act_k, z;
};
template <int NT> __device__ __forceinline__ bool find_tile(Tile &tl, const MmaArgs &a, int tile, bool grouped) {
  if (!grouped) {
    tl.W = a.W;
    tl.pos = tile * 8 * NT;
    tl.act_first = 0;
    tl.act_tiles = (a.M + a.th - 1) / a.th;
    tl.act_k = tile * NT;
    tl.rows = min(8 * NT, a.M - tl.pos);
    return true;
  }
  // the expert whose tiles of 8 * NT rows hold this one: the last one that starts at or before it. All offsets are loaded at
  // once (one round trip; a binary search is a chain of five to eight, a third of a small CTA's life).
  const int lane = threadIdx.x & 31, end = a.tile_off[a.n_experts];
  int lo = -1;
#pragma unroll
  for (int i = 0; i < 8; ++i) { // at most 256 experts
    const int x = 32 * i + lane;
    lo += __popc(__ballot_sync(FULL, x < a.n_experts && a.tile_off[x < a.n_experts ? x : 0] <= tile));
  }
  if (tile >= end)
    return false;
  const int k = tile - a.tile_off[lo], first = k * 8 * NT;
  tl.W = (tl.z ? a.w_table[1] : a.w_table[0])[lo];
  tl.pos = a.off[lo] + first;
  const int all = a.off[lo + 1] - a.off[lo];
  tl.act_first = a.act_off[lo];
  tl.act_tiles = (all + 7) >> 3;
  tl.act_k = k * NT;
  tl.rows = min(8 * NT, all - first);
  return tl.rows > 0 && tl.W; // a null weight: expert of another rank
}
__device__ __forceinline__ float *out_row(const MmaArgs &a, const Tile &tl, int i, bool grouped) {
  const int row = grouped ? a.perm[tl.pos + i] * a.c_mul + tl.z : tl.pos + i;
  return a.C + (size_t)row * a.ldc;
}

/** One unit of a warp's 16 rows against up to 8 * NT activation rows in shared memory, chains in registers. The pair of
 *  sub-blocks is the outer loop, so that its fragments and factors are unpacked once for all tiles.
 *  CHAIN_FOUR: four steps per super-block; CHAIN_ONE: one; CHAIN_MIXED: four for the rows below m4 of the tile, one behind.
 *  Scales meet the sums as integers: |sc * I| summed over a super-block stays below 2^25, and its one conversion rounds as the
 *  reference's does. */
enum { CHAIN_FOUR, CHAIN_ONE, CHAIN_MIXED };
template <int N_TILES, int CHAIN, bool TH8, int NT>
__device__ __forceinline__ void q4k_unit(float (&acc)[NT][4], float (&accm)[NT][4], const Q4KScales &sc, const BlockQ4Kx8 *w0,
                                         const BlockQ4Kx8 *w1, const uint8_t *act, int th, int m4, int g, int t,
                                         int lane) {
  int sum[N_TILES][4];                  // one-step rows: of the super-block so far
  float2 s1[N_TILES][2], s2[N_TILES][2]; // four-step rows: d * da and dmin * da of the rows 2t, 2t + 1
  uint32_t bs[N_TILES][2];
#pragma unroll
  for (int i = 0; i < N_TILES; ++i) {
    const uint8_t *unit = act + i * (8 * act_row_bytes(NNTR_Q4_K));
    if (CHAIN != CHAIN_ONE) {
      const uint32_t sums = act_sums<TH8>(unit, th, lane);
      bs[i][0] = sum_halves<0>(sums);
      bs[i][1] = sum_halves<1>(sums);
      const float2 d = act_d<TH8>(unit, th, t);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        s1[i][r] = mul2(sc.dw[r], sc.dw[r], d.x, d.y);
        s2[i][r] = mul2(sc.dm[r], sc.dm[r], d.x, d.y);
      }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
      sum[i][c] = 0;
  }
  auto pair = [&](auto P) {
    constexpr int p = decltype(P)::value;
    const uint2 q0 = *reinterpret_cast<const uint2 *>(w0->qs + ((4 * p + t) * 8 + g) * 8),
                q1 = *reinterpret_cast<const uint2 *>(w1->qs + ((4 * p + t) * 8 + g) * 8);
    const uint32_t lo[4] = {q0.x & 0x0f0f0f0fu, q1.x & 0x0f0f0f0fu, q0.y & 0x0f0f0f0fu, q1.y & 0x0f0f0f0fu};
    const uint32_t hi[4] = {(q0.x >> 4) & 0x0f0f0f0fu, (q1.x >> 4) & 0x0f0f0f0fu, (q0.y >> 4) & 0x0f0f0f0fu,
                            (q1.y >> 4) & 0x0f0f0f0fu};
    const int f0[2] = {q4k_scale_int<2 * p>(sc, 0), q4k_scale_int<2 * p>(sc, 1)},
              f1[2] = {q4k_scale_int<2 * p + 1>(sc, 0), q4k_scale_int<2 * p + 1>(sc, 1)};
    const bool own = (t >> 1) == (p & 1); // the lanes that hold the mins of this pair
    const uint32_t m0 = own ? sc.mn[2 * (p >> 1)] : 0u, m1 = own ? sc.mn[2 * (p >> 1) + 1] : 0u;
#pragma unroll
    for (int i = 0; i < N_TILES; ++i) {
      const uint4 x = act_frag<TH8>(act + i * (8 * act_row_bytes(NNTR_Q4_K)), p, th, lane);
      int lo_sum[4], hi_sum[4];
      mma_u8s8(lo_sum, lo[0], lo[1], lo[2], lo[3], x.x, x.y);
      mma_u8s8(hi_sum, hi[0], hi[1], hi[2], hi[3], x.z, x.w);
      if (CHAIN == CHAIN_ONE) {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          sum[i][c] += f0[c >> 1] * lo_sum[c] + f1[c >> 1] * hi_sum[c];
        continue;
      }
      int v[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        v[c] = f0[c >> 1] * lo_sum[c] + f1[c >> 1] * hi_sum[c]; // below 2^23: exact as a float
      float j[4];
      mma_f16_k8(j, m0, m1, bs[i][p >> 1]);
      if (CHAIN == CHAIN_FOUR) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          fma2(acc[i][2 * r], acc[i][2 * r + 1], (float)v[2 * r], (float)v[2 * r + 1], s1[i][r].x, s1[i][r].y);
          fma2(accm[i][2 * r], accm[i][2 * r + 1], j[2 * r], j[2 * r + 1], s2[i][r].x, s2[i][r].y);
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (8 * i + 2 * t + (c & 1) < m4) {
            acc[i][c] = __fmaf_rn((float)v[c], (c & 1) ? s1[i][c >> 1].y : s1[i][c >> 1].x, acc[i][c]);
            accm[i][c] = __fmaf_rn(j[c], (c & 1) ? s2[i][c >> 1].y : s2[i][c >> 1].x, accm[i][c]);
          }
          sum[i][c] += v[c];
        }
      }
    }
  };
  pair(std::integral_constant<int, 0>{});
  pair(std::integral_constant<int, 1>{});
  pair(std::integral_constant<int, 2>{});
  pair(std::integral_constant<int, 3>{});
  if (CHAIN != CHAIN_FOUR) {
#pragma unroll
    for (int i = 0; i < N_TILES; ++i) {
      const uint8_t *unit = act + i * (8 * act_row_bytes(NNTR_Q4_K));
      const uint32_t sums = act_sums<TH8>(unit, th, lane);
      const float2 d = act_d<TH8>(unit, th, t);
      float j[4];
      mma_f16_k16(j, sc.mn[0], sc.mn[1], sc.mn[2], sc.mn[3], sum_halves<0>(sums), sum_halves<1>(sums));
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const float2 e1 = mul2(sc.dw[r], sc.dw[r], d.x, d.y), e2 = mul2(sc.dm[r], sc.dm[r], d.x, d.y);
        if (CHAIN == CHAIN_ONE) { // one rounding of the exact sum of the super-block
          fma2(acc[i][2 * r], acc[i][2 * r + 1], __int2float_rn(sum[i][2 * r]), __int2float_rn(sum[i][2 * r + 1]), e1.x, e1.y);
          fma2(accm[i][2 * r], accm[i][2 * r + 1], j[2 * r], j[2 * r + 1], e2.x, e2.y);
        } else {
#pragma unroll
          for (int k = 0; k < 2; ++k)
            if (8 * i + 2 * t + k >= m4) {
              const int c = 2 * r + k;
              acc[i][c] = __fmaf_rn(__int2float_rn(sum[i][c]), k ? e1.y : e1.x, acc[i][c]);
              accm[i][c] = __fmaf_rn(j[c], k ? e2.y : e2.x, accm[i][c]);
            }
        }
      }
    }
  }
}

/** Q4_0: the n blocks of a unit, two at a time. FULL: n is 8, no branches between them. */
template <int N_TILES, bool FULL, int NT>
__device__ __forceinline__ void q40_unit(float (&acc)[NT][4], const BlockQ40x8 *w0, const BlockQ40x8 *w1, const uint8_t *act,
                                         int n, int g, int t, int lane) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    if (!FULL && 2 * p >= n)
      break;
    uint32_t q[2][4];
    uint16_t dw[2][2];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int row = 0; row < 2; ++row) {
        // a block past the end of the row: what the shared memory holds, with scale 0
        const BlockQ40x8 *blk = (row ? w1 : w0) + 2 * p + j;
        const uint32_t w = *reinterpret_cast<const uint32_t *>(blk->qs + (t >> 1) * 64 + g * 8 + (t & 1) * 4);
        q[j][row] = (w << 4) & 0xf0f0f0f0u;
        q[j][row + 2] = w & 0xf0f0f0f0u;
        dw[j][row] = FULL || 2 * p + j < n ? blk->d[g] : (uint16_t)0;
      }
#pragma unroll
    for (int i = 0; i < N_TILES; ++i) {
      const uint8_t *unit = act + i * (8 * act_row_bytes(NNTR_Q4_0));
      const uint4 x = act_frag<true>(unit, p, 8, lane);
      const uint2 da = act_d2(unit, p, t);
      auto block = [&](auto J) {
        constexpr int j = decltype(J)::value;
        float v[4], s[4];
        q40_terms<j>(v, s, q[j], j ? x.z : x.x, j ? x.w : x.y, dw[j][0], dw[j][1], da);
#pragma unroll
        for (int r = 0; r < 2; ++r)
          fma2(acc[i][2 * r], acc[i][2 * r + 1], v[2 * r], v[2 * r + 1], s[2 * r], s[2 * r + 1]);
      };
      block(std::integral_constant<int, 0>{});
      block(std::integral_constant<int, 1>{});
    }
  }
}

/** f(integral_constant<1 .. NT>) for n tiles: the loops over tiles are then free of branches */
template <int NT, typename F> __device__ __forceinline__ void with_tiles(int n, F f) {
  if constexpr (NT > 1)
    if (n < NT)
      return with_tiles<NT - 1>(n, f);
  f(std::integral_constant<int, NT>{});
}

/* --------------------------------------------------- a warp owns its rows */
constexpr int ROWS_WARPS = 4;                                    // that compute; a fifth one brings the data in
constexpr int ROWS_W = ROWS_WARPS * 2 * (int)sizeof(BlockQ4Kx8); // the weights of a unit: 8 row groups (Q4_0: 8 blocks of 144)

__device__ int g_mma_status = 0;

/* Units in flight per CTA and the CTAs per SM that registers and shared memory are held to. More warps hide more latency until
 * registers spill by much or the ring gets too short; measured with 2 to 5 stages and 2 to 9 CTAs. Q4_0 1000 x 8000 x 4096 with 3 / 4 / 5
 * CTAs of 32 rows 226 / 201 / 230 us; Q4_K (12 of 16 warps' worth of registers) 31 x 24576 x 4096 with 3 / 4: 51 / 70; 16 rows, 16 x 24576
 * x 4096 with 3 / 4: 23 / 28. The third CTA of Q4_K's 32 rows costs 120 bytes of spills and pays for them: with 2 CTAs and none
 * 31 x 24576 x 4096 60.5 us instead of 48.1, 255 x 9728 x 2560 85.8 instead of 77.2.
 * Q4_0 tiles of 8 rows per expert: as many as the kernel's 55 registers allow, seven. Which number wins at one batch size depends on
 * how the last round fills, so over sizes: 4 of 32 experts of 2880 x 2880, 17 batches of 5 to 48 tokens, 4 of 32 of 1024 x 1440 (9), 2 of
 * 16 of 4096 x 4096 (6), 4 of 64 of 1024 x 2880 (8 batches, 5 to 96): six take 1.008 / 1.009 / 0.995 / 0.974 times as long as seven in the
 * geometric mean, eight 1.046 / 1.001 / 1.036 / 0.982; single batches differ by up to 15 % either way (8 tokens of the first layer
 * with 6 / 7 / 8: 94.9 / 88.8 / 97.1 us, 16 tokens 113 / 122 / 124, 24 tokens of the third 131 / 118 / 129). */
template <int QT, int NT, bool GROUPED> constexpr int rows_stages() { return QT == NNTR_Q4_0 && NT == 1 && GROUPED ? 2 : 3; }
template <int QT, int NT, bool GROUPED> constexpr int rows_ctas() {
  return QT == NNTR_Q4_0 ? (NT >= 2 ? 4 : GROUPED ? 7 : 5) : (NT == 4 ? 3 : NT == 2 ? 3 + GROUPED : 4);
}

/** Up to 64 weight rows, `groups` row groups from group0 on, against the rows of a Tile; with every unit of 256 of K in the ring. */
struct RowsItem {
  Tile tl; // rows == 0: no more units
  int group0, groups, b;
};
template <int NT, int STAGES> struct RowsShared {
  alignas(16) uint8_t w[STAGES][ROWS_W];
  alignas(16) uint8_t act[STAGES][NT * 8 * act_row_bytes(NNTR_Q4_K)];
  alignas(8) unsigned long long full[STAGES], empty[STAGES];
  RowsItem item[STAGES];
  int abort_flag;
};

template <int QT, int NT, bool GROUPED, bool TH8, int STAGES>
__global__ void __launch_bounds__(ROWS_WARPS * 32 + 32, rows_ctas<QT, NT, GROUPED>()) gemm_mma_rows_kernel(const MmaArgs a, int n_tiles, int n_z) {
  extern __shared__ __align__(16) uint8_t rows_smem[];
  RowsShared<NT, STAGES> &sh = *reinterpret_cast<RowsShared<NT, STAGES> *>(rows_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int n_groups = a.N / 8, nb = a.nb;
  const int th = TH8 ? 8 : a.th;
  volatile int *abort_flag = &sh.abort_flag;
  const uint32_t full0 = smem_u32(sh.full), empty0 = smem_u32(sh.empty);
  if (tid == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(full0 + 8 * s, 1);
      mbar_init(empty0 + 8 * s, ROWS_WARPS);
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (GROUPED)
    pdl_wait(); // tables and activation tiles come from the kernels before
  else if (NT > 2 || (n_groups + 2 * ROWS_WARPS - 1) / (2 * ROWS_WARPS) * n_tiles * n_z > (int)gridDim.x)
    // The next launch's CTAs are let in beside the products. Up to 16 rows and no CTA with a second item: not, 5 x 24576 x 4096 Q4_K 24.4 us,
    // so 20.9, 8 x 24576 x 4096 Q4_0 18.5 and 17.1; more rows: 31 x 20000 x 4096 Q4_0 26.4 us, without 31.9, 40 x 9728 x 2560 Q4_K 21.7 and 23.7.
    // (Grouped: 64 tokens, 8 of 128 experts 113 -> 132 us.)
    pdl_launch_dependents();
  int slot = 0;
  uint32_t par = 0;
  bool ok = true;
  auto next_slot = [&]() {
    if (++slot == STAGES)
      slot = 0, par ^= 1;
  };
  auto wait = [&](uint32_t bar, uint32_t parity) {
    if (!__all_sync(FULL, mbar_try_wait(bar + 8 * slot, parity)))
      ok = __all_sync(FULL, mbar_wait_bounded(bar + 8 * slot, parity, abort_flag, &g_mma_status, 1u << 22, 2048));
    return ok;
  };
  if (warp == ROWS_WARPS) {
    /* ---- A warp brings the units of all items in, a lane per copy. A bulk copy holds its warp for 50 ns, so the nine of a unit are
     * kept away from the warps that compute. */
    if (GROUPED)
      n_tiles = a.tile_off[a.n_experts];
    const int row_blocks = (n_groups + 2 * ROWS_WARPS - 1) / (2 * ROWS_WARPS), n_items = n_tiles * row_blocks * n_z;
    const size_t row = QT == NNTR_Q4_K ? (size_t)nb * sizeof(BlockQ4Kx8) : (size_t)a.nblk * sizeof(BlockQ40x8);
    auto fetch_act = [&](const RowsItem &it, int s) {
      if (lane == 31)
        bulk_g2s(smem_u32(sh.act[s]), act_unit<QT>(a.act, it.tl.act_first, it.tl.act_tiles, it.tl.act_k, th, nb, it.b),
                 ((it.tl.rows + 7) >> 3) * th * act_row_bytes(QT), full0 + 8 * s);
    };
    int u = 0; // units so far; the activations of the first STAGES wait for the kernel that writes them
    auto first_acts = [&]() {
      if (!GROUPED)
        pdl_wait();
      for (int s = 0; s < u && s < STAGES; ++s)
        fetch_act(sh.item[s], s);
    };
    // Whole rounds of items first. Those that are left over are cut into 2 or 4 parts of 32 or 16 weight rows where there are
    // CTAs enough, so that the last round is shared by all of them.
    const int rounds = n_items / (int)gridDim.x, left = n_items - rounds * (int)gridDim.x;
    const int cut = left * 4 <= (int)gridDim.x ? 4 : left * 2 <= (int)gridDim.x ? 2 : 1;
    for (int k = 0; k <= rounds && ok; ++k) { // tiles fastest: neighbouring CTAs share their weights
      const bool whole = k < rounds;
      if (!whole && (int)blockIdx.x >= left * cut)
        break;
      const int item = k * (int)gridDim.x + (int)blockIdx.x / (whole ? 1 : cut);
      const int part = whole ? 0 : (int)blockIdx.x % cut, part_groups = 2 * ROWS_WARPS / (whole ? 1 : cut);
      RowsItem it;
      const int rest = item / n_tiles;
      it.tl.z = rest / row_blocks;
      it.group0 = (rest - it.tl.z * row_blocks) * (2 * ROWS_WARPS) + part * part_groups;
      if (it.group0 >= n_groups)
        continue;
      if (!find_tile<NT>(it.tl, a, item - rest * n_tiles, GROUPED))
        continue;
      if (GROUPED && (reinterpret_cast<uintptr_t>(it.tl.W) & 15)) { // from a table in device memory: not seen by the launcher
        if (lane == 0)
          atomicExch(&g_mma_status, NNTR_CUDA_ERR_INVALID);
        continue;
      }
      const int groups = min(part_groups, n_groups - it.group0), tiles = (it.tl.rows + 7) >> 3;
      it.groups = groups;
      const uint8_t *w = static_cast<const uint8_t *>(it.tl.W) + (size_t)(it.group0 + min(lane, groups - 1)) * row;
      for (int b = 0; b < nb; ++b, ++u) {
        if (u >= STAGES && !wait(empty0, par ^ 1))
          break;
        it.b = b;
        const int bytes = QT == NNTR_Q4_K ? (int)sizeof(BlockQ4Kx8) : min(8, a.nblk - 8 * b) * (int)sizeof(BlockQ40x8);
        if (lane == 0) {
          sh.item[slot] = it;
          mbar_expect_tx(full0 + 8 * slot, groups * bytes + tiles * th * act_row_bytes(QT));
        }
        __syncwarp();
        if (lane < groups)
          bulk_g2s(smem_u32(sh.w[slot]) + lane * (int)sizeof(BlockQ4Kx8), w + (size_t)b * sizeof(BlockQ4Kx8), bytes, full0 + 8 * slot);
        if (u >= STAGES)
          fetch_act(it, slot);
        else if (u == STAGES - 1) {
          ++u;
          first_acts();
          --u;
        }
        next_slot();
      }
    }
    if (u < STAGES)
      first_acts();
    if (ok && (u < STAGES || wait(empty0, par ^ 1)) && lane == 0) {
      sh.item[slot].tl.rows = 0;
      mbar_arrive(full0 + 8 * slot);
    }
  } else {
    float acc[NT][4], accm[QT == NNTR_Q4_K ? NT : 1][4];
    while (wait(full0, par)) {
      const Tile tl = sh.item[slot].tl;
      const int group0 = sh.item[slot].group0, groups = sh.item[slot].groups;
      if (tl.rows == 0)
        break;
      // this warp's two row groups inside the CTA's (past the end of N the last group is repeated and not stored)
      const int wg0 = 2 * warp, wg1 = min(2 * warp + 1, groups - 1);
      const int nt = wg0 < groups ? (tl.rows + 7) >> 3 : 0; // 0: nothing for this warp
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc[i][c] = 0.f;
          if constexpr (QT == NNTR_Q4_K)
            accm[i][c] = 0.f;
        }
      for (int b = 0; b < nb; ++b) {
        if (b > 0 && !wait(full0, par))
          break;
        const uint8_t *act = sh.act[slot];
        if (nt == 0) {
        } else if constexpr (QT == NNTR_Q4_K) {
          const BlockQ4Kx8 *w0 = reinterpret_cast<const BlockQ4Kx8 *>(sh.w[slot]) + wg0,
                           *w1 = reinterpret_cast<const BlockQ4Kx8 *>(sh.w[slot]) + wg1;
          Q4KScales sc;
          q4k_scales(sc, w0, w1, g, t, lane);
          with_tiles<NT>(nt, [&](auto N) {
            constexpr int n = decltype(N)::value;
            if constexpr (GROUPED)
              q4k_unit<n, CHAIN_ONE, true>(acc, accm, sc, w0, w1, act, 8, 0, g, t, lane);
            else if (TH8 && tl.pos + tl.rows <= a.M4)
              q4k_unit<n, CHAIN_FOUR, true>(acc, accm, sc, w0, w1, act, 8, 0, g, t, lane);
            else if (TH8 && tl.pos >= a.M4)
              q4k_unit<n, CHAIN_ONE, true>(acc, accm, sc, w0, w1, act, 8, 0, g, t, lane);
            else // the last tile, with up to three rows of the one-step chain
              q4k_unit<n, CHAIN_MIXED, TH8>(acc, accm, sc, w0, w1, act, th, a.M4 - tl.pos, g, t, lane);
          });
        } else {
          const int n = min(8, a.nblk - 8 * b);
          const BlockQ40x8 *w0 = reinterpret_cast<const BlockQ40x8 *>(sh.w[slot] + wg0 * sizeof(BlockQ4Kx8)),
                           *w1 = reinterpret_cast<const BlockQ40x8 *>(sh.w[slot] + wg1 * sizeof(BlockQ4Kx8));
          with_tiles<NT>(nt, [&](auto N) {
            if (n == 8)
              q40_unit<decltype(N)::value, true>(acc, w0, w1, act, 8, g, t, lane);
            else
              q40_unit<decltype(N)::value, false>(acc, w0, w1, act, n, g, t, lane);
          });
        }
        // every lane's loads have been performed before the slot is given back (loads_before_refill() does the same here and costs
        // 0.4 % of the grouped products)
        __threadfence_block();
        __syncwarp();
        if (lane == 0)
          mbar_arrive(empty0 + 8 * slot);
        next_slot();
      }
      if (!ok)
        break;
#pragma unroll
      for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = 8 * i + 2 * t + h;
          if (m < tl.rows) {
            float *out = out_row(a, tl, m, GROUPED) + (size_t)(group0 + 2 * warp) * 8 + g;
#pragma unroll
            for (int r = 0; r < 2; ++r)
              if (wg0 + r < groups) {
                const int c = 2 * r + h;
                out[8 * r] = QT == NNTR_Q4_K ? __fsub_rn(acc[i][c], accm[QT == NNTR_Q4_K ? i : 0][c]) : acc[i][c] * 0.0625f;
              }
          }
        }
    }
  }
  if (!ok) { // a wait ran out: give the copies in flight time to land in this CTA's shared memory
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
  }
}

/* ------------------------------------------- eight warps along K, one tile */
constexpr int KS_WARPS = 8;
constexpr int KS_RING = 3;                                    // rounds of weights in flight
constexpr int KS_W = 2 * KS_WARPS * (int)sizeof(BlockQ4Kx8);  // the weights of a round: 2 row groups x 8 units

template <int NT> struct KsShared {
  alignas(16) uint8_t w[KS_RING][KS_W];
  alignas(16) float4 chain[KS_WARPS][NT][2][32]; // what the warp in front has added up, a lane's outputs each
  alignas(8) unsigned long long full[KS_RING];
  int abort_flag;
};

/** COPIES: the weights start at a multiple of 16 and bulk copies bring them in; otherwise they start at a multiple of 8 and every
 *  warp brings its own units in by 8-byte copies. Instances of their own: as branches of one they cost Q4_K with two tiles 2 to 3 %
 *  (16 x 4096 x 4096 9.8 -> 10.1 us). Q4_K at a multiple of 8, 8 x 2560 x 9728 13.0 us, 256 x 4096 x 4096 101 (loads into registers one
 *  round ahead: 18.7 and 135; every warp's loads and then its products: 19.8 and 141). */
template <int QT, int NT, bool GROUPED, bool TH8, bool COPIES>
__global__ void __launch_bounds__(KS_WARPS * 32, 2) gemm_mma_ksplit_kernel(const MmaArgs a) {
  extern __shared__ __align__(16) uint8_t ks_smem[];
  static_assert(KS_WARPS * NT <= 16, "a hand-over barrier per warp and tile"); // with 16, nothing in the loop may be a barrier of the CTA
  KsShared<NT> &sh = *reinterpret_cast<KsShared<NT> *>(ks_smem);
  volatile int *abort_flag = &sh.abort_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int rt = blockIdx.y, nb = a.nb;
  const bool second = rt * 16 + 8 < a.N;
  const int per = (nb + KS_WARPS - 1) / KS_WARPS; // rounds
  const int upr = (nb + per - 1) / per;           // units per round, the same in every round but the last
  const size_t row = QT == NNTR_Q4_K ? (size_t)nb * sizeof(BlockQ4Kx8) : (size_t)a.nblk * sizeof(BlockQ40x8); // bytes of a row group
  if (tid == 0) {
    for (int i = 0; i < KS_RING; ++i)
      mbar_init(smem_u32(sh.full + i), 1);
    sh.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  Tile tl;
  tl.z = GROUPED ? blockIdx.z : 0;
  if (GROUPED)
    pdl_wait();
  if (!find_tile<NT>(tl, a, blockIdx.x, GROUPED))
    return;
  if (GROUPED && (reinterpret_cast<uintptr_t>(tl.W) & 15)) { // from a table in device memory: not seen by the launcher
    if (tid == 0)
      atomicExch(&g_mma_status, NNTR_CUDA_ERR_INVALID);
    return;
  }
  const uint8_t *w = static_cast<const uint8_t *>(tl.W) + (size_t)(2 * rt) * row;
  auto round_bytes = [&](int rd) { return (int)min((size_t)upr * sizeof(BlockQ4Kx8), row - (size_t)rd * upr * sizeof(BlockQ4Kx8)); };
  auto fetch = [&](int rd, int slot) { // thread 0: a row group's units of a round are one piece of memory
    const uint32_t bar = smem_u32(sh.full + slot), dst = smem_u32(sh.w[slot]);
    const int bytes = round_bytes(rd);
    mbar_expect_tx(bar, bytes * (1 + second));
    for (int h = 0; h < 1 + second; ++h)
      bulk_g2s(dst + h * (KS_W / 2), w + h * row + (size_t)rd * upr * sizeof(BlockQ4Kx8), bytes, bar);
  };
  auto fetch_own = [&](int rd, int slot) { // all lanes: this warp's unit of a round, one group of copies
    const int b = rd * upr + warp;
    if (warp < upr && b < nb) {
      const int bytes = QT == NNTR_Q4_K ? (int)sizeof(BlockQ4Kx8) : min(8, a.nblk - 8 * b) * (int)sizeof(BlockQ40x8);
      const uint32_t dst = smem_u32(sh.w[slot]) + warp * (int)sizeof(BlockQ4Kx8);
      for (int h = 0; h < 1 + second; ++h)
        for (int i = lane * 8; i < bytes; i += 32 * 8)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + h * (KS_W / 2) + i),
                       "l"(w + h * row + (size_t)b * sizeof(BlockQ4Kx8) + i)
                       : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // the weights do not depend on the quantizer's kernel: fetched while it runs
  if (!COPIES)
    for (int rd = 0; rd < KS_RING - 1; ++rd)
      fetch_own(rd, rd);
  else if (tid == 0)
    for (int rd = 0; rd < KS_RING && rd < per; ++rd)
      fetch(rd, rd);
  if (!GROUPED) {
    pdl_wait();
    pdl_launch_dependents();
  }
  __syncthreads();
  const int nt = (tl.rows + 7) >> 3, th = TH8 ? 8 : a.th;
  using Act = std::conditional_t<QT == NNTR_Q4_K, ActQ4K, ActQ40>;
  Act next; // activations of the step that comes next
  auto load_act = [&](int rd, int i) {
    if (warp < upr && rd * upr + warp < nb)
      act_load<TH8>(next, act_unit<QT>(a.act, tl.act_first, tl.act_tiles, tl.act_k + i, th, nb, rd * upr + warp), th, lane);
  };
  load_act(0, 0);
  bool ok = true;
  int slot = 0;
  uint32_t par = 0;
  for (int rd = 0; rd < per; ++rd) {
    const int b = rd * upr + warp;
    uint8_t *wr = sh.w[slot];
    if (warp < upr && b < nb) {
      if (!COPIES) {
        __syncwarp(); // all lanes are done with the unit in front
        fetch_own(rd + KS_RING - 1, slot ? slot - 1 : KS_RING - 1);
        asm volatile("cp.async.wait_group %0;" ::"n"(KS_RING - 1) : "memory");
      } else if (!__all_sync(FULL, mbar_try_wait(smem_u32(sh.full + slot), par))) {
        ok = mbar_wait_bounded(smem_u32(sh.full + slot), par, abort_flag, &g_mma_status, 1u << 22, 2048) && ok;
      }
      __syncwarp();
      const uint8_t *u0 = wr + warp * sizeof(BlockQ4Kx8), *u1 = u0 + (second ? KS_W / 2 : 0);
      Q4KScales sc;
      if constexpr (QT == NNTR_Q4_K)
        q4k_scales(sc, reinterpret_cast<const BlockQ4Kx8 *>(u0), reinterpret_cast<const BlockQ4Kx8 *>(u1), g, t, lane);
      const int to_warp = warp + 1 < upr ? warp + 1 : 0;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        if (i >= nt)
          break;
        const Act x = next;
        if (i + 1 < nt)
          load_act(rd, i + 1);
        else if (rd + 1 < per)
          load_act(rd + 1, 0);
        float acc[4], accm[4];
        /* The chains go through the warps: this one takes them over when the units in front have been added. */
        auto receive = [&]() {
          if (b == 0) {
#pragma unroll
            for (int c = 0; c < 4; ++c)
              acc[c] = accm[c] = 0.f;
            return;
          }
          pair_sync(warp * NT + i);
          const float4 f = sh.chain[warp][i][0][lane];
          acc[0] = f.x, acc[1] = f.y, acc[2] = f.z, acc[3] = f.w;
          if constexpr (QT == NNTR_Q4_K) {
            const float4 m = sh.chain[warp][i][1][lane];
            accm[0] = m.x, accm[1] = m.y, accm[2] = m.z, accm[3] = m.w;
          }
        };
        if constexpr (QT == NNTR_Q4_K) {
          int v[4][4];
          auto pair = [&](auto P) {
            constexpr int p = decltype(P)::value;
            const uint2 q0 = *reinterpret_cast<const uint2 *>(reinterpret_cast<const BlockQ4Kx8 *>(u0)->qs + ((4 * p + t) * 8 + g) * 8),
                        q1 = *reinterpret_cast<const uint2 *>(reinterpret_cast<const BlockQ4Kx8 *>(u1)->qs + ((4 * p + t) * 8 + g) * 8);
            int lo[4], hi[4];
            mma_u8s8(lo, q0.x & 0x0f0f0f0fu, q1.x & 0x0f0f0f0fu, q0.y & 0x0f0f0f0fu, q1.y & 0x0f0f0f0fu, x.b[p].x, x.b[p].y);
            mma_u8s8(hi, (q0.x >> 4) & 0x0f0f0f0fu, (q1.x >> 4) & 0x0f0f0f0fu, (q0.y >> 4) & 0x0f0f0f0fu, (q1.y >> 4) & 0x0f0f0f0fu,
                     x.b[p].z, x.b[p].w);
#pragma unroll
            for (int c = 0; c < 4; ++c)
              v[p][c] = q4k_scale_int<2 * p>(sc, c >> 1) * lo[c] + q4k_scale_int<2 * p + 1>(sc, c >> 1) * hi[c];
          };
          pair(std::integral_constant<int, 0>{});
          pair(std::integral_constant<int, 1>{});
          pair(std::integral_constant<int, 2>{});
          pair(std::integral_constant<int, 3>{});
          const uint32_t bs[2] = {sum_halves<0>(x.sums), sum_halves<1>(x.sums)};
          float2 s1[2], s2[2];
#pragma unroll
          for (int r = 0; r < 2; ++r) {
            s1[r] = mul2(sc.dw[r], sc.dw[r], x.d.x, x.d.y);
            s2[r] = mul2(sc.dm[r], sc.dm[r], x.d.x, x.d.y);
          }
          const int m4 = GROUPED ? 0 : a.M4 - tl.pos - 8 * i; // rows of the tile below it take four steps, the others one
          float vf[4][4], jf[4][4], v1[4], j1[4];
          if (m4 > 0) {
#pragma unroll
            for (int p = 0; p < 4; ++p) {
              mma_f16_k8(jf[p], sc.mn[2 * (p >> 1)], sc.mn[2 * (p >> 1) + 1], (t >> 1) == (p & 1) ? bs[p >> 1] : 0u);
#pragma unroll
              for (int c = 0; c < 4; ++c)
                vf[p][c] = (float)v[p][c]; // below 2^23: exact
            }
          }
          if (m4 < 8) {
            mma_f16_k16(j1, sc.mn[0], sc.mn[1], sc.mn[2], sc.mn[3], bs[0], bs[1]);
#pragma unroll
            for (int c = 0; c < 4; ++c)
              v1[c] = __int2float_rn((v[0][c] + v[1][c]) + (v[2][c] + v[3][c])); // one rounding of the exact sum
          }
          receive();
          if (m4 >= 8) {
#pragma unroll
            for (int p = 0; p < 4; ++p)
#pragma unroll
              for (int r = 0; r < 2; ++r) {
                fma2(acc[2 * r], acc[2 * r + 1], vf[p][2 * r], vf[p][2 * r + 1], s1[r].x, s1[r].y);
                fma2(accm[2 * r], accm[2 * r + 1], jf[p][2 * r], jf[p][2 * r + 1], s2[r].x, s2[r].y);
              }
          } else if (m4 <= 0) {
#pragma unroll
            for (int r = 0; r < 2; ++r) {
              fma2(acc[2 * r], acc[2 * r + 1], v1[2 * r], v1[2 * r + 1], s1[r].x, s1[r].y);
              fma2(accm[2 * r], accm[2 * r + 1], j1[2 * r], j1[2 * r + 1], s2[r].x, s2[r].y);
            }
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float e1 = (c & 1) ? s1[c >> 1].y : s1[c >> 1].x, e2 = (c & 1) ? s2[c >> 1].y : s2[c >> 1].x;
              if (2 * t + (c & 1) < m4) {
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                  acc[c] = __fmaf_rn(vf[p][c], e1, acc[c]);
                  accm[c] = __fmaf_rn(jf[p][c], e2, accm[c]);
                }
              } else {
                acc[c] = __fmaf_rn(v1[c], e1, acc[c]);
                accm[c] = __fmaf_rn(j1[c], e2, accm[c]);
              }
            }
          }
        } else {
          const int n = min(8, a.nblk - 8 * b);
          float v[8][4], s[8][4];
          auto block = [&](auto J) {
            constexpr int j = decltype(J)::value;
            // a block past the end of the row: what the shared memory holds, with scale 0
            const BlockQ40x8 *k0 = reinterpret_cast<const BlockQ40x8 *>(u0) + j, *k1 = reinterpret_cast<const BlockQ40x8 *>(u1) + j;
            const uint4 bb = x.b[j >> 1];
            const uint32_t at = (t >> 1) * 64 + g * 8 + (t & 1) * 4;
            const uint32_t w0 = *reinterpret_cast<const uint32_t *>(k0->qs + at), w1 = *reinterpret_cast<const uint32_t *>(k1->qs + at);
            const uint32_t qq[4] = {(w0 << 4) & 0xf0f0f0f0u, (w1 << 4) & 0xf0f0f0f0u, w0 & 0xf0f0f0f0u, w1 & 0xf0f0f0f0u};
            q40_terms<j & 1>(v[j], s[j], qq, (j & 1) ? bb.z : bb.x, (j & 1) ? bb.w : bb.y,
                             j < n ? k0->d[g] : (uint16_t)0, j < n ? k1->d[g] : (uint16_t)0, x.d[j >> 1]);
          };
          block(std::integral_constant<int, 0>{});
          block(std::integral_constant<int, 1>{});
          block(std::integral_constant<int, 2>{});
          block(std::integral_constant<int, 3>{});
          block(std::integral_constant<int, 4>{});
          block(std::integral_constant<int, 5>{});
          block(std::integral_constant<int, 6>{});
          block(std::integral_constant<int, 7>{});
          receive();
#pragma unroll
          for (int j = 0; j < 8; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r)
              fma2(acc[2 * r], acc[2 * r + 1], v[j][2 * r], v[j][2 * r + 1], s[j][2 * r], s[j][2 * r + 1]);
        }
        if (b + 1 < nb) {
          sh.chain[to_warp][i][0][lane] = make_float4(acc[0], acc[1], acc[2], acc[3]);
          if constexpr (QT == NNTR_Q4_K)
            sh.chain[to_warp][i][1][lane] = make_float4(accm[0], accm[1], accm[2], accm[3]);
          pair_arrive(to_warp * NT + i);
        } else if (nobody_gave_up(ok, abort_flag)) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int m = 8 * i + 2 * t + (c & 1);
            if (m < tl.rows && (c < 2 || second))
              out_row(a, tl, m, GROUPED)[rt * 16 + g + 8 * (c >> 1)] = QT == NNTR_Q4_K ? __fsub_rn(acc[c], accm[c]) : acc[c] * 0.0625f;
          }
        }
      }
      // The chains of this round's first unit have come through every unit of the round before, so nobody reads its weights any more.
      if (COPIES && warp == 0 && rd > 0 && rd - 1 + KS_RING < per) {
        __syncwarp();
        if (lane == 0 && ok) {
          loads_before_refill();
          fetch(rd - 1 + KS_RING, slot ? slot - 1 : KS_RING - 1);
        }
      }
    }
    if (++slot == KS_RING)
      slot = 0, par ^= 1;
  }
  if (!ok) { // a wait ran out: give the copies in flight time to land in this CTA's shared memory
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
  }
}

/* ----------------------------------------------------- activation tiles */
/** The 256 elements from element 256 * b of a row, a lane's eight of them quantized (rule: the quantizer's of Q4_K). */
template <int QT> __device__ __forceinline__ auto quantize_unit(const float *row, int b, int K, int rule, int lane) {
  const float *src = row + (int64_t)b * QK_K + lane * 8;
  if constexpr (QT == NNTR_Q4_K) {
    return q8K_quantize_warp(*reinterpret_cast<const float4 *>(src), *reinterpret_cast<const float4 *>(src + 4), lane, rule);
  } else {
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
    if (b * QK_K + lane * 8 < K) { // blocks past K are zeros
      v0 = *reinterpret_cast<const float4 *>(src);
      v1 = *reinterpret_cast<const float4 *>(src + 4);
    }
    return q80_quantize_warp(v0, v1);
  }
}
/** fp32 rows -> activation tiles; one warp per (row, unit). */
template <int QT>
__global__ void __launch_bounds__(256)
act_tiles_kernel(const float *__restrict__ x, int64_t ldx, uint8_t *__restrict__ act, int M, int M4, int nb, int K, int th) {
  pdl_wait();
  pdl_launch_dependents(); // the GEMM behind fetches weights, which a kernel in front of this one may have written, and waits for the rest
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (w >= (int64_t)M * nb)
    return;
  const int row = (int)(w / nb), b = (int)(w - (int64_t)row * nb), tile = row / th;
  uint8_t *unit = act_unit<QT>(act, 0, (M + th - 1) / th, tile, th, nb, b);
  const auto q = quantize_unit<QT>(x + (int64_t)row * ldx, b, K, row < M4 ? 1 : 0, lane);
  if constexpr (QT == NNTR_Q4_K)
    put_q8K(unit, th, row - tile * th, q, lane);
  else
    put_q80(unit, th, row - tile * th, q, lane);
}
/** The same for the rows of every expert: a token's row goes into the tiles of its topk experts. One warp per (token, unit), so that it
 *  is quantized once and not once per expert (2048 rows of 2048 were 10.9 us of a layer's 200, cold). Lane k looks up where the
 *  k-th copy goes. */
template <int QT>
__global__ void __launch_bounds__(256)
act_tiles_grouped_kernel(const float *__restrict__ x, uint8_t *__restrict__ act, int T, int nb, int K, int topk, const int *__restrict__ inv,
                         const int *__restrict__ idx, const int *__restrict__ off, const int *__restrict__ act_off) {
  pdl_launch_dependents();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (w >= (int64_t)T * nb)
    return;
  const int t = (int)(w / nb), b = (int)(w - (int64_t)t * nb);
  int i = 0, first = 0, n_tiles = 0;
  if (lane < topk) { // topk <= 32
    const int e = idx[t * topk + lane], o = off[e];
    i = inv[t * topk + lane] - o;
    first = act_off[e];
    n_tiles = (off[e + 1] - o + 7) >> 3;
  }
  const auto q = quantize_unit<QT>(x + (int64_t)t * K, b, K, 0, lane);
  for (int k = 0; k < topk; ++k) {
    const int row = __shfl_sync(FULL, i, k);
    uint8_t *unit = act_unit<QT>(act, __shfl_sync(FULL, first, k), __shfl_sync(FULL, n_tiles, k), row >> 3, 8, nb, b);
    if constexpr (QT == NNTR_Q4_K)
      put_q8K(unit, 8, row & 7, q, lane);
    else
      put_q80(unit, 8, row & 7, q, lane);
  }
}

template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

template <int QT, int NT, bool GROUPED, bool TH8>
int run_tiles(const MmaArgs &a, unsigned tiles, unsigned z, bool ksplit, bool misaligned, cudaStream_t st) {
  const unsigned row_tiles = (unsigned)((a.N + 15) / 16);
  constexpr int stages = rows_stages<QT, NT, GROUPED>(), ctas = rows_ctas<QT, NT, GROUPED>();
  constexpr size_t smem = sizeof(RowsShared<NT, stages>);
  static bool attr_set[64] = {};
  int dev = 0;
  NNTR_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !attr_set[dev]) {
    if constexpr (NT <= 2) {
      NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8, true>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KsShared<NT>)));
      NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8, GROUPED>,
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(KsShared<NT>)));
    }
    NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_mma_rows_kernel<QT, NT, GROUPED, TH8, stages>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev] = true;
  }
  cudaError_t e = cudaSuccess;
  if (NT <= 2 && ksplit) {
    if constexpr (NT <= 2)
      e = launch(misaligned ? gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8, GROUPED> : gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8, true>,
                 dim3(tiles, row_tiles, z), KS_WARPS * 32, sizeof(KsShared<NT>), st, a);
  } else {
    const uint64_t items = (uint64_t)tiles * ((row_tiles + ROWS_WARPS - 1) / ROWS_WARPS) * z;
    const uint64_t slots = (uint64_t)ctas * (unsigned)sm_count();
    e = launch(gemm_mma_rows_kernel<QT, NT, GROUPED, TH8, stages>, dim3((unsigned)(4 * items < slots ? 4 * items : slots)), ROWS_WARPS * 32 + 32,
               smem, st, a, (int)tiles, (int)z);
  }
  count_launch();
  return check_cuda(e, "gemm (integer warp MMA) launch");
}

} // namespace

size_t gemm_mma_workspace_bytes(int qtype, unsigned M, unsigned K) {
  return (size_t)((M + 7) / 8 * 8) * ((K + 255) / 256) * act_row_bytes(qtype);
}

int launch_gemm_mma(int qtype, unsigned M, unsigned M4, unsigned N, unsigned K, const float *A, const void *B, float *C,
                    unsigned ldc, void *ws, size_t ws_bytes, cudaStream_t st) {
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(ws) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm: activations and workspace must be 16-byte aligned");
  if (reinterpret_cast<uintptr_t>(B) & 7)
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm: weights must be 8-byte aligned");
  MmaArgs a = {};
  a.act = static_cast<const uint8_t *>(ws);
  a.W = B;
  a.C = C;
  a.ldc = (int)ldc;
  a.M = (int)M;
  a.M4 = (int)M4;
  a.N = (int)N;
  a.nb = (int)((K + 255) / 256);
  a.nblk = (int)(K / 32);
  a.th = M < 8 && ws_bytes < gemm_mma_workspace_bytes(qtype, M, K) ? (int)M : 8;
  const unsigned grid = (unsigned)(((int64_t)M * a.nb + 7) / 8);
  const auto quantize = qtype == NNTR_Q4_K ? act_tiles_kernel<NNTR_Q4_K> : act_tiles_kernel<NNTR_Q4_0>;
  NNTR_CHECK_CUDA(launch(quantize, dim3(grid), 256, 0, st, A, (int64_t)K, static_cast<uint8_t *>(ws), a.M, a.M4, a.nb, (int)K, a.th));
  count_launch();
  // Weights that are not 16-byte aligned cannot be fetched by bulk copies: the shared tile has 8-byte copies for them.
  const bool misaligned = reinterpret_cast<uintptr_t>(B) & 15;
  const unsigned row_tiles = (N + 15) / 16, row_blocks = (N + 63) / 64, sms = (unsigned)sm_count();
  const auto tiles_of = [&](unsigned nt) { return (M + 8 * nt - 1) / (8 * nt); };
  // One CTA per tile of 8 or 16 rows as long as all of them run at once, two per SM. Beyond that a warp per tile: of 32 rows (the
  // weights are unpacked once for them) where CTAs of 64 weight rows still give every SM work, else of 16, else of 8. Measured on both
  // sides: Q4_K 8 x 2560 x 2560 (160 CTAs) 5.9 us, a warp per tile 8.4; 8 x 4736 x 2560 (296) 5.9 and 9.1; 8 x 6144 x 2560 (384) 9.7 and
  // 9.2; 31 x 2560 x 2560 (320 of 16 rows) 12.3 and 11.4. A warp per tile of 16 / 32 rows: Q4_K 31 x 12288 x 4096 (192 items of 32) 27.1 /
  // 36.9 us, 64 x 9728 x 2560 (304) 24.2 / 24.4, 63 through gemv_rows 22.7 / 21.9; Q4_0 31 x 2560 x 2560 (40) 9.3 / 11.1, 64 x 2880 x 2880
  // (90) 12.8 / 12.5, 31 x 12288 x 4096 (192) 23.6 / 20.7; of 8 / 16 rows: Q4_K 31 x 2560 x 2560 (80 of 16) 11.4 / 11.9, 16 x 6144 x 2560
  // (96) 10.8 / 10.6.
  const bool ksplit = misaligned || (uint64_t)tiles_of(2) * row_tiles <= 2u * sms;
  unsigned nt;
  if (ksplit)
    nt = (uint64_t)tiles_of(1) * row_tiles <= 2u * sms ? 1 : 2;
  else if (qtype == NNTR_Q4_K)
    nt = M <= 8 ? 1 : M > 16 && tiles_of(4) * row_blocks >= 2 * sms ? 4 : 3 * tiles_of(2) * row_blocks >= 2 * sms ? 2 : 1;
  else
    nt = M <= 8 ? 1 : M > 16 && 3 * tiles_of(4) * row_blocks >= 2 * sms ? 4 : 2;
  const unsigned tiles = tiles_of(a.th < 8 ? 1 : nt);
  if (a.th < 8)
    return run_tiles<NNTR_Q4_K, 1, false, false>(a, tiles, 1, ksplit, misaligned, st);
#define NNTR_MMA_RUN(QT)                                                                                               \
  (nt == 1   ? run_tiles<QT, 1, false, true>(a, tiles, 1, ksplit, misaligned, st)                                                  \
   : nt == 2 ? run_tiles<QT, 2, false, true>(a, tiles, 1, ksplit, misaligned, st)                                                  \
             : run_tiles<QT, 4, false, true>(a, tiles, 1, ksplit, misaligned, st))
  return qtype == NNTR_Q4_K ? NNTR_MMA_RUN(NNTR_Q4_K) : NNTR_MMA_RUN(NNTR_Q4_0);
#undef NNTR_MMA_RUN
}

int grouped_tile_rows(int qtype, unsigned pairs, unsigned n_experts) {
  // Tiles of about what an expert gets, so that few experts need a second tile (which fetches and unpacks the expert's weights
  // again). A warp skips the rows that a tile lacks, so a large tile costs registers only. Q4_K, 8 of 128 experts of 2048 x 768, 32 /
  // 100 / 200 / 256 tokens in tiles of 16 and of 32: 105 / 123 / 153 / 184 us and 119 / 138 / 160 / 178; tiles of 8 are behind or
  // level (109 / 132 / 204 / 242). Q4_0, 4 of 32 of 2880 x 2880, 8 / 40 / 64 / 100 tokens in tiles of 8 and of 32: 89 / 133 / 147 /
  // 203 us and 101 / 140 / 142 / 161; 16 is between them (99 / 138 / 142 / 170).
  return qtype == NNTR_Q4_K ? (pairs <= 14 * n_experts ? 16 : 32) : (pairs <= 6 * n_experts ? 8 : 32);
}

int launch_act_tiles_grouped(int qtype, const float *x, unsigned tokens, unsigned topk, unsigned K, void *act, const int *inv, const int *idx,
                             const int *off, const int *act_off, cudaStream_t st) {
  const int nb = (int)((K + 255) / 256);
  const dim3 grid((unsigned)(((int64_t)tokens * nb + 7) / 8));
  const auto kernel = qtype == NNTR_Q4_K ? act_tiles_grouped_kernel<NNTR_Q4_K> : act_tiles_grouped_kernel<NNTR_Q4_0>;
  const cudaError_t e = launch(kernel, grid, 256, 0, st, x, static_cast<uint8_t *>(act), (int)tokens, nb, (int)K, (int)topk, inv, idx, off,
                               act_off);
  count_launch();
  return check_cuda(e, "activation tiles launch");
}

int launch_gemm_grouped(int qtype, unsigned N, unsigned K, const void *act, float *C, unsigned ldc,
                        const void *const *w_table0, const void *const *w_table1, const int *off, const int *tile_off,
                        const int *act_off, const int *perm, int n_experts, int c_mul, int tile_rows, unsigned pairs,
                        cudaStream_t st) {
  if (!act || !C || !w_table0 || !off || !tile_off || !act_off || !perm)
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm_grouped: null pointer");
  if (pairs == 0 || N == 0)
    return NNTR_CUDA_OK;
  MmaArgs a = {};
  a.act = static_cast<const uint8_t *>(act);
  a.C = C;
  a.ldc = (int)ldc;
  a.N = (int)N;
  a.nb = (int)((K + 255) / 256);
  a.nblk = (int)(K / 32);
  a.th = 8;
  a.w_table[0] = w_table0;
  a.w_table[1] = w_table1 ? w_table1 : w_table0;
  a.off = off;
  a.tile_off = tile_off;
  a.act_off = act_off;
  a.perm = perm;
  a.n_experts = n_experts;
  a.c_mul = c_mul;
  // sum over the experts of ceil(count / tile_rows), at most one tile per pair
  const unsigned tiles = pairs < pairs / tile_rows + n_experts ? pairs : pairs / tile_rows + n_experts;
  const unsigned z = w_table1 ? 2 : 1;
  const bool ksplit = tile_rows <= 16 && (uint64_t)tiles * z * ((N + 15) / 16) <= 2u * (unsigned)sm_count();
  if (qtype == NNTR_Q4_K)
    return tile_rows <= 16 ? run_tiles<NNTR_Q4_K, 2, true, true>(a, tiles, z, ksplit, false, st)
                           : run_tiles<NNTR_Q4_K, 4, true, true>(a, tiles, z, ksplit, false, st);
  if (qtype == NNTR_Q4_0)
    return tile_rows <= 8 ? run_tiles<NNTR_Q4_0, 1, true, true>(a, tiles, z, ksplit, false, st)
                          : run_tiles<NNTR_Q4_0, 4, true, true>(a, tiles, z, ksplit, false, st);
  return set_error(NNTR_CUDA_ERR_UNSUPPORTED, "gemm_grouped: expert weights must be Q4_K or Q4_0");
}

int read_mma_status(int *out) {
  int v = 0;
  NNTR_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_mma_status, sizeof(int)));
  *out = v;
  return NNTR_CUDA_OK;
}
int clear_mma_status() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_mma_status, &zero, sizeof(int)), "clear_mma_status");
}

} // namespace nntr
