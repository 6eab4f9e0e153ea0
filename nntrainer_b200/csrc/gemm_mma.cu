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
 * high nibbles of 4 bytes each, one logic op per fragment register and no trip through shared memory.
 *
 * sc0 * I0 + sc1 * I1 of a pair of sub-blocks is computed in fp32: |I| <= 15 * 127 * 32 and sc <= 63, so every product
 * and the sum (below 2^23) are exact. High nibbles enter in place, as 16 times their value, and meet sc1 / 16. (Seeding
 * the MMA with the bits of 1.5 * 2^23, so that its result is a float already, was measured: the four moves that set the
 * operand up for each MMA cost more than the conversions.) The sums of the mins term come from one fp16 MMA
 * of [min, 64 min] with the sums of 32 activations split into [sum & 63, sum >> 6], all of them integers fp16 holds.
 *
 * Two splits of the work:
 *   gemm_mma_rows_kernel   a warp owns 16 weight rows and up to 32 activation rows over all of K; the CTA's four warps share
 *                          the unit's activation tiles and weights, which bulk copies bring into a ring. For problems with
 *                          enough such tiles to fill the machine. Bound by too few warps in flight: at 32 rows per tile 142 (Q4_0) to
 *                          168 registers and 55 KB hold three CTAs per SM, and Q4_0 509 x 2880 x 2880 (720 CTAs, 1.6 waves) issues
 *                          in 54 % of the active clocks with 2.5 warps per scheduler, a third of the waiting being for memory
 *                          (the conversions and the chains are about 100 of the 220 instructions per 16 x 8 x 256): 256 x 24576 x 4096 286 us, 180 TOP/s
 *                          (CUDA-core kernel before: 2981 us); Q4_0 509 x 2880 x 2880 58 us (551).
 *   gemm_mma_ksplit_kernel eight warps share the tile and take every eighth unit of 256 along K; the terms of the chains
 *                          go through shared memory and one thread per chain adds them in order. For the others: bound by
 *                          latency. 8 x 6144 x 2560 12.2 us including the quantizer's launch (25.5), 8 x 2560 x 9728
 *                          18.9 us (77.6).
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
/** (v, 64 v) of a 6-bit value as half2; 0x64vv is 1024 + v */
__device__ __forceinline__ uint32_t min_halves(uint32_t v) {
  return h2_bits(__hmul2(__hsub2(bits_h2(v * 0x10001u | 0x64006400u), bits_h2(0x64006400u)), __floats2half2_rn(1.f, 64.f)));
}
/** (lo, hi - 64) of one 16-bit half K of an activation row's word as half2 */
template <int K> __device__ __forceinline__ uint32_t sum_halves(uint32_t w) {
  return h2_bits(__hsub2(bits_h2(__byte_perm(w, 0x64646464u, K ? 0x4342 : 0x4140)), __floats2half2_rn(1024.f, 1088.f)));
}

/* ------------------------------------------------------------------ Q4_K */
/** The weights of 16 rows x 256 as a lane holds them: g = lane / 4 picks the rows g and g + 8, t = lane % 4 the 8-byte
 *  chunk 4p + t of pair p, i.e. elements 8t .. 8t+7 of the pair's two sub-blocks. */
struct Q4KRaw {
  uint2 q[4][2];       // [pair][row g / g + 8]
  uint32_t head[2][2][3]; // [row][sub-block t / t + 4]: the 12-byte group with scales and mins of the row's 8-row group
  uint32_t d[2];       // d | dmin << 16
};
__device__ __forceinline__ void q4k_load(Q4KRaw &r, const BlockQ4Kx8 *lo, const BlockQ4Kx8 *hi, int g, int t) {
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    r.q[p][0] = ldg_stream_u2(lo->qs + ((4 * p + t) * 8 + g) * 8);
    r.q[p][1] = ldg_stream_u2(hi->qs + ((4 * p + t) * 8 + g) * 8);
  }
#pragma unroll
  for (int row = 0; row < 2; ++row) {
    const BlockQ4Kx8 *b = row ? hi : lo;
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
      for (int i = 0; i < 3; ++i)
        r.head[row][s][i] = __ldg(reinterpret_cast<const uint32_t *>(b->scales + 12 * (t + 4 * s)) + i);
    r.d[row] = (uint32_t)__ldg(&b->d[g]) | ((uint32_t)__ldg(&b->dmin[g]) << 16);
  }
}
/** What the MMAs and chains need besides the nibbles. */
struct Q4KScales {
  uint32_t sc[4];  // gathered from the quad: word t' = scales of sub-blocks t' and t' + 4 of row g (bytes 0, 1), row g + 8 (2, 3)
  uint32_t mn[4];  // A fragment of the mins: [row g, t], [row g + 8, t], [row g, t + 4], [row g + 8, t + 4]
  float dw[2], dm[2];
};
__device__ __forceinline__ void q4k_scales(Q4KScales &s, const uint32_t (&head)[2][2][3], const uint32_t (&d)[2], int g, int lane) {
  const int sh = 8 * (g & 3);
  uint32_t own = 0;
#pragma unroll
  for (int row = 0; row < 2; ++row)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const uint32_t b0 = (head[row][k][0] >> sh) & 0xff, b1 = (head[row][k][1] >> sh) & 0xff,
                     b2 = (head[row][k][2] >> sh) & 0xff;
      const uint32_t sc = g < 4 ? (b0 & 63) : ((b2 & 0xf) | ((b0 >> 6) << 4));
      const uint32_t mn = g < 4 ? (b1 & 63) : ((b2 >> 4) | ((b1 >> 6) << 4));
      own |= sc << (8 * k + 16 * row);
      s.mn[row + 2 * k] = min_halves(mn);
    }
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
/** scale of sub-block J of row g + 8 * row as a float (even J: as it is; odd J: over 16, because the high nibbles enter
 *  the MMA times 16): 0x4B0000bb is 2^23 + b, 0x490000bb is 2^19 + b / 16 */
template <int J> __device__ __forceinline__ float q4k_scale(const Q4KScales &s, int row) {
  const uint32_t w = __byte_perm(s.sc[J & 3], (J & 1) ? 0x49000000u : 0x4B000000u, 0x7440 | ((J >> 2) + 2 * row));
  return __uint_as_float(w) - ((J & 1) ? 524288.f : 8388608.f);
}
struct Q4KFactors { // per pair and row: the two scales
  float s0[4][2], s1[4][2];
};
__device__ __forceinline__ void q4k_factors(Q4KFactors &f, const Q4KScales &s) {
  auto pair = [&](auto P) {
    constexpr int p = decltype(P)::value;
#pragma unroll
    for (int row = 0; row < 2; ++row) {
      f.s0[p][row] = q4k_scale<2 * p>(s, row);
      f.s1[p][row] = q4k_scale<2 * p + 1>(s, row);
    }
  };
  pair(std::integral_constant<int, 0>{});
  pair(std::integral_constant<int, 1>{});
  pair(std::integral_constant<int, 2>{});
  pair(std::integral_constant<int, 3>{});
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

/** Pair p of a 16 x 8 tile: f[c] = sc0 * I0 + sc1 * I1 (exact). c = 0..3: row g + 8 * (c / 2), activation row 2t + c % 2. */
__device__ __forceinline__ void q4k_pair(float (&f)[4], const uint32_t (&al)[4], const uint32_t (&ah)[4], const uint4 &b,
                                         const float (&s0)[2], const float (&s1)[2]) {
  int lo[4], hi[4];
  mma_u8s8(lo, al[0], al[1], al[2], al[3], b.x, b.y);
  mma_u8s8(hi, ah[0], ah[1], ah[2], ah[3], b.z, b.w);
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const int row = c >> 1;
    f[c] = fmaf(s1[row], (float)hi[c], s0[row] * (float)lo[c]);
  }
}

/* ------------------------------------------------------------------ Q4_0 */
/** 16 rows x 256: word t of every 32-block of the rows g and g + 8 (elements 4t.. as low and 16 + 4t.. as high nibbles). */
struct Q40Raw {
  uint32_t q[8][2];
  uint16_t d[8][2];
};
__device__ __forceinline__ void q40_load(Q40Raw &r, const BlockQ40x8 *lo, const BlockQ40x8 *hi, int n, int g, int t) {
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int row = 0; row < 2; ++row) {
      const BlockQ40x8 *b = (row ? hi : lo) + (j < n ? j : n - 1);
      r.q[j][row] = ldg_stream_u32(b->qs + (t >> 1) * 64 + g * 8 + (t & 1) * 4);
      r.d[j][row] = __ldg(&b->d[g]);
    }
}
struct ActQ40 {
  uint4 b[4];
  float d[2][8]; // rows 2t, 2t + 1
};
/** scales of the blocks 4h .. 4h + 3 of row i */
__device__ __forceinline__ float4 act_d4(const uint8_t *unit, int i, int h) {
  const uint2 d = *reinterpret_cast<const uint2 *>(unit + 256 * 8 + 16 * i + 8 * h);
  const float2 lo = __half22float2(bits_h2(d.x)), hi = __half22float2(bits_h2(d.y));
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}
template <bool TH8> __device__ __forceinline__ void act_load(ActQ40 &a, const uint8_t *unit, int, int lane) {
  static_assert(TH8, "only Q4_K has a call with short tiles");
#pragma unroll
  for (int p = 0; p < 4; ++p)
    a.b[p] = act_frag<true>(unit, p, 8, lane);
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const float4 d = act_d4(unit, 2 * (lane & 3) + c, h);
      a.d[c][4 * h] = d.x, a.d[c][4 * h + 1] = d.y, a.d[c][4 * h + 2] = d.z, a.d[c][4 * h + 3] = d.w;
    }
}
/** Block of a 16 x 8 tile: x[c] = 16 * (sum of (q - 8) * a). The stored nibble (q ^ 8) is q - 8 in two's complement, so
 *  in the upper half of a byte it is that times 16. q: low nibbles of rows g, g + 8, high nibbles of them, all moved there. */
__device__ __forceinline__ void q40_block(float (&x)[4], const uint32_t (&q)[4], uint32_t b0, uint32_t b1) {
  int v[4];
  mma_s8s8(v, q[0], q[1], q[2], q[3], b0, b1);
#pragma unroll
  for (int c = 0; c < 4; ++c)
    x[c] = (float)v[c];
}

/* ------------------------------------------------------- where a tile lies */
/** Activation rows of one warp (or CTA): `rows` of them, outputs from position `pos`, tiles from `act_tile`; weights W. */
struct Tile {
  const void *W;
  int pos, rows, act_tile, z;
};
template <int NT> __device__ __forceinline__ bool find_tile(Tile &tl, const MmaArgs &a, int tile, bool grouped) {
  if (!grouped) {
    tl.W = a.W;
    tl.pos = tile * 8 * NT;
    tl.act_tile = tile * NT;
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
  tl.act_tile = a.act_off[lo] + k * NT;
  tl.rows = min(8 * NT, a.off[lo + 1] - a.off[lo] - first);
  return tl.rows > 0 && tl.W; // a null weight: expert of another rank
}
__device__ __forceinline__ float *out_row(const MmaArgs &a, const Tile &tl, int i, bool grouped) {
  const int row = grouped ? a.perm[tl.pos + i] * a.c_mul + tl.z : tl.pos + i;
  return a.C + (size_t)row * a.ldc;
}

/** One unit of a warp's 16 rows against up to 8 * NT activation rows in shared memory, chains in registers. The pair of
 *  sub-blocks is the outer loop, so that its fragments and factors are unpacked once for all tiles.
 *  CHAIN_FOUR: four steps per super-block; CHAIN_ONE: one; CHAIN_MIXED: four for the rows below m4 of the tile, one behind. */
enum { CHAIN_FOUR, CHAIN_ONE, CHAIN_MIXED };
template <int N_TILES, int CHAIN, bool TH8, int NT>
__device__ __forceinline__ void q4k_unit(float (&acc)[NT][4], float (&accm)[NT][4], const Q4KScales &sc, const BlockQ4Kx8 *w0,
                                         const BlockQ4Kx8 *w1, const uint8_t *act, int th, int m4, int g, int t,
                                         int lane) {
  float s1[N_TILES][4], s2[N_TILES][4]; // four-step rows: d * da and dmin * da; one-step rows: the sums of pairs 0 + 1 and 2 + 3 (exact)
  uint32_t bs[N_TILES][2];
  auto four = [&](int i, int c) { return CHAIN == CHAIN_FOUR || (CHAIN == CHAIN_MIXED && 8 * i + 2 * t + (c & 1) < m4); };
#pragma unroll
  for (int i = 0; i < N_TILES; ++i) {
      const uint8_t *unit = act + i * (8 * act_row_bytes(NNTR_Q4_K));
      const uint32_t sums = act_sums<TH8>(unit, th, lane);
      bs[i][0] = sum_halves<0>(sums);
      bs[i][1] = sum_halves<1>(sums);
      if (CHAIN != CHAIN_ONE) {
        const float2 d = act_d<TH8>(unit, th, t);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s1[i][c] = four(i, c) ? __fmul_rn(sc.dw[c >> 1], (c & 1) ? d.y : d.x) : 0.f;
          s2[i][c] = four(i, c) ? __fmul_rn(sc.dm[c >> 1], (c & 1) ? d.y : d.x) : 0.f;
        }
      } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
          s1[i][c] = s2[i][c] = 0.f;
      }
    }
  auto pair = [&](auto P) {
    constexpr int p = decltype(P)::value;
    const uint2 q0 = *reinterpret_cast<const uint2 *>(w0->qs + ((4 * p + t) * 8 + g) * 8),
                q1 = *reinterpret_cast<const uint2 *>(w1->qs + ((4 * p + t) * 8 + g) * 8);
    const uint32_t lo[4] = {q0.x & 0x0f0f0f0fu, q1.x & 0x0f0f0f0fu, q0.y & 0x0f0f0f0fu, q1.y & 0x0f0f0f0fu};
    const uint32_t hi[4] = {q0.x & 0xf0f0f0f0u, q1.x & 0xf0f0f0f0u, q0.y & 0xf0f0f0f0u, q1.y & 0xf0f0f0f0u};
    float f0[2], f1[2];
#pragma unroll
    for (int row = 0; row < 2; ++row) {
      f0[row] = q4k_scale<2 * p>(sc, row);
      f1[row] = q4k_scale<2 * p + 1>(sc, row);
    }
    const bool own = (t >> 1) == (p & 1); // the lanes that hold the mins of this pair
    const uint32_t m0 = own ? sc.mn[2 * (p >> 1)] : 0u, m1 = own ? sc.mn[2 * (p >> 1) + 1] : 0u;
#pragma unroll
    for (int i = 0; i < N_TILES; ++i) {
        const uint4 x = act_frag<TH8>(act + i * (8 * act_row_bytes(NNTR_Q4_K)), p, th, lane);
        float v[4], j[4];
        q4k_pair(v, lo, hi, x, f0, f1);
        if (CHAIN != CHAIN_ONE)
          mma_f16_k8(j, m0, m1, bs[i][p >> 1]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (CHAIN == CHAIN_FOUR || (CHAIN == CHAIN_MIXED && four(i, c))) {
            acc[i][c] = __fmaf_rn(v[c], s1[i][c], acc[i][c]);
            accm[i][c] = __fmaf_rn(j[c], s2[i][c], accm[i][c]);
          } else if (p < 2) {
            s1[i][c] += v[c];
          } else {
            s2[i][c] += v[c];
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
        const float2 d = act_d<TH8>(act + i * (8 * act_row_bytes(NNTR_Q4_K)), th, t);
        float j[4];
        mma_f16_k16(j, sc.mn[0], sc.mn[1], sc.mn[2], sc.mn[3], bs[i][0], bs[i][1]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          if (CHAIN == CHAIN_ONE || !four(i, c)) { // one rounding of the exact sum of the super-block
            const float da = (c & 1) ? d.y : d.x;
            acc[i][c] = __fmaf_rn(__fadd_rn(s1[i][c], s2[i][c]), __fmul_rn(sc.dw[c >> 1], da), acc[i][c]);
            accm[i][c] = __fmaf_rn(j[c], __fmul_rn(sc.dm[c >> 1], da), accm[i][c]);
          }
      }
  }
}

/** Q4_0: the n blocks of a unit, four at a time. */
template <int N_TILES, int NT>
__device__ __forceinline__ void q40_unit(float (&acc)[NT][4], const BlockQ40x8 *w0, const BlockQ40x8 *w1, const uint8_t *act,
                                         int n, int g, int t, int lane) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (4 * h >= n)
      break;
    uint32_t q[4][4];
    float dw[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int row = 0; row < 2; ++row) {
        // blocks past the end of the row: what the shared memory holds, with scale 0
        const BlockQ40x8 *blk = (row ? w1 : w0) + 4 * h + j;
        const uint32_t w = *reinterpret_cast<const uint32_t *>(blk->qs + (t >> 1) * 64 + g * 8 + (t & 1) * 4);
        q[j][row] = (w << 4) & 0xf0f0f0f0u;
        q[j][row + 2] = w & 0xf0f0f0f0u;
        dw[j][row] = 4 * h + j < n ? half_bits_to_float(blk->d[g]) * 0.0625f : 0.f; // the sums come times 16
      }
    }
#pragma unroll
    for (int i = 0; i < N_TILES; ++i) {
      const uint8_t *unit = act + i * (8 * act_row_bytes(NNTR_Q4_0));
      const uint4 x[2] = {act_frag<true>(unit, 2 * h, 8, lane), act_frag<true>(unit, 2 * h + 1, 8, lane)};
      const float4 d0 = act_d4(unit, 2 * t, h), d1 = act_d4(unit, 2 * t + 1, h);
      const float da[4][2] = {{d0.x, d1.x}, {d0.y, d1.y}, {d0.z, d1.z}, {d0.w, d1.w}};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float v[4];
        q40_block(v, q[j], (j & 1) ? x[j >> 1].z : x[j >> 1].x, (j & 1) ? x[j >> 1].w : x[j >> 1].y);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          acc[i][c] = __fmaf_rn(v[c], __fmul_rn(dw[j][c >> 1], da[j][c & 1]), acc[i][c]);
      }
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
constexpr int ROWS_WARPS = 4;
constexpr int ROWS_W = ROWS_WARPS * 2 * (int)sizeof(BlockQ4Kx8); // the weights of a unit: 8 row groups (Q4_0: 8 blocks of 144)

__device__ int g_mma_status = 0;

template <int NT, int STAGES> struct RowsShared { // STAGES: units in flight per CTA
  alignas(16) uint8_t w[STAGES][ROWS_W];
  alignas(16) uint8_t act[STAGES][NT * 8 * act_row_bytes(NNTR_Q4_K)];
  alignas(8) unsigned long long full[STAGES], empty[STAGES];
  int abort_flag;
};

template <int QT, int NT, bool GROUPED, bool TH8, int STAGES>
__global__ void __launch_bounds__(ROWS_WARPS * 32, NT == 4 ? 3 : 4) gemm_mma_rows_kernel(const MmaArgs a) {
  extern __shared__ __align__(16) uint8_t rows_smem[];
  RowsShared<NT, STAGES> &sh = *reinterpret_cast<RowsShared<NT, STAGES> *>(rows_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int n_groups = a.N / 8, group0 = blockIdx.y * (2 * ROWS_WARPS), groups = min(2 * ROWS_WARPS, n_groups - group0);
  // this warp's two row groups inside the CTA's (past the end of N the last group is repeated and not stored)
  const int wg0 = min(2 * warp, groups - 1), wg1 = min(2 * warp + 1, groups - 1);
  const int nb = a.nb;
  Tile tl;
  tl.z = GROUPED ? blockIdx.z : 0;
  if (GROUPED)
    pdl_wait(); // tables and activation tiles come from the kernels before
  if (!find_tile<NT>(tl, a, blockIdx.x, GROUPED))
    return;
  if (GROUPED && (reinterpret_cast<uintptr_t>(tl.W) & 15)) { // from a table in device memory: not seen by the launcher
    if (tid == 0)
      atomicExch(&g_mma_status, NNTR_CUDA_ERR_INVALID);
    return;
  }
  const int nt = (tl.rows + 7) >> 3, th = TH8 ? 8 : a.th;
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
  /* thread 0: the copies of unit b, weights and activations apart so that the first weights need not wait for the
   * kernel that writes the activations */
  auto unit_bytes = [&](int b) { return QT == NNTR_Q4_K ? (int)sizeof(BlockQ4Kx8) : min(8, a.nblk - 8 * b) * (int)sizeof(BlockQ40x8); };
  auto fetch_w = [&](int b) {
    const int s = b % STAGES, bytes = unit_bytes(b);
    const size_t row = QT == NNTR_Q4_K ? (size_t)nb * sizeof(BlockQ4Kx8) : (size_t)a.nblk * sizeof(BlockQ40x8);
    const uint8_t *src = static_cast<const uint8_t *>(tl.W) + (size_t)group0 * row + (size_t)b * sizeof(BlockQ4Kx8);
    mbar_expect_tx(full0 + 8 * s, groups * bytes + nt * th * act_row_bytes(QT));
    for (int i = 0; i < groups; ++i)
      bulk_g2s(smem_u32(sh.w[s]) + i * (int)sizeof(BlockQ4Kx8), src + i * row, bytes, full0 + 8 * s);
  };
  auto fetch_act = [&](int b) {
    const int s = b % STAGES;
    for (int i = 0; i < nt; ++i)
      bulk_g2s(smem_u32(sh.act[s]) + i * (8 * act_row_bytes(QT)), act_unit<QT>(a.act, tl.act_tile + i, th, nb, b),
               th * act_row_bytes(QT), full0 + 8 * s);
  };
  auto wait = [&](uint32_t bar, int use) {
    return mbar_wait_bounded(bar, use & 1, abort_flag, &g_mma_status, 1u << 22, 2048);
  };
  if (tid == 0) {
    for (int b = 0; b < STAGES - 1 && b < nb; ++b)
      fetch_w(b);
    if (!GROUPED)
      pdl_wait(); // only this thread reads what the kernel before wrote
    for (int b = 0; b < STAGES - 1 && b < nb; ++b)
      fetch_act(b);
  }
  float acc[NT][4], accm[QT == NNTR_Q4_K ? NT : 1][4];
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      acc[i][c] = 0.f;
      if constexpr (QT == NNTR_Q4_K)
        accm[i][c] = 0.f;
    }
  bool ok = true;
  for (int b = 0; b < nb; ++b) {
    // refill the slot that unit b - 1 left, then wait for this unit's own data
    if (tid == 0 && b + STAGES - 1 < nb) {
      if (b > 0)
        ok = wait(empty0 + 8 * ((b - 1) % STAGES), (b - 1) / STAGES);
      if (ok) {
        fetch_w(b + STAGES - 1);
        fetch_act(b + STAGES - 1);
      }
    }
    const int s = b % STAGES;
    ok = ok && wait(full0 + 8 * s, b / STAGES);
    if (!(ok = __all_sync(FULL, ok)))
      break;
    const uint8_t *act = sh.act[s];
    if constexpr (QT == NNTR_Q4_K) {
      const BlockQ4Kx8 *w0 = reinterpret_cast<const BlockQ4Kx8 *>(sh.w[s]) + wg0,
                       *w1 = reinterpret_cast<const BlockQ4Kx8 *>(sh.w[s]) + wg1;
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
      const BlockQ40x8 *w0 = reinterpret_cast<const BlockQ40x8 *>(sh.w[s] + wg0 * sizeof(BlockQ4Kx8)),
                       *w1 = reinterpret_cast<const BlockQ40x8 *>(sh.w[s] + wg1 * sizeof(BlockQ4Kx8));
      with_tiles<NT>(nt, [&](auto N) { q40_unit<decltype(N)::value>(acc, w0, w1, act, n, g, t, lane); });
    }
    // every lane's loads have been performed before the slot is given back (loads_before_refill() does the same here and costs 0.4 %
    // of the grouped products)
    __threadfence_block();
    __syncwarp();
    if (lane == 0)
      mbar_arrive(empty0 + 8 * s);
  }
  if (!ok) { // a wait ran out: give the copies in flight time to land in this CTA's shared memory
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
    return;
  }
#pragma unroll
  for (int i = 0; i < NT; ++i)
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const int m = 8 * i + 2 * t + k;
      if (m < tl.rows) {
        float *out = out_row(a, tl, m, GROUPED) + (size_t)(group0 + 2 * warp) * 8 + g;
#pragma unroll
        for (int row = 0; row < 2; ++row)
          if (2 * warp + row < groups) {
            const int c = 2 * row + k;
            out[8 * row] = QT == NNTR_Q4_K ? __fsub_rn(acc[i][c], accm[QT == NNTR_Q4_K ? i : 0][c]) : acc[i][c];
          }
      }
    }
}

/* ------------------------------------------- eight warps along K, one tile */
constexpr int KS_WARPS = 8;
constexpr int KS_BUF = KS_WARPS * 2 * 128 * 16;          // terms of one step: [unit][half][output] float4
constexpr int KS_DW = KS_WARPS * 16 * 8 * 4;             // [unit][row][8] floats (Q4_K uses two of them)
constexpr int KS_DA = KS_WARPS * 8 * 8 * 4;              // [unit][activation row][8] floats (Q4_K uses one)
constexpr int KS_SMEM = 2 * (KS_BUF + KS_DW + KS_DA);

template <int QT, int NT, bool GROUPED, bool TH8>
__global__ void __launch_bounds__(KS_WARPS * 32) gemm_mma_ksplit_kernel(const MmaArgs a) {
  extern __shared__ __align__(16) uint8_t ks_smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int rt = blockIdx.y, nb = a.nb;
  const bool second = rt * 16 + 8 < a.N;
  const int per = (nb + KS_WARPS - 1) / KS_WARPS; // rounds
  const int upr = (nb + per - 1) / per;           // units per round, the same in every round but the last
  Tile tl;
  tl.z = GROUPED ? blockIdx.z : 0;
  Q4KRaw rk;
  Q40Raw r0;
  auto load = [&](int b) {
    if constexpr (QT == NNTR_Q4_K) {
      const BlockQ4Kx8 *w0 = static_cast<const BlockQ4Kx8 *>(tl.W) + (size_t)(2 * rt) * nb;
      q4k_load(rk, w0 + b, (second ? w0 + nb : w0) + b, g, t);
    } else {
      const BlockQ40x8 *w0 = static_cast<const BlockQ40x8 *>(tl.W) + (size_t)(2 * rt) * a.nblk;
      q40_load(r0, w0 + 8 * b, (second ? w0 + a.nblk : w0) + 8 * b, min(8, a.nblk - 8 * b), g, t);
    }
  };
  if constexpr (!GROUPED) { // the weights do not depend on the quantizer's kernel: fetched while it runs
    find_tile<NT>(tl, a, blockIdx.x, false);
    if (warp < upr)
      load(warp);
    pdl_wait();
  } else {
    pdl_wait();
    if (!find_tile<NT>(tl, a, blockIdx.x, true))
      return;
    if (warp < upr)
      load(warp);
  }
  const int nt = (tl.rows + 7) >> 3, th = TH8 ? 8 : a.th;
  // the chain of this thread: output o of the tile (row g + 8 * (o / 64), activation row 2t + (o / 32) % 2 with g, t of
  // lane o % 32); Q4_K: threads 128.. add the mins term
  const int o = tid & 127, kind = tid >> 7, oq = o >> 5, og = (o & 31) >> 2, ot = o & 3;
  const int orow = og + 8 * (oq >> 1), oact = 2 * ot + (oq & 1);
  float acc[NT];
#pragma unroll
  for (int i = 0; i < NT; ++i)
    acc[i] = 0.f;
  int step = 0;
  for (int rd = 0; rd < per; ++rd) {
    const int b = rd * upr + warp;
    const bool have = warp < upr && b < nb;
    const int n_units = min(upr, nb - rd * upr);
    float *dws = reinterpret_cast<float *>(ks_smem + 2 * KS_BUF + (rd & 1) * KS_DW);
    Q4KScales sc;
    Q4KFactors f;
    uint2 qk[4][2];
    uint32_t q0[8][2];
    int n = 0;
    if (have) {
      if constexpr (QT == NNTR_Q4_K) {
        q4k_scales(sc, rk.head, rk.d, g, lane);
        q4k_factors(f, sc);
#pragma unroll
        for (int p = 0; p < 4; ++p)
          qk[p][0] = rk.q[p][0], qk[p][1] = rk.q[p][1];
        if (t == 0) {
#pragma unroll
          for (int row = 0; row < 2; ++row)
            *reinterpret_cast<float2 *>(dws + (warp * 16 + g + 8 * row) * 8) = make_float2(sc.dw[row], sc.dm[row]);
        }
      } else {
        n = min(8, a.nblk - 8 * b);
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int row = 0; row < 2; ++row) {
            q0[j][row] = r0.q[j][row];
            if (t == (j >> 1)) // a missing block of the last unit: scale 0, the chain adds nothing
              dws[(warp * 16 + g + 8 * row) * 8 + j] = j < n ? half_bits_to_float(r0.d[j][row]) * 0.0625f : 0.f;
          }
      }
      if (rd + 1 < per && b + upr < nb)
        load(b + upr);
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) {
      if (i >= nt)
        break;
      float4 *buf = reinterpret_cast<float4 *>(ks_smem + (step & 1) * KS_BUF);
      float *das = reinterpret_cast<float *>(ks_smem + 2 * (KS_BUF + KS_DW) + (step & 1) * KS_DA);
      ++step;
      if (have) {
        const uint8_t *unit = act_unit<QT>(a.act, tl.act_tile + i, th, nb, b);
        float4 *mine = buf + warp * 256 + lane;
        if constexpr (QT == NNTR_Q4_K) {
          ActQ4K x;
          act_load<TH8>(x, unit, th, lane);
          if (g == 0)
            das[(warp * 8 + 2 * t) * 8] = x.d.x, das[(warp * 8 + 2 * t + 1) * 8] = x.d.y;
          const uint32_t bs0 = sum_halves<0>(x.sums), bs1 = sum_halves<1>(x.sums);
          float v[4][4], j[4][4];
#pragma unroll
          for (int p = 0; p < 4; ++p) {
            const uint32_t lo[4] = {qk[p][0].x & 0x0f0f0f0fu, qk[p][1].x & 0x0f0f0f0fu, qk[p][0].y & 0x0f0f0f0fu, qk[p][1].y & 0x0f0f0f0fu};
            const uint32_t hi[4] = {qk[p][0].x & 0xf0f0f0f0u, qk[p][1].x & 0xf0f0f0f0u, qk[p][0].y & 0xf0f0f0f0u, qk[p][1].y & 0xf0f0f0f0u};
            q4k_pair(v[p], lo, hi, x.b[p], f.s0[p], f.s1[p]);
            mma_f16_k8(j[p], sc.mn[2 * (p >> 1)], sc.mn[2 * (p >> 1) + 1], (t >> 1) == (p & 1) ? (p < 2 ? bs0 : bs1) : 0u);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            mine[32 * c] = make_float4(v[0][c], v[1][c], v[2][c], v[3][c]);
            mine[128 + 32 * c] = make_float4(j[0][c], j[1][c], j[2][c], j[3][c]);
          }
        } else {
          ActQ40 x;
          act_load<TH8>(x, unit, th, lane);
          if (g == 0) {
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
              for (int j = 0; j < 8; ++j)
                das[(warp * 8 + 2 * t + c) * 8 + j] = x.d[c][j];
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            float v[4][4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 bb = x.b[2 * h + (j >> 1)];
              const uint32_t w0 = q0[4 * h + j][0], w1 = q0[4 * h + j][1];
              const uint32_t qq[4] = {(w0 << 4) & 0xf0f0f0f0u, (w1 << 4) & 0xf0f0f0f0u, w0 & 0xf0f0f0f0u, w1 & 0xf0f0f0f0u};
              q40_block(v[j], qq, (j & 1) ? bb.z : bb.x, (j & 1) ? bb.w : bb.y);
            }
#pragma unroll
            for (int c = 0; c < 4; ++c)
              mine[128 * h + 32 * c] = make_float4(v[0][c], v[1][c], v[2][c], v[3][c]);
          }
        }
      }
      __syncthreads();
      // the chains: terms in ascending K order
      if constexpr (QT == NNTR_Q4_K) {
        const bool four = !GROUPED && tl.pos + 8 * i + oact < a.M4;
        for (int u = 0; u < n_units; ++u) {
          const float4 v = buf[u * 256 + 128 * kind + o];
          const float s = __fmul_rn(dws[(u * 16 + orow) * 8 + kind], das[(u * 8 + oact) * 8]);
          if (four) {
            acc[i] = __fmaf_rn(v.x, s, acc[i]);
            acc[i] = __fmaf_rn(v.y, s, acc[i]);
            acc[i] = __fmaf_rn(v.z, s, acc[i]);
            acc[i] = __fmaf_rn(v.w, s, acc[i]);
          } else { // one rounding of the exact sum: the halves stay below 2^24
            acc[i] = __fmaf_rn(__fadd_rn(v.x + v.y, v.z + v.w), s, acc[i]);
          }
        }
      } else if (kind == 0) {
        for (int u = 0; u < n_units; ++u) {
          const float4 v0 = buf[u * 256 + o], v1 = buf[u * 256 + 128 + o];
          const float4 *dw = reinterpret_cast<const float4 *>(dws + (u * 16 + orow) * 8);
          const float4 *da = reinterpret_cast<const float4 *>(das + (u * 8 + oact) * 8);
          const float4 w0 = dw[0], w1 = dw[1], a0 = da[0], a1 = da[1];
          acc[i] = __fmaf_rn(v0.x, __fmul_rn(w0.x, a0.x), acc[i]);
          acc[i] = __fmaf_rn(v0.y, __fmul_rn(w0.y, a0.y), acc[i]);
          acc[i] = __fmaf_rn(v0.z, __fmul_rn(w0.z, a0.z), acc[i]);
          acc[i] = __fmaf_rn(v0.w, __fmul_rn(w0.w, a0.w), acc[i]);
          acc[i] = __fmaf_rn(v1.x, __fmul_rn(w1.x, a1.x), acc[i]);
          acc[i] = __fmaf_rn(v1.y, __fmul_rn(w1.y, a1.y), acc[i]);
          acc[i] = __fmaf_rn(v1.z, __fmul_rn(w1.z, a1.z), acc[i]);
          acc[i] = __fmaf_rn(v1.w, __fmul_rn(w1.w, a1.w), acc[i]);
        }
      }
    }
  }
  float *fin = reinterpret_cast<float *>(ks_smem);
  if constexpr (QT == NNTR_Q4_K) {
    __syncthreads(); // the last chains have read the buffers
    if (kind)
#pragma unroll
      for (int i = 0; i < NT; ++i)
        fin[i * 128 + o] = acc[i];
    __syncthreads();
  }
  if (kind == 0 && (orow < 8 || second)) {
#pragma unroll
    for (int i = 0; i < NT; ++i)
      if (8 * i + oact < tl.rows) {
        float *out = out_row(a, tl, 8 * i + oact, GROUPED) + rt * 16 + orow;
        *out = QT == NNTR_Q4_K ? __fsub_rn(acc[i], fin[i * 128 + o]) : acc[i];
      }
  }
}

/* ----------------------------------------------------- activation tiles */
/** fp32 rows -> activation tiles; one warp per (row, unit). perm != nullptr: position p of an expert's range is the row
 *  perm[p] / a_div of x and goes to the expert's own tiles. */
template <int QT>
__global__ void __launch_bounds__(256)
act_tiles_kernel(const float *__restrict__ x, int64_t ldx, uint8_t *__restrict__ act, int M, int M4, int nb, int K, int th,
                 const int *__restrict__ perm, const int *__restrict__ idx, const int *__restrict__ off,
                 const int *__restrict__ act_off, int a_div) {
  pdl_launch_dependents();
  const int lane = threadIdx.x & 31;
  const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (w >= (int64_t)M * nb)
    return;
  const int pos = (int)(w / nb), b = (int)(w - (int64_t)pos * nb);
  int row = pos, tile = pos / th, i = pos - tile * th;
  if (perm) {
    pdl_wait();
    const int pair = perm[pos], e = idx[pair];
    row = pair / a_div;
    i = pos - off[e];
    tile = act_off[e] + (i >> 3);
    i &= 7;
  }
  uint8_t *unit = act_unit<QT>(act, tile, th, nb, b);
  const float *src = x + (int64_t)row * ldx + (int64_t)b * QK_K + lane * 8;
  if constexpr (QT == NNTR_Q4_K) {
    put_q8K(unit, th, i, q8K_quantize_warp(*reinterpret_cast<const float4 *>(src), *reinterpret_cast<const float4 *>(src + 4),
                                           lane, row < M4 ? 1 : 0),
            lane);
  } else {
    float4 v0 = make_float4(0.f, 0.f, 0.f, 0.f), v1 = v0;
    if (b * QK_K + lane * 8 < K) { // blocks past K are zeros
      v0 = *reinterpret_cast<const float4 *>(src);
      v1 = *reinterpret_cast<const float4 *>(src + 4);
    }
    put_q80(unit, th, i, q80_quantize_warp(v0, v1), lane);
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
int run_tiles(const MmaArgs &a, unsigned tiles, unsigned z, bool ksplit, bool shallow, cudaStream_t st) {
  const unsigned row_tiles = (unsigned)((a.N + 15) / 16);
  static bool attr_set[64] = {};
  int dev = 0;
  NNTR_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && !attr_set[dev]) {
    NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, KS_SMEM));
    NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_mma_rows_kernel<QT, NT, GROUPED, TH8, 3>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(RowsShared<NT, 3>)));
    attr_set[dev] = true;
  }
  const dim3 rows_grid(tiles, (row_tiles + ROWS_WARPS - 1) / ROWS_WARPS, z);
  cudaError_t e;
  if (ksplit) {
    e = launch(gemm_mma_ksplit_kernel<QT, NT, GROUPED, TH8>, dim3(tiles, row_tiles, z), KS_WARPS * 32, KS_SMEM, st, a);
  } else {
    auto kernel = gemm_mma_rows_kernel<QT, NT, GROUPED, TH8, 3>;
    size_t smem = sizeof(RowsShared<NT, 3>);
    if constexpr (QT == NNTR_Q4_0 && NT == 1 && GROUPED) // 23 KB: no opt-in
      if (shallow)
        kernel = gemm_mma_rows_kernel<QT, NT, GROUPED, TH8, 2>, smem = sizeof(RowsShared<NT, 2>);
    e = launch(kernel, rows_grid, ROWS_WARPS * 32, smem, st, a);
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
  quantize<<<grid, 256, 0, st>>>(A, K, static_cast<uint8_t *>(ws), a.M, a.M4, a.nb, (int)K, a.th, nullptr, nullptr, nullptr,
                                 nullptr, 1);
  count_launch();
  NNTR_CHECK_CUDA(cudaGetLastError());
  const int nt = M <= 8 ? 1 : M <= 16 ? 2 : 4;
  const unsigned tiles = (M + 8 * nt - 1) / (8 * nt);
  // a warp per 16 x 8nt tile fills the machine from about 8 warps per SM up; below, the warps of a CTA share the tile. Weights
  // that are not 16-byte aligned cannot be fetched by bulk copies: the shared tile's loads of at most 8 bytes take them all.
  const bool ksplit = (uint64_t)tiles * ((N + 15) / 16) < 8u * (unsigned)sm_count() || (reinterpret_cast<uintptr_t>(B) & 15);
  if (a.th < 8)
    return run_tiles<NNTR_Q4_K, 1, false, false>(a, tiles, 1, ksplit, false, st);
#define NNTR_MMA_RUN(QT)                                                                                               \
  (nt == 1   ? run_tiles<QT, 1, false, true>(a, tiles, 1, ksplit, false, st)                                                  \
   : nt == 2 ? run_tiles<QT, 2, false, true>(a, tiles, 1, ksplit, false, st)                                                  \
             : run_tiles<QT, 4, false, true>(a, tiles, 1, ksplit, false, st))
  return qtype == NNTR_Q4_K ? NNTR_MMA_RUN(NNTR_Q4_K) : NNTR_MMA_RUN(NNTR_Q4_0);
#undef NNTR_MMA_RUN
}

int grouped_tile_rows(unsigned pairs, unsigned n_experts) {
  // tiles of 8, 16 or 32 rows: about what an expert gets, so that few experts need a second tile (which fetches the
  // expert's weights again) and short ones carry little padding
  return pairs <= 6 * n_experts ? 8 : pairs <= 12 * n_experts ? 16 : 32;
}

int launch_act_tiles_grouped(int qtype, const float *x, unsigned rows, unsigned K, void *act, const int *perm, const int *idx,
                             const int *off, const int *act_off, int a_div, cudaStream_t st) {
  const int nb = (int)((K + 255) / 256);
  const dim3 grid((unsigned)(((int64_t)rows * nb + 7) / 8));
  const auto kernel = qtype == NNTR_Q4_K ? act_tiles_kernel<NNTR_Q4_K> : act_tiles_kernel<NNTR_Q4_0>;
  const cudaError_t e = launch(kernel, grid, 256, 0, st, x, (int64_t)K, static_cast<uint8_t *>(act), (int)rows, 0, nb, (int)K,
                               8, perm, idx, off, act_off, a_div);
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
  const bool ksplit = (uint64_t)tiles * z * ((N + 15) / 16) < 8u * (unsigned)sm_count();
  // Q4_0's small tile: 55 registers, so shared memory sets the CTAs per SM, six with three units in flight and nine with two.
  // From a pair per expert up the grid is two and more waves of six, and nine win: 4 of 32 experts of 2880 x 2880, 8 tokens
  // 107 -> 100 us; 5 tokens (a wave and a half) 87.7 -> 89.3, so those keep three. Q4_K's tile is held to five by registers.
  // The line holds for experts of that size (7 tokens, below it: three in flight 109.8 us, two 102.6) and of half the width (8 / 12 /
  // 16 tokens 75.9 / 82.2 / 85.3 us with three, 70.9 / 74.9 / 77.5 with two). Elsewhere two in flight cost a little: 2 of 16 experts of
  // 4096 x 4096, 12 tokens 117.3 -> 120.0; 4 of 64 experts of 1024 x 2880, 16 / 32 tokens 85.3 / 101 -> 88.8 / 103.
  const bool shallow = pairs >= (unsigned)n_experts;
#define NNTR_MMA_RUN(QT)                                                                                               \
  (tile_rows == 8    ? run_tiles<QT, 1, true, true>(a, tiles, z, ksplit, shallow, st)                                           \
   : tile_rows == 16 ? run_tiles<QT, 2, true, true>(a, tiles, z, ksplit, shallow, st)                                           \
                     : run_tiles<QT, 4, true, true>(a, tiles, z, ksplit, shallow, st))
  if (qtype == NNTR_Q4_K)
    return NNTR_MMA_RUN(NNTR_Q4_K);
  if (qtype == NNTR_Q4_0)
    return NNTR_MMA_RUN(NNTR_Q4_0);
#undef NNTR_MMA_RUN
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
