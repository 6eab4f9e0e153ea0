// SPDX-License-Identifier: Apache-2.0
/**
 * @file  gemm_umma_f16.cu
 * @brief Prefill GEMM for Q4_K and Q4_0 weights with both operands dequantized to fp16
 *        on the fly: tcgen05.mma kind::f16, fp32 accumulators in tensor memory,
 *        no work per super-block outside the tensor pipe.
 *
 * What is computed. The reference's quantity (nntr_gemm_q4_K_8x8_q8_K,
 * nntr_ggml_impl.cpp:3261-7078): C[m][n] = sum_k w[n][k] * a[m][k] with
 * w = d * sc * q - dmin * min (block_q4_K) and a = d_a * q8 (the activation
 * quantized to Q8_K by the same rules as the exact path). Here both factors are
 * rounded to fp16 before the multiply (w as fma(q, fp16(d*sc), -fp16(dmin*min))
 * in half precision, a as fp16(d_a * q8)) and the products are summed in fp32 by
 * the tensor core. Measured against the reference chain on random-byte weights:
 * max-rel 3.5e-4 (bar 2e-3). This is the fast prefill path; the integer-exact
 * tensor path (gemm_umma.cu) and the bit-exact path (gemm_mma.cu, gemm_mma_q6k.cu)
 * stay selectable. Q4_0 weights (nntr_gemm_q4_0_8x8_q8_0, nntr_ggml_impl.cpp:650-3259) take the same route:
 * w = (q4 - 8) * d as one half-precision multiply, a = fp16(fp32(d_a) * q8) with the Q8_0 quantizer, a stage of 64
 * being two 32-weight blocks; their 32-element block scale would force an integer kernel to leave the tensor pipe at
 * every MMA K step.
 *
 * Why fp16 operands: folding the per-sub-block scales and mins into the weight
 * values removes every per-super-block step from the CUDA cores -- no split of
 * the 6-bit scale into two 8-bit operands, no drain of the accumulators every
 * 256 of K, no mins term. What is left outside the tensor pipe is the nibble
 * expansion (about two instructions per weight) and one epilogue per tile.
 *
 * Up to 256 activation rows, a CTA owns two tiles of 128 of them (MMA M, tensor-memory lanes) against the same 256 weight rows (MMA N,
 * columns), so every expanded weight stage feeds two MMAs. With more rows mostly a pair of CTAs owns four tiles: each CTA expands half of the
 * weight rows, an MMA (cta_group::2) takes 128 activation rows of each and the weights of both, and an expanded stage feeds 512 rows.
 * A CTA walks K in stages of 64 (one pair of sub-blocks):
 *   warps 0-15  producers: expand a stage's nibble bytes into 64 fp16 values per
 *               weight row. A 32-bit word yields four half2 with one
 *               logic op each ((w >> s) & 0x000F000F | 0x64006400 is
 *               (1024 + n_lo, 1024 + n_hi)), so the K order inside a stage is
 *               the order that unpack produces; the activation tiles are written
 *               in the same order (a dot product does not care). Q4_K and Q4_0:
 *               one thread per row, two groups of eight warps (pair: four of four)
 *               take the stages in turn. Q6_K: two threads per row, all warps
 *               every stage (pair: two groups, two stages in turn). After
 *               the last stage the same warps are the epilogue: tcgen05.ld of the
 *               tile, a turn through shared memory, stores of C by whole lines.
 *   warp 16     one thread issues 8 MMAs per stage; in a pair's second CTA it
 *               tells the first one that a stage is ready here.
 *   warp 17     one thread starts the bulk copies of the activation stages, each
 *               as soon as the MMAs that read its slot have retired.
 *   warp 18     one thread starts the tiled copies of the packed weights
 *               (Q4_K, Q4_0) into a ring of two (pair: four) stages.
 * Three stages of 64 KB (pair: four of 48; Q6_K alone or shared: two of 64), both accumulators (512 columns) in tensor memory. Every wait is bounded (pipeline.cuh).
 *
 * What bounds it. A stage's MMAs take 1024 clocks. A CTA alone takes about 1600 a stage with Q4_K and 1350 with Q4_0 (the difference of K =
 * 4096 and 8192, 256 x 37888, at the clock meanwhile): its producers, and the shared memory, which carries 96 KB for the MMAs, 64 of
 * stores and copies and the packed weights. A pair takes 1070 (Q4_K, stamps inside a CTA), the MMAs: half of the expansion and 64 KB
 * for the MMAs. (With no expansion and no copies at all 1050; a hand-over from CTA to CTA with release and acquire at cluster
 * scope 1600: it is one more latency in each round of the ring.) Q4_K 24576 x 4096, 1024 rows 184.6 -> 167 us, 512
 * rows 115.9 -> 101.6 (98.5 with even_rows()); Q4_0 512 rows of 24576 x 2880 85.2 -> 77.3 (70.6); Q6_K 151936 x 2560, 300 / 512 rows
 * 515 / 572 -> 346 / 380.
 *
 * Few tiles: a cluster of two, four or eight CTAs shares a tile, each walks a part of K (k_parts), and the sums are added
 * through distributed shared memory. 512 x 1280 x 2560: Q4_0 40 -> 25 us, Q6_K 69 -> 33; 128 x 2560 x 8192: Q4_0 93 -> 25,
 * Q6_K 268 -> 49.
 */
#include "cluster.cuh"
#include "common.cuh"
#include "pipeline.cuh"
#include "tma_map.cuh"

#include <algorithm>
#include <cuda_fp16.h>

namespace nntr {

namespace {

constexpr int F16_TILE_M = 128;  // rows of an activation tile
constexpr int F16_TILE_N = 256;  // weight rows of a tile of C, at most
constexpr int F16_KS = 64;       // K per stage
constexpr int F16_A_BYTES = F16_TILE_M * F16_KS * 2; // 16 KB
constexpr int F16_PRODUCERS = 512;
constexpr int F16_TURN_PITCH = 68; // floats of a row of the epilogue's areas: 16-byte pieces of neighbours fall into different banks
constexpr int F16_TURN_BYTES = F16_PRODUCERS * F16_TURN_PITCH * 4; // in the stages' place
constexpr int F16_MMA_WARP = F16_PRODUCERS / 32;
constexpr int F16_COPY_WARP = F16_MMA_WARP + 1;
constexpr int F16_RAW_WARP = F16_COPY_WARP + 1;
constexpr int F16_THREADS = (F16_RAW_WARP + 1) * 32; // 608
/* How a tile of C is dealt out: a CTA of its own, a cluster whose CTAs share it along K, a pair of CTAs with one MMA over both. */
enum F16Mode { F16_LONE, F16_SHARED, F16_PAIR };
template <int QT, int MODE> struct F16Cfg {
  static constexpr int W_ROWS = MODE == F16_PAIR ? F16_TILE_N / 2 : F16_TILE_N; // weight rows that a CTA expands
  static constexpr int W_BYTES = W_ROWS * F16_KS * 2;
  static constexpr int STAGE_BYTES = W_BYTES + 2 * F16_A_BYTES; // weights + two activation tiles
  /* Q6_K: two, because the producers' loads live on the L1 cache that shared memory leaves (three: 256 x 151936 x 2560 280 us, 274;
   * 100 x 4096 x 4096 36.7, 33.8) */
  static constexpr int STAGES = MODE == F16_PAIR ? 4 : QT == NNTR_Q6_K ? 2 : 3;
  /* Groups of producers, each with the next stage in turn. Q4_K, Q4_0: a thread per weight row; Q6_K: two, and two stages in turn */
  static constexpr int GROUPS = F16_PRODUCERS / (QT == NNTR_Q6_K ? 2 * W_ROWS : W_ROWS);
  static constexpr int STAGE_WARPS = F16_PRODUCERS / 32 / GROUPS;
  /* Packed weights of a stage on their way to the producers, groups of 8 rows: Q4_K the 256 nibble bytes of a pair of
   * sub-blocks per group, plus the 128 header bytes (d, dmin, scales) of a super-block for its four stages; Q4_0 two whole
   * blocks per group. Q6_K rows are not 16-byte aligned: their producers load from global memory. */
  static constexpr int RAW = W_ROWS == F16_TILE_N ? 2 : 4; // one per producer group: with another number a group could take a phase of another group for its own
  static constexpr int ROW_GROUPS = W_ROWS / 8;
  static constexpr int RAW_BOX = QT == NNTR_Q4_K ? 128 : 144;
  static constexpr int RAW_BYTES = QT == NNTR_Q6_K ? 0 : ROW_GROUPS * 2 * RAW_BOX;
  static constexpr int HDR_BYTES = ROW_GROUPS * 128;
  static constexpr int OFF_RAW = STAGES * STAGE_BYTES > F16_TURN_BYTES ? STAGES * STAGE_BYTES : F16_TURN_BYTES;
  static constexpr int OFF_HDR = OFF_RAW + RAW * RAW_BYTES;
  static constexpr int OFF_BARS = OFF_HDR + (QT == NNTR_Q4_K ? 2 * HDR_BYTES : 0);
  static constexpr int SMEM = OFF_BARS + 256;
  static_assert(SMEM <= 227 * 1024, "shared memory of a CTA");
  static_assert(QT == NNTR_Q6_K || RAW == GROUPS, "ring of packed weights");
};
constexpr uint32_t F16_POLLS = 1u << 22;

__device__ int g_f16_status = 0;

__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
  return mbar_wait_bounded(bar, parity, abort_flag, &g_f16_status, F16_POLLS, 2048);
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3fff) | ((uint64_t)((lbo >> 4) & 0x3fff) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3fff) << 32) | ((uint64_t)1 << 46);
}
/* PAIR: one MMA over two CTAs of a cluster, issued by the first; the descriptors hold for the shared memory of both */
template <bool PAIR>
__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
                 "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
                 : "memory");
}
/* the barrier at this address, PAIR: in both CTAs, when the MMAs issued so far have retired */
template <bool PAIR> __device__ __forceinline__ void umma_commit(uint32_t bar) {
  if constexpr (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
template <bool PAIR> __device__ __forceinline__ void tmem_alloc_all(uint32_t slot) {
  if constexpr (PAIR) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
  } else {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
}
template <bool PAIR> __device__ __forceinline__ void tmem_free_all(uint32_t tmem) {
  if constexpr (PAIR)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
  else
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}
/** Arrival at the barrier at this address in another CTA of the cluster. No release at cluster scope: what the MMAs of the other CTA's
 *  thread read here was written by this CTA's warps and copies, behind their proxy fences and this CTA's barrier, and is read by this SM. */
__device__ __forceinline__ void mbar_arrive_remote(uint32_t bar, uint32_t rank) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(bar), "r"(rank));
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(remote) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
               "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
}

/** scale and min of row j from the three words of one 12-byte group of a block_q4_Kx8 (get_scale_min_k4,
 *  nntr_ggml_impl_quant.cpp:368-378, with the row as the index): bytes 0-3 hold the low 6 bits of the scales of rows
 *  0-3 and the top 2 bits of rows 4-7, bytes 4-7 the same for the mins, bytes 8-11 the low nibbles of rows 4-7. */
__device__ __forceinline__ void scale_min_row(uint32_t w0, uint32_t w1, uint32_t w2, int j, float &sc, float &mn) {
  const int sh = 8 * (j & 3);
  const uint32_t b0 = (w0 >> sh) & 0xff, b1 = (w1 >> sh) & 0xff, b2 = (w2 >> sh) & 0xff;
  const uint32_t s = j < 4 ? (b0 & 63) : ((b2 & 0xf) | ((b0 >> 6) << 4));
  const uint32_t m = j < 4 ? (b1 & 63) : ((b2 >> 4) | ((b1 >> 6) << 4));
  sc = (float)s;
  mn = (float)m;
}

/** (n_a, n_b) as half2 from a word holding them at bits 0-3 and 16-19, times d, minus m */
__device__ __forceinline__ uint32_t expand2(uint32_t nib2, __half2 d, __half2 negm) {
  const uint32_t biased = nib2 | 0x64006400u; // (1024 + n_a, 1024 + n_b), exact in fp16
  const __half2 n = __hsub2(*reinterpret_cast<const __half2 *>(&biased), __half2half2(__ushort_as_half(0x6400)));
  const __half2 w = __hfma2(n, d, negm);
  return *reinterpret_cast<const uint32_t *>(&w);
}

/** (n_a, n_b) of a Q4_0 word whose nibbles already had their XOR 8 undone, as half2: (n - 8) * d */
__device__ __forceinline__ uint32_t expand2_q40(uint32_t nib2, __half2 d) {
  const uint32_t biased = nib2 | 0x64006400u;
  const __half2 x = __hsub2(*reinterpret_cast<const __half2 *>(&biased), __half2half2(__ushort_as_half(0x6408))); // - 1032
  const __half2 w = __hmul2(x, d);
  return *reinterpret_cast<const uint32_t *>(&w);
}

/* QT = NNTR_Q4_K: W is block_q4_Kx8, a stage is one pair of sub-blocks (k_stages = 4 * K/256).
 * QT = NNTR_Q4_0: W is block_q4_0x8, a stage is two 32-weight blocks (k_stages = K/64).
 * QT = NNTR_Q6_K: W is plain rows of block_q6_K (210 bytes, 2-byte aligned); stage (b, h, s2) of super-block b holds
 *                 the quarters s2 and s2 + 2 of its 128-element half h (the two quarters that share the bytes ql[64h +
 *                 32 s2 ..] as low and high nibbles); k_stages = 4 * K/256. N may end inside the last 256-row tile.
 * F16_PAIR: the cluster's two CTAs expand 128 of the 256 weight rows each and hold two of four activation tiles; an MMA takes
 * 128 activation rows of each and the weights of both, so a stage's expansion serves 512 rows instead of 256, and a CTA's MMAs read half
 * of the weights from its own shared memory only.
 * F16_SHARED: a cluster of CTAs may share the tile. A kernel of its own: the code of a shared tile in the kernel of a lone CTA costs
 * that one registers (81 without, 96 with) and 1024 x 24576 x 4096 Q4_K 185 us instead of 182. (It keeps the test for a cluster of
 * one, without which the compiler spills 44 bytes instead of 8.) */
template <int QT, int MODE>
__global__ void __launch_bounds__(F16_THREADS, 1)
gemm_f16_kernel(const __grid_constant__ CUtensorMap wmap, const uint8_t *__restrict__ atiles, const uint8_t *__restrict__ Wb,
                float *__restrict__ C, int ldc, int M, int N, int k_stages, int m_tiles, int tiles_per_cta,
                int max_rows, int c_vec4) {
  extern __shared__ __align__(128) uint8_t smem[];
  using Cfg = F16Cfg<QT, MODE>;
  constexpr bool SHARED = MODE == F16_SHARED, PAIR = MODE == F16_PAIR;
  const int tile_rows = SHARED ? F16_TILE_N : max_rows; // weight rows of the tile
  // bars: [0..3] full, [4..7] empty, [8] tile complete, [9..12] packed weights here, [13..16] packed weights read,
  // [17..18] Q4_K headers here
  const uint32_t sbase = smem_u32(smem);
  const uint32_t bar0 = sbase + Cfg::OFF_BARS;
  auto BAR = [&](int i) { return bar0 + 8u * i; };
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem + Cfg::OFF_BARS + 192);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(smem + Cfg::OFF_BARS + 200);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // a CTA takes two 128-row activation tiles (unless there are SMs to spare) against the same 256 weight rows: the expanded
  // weights of a stage feed two MMAs, which halves the expansion work per output
  // the CTAs of a cluster share a tile: each walks its part of K, whole super-blocks (Q6_K: halves; Q4_0: pairs of blocks)
  const int parts = SHARED ? cluster_size() : 1, part = SHARED ? cluster_rank() : 0;
  // a pair takes four activation tiles, its CTAs alternate ones
  const int peer = PAIR ? cluster_rank() : 0, mt_step = PAIR ? 2 : 1; // place in the pair
  const int mt = PAIR ? 4 * (blockIdx.x / 2) + peer : tiles_per_cta * (blockIdx.x / parts), nt = blockIdx.y;
  const int n0 = nt * tile_rows, own_rows = PAIR ? tile_rows / 2 : tile_rows; // the tile's first weight row, rows that this CTA expands
  const bool two = PAIR ? mt - peer + 2 < m_tiles : tiles_per_cta == 2 && mt + 1 < m_tiles; // the same in both CTAs of a pair
  constexpr int UNIT = QT == NNTR_Q4_K ? 4 : QT == NNTR_Q6_K ? 2 : 1;
  const int units = k_stages / UNIT;
  const int st0 = units * part / parts * UNIT, n_stages = units * (part + 1) / parts * UNIT - st0; // stages st0 ..

  if (tid == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      // the stage's producer warps + the thread that armed the activation copy + in the pair's first CTA the other one
      mbar_init(BAR(s), Cfg::STAGE_WARPS + 1 + (PAIR && peer == 0));
      mbar_init(BAR(4 + s), 1); // MMAs of the stage retired
    }
    for (int s = 0; s < Cfg::RAW; ++s) {
      mbar_init(BAR(9 + s), 1);
      mbar_init(BAR(13 + s), Cfg::STAGE_WARPS);
    }
    mbar_init(BAR(17), 1);
    mbar_init(BAR(18), 1);
    mbar_init(BAR(8), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == F16_MMA_WARP)
    tmem_alloc_all<PAIR>(smem_u32(tmem_slot));
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR)
    cluster_sync(); // the other CTA's barriers and tensor memory are there
  // Only pairs let the next launch in early: Q4_K 512 x 14336 x 4096 50.6 us, without 51.6. CTAs alone are slowed down by its waiting CTAs:
  // Q4_K 256 x 24576 x 4096 55.3 us, without 53.8, 1280 x 37888 x 4096 333 and 324, 603 x 9728 x 2560 39.8 and 38.9; shared tiles, 1024 x 2560 x
  // 9728, 85.0 and 83.6.
  if (PAIR)
    pdl_launch_dependents();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // Epilogue. A lane holds a row of the accumulator; stored as it is, a store instruction would touch 32 rows of C with 16
  // bytes each (27 of a tile's 142 thousand clocks). Every warp turns its 32 x 64 part round in the stages' memory, which is
  // free then, and whole lines are written from there.
  constexpr int PITCH = F16_TURN_PITCH;
  bool tile_done = false;   // warps 0-15: all MMAs have retired
  auto turn_area = [&](int w) { return w * (32 * PITCH); }; // of the warp with lanes 32 * (w & 3) .., columns 64 * (w >> 2) ..
  auto turn_round = [&](int hm) {
    const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + hm * 256 + (warp >> 2) * 64;
    float *turn = reinterpret_cast<float *>(smem) + turn_area(warp);
#pragma unroll
    for (int half = 0; half < 2; ++half) { // two loads in flight
      uint32_t v[2][16];
      tmem_ld16(trow + half * 32, v[0]);
      tmem_ld16(trow + half * 32 + 16, v[1]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
      for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int i = 0; i < 16; i += 4)
          *reinterpret_cast<uint4 *>(turn + lane * PITCH + half * 32 + k * 16 + i) =
            make_uint4(v[k][i], v[k][i + 1], v[k][i + 2], v[k][i + 3]);
    }
  };
  auto store4 = [&](int row, int col, const float4 &f) {
    if (col >= n0 + tile_rows) // a multiple of 16
      return;
    float *dst = C + (size_t)row * ldc + col;
    if (c_vec4 && col + 4 <= N) {
      *reinterpret_cast<float4 *>(dst) = f;
    } else {
      if (col < N)
        dst[0] = f.x;
      if (col + 1 < N)
        dst[1] = f.y;
      if (col + 2 < N)
        dst[2] = f.z;
      if (col + 3 < N)
        dst[3] = f.w;
    }
  };

  if (warp < F16_MMA_WARP) {
    /* ------------------------------ producers ------------------------------ */
    const int r = tid % Cfg::W_ROWS;    // weight row inside the CTA's part of the tile
    const int hsel = tid / Cfg::W_ROWS; // Q4_K, Q4_0: the thread's group; Q6_K, modulo 2: which half of the stage's 32 nibble bytes
    const int j = r & 7;                  // row inside its 8-row group
    bool ok = true;
    auto slot_wait = [&](int st) { // the MMAs that read the slot have retired
      const int use = st / Cfg::STAGES;
      const bool go = use == 0 || mbar_wait(BAR(4 + st % Cfg::STAGES), (use - 1) & 1, abort_flag);
      return __all_sync(0xffffffffu, go) != 0; // the warp leaves together: its lanes meet at the arrives below
    };
    auto raw_wait = [&](int st) { // the stage's packed weights are here (Q4_K: half the lanes ask for the super-block's header)
      const bool head = QT == NNTR_Q4_K && lane >= 16;
      return __all_sync(0xffffffffu, mbar_wait(head ? BAR(17 + ((st >> 2) & 1)) : BAR(9 + st % Cfg::RAW),
                                               (head ? st >> 3 : st / Cfg::RAW) & 1, abort_flag)) != 0;
    };
    auto stage_done = [&](int st) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp(); // every lane's writes are fenced; one arrival per warp keeps the barrier word off the critical path
      if (lane == 0)
        mbar_arrive(BAR(st % Cfg::STAGES));
    };
    auto raw_done = [&](int st) { // the packed words are on their way to registers: the slot may be refilled when they are there
      loads_before_refill();
      __syncwarp();
      if (lane == 0)
        mbar_arrive(BAR(13 + st % Cfg::RAW));
    };
    if constexpr (QT == NNTR_Q4_K) {
      // neighbouring groups read pairs of nibble chunks in opposite order: 128 bytes apart, they would meet in the same banks
      const int grp = r >> 3, sw = grp & 1;
      const uint8_t *nq = smem + Cfg::OFF_RAW + grp * 128 + 8 * j;
      const uint8_t *hdr = smem + Cfg::OFF_HDR + grp * 128;
      // the next stage's words go to registers as soon as this one's are expanded, so that its ring slot refills meanwhile
      uint2 w[4], g0, g1, g2;
      float dw, dmw;
      auto fetch = [&](int st) {
        if (!raw_wait(st))
          return false;
#pragma unroll
        for (int c = 0; c < 4; ++c)
          w[c] = *reinterpret_cast<const uint2 *>(nq + (st % Cfg::RAW) * Cfg::RAW_BYTES + (c >> 1) * (Cfg::ROW_GROUPS * 128) + 64 * ((c & 1) ^ sw));
        const uint8_t *h = hdr + ((st >> 2) & 1) * Cfg::HDR_BYTES;
        g0 = *reinterpret_cast<const uint2 *>(h + 32 + 24 * (st & 3));
        g1 = *reinterpret_cast<const uint2 *>(h + 40 + 24 * (st & 3));
        g2 = *reinterpret_cast<const uint2 *>(h + 48 + 24 * (st & 3));
        dw = half_bits_to_float(*reinterpret_cast<const uint16_t *>(h + 2 * j));
        dmw = half_bits_to_float(*reinterpret_cast<const uint16_t *>(h + 16 + 2 * j));
        raw_done(st);
        return true;
      };
      ok = hsel >= n_stages || fetch(hsel);
      for (int st = hsel; st < n_stages && ok; st += Cfg::GROUPS) {
        float sc0, mn0, sc1, mn1;
        scale_min_row(g0.x, g0.y, g1.x, j, sc0, mn0);
        scale_min_row(g1.y, g2.x, g2.y, j, sc1, mn1);
        const __half2 d_lo = __float2half2_rn(dw * sc0), d_hi = __float2half2_rn(dw * sc1);
        const __half2 m_lo = __float2half2_rn(-(dmw * mn0)), m_hi = __float2half2_rn(-(dmw * mn1));
        if (!(ok = slot_wait(st)))
          break;
        uint8_t *wdst = smem + (st % Cfg::STAGES) * Cfg::STAGE_BYTES + r * 16;
        if (r < own_rows) {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            // word -> 8 halves in the order [lo b0, lo b2, lo b1, lo b3, hi b0, hi b2, hi b1, hi b3]
            const uint32_t wx = w[c].x, wy = w[c].y;
            uint8_t *d = wdst + (2 * (c ^ sw)) * (Cfg::W_ROWS * 16);
            *reinterpret_cast<uint4 *>(d) =
              make_uint4(expand2(wx & 0x000f000fu, d_lo, m_lo), expand2((wx >> 8) & 0x000f000fu, d_lo, m_lo),
                         expand2((wx >> 4) & 0x000f000fu, d_hi, m_hi), expand2((wx >> 12) & 0x000f000fu, d_hi, m_hi));
            *reinterpret_cast<uint4 *>(d + Cfg::W_ROWS * 16) =
              make_uint4(expand2(wy & 0x000f000fu, d_lo, m_lo), expand2((wy >> 8) & 0x000f000fu, d_lo, m_lo),
                         expand2((wy >> 4) & 0x000f000fu, d_hi, m_hi), expand2((wy >> 12) & 0x000f000fu, d_hi, m_hi));
          }
        }
        stage_done(st);
        ok = st + Cfg::GROUPS >= n_stages || fetch(st + Cfg::GROUPS);
      }
    } else if constexpr (QT == NNTR_Q6_K) {
      const int n_row = n0 + peer * own_rows + r, qhalf = hsel & 1;
      const bool have_row = r < own_rows && n_row < N; // rows beyond N: scale 0, so zero weights (their columns are not stored either)
      const int nb = k_stages / 4, n_groups = n_stages / 2, g0 = st0 / 2;
      const uint8_t *wrow = Wb + (size_t)(have_row ? n_row : 0) * nb * sizeof(BlockQ6K);
      // A group is the two stages of one half h of a super-block: they share the 32 qh bytes. This thread: bytes
      // 16*hsel .. +15 of each stage's 32 ql bytes and of the qh bytes, each read as five aligned words and
      // funnel-shifted (blocks are 2-byte aligned), the four scales of its 16-element slices, and d.
      uint32_t rl[2][5], rh[5], rs = 0, rd = 0;
      auto fetch = [&](int g) {
        const int b = (g0 + g) >> 1, h = (g0 + g) & 1;
        const uint8_t *blk = wrow + (size_t)b * sizeof(BlockQ6K);
        const uint32_t *al =
          reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(blk + 64 * h + 16 * qhalf) & ~(uintptr_t)3);
        const uint32_t *ah =
          reinterpret_cast<const uint32_t *>(reinterpret_cast<uintptr_t>(blk + 128 + 32 * h + 16 * qhalf) & ~(uintptr_t)3);
#pragma unroll
        for (int k = 0; k < 5; ++k) {
          rl[0][k] = __ldg(al + k);
          rl[1][k] = __ldg(al + 8 + k);
          rh[k] = __ldg(ah + k);
        }
        const uint8_t *sc = blk + 192 + 8 * h + qhalf; // scale of quarter w: sc[2 w]
        rs = (uint32_t)__ldg(sc) | ((uint32_t)__ldg(sc + 2) << 8) | ((uint32_t)__ldg(sc + 4) << 16) | ((uint32_t)__ldg(sc + 6) << 24);
        rd = __ldg(reinterpret_cast<const uint16_t *>(blk + 208));
      };
      const int first = hsel / 2;
      fetch(first < n_groups ? first : 0);
      for (int g = first; g < n_groups && ok; g += Cfg::GROUPS) {
        const uint32_t sh = (uint32_t)((reinterpret_cast<uintptr_t>(wrow) + (size_t)((g0 + g) >> 1) * sizeof(BlockQ6K)) & 2) * 8;
        uint32_t ql[2][4], qh[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          ql[0][k] = __funnelshift_r(rl[0][k], rl[0][k + 1], sh);
          ql[1][k] = __funnelshift_r(rl[1][k], rl[1][k + 1], sh);
          qh[k] = __funnelshift_r(rh[k], rh[k + 1], sh);
        }
        const float d = have_row ? half_bits_to_float((uint16_t)rd) : 0.f;
        const uint32_t scs = rs;
        fetch(g + Cfg::GROUPS < n_groups ? g + Cfg::GROUPS : g); // the next group travels while this one is expanded
#pragma unroll
        for (int s2 = 0; s2 < 2; ++s2) {
          const int st = 2 * g + s2, s = st % Cfg::STAGES, use = st / Cfg::STAGES;
          const __half2 d_lo = __float2half2_rn(d * (float)(int)(int8_t)(scs >> (8 * s2)));
          const __half2 d_hi = __float2half2_rn(d * (float)(int)(int8_t)(scs >> (8 * s2 + 16)));
          if (use > 0 && !mbar_wait(BAR(4 + s), (use - 1) & 1, abort_flag))
            ok = false;
          ok = __all_sync(0xffffffffu, ok); // the warp leaves together: its lanes meet at the arrive below
          if (!ok)
            break;
          uint8_t *wdst = smem + s * Cfg::STAGE_BYTES + r * 16 + (4 * qhalf) * (Cfg::W_ROWS * 16);
          const __half2 off = __half2half2(__ushort_as_half(0x6420)); // 1024 + 32
          if (r < own_rows) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t l = ql[s2][i], hq = qh[i];
              // the 6-bit values as bytes: low nibbles + qh bits (2 s2, 2 s2 + 1) for quarter s2, high nibbles + qh bits
              // (2 s2 + 4, + 5) for quarter s2 + 2; a byte permute with 0x64 makes (1024 + q) halves: elements {0, 2}, {1, 3}
              const uint32_t qlo = (l & 0x0f0f0f0fu) | ((hq << (4 - 2 * s2)) & 0x30303030u);
              const uint32_t qhi = ((l >> 4) & 0x0f0f0f0fu) | ((hq >> (2 * s2)) & 0x30303030u);
              const uint32_t t0 = __byte_perm(qlo, 0x64646464u, 0x4240), t1 = __byte_perm(qlo, 0x64646464u, 0x4341);
              const uint32_t t2 = __byte_perm(qhi, 0x64646464u, 0x4240), t3 = __byte_perm(qhi, 0x64646464u, 0x4341);
              const __half2 w0 = __hmul2(__hsub2(*reinterpret_cast<const __half2 *>(&t0), off), d_lo);
              const __half2 w1 = __hmul2(__hsub2(*reinterpret_cast<const __half2 *>(&t1), off), d_lo);
              const __half2 w2 = __hmul2(__hsub2(*reinterpret_cast<const __half2 *>(&t2), off), d_hi);
              const __half2 w3 = __hmul2(__hsub2(*reinterpret_cast<const __half2 *>(&t3), off), d_hi);
              *reinterpret_cast<uint4 *>(wdst + i * (Cfg::W_ROWS * 16)) =
                make_uint4(*reinterpret_cast<const uint32_t *>(&w0), *reinterpret_cast<const uint32_t *>(&w1),
                           *reinterpret_cast<const uint32_t *>(&w2), *reinterpret_cast<const uint32_t *>(&w3));
            }
          }
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp(); // every lane's writes are fenced; one arrival per warp keeps the barrier word off the critical path
          if (lane == 0)
            mbar_arrive(BAR(s));
        }
      }
    } else {
      // the two blocks of a stage: 16 nibble bytes each = four words = four 16-byte chunks of halves
      const uint8_t *blk0 = smem + Cfg::OFF_RAW + (r >> 3) * 144;
      uint2 q[4];
      uint16_t dbits[2];
      auto fetch = [&](int st) {
        if (!raw_wait(st))
          return false;
        const uint8_t *blk = blk0 + (st % Cfg::RAW) * Cfg::RAW_BYTES;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          q[2 * k] = *reinterpret_cast<const uint2 *>(blk + k * (Cfg::ROW_GROUPS * 144) + 16 + 8 * j);
          q[2 * k + 1] = *reinterpret_cast<const uint2 *>(blk + k * (Cfg::ROW_GROUPS * 144) + 80 + 8 * j);
          dbits[k] = *reinterpret_cast<const uint16_t *>(blk + k * (Cfg::ROW_GROUPS * 144) + 2 * j);
        }
        raw_done(st);
        return true;
      };
      ok = hsel >= n_stages || fetch(hsel); // n_stages may be odd (K = 2880)
      for (int st = hsel; st < n_stages && ok; st += Cfg::GROUPS) {
        if (!(ok = slot_wait(st)))
          break;
        uint8_t *wdst = smem + (st % Cfg::STAGES) * Cfg::STAGE_BYTES + r * 16;
        if (r < own_rows) {
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            const __half2 d2 = __half2half2(__ushort_as_half(dbits[k]));
            const uint32_t w[4] = {q[2 * k].x ^ 0x88888888u, q[2 * k].y ^ 0x88888888u, q[2 * k + 1].x ^ 0x88888888u,
                                   q[2 * k + 1].y ^ 0x88888888u};
#pragma unroll
            for (int wi = 0; wi < 4; ++wi) // chunk wi: elements 4wi + {0,2,1,3} then 16 + 4wi + {0,2,1,3} of the block
              *reinterpret_cast<uint4 *>(wdst + (4 * k + wi) * (Cfg::W_ROWS * 16)) =
                make_uint4(expand2_q40(w[wi] & 0x000f000fu, d2), expand2_q40((w[wi] >> 8) & 0x000f000fu, d2),
                           expand2_q40((w[wi] >> 4) & 0x000f000fu, d2), expand2_q40((w[wi] >> 12) & 0x000f000fu, d2));
          }
        }
        stage_done(st);
        ok = st + Cfg::GROUPS >= n_stages || fetch(st + Cfg::GROUPS);
      }
    }
    /* ------------------------------ epilogue ------------------------------- */
    tile_done = __all_sync(0xffffffffu, ok && mbar_wait(BAR(8), 0, abort_flag)) != 0;
    if (tile_done) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (parts == 1) {
        const float *turn = reinterpret_cast<const float *>(smem) + turn_area(warp);
        const int cc = n0 + (warp >> 2) * 64 + 4 * (lane & 15);
        for (int hm = 0; hm < ((warp >> 2) * 64 >= tile_rows ? 0 : two ? 2 : 1); ++hm) {
          const int row0 = (mt + mt_step * hm) * F16_TILE_M + (warp & 3) * 32;
          turn_round(hm);
          __syncwarp();
#pragma unroll 4
          for (int i = 0; i < 16; ++i) { // two rows of 256 bytes per instruction
            const int rr = 2 * i + (lane >> 4);
            const float4 f = *reinterpret_cast<const float4 *>(turn + rr * PITCH + 4 * (lane & 15));
            if (row0 + rr < M)
              store4(row0 + rr, cc, f);
          }
          __syncwarp(); // the area is rewritten by the second activation tile
        }
      }
    }
  } else if (warp == F16_COPY_WARP) {
    /* -------------------------- activation copies -------------------------- */
    // A warp of its own keeps the activation stages as far ahead as the ring allows: a slot's copy starts the moment
    // its MMAs have retired, whatever the producers are doing.
    if (lane == 0) {
      const uint8_t *asrc = atiles + ((size_t)mt * k_stages + st0) * F16_A_BYTES;
      // a pair's last tiles may lack partners: what the MMA makes of the memory there is not stored
      const bool have0 = mt < m_tiles, have1 = two && mt + mt_step < m_tiles;
      pdl_wait(); // the quantizer's tiles; the weights do not depend on the kernel before
      for (int st = 0; st < n_stages; ++st) {
        const int s = st % Cfg::STAGES, use = st / Cfg::STAGES;
        if (use > 0 && !mbar_wait(BAR(4 + s), (use - 1) & 1, abort_flag))
          break;
        mbar_expect_tx(BAR(s), (have0 + have1) * F16_A_BYTES);
        const uint32_t dst = sbase + s * Cfg::STAGE_BYTES + Cfg::W_BYTES;
        if (have0)
          bulk_g2s(dst, asrc + (size_t)st * F16_A_BYTES, F16_A_BYTES, BAR(s));
        if (have1)
          bulk_g2s(dst + F16_A_BYTES, asrc + ((size_t)mt_step * k_stages + st) * F16_A_BYTES, F16_A_BYTES, BAR(s));
      }
    }
    __syncwarp();
  } else if (warp == F16_RAW_WARP) {
    /* ---------------------------- packed weights ---------------------------- */
    // The latency of HBM and L2 is in this ring and the producers never wait for a load they issued themselves. Tiled
    // copies, a box of all row groups that the CTA expands x 128 (Q4_0: 144) bytes each: 32 untiled copies of 256 bytes per stage measured 1.6 times
    // slower than no ring at all.
    if (QT != NNTR_Q6_K && lane == 0) {
      const int y = (n0 + peer * own_rows) / 8;
      const uint32_t box = own_rows / 8 * Cfg::RAW_BOX; // bytes of a copy
      for (int st = 0; st < n_stages; ++st) {
        const int rs = st % Cfg::RAW, use = st / Cfg::RAW;
        if (use > 0 && !mbar_wait(BAR(13 + rs), (use - 1) & 1, abort_flag))
          break;
        mbar_expect_tx(BAR(9 + rs), 2 * box);
        const uint32_t dst = sbase + Cfg::OFF_RAW + rs * Cfg::RAW_BYTES;
        int x = (st0 + st) * 2 * (int)sizeof(BlockQ40x8);
        if (QT == NNTR_Q4_K) {
          x = ((st0 + st) >> 2) * (int)sizeof(BlockQ4Kx8);
          if ((st & 3) == 0) { // two headers: the stages up to st - RAW have been read, the one replaced served those up to st - 5
            const int hb = (st >> 2) & 1;
            mbar_expect_tx(BAR(17 + hb), box);
            tma_tile(sbase + Cfg::OFF_HDR + hb * Cfg::HDR_BYTES, &wmap, x, y, BAR(17 + hb));
          }
          x += 128 + 256 * (st & 3);
        }
        tma_tile(dst, &wmap, x, y, BAR(9 + rs));
        tma_tile(dst + Cfg::ROW_GROUPS * Cfg::RAW_BOX, &wmap, x + Cfg::RAW_BOX, y, BAR(9 + rs));
      }
    }
    __syncwarp();
  } else {
    /* ------------------------------ MMA issue ------------------------------ */
    if (lane == 0 && peer) { // the first CTA issues the MMAs: it is told what is ready here
      for (int st = 0; st < n_stages; ++st) {
        const int s = st % Cfg::STAGES;
        if (!mbar_wait(BAR(s), (st / Cfg::STAGES) & 1, abort_flag))
          break;
        mbar_arrive_remote(BAR(s), 0);
      }
    } else if (lane == 0) {
      // D = F32; A = activations (F16, 128 rows = lanes, PAIR: of each CTA); B = weights (F16, tile_rows rows = columns); both K-major
      const uint32_t idesc = (1u << 4) | (0u << 7) | (0u << 10) | ((uint32_t)(tile_rows >> 3) << 17) |
                             ((uint32_t)((PAIR ? 2 : 1) * F16_TILE_M >> 4) << 24);
      bool ok = true;
      for (int st = 0; st < n_stages && ok; ++st) {
        const int s = st % Cfg::STAGES, use = st / Cfg::STAGES;
        if (!mbar_wait(BAR(s), use & 1, abort_flag)) {
          ok = false;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint32_t ws = sbase + s * Cfg::STAGE_BYTES, as = ws + Cfg::W_BYTES;
#pragma unroll
        for (int ks = 0; ks < 4; ++ks) { // K = 16 per instruction: two 16-byte core-matrix columns
          const uint64_t db = umma_desc(ws + ks * 2 * (Cfg::W_ROWS * 16), Cfg::W_ROWS * 16, 128);
          umma_f16<PAIR>(tmem, umma_desc(as + ks * 2 * (F16_TILE_M * 16), F16_TILE_M * 16, 128), db, idesc, (st | ks) != 0);
          if (two)
            umma_f16<PAIR>(tmem + 256, umma_desc(as + F16_A_BYTES + ks * 2 * (F16_TILE_M * 16), F16_TILE_M * 16, 128), db,
                     idesc, (st | ks) != 0);
        }
        umma_commit<PAIR>(BAR(4 + s));
      }
      if (ok)
        umma_commit<PAIR>(BAR(8));
    }
    __syncwarp();
  }

  /* ------------------------------ a shared tile ------------------------------ */
  // Every CTA of the cluster leaves its sums in its own shared memory; the rows are dealt out, and a CTA adds its rows' parts in
  // the order of K. All threads pass all barriers, whatever went wrong before.
  if (SHARED && parts > 1) {
    for (int hm = 0; hm < (two ? 2 : 1); ++hm) {
      if (tile_done)
        turn_round(hm);
      cluster_sync();
      const int row0 = (mt + hm) * F16_TILE_M, rows = min(F16_TILE_M, M - row0);
      if (tile_done) {
        const uint32_t raised = neighbour_raised(smem_u32(const_cast<int *>(abort_flag)), lane);
        for (int i = tid; part + (i >> 6) * parts < rows; i += F16_PRODUCERS) {
          const int r = part + (i >> 6) * parts, c = 4 * (i & 63);
          const uint32_t at = sbase + 4u * (turn_area((r >> 5) + 4 * (c >> 6)) + (r & 31) * PITCH + (c & 63));
          float4 v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k)
            if (k < parts)
              v[k] = ld_cluster4(at, k);
#pragma unroll
          for (int k = 1; k < 8; ++k)
            if (k < parts)
              v[0] = make_float4(v[0].x + v[k].x, v[0].y + v[k].y, v[0].z + v[k].z, v[0].w + v[k].w);
          if (__any_sync(0xffffffffu, raised)) // a part is missing: C stays as it is
            break;
          store4(row0 + r, n0 + c, v[0]);
        }
      }
      cluster_sync(); // the area is rewritten by the second activation tile, and nobody leaves while it is read
    }
  }

  /* common tail: on an abort give copies and MMAs in flight time to land before the memory is released */
  if (*abort_flag)
    for (int i = 0; i < 1000; ++i)
      __nanosleep(1000);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR)
    cluster_sync(); // neither CTA leaves, or frees the tensor memory, while the other needs it
  if (warp == F16_MMA_WARP)
    tmem_free_all<PAIR>(tmem);
}

/* Activation tiles for the fp16 path: per (128 activation rows, 64 of K) 16 KB, core-matrix layout (8 halves = one
 * 16-byte row of a core matrix): chunk wi of row m at wi*2048 + m*16. Chunk wi of stage (b, p) holds, in this order,
 * the elements 64p + 4wi + {0,2,1,3} and 64p + 32 + 4wi + {0,2,1,3} of super-block b -- the order in which the weight
 * producer's unpack delivers them. Values: fp16(d_a * q8), Q8_K quantization as in the exact path (rows below M4 with
 * the 4-row quantizer's sign rule). Rows at or beyond M are zero. One warp per (row, super-block). */
__global__ void __launch_bounds__(256)
quantize_q8_K_f16_tiles_kernel(const float *__restrict__ x, int64_t ldx, uint8_t *__restrict__ tiles, int M, int M4,
                               int Mpad, int nb, int q6_order) {
  pdl_wait();
  pdl_launch_dependents(); // the GEMM behind fetches weights, which a kernel in front of this one may have written, and waits for the rest
  const int lane = threadIdx.x & 31;
  const int64_t blk = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (blk >= (int64_t)Mpad * nb)
    return;
  const int b = (int)(blk / Mpad);
  const int row = (int)(blk - (int64_t)b * Mpad);
  const int m = row % F16_TILE_M;
  float v[8];
  if (row < M) {
    const float *src = x + (int64_t)row * ldx + (int64_t)b * QK_K + lane * 8;
    const float4 a = *reinterpret_cast<const float4 *>(src);
    const float4 c = *reinterpret_cast<const float4 *>(src + 4);
    const Q8KLane q = q8K_quantize_warp(a, c, lane, row < M4 ? 1 : 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      v[i] = __fmul_rn(q.d, (float)(int)(int8_t)(q.w0 >> (8 * i)));
      v[4 + i] = __fmul_rn(q.d, (float)(int)(int8_t)(q.w1 >> (8 * i)));
    }
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i)
      v[i] = 0.f;
  }
  // lane's elements 8*lane + i: p = lane/8, half = (lane%8)/4, wi = 2*(lane%4) + i/4, position j = i%4 -> slot {0,2,1,3}
  int p = lane >> 3, hf = (lane & 7) >> 2, wi0 = 2 * (lane & 3);
  if (q6_order) {
    // Q6_K stages: element e = 8*lane + i: half h = lane/16, quarter w = (lane%16)/4, l = 8*(lane%4) + i inside it;
    // stage 2h + w%2, slot half w/2, chunk 4*(l/16) + (l%16)/4
    p = 2 * (lane >> 4) + ((lane >> 2) & 1);
    hf = (lane >> 3) & 1;
    wi0 = 4 * ((lane >> 1) & 1) + 2 * (lane & 1);
  }
  uint8_t *tile = tiles + ((size_t)(row / F16_TILE_M) * (nb * 4) + (size_t)b * 4 + p) * F16_A_BYTES;
#pragma unroll
  for (int h2 = 0; h2 < 2; ++h2) {
    const __half2 lo = __floats2half2_rn(v[4 * h2 + 0], v[4 * h2 + 2]); // slots 0,1 = j0, j2
    const __half2 hi = __floats2half2_rn(v[4 * h2 + 1], v[4 * h2 + 3]); // slots 2,3 = j1, j3
    *reinterpret_cast<uint2 *>(tile + (wi0 + h2) * (F16_TILE_M * 16) + m * 16 + hf * 8) =
      make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
  }
}

/* Activation tiles for Q4_0 weights: Q8_0 quantization (32-element blocks, fp16 scale; the x86 SIMD form the
 * reference's GEMM uses), values fp16(fp32(d_a) * q8), same tile geometry. A stage is two blocks; chunk 4h + wi of stage
 * st holds the elements 4wi + {0,2,1,3} and 16 + 4wi + {0,2,1,3} of block 2 st + h. One warp per (row, 256 elements);
 * K % 64 == 0, elements at or beyond K belong to no stage. */
__global__ void __launch_bounds__(256)
quantize_q8_0_f16_tiles_kernel(const float *__restrict__ x, int64_t ldx, uint8_t *__restrict__ tiles, int M, int Mpad,
                               int K) {
  pdl_wait();
  pdl_launch_dependents(); // the GEMM behind fetches weights, which a kernel in front of this one may have written, and waits for the rest
  const int lane = threadIdx.x & 31;
  const int nu = (K + 255) / 256, n_stages = K / 64;
  const int64_t unit = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (unit >= (int64_t)Mpad * nu)
    return;
  const int u = (int)(unit / Mpad);
  const int row = (int)(unit - (int64_t)u * Mpad);
  const int m = row % F16_TILE_M;
  const int e0 = u * 256 + lane * 8;
  const bool valid = e0 < K;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), c = a;
  if (valid && row < M) {
    const float *src = x + (int64_t)row * ldx + e0;
    a = *reinterpret_cast<const float4 *>(src);
    c = *reinterpret_cast<const float4 *>(src + 4);
  }
  const Q80Lane q = q80_quantize_warp(a, c);
  if (!valid)
    return;
  const float d = half_bits_to_float(q.d_bits);
  float v[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[i] = __fmul_rn(d, (float)(int)(int8_t)(q.w0 >> (8 * i)));
    v[4 + i] = __fmul_rn(d, (float)(int)(int8_t)(q.w1 >> (8 * i)));
  }
  // lane's elements: block (lane/4) of the unit, e = 8*(lane%4) + i inside it
  const int st = u * 4 + (lane >> 3), h = (lane >> 2) & 1, hf = (lane & 3) >> 1, wi0 = 2 * (lane & 1);
  uint8_t *tile = tiles + ((size_t)(row / F16_TILE_M) * n_stages + st) * F16_A_BYTES;
#pragma unroll
  for (int h2 = 0; h2 < 2; ++h2) {
    const __half2 lo = __floats2half2_rn(v[4 * h2 + 0], v[4 * h2 + 2]);
    const __half2 hi = __floats2half2_rn(v[4 * h2 + 1], v[4 * h2 + 3]);
    *reinterpret_cast<uint2 *>(tile + (4 * h + wi0 + h2) * (F16_TILE_M * 16) + m * 16 + hf * 8) =
      make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
  }
}

/** Into how many parts K is cut, so that few tiles still use the machine. A CTA alone walks K at 0.8 us (Q4_0 0.7, Q6_K 1.4 and more) a stage
 *  however many SMs are idle; the parts' sums cost about 2 us at the end. As many as still run in one wave of clusters, of at
 *  least four stages each. */
template <int QT> int k_parts(int tiles, int k_stages) {
  static ClusterFit fit;
  for (int parts = 8; parts > 1; parts /= 2)
    if (k_stages >= 4 * parts && tiles <= fit(gemm_f16_kernel<QT, F16_SHARED>, parts, F16_THREADS, F16Cfg<QT, F16_SHARED>::SMEM))
      return parts;
  return 1;
}

} // namespace

size_t umma_f16_workspace_bytes(unsigned M, unsigned K) {
  return (size_t)((M + F16_TILE_M - 1) / F16_TILE_M) * F16_TILE_M * K * 2;
}

bool umma_f16_supported(int qtype, unsigned M, unsigned N, unsigned K) {
  if (M < 2 || K == 0 || N == 0)
    return false;
  if (qtype == NNTR_Q6_K) // plain rows: any N; the last tile may be ragged
    return K % QK_K == 0;
  if (N % F16_TILE_N)
    return false;
  return (qtype == NNTR_Q4_K && K % QK_K == 0) || (qtype == NNTR_Q4_0 && K % F16_KS == 0);
}

namespace {

template <int QT, int MODE>
int launch_mode(dim3 grid, int cluster, cudaStream_t st, const CUtensorMap &wmap, const uint8_t *tiles, const uint8_t *W, float *C,
                int ldc, int M, int N, int k_stages, int m_tiles, int tiles_per_cta, int tile_rows, int c_vec4) {
  NNTR_CHECK_CUDA(launch_in_clusters(gemm_f16_kernel<QT, MODE>, grid, cluster, F16_THREADS, F16Cfg<QT, MODE>::SMEM, st, wmap, tiles, W,
                                     C, ldc, M, N, k_stages, m_tiles, tiles_per_cta, tile_rows, c_vec4));
  return NNTR_CUDA_OK;
}

/** Weight rows of a tile, so that the tiles of m_groups rows of them fill the waves of `slots` that they need anyway: with 256 rows a
 *  last wave can be nearly empty. A multiple of step, at least 128 (the copies of the activations cost the same for fewer rows). Q4_K
 *  1024 x 9728 x 2560 71.8 -> 66.7 us, 256 x 24576 x 4096 58.0 -> 54.5, Q4_0 200 x 24576 x 4096 55.3 -> 49.8, Q6_K 256 x 151936 x 2560
 *  320 -> 282, 700 x 12288 x 4096 125 -> 109; Q4_K 1024 x 24576 x 4096, whose last wave was 60 % full, 167 and 168. */
int even_rows(int m_groups, int N, int slots, int step) {
  const int tiles = m_groups * ((N + F16_TILE_N - 1) / F16_TILE_N);
  if (slots < m_groups)
    return F16_TILE_N;
  const int n_tiles = (tiles + slots - 1) / slots * slots / m_groups, rows = (N + n_tiles - 1) / n_tiles;
  return std::min(F16_TILE_N, std::max(128, (rows + step - 1) / step * step));
}

/** What the tiles of m_groups rows of them take, in units of a stage of a tile: rounds over the slots that run at a time, each as long as
 *  its tiles are high. */
int64_t rounds_cost(int m_groups, int N, int slots, int tile_rows) {
  return ((int64_t)m_groups * ((N + tile_rows - 1) / tile_rows) + slots - 1) / slots * (224 + tile_rows);
}

/** allows every form of the kernel its shared memory, once per device */
template <int QT> int allow_smem() {
  static std::atomic<uint64_t> done{0};
  int dev = 0;
  NNTR_CHECK_CUDA(cudaGetDevice(&dev));
  if (dev < 64 && (done.load(std::memory_order_acquire) >> dev & 1))
    return NNTR_CUDA_OK;
  NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_f16_kernel<QT, F16_LONE>, cudaFuncAttributeMaxDynamicSharedMemorySize, F16Cfg<QT, F16_LONE>::SMEM));
  NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_f16_kernel<QT, F16_SHARED>, cudaFuncAttributeMaxDynamicSharedMemorySize, F16Cfg<QT, F16_SHARED>::SMEM));
  NNTR_CHECK_CUDA(cudaFuncSetAttribute(gemm_f16_kernel<QT, F16_PAIR>, cudaFuncAttributeMaxDynamicSharedMemorySize, F16Cfg<QT, F16_PAIR>::SMEM));
  if (dev < 64)
    done.fetch_or(1ull << dev, std::memory_order_release);
  return NNTR_CUDA_OK;
}

template <int QT>
int launch_typed(unsigned M, unsigned N, unsigned K, const uint8_t *tiles, const void *B, float *C, unsigned ldc, cudaStream_t st) {
  const int mtiles = (int)((M + F16_TILE_M - 1) / F16_TILE_M), n_tiles = (int)((N + F16_TILE_N - 1) / F16_TILE_N);
  const int k_stages = (int)(K / F16_KS), c_vec4 = (ldc % 4 == 0) && !(reinterpret_cast<uintptr_t>(C) & 15);
  int cta_m = (mtiles + 1) / 2, tiles_per_cta = 2;
  if (const int rc = allow_smem<QT>())
    return rc;
  const int parts = k_parts<QT>(cta_m * n_tiles, k_stages);
  bool pair = false;
  int tile_rows = F16_TILE_N;
  if (parts == 1) {
    tile_rows = even_rows(cta_m, (int)N, sm_count(), 16);
    // Pairs where their rounds take less: a stage of a tile of r weight rows takes them about (224 + r) units and a CTA alone 1.2 (Q6_K:
    // 1.5) times as many, but a pair that has fewer than four tiles of activations works for the missing ones too, and its rounds hold
    // half as many tiles. Q4_K, pairs / CTAs alone: 300 x 24576 x 4096 91.4 / 103.8 us, 512 95.5 / 107, 603 140.7 / 117.8, 768 143.5 / 129.6,
    // 859 157 / 169.6, 1024 161 / 182.6; 9728 x 2560 512 / 768 / 1024 rows 33.4 / 37.0, 61.9 / 40.2, 64.8 / 70.2; 8192 x 8192 768 rows 93.7 / 106.5;
    // Q4_0 19456 x 2560 768 / 1280 / 1792 rows 90.5 / 73.5, 126.3 / 115.1, 161.6 / 156.3; Q6_K 9728 x 2560 768 rows 64.4 / 58.4, 1280
    // 76.8 / 101.2. Of 296 sizes of 257 to 2048 rows the other form is by no more than 3 % the faster one.
    if (mtiles > 2) {
      static ClusterFit fit;
      const int quads = (mtiles + 3) / 4, slots = fit(gemm_f16_kernel<QT, F16_PAIR>, 2, F16_THREADS, F16Cfg<QT, F16_PAIR>::SMEM);
      const int pair_rows = even_rows(quads, (int)N, slots, 32);
      pair = slots > 0 && 10 * rounds_cost(quads, (int)N, slots, pair_rows) <=
                            (QT == NNTR_Q6_K ? 15 : 12) * rounds_cost(cta_m, (int)N, sm_count(), tile_rows);
      if (pair)
        cta_m = quads, tile_rows = pair_rows;
    }
  } else if (mtiles > 1 && parts == k_parts<QT>(mtiles * n_tiles, k_stages)) {
    // tiles one by one if they run in the same wave as the pairs: 128 instead of 256 columns of MMAs per stage and one sum at the
    // end instead of two (256 x 1280 x 2560 Q4_0: 24 -> 16 us)
    tiles_per_cta = 1;
    cta_m = mtiles;
  }
  CUtensorMap wmap = {};
  if (QT != NNTR_Q6_K) { // rows of 8-row groups of packed weights
    const uint64_t row = QT == NNTR_Q4_K ? (uint64_t)(K / QK_K) * sizeof(BlockQ4Kx8) : (uint64_t)(K / 32) * sizeof(BlockQ40x8);
    const int rc = encode_map_2d(&wmap, B, 1, row, N / 8, row, F16Cfg<QT, F16_LONE>::RAW_BOX, (unsigned)(pair ? tile_rows / 2 : tile_rows) / 8, false);
    if (rc)
      return rc;
  }
  const uint8_t *W = static_cast<const uint8_t *>(B);
  const dim3 grid(cta_m, ((int)N + tile_rows - 1) / tile_rows);
  const auto launch = pair ? launch_mode<QT, F16_PAIR> : parts > 1 ? launch_mode<QT, F16_SHARED> : launch_mode<QT, F16_LONE>;
  return launch(grid, pair ? 2 : parts, st, wmap, tiles, W, C, (int)ldc, (int)M, (int)N, k_stages, mtiles, tiles_per_cta, tile_rows, c_vec4);
}

} // namespace

int launch_gemm_f16(int qtype, unsigned M, unsigned N, unsigned K, const float *A, const void *B, float *C, unsigned ldc,
                    void *ws, cudaStream_t st) {
  const int mtiles = (int)((M + F16_TILE_M - 1) / F16_TILE_M), Mpad = mtiles * F16_TILE_M;
  if ((reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(ws) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm (fp16 tensor path): activations and workspace must be 16-byte aligned");
  if (qtype != NNTR_Q6_K && (reinterpret_cast<uintptr_t>(B) & 15))
    return set_error(NNTR_CUDA_ERR_INVALID, "gemm (fp16 tensor path): weights must be 16-byte aligned");
  uint8_t *tiles = static_cast<uint8_t *>(ws);
  int rc;
  if (qtype == NNTR_Q4_K || qtype == NNTR_Q6_K) {
    const int nb = (int)(K / QK_K);
    // Q4_K: rows below 4*floor(M/4) with the 4-row quantizer's sign rule; Q6_K: the row quantizer for every row
    // (ggml_interface_omp.cpp:545-551)
    const unsigned M4 = qtype == NNTR_Q4_K ? (M / 4) * 4 : 0;
    const int64_t nwarps = (int64_t)Mpad * nb;
    NNTR_CHECK_CUDA(launch_in_clusters(quantize_q8_K_f16_tiles_kernel, dim3((unsigned)((nwarps + 7) / 8)), 1, 256, 0, st, A, (int64_t)K, tiles,
                                       (int)M, (int)M4, Mpad, nb, (int)(qtype == NNTR_Q6_K)));
    count_launch();
    rc = qtype == NNTR_Q4_K ? launch_typed<NNTR_Q4_K>(M, N, K, tiles, B, C, ldc, st) : launch_typed<NNTR_Q6_K>(M, N, K, tiles, B, C, ldc, st);
  } else {
    const int64_t nwarps = (int64_t)Mpad * ((K + 255) / 256);
    NNTR_CHECK_CUDA(launch_in_clusters(quantize_q8_0_f16_tiles_kernel, dim3((unsigned)((nwarps + 7) / 8)), 1, 256, 0, st, A, (int64_t)K, tiles,
                                       (int)M, Mpad, (int)K));
    count_launch();
    rc = launch_typed<NNTR_Q4_0>(M, N, K, tiles, B, C, ldc, st);
  }
  if (rc)
    return rc;
  count_launch();
  return check_cuda(cudaGetLastError(), "gemm fp16 tensor-path launch");
}

int read_f16_status(int *out) {
  int v = 0;
  NNTR_CHECK_CUDA(cudaMemcpyFromSymbol(&v, g_f16_status, sizeof(int)));
  *out = v;
  return NNTR_CUDA_OK;
}
int clear_f16_status() {
  const int zero = 0;
  return check_cuda(cudaMemcpyToSymbol(g_f16_status, &zero, sizeof(int)), "clear_f16_status");
}

} // namespace nntr
