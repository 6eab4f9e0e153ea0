// SPDX-License-Identifier: Apache-2.0
/**
 * @file  pipeline.cuh
 * @brief Device primitives shared by the streaming kernels: mbarriers with
 *        bounded waits, bulk copies into shared memory, explicit shared-space
 *        accesses by 32-bit address.
 *
 * Every wait on another agent (a bulk copy, another warp, the tensor pipe) goes
 * through mbar_wait_bounded: a fixed number of polls, after which the caller's
 * abort flag and the translation unit's status word are raised and the wait
 * returns false, so a lost signal ends the kernel instead of hanging the GPU.
 */
#pragma once

#include "common.cuh"

namespace nntr {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\t"
               "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
/** try_wait that lets the hardware park the thread for up to `ns` nanoseconds per try */
__device__ __forceinline__ bool mbar_try_wait_hint(uint32_t bar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\t"
               "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
               "selp.u32 %0, 1, 0, p;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity), "r"(ns)
               : "memory");
  return ok != 0;
}

/** Bounded wait for the phase with `parity` of an mbarrier. After `spin` polls it also watches the CTA's abort flag and
 *  backs off. False when the CTA is aborting, or (after `polls` polls) when the phase never completed: then the abort
 *  flag and *status are raised. hint_ns != 0 uses the parked form of try_wait. */
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status,
                                                  uint32_t polls, uint32_t spin, uint32_t hint_ns = 0) {
  for (uint32_t it = 0; it < polls; ++it) {
    if (hint_ns ? mbar_try_wait_hint(bar, parity, hint_ns) : mbar_try_wait(bar, parity))
      return true;
    if (it > spin) {
      if (*abort_flag)
        return false;
      __nanosleep(32);
    }
  }
  *abort_flag = 1;
  atomicExch(status, NNTR_CUDA_ERR_TIMEOUT);
  return false;
}

/** The same for all lanes of a warp: true in every one or in none. Two lanes may learn of the phase's end and of the abort flag in
 *  turn; in front of an instruction that takes the whole warp (ldmatrix, __syncwarp) they have to leave together. */
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity, volatile int *abort_flag, int *status, uint32_t polls,
                                               uint32_t spin) {
  return __all_sync(FULL, mbar_wait_bounded(bar, parity, abort_flag, status, polls, spin)) != 0;
}

/** A chain that goes from warp to warp: the warp in front arrives at barrier `id`, the one behind waits for it. Number 0 is the
 *  barrier of __syncthreads(): where it is used for a hand-over, no barrier of the whole CTA may lie between the first and the last. */
__device__ __forceinline__ void pair_arrive(int id) { asm volatile("barrier.cta.arrive %0, 64;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void pair_sync(int id) { asm volatile("barrier.cta.sync %0, 64;" ::"r"(id) : "memory"); }
/** For the last warp of such a chain, behind its hand-over: whether its own waits and those of every warp in front (that raise the
 *  flag before they hand over) came to their end. Without that the sums are incomplete and must not be stored. */
__device__ __forceinline__ bool nobody_gave_up(bool ok, const volatile int *abort_flag) { return ok && !*abort_flag; }

/** Bulk copy global -> shared memory of this CTA, completion counted in bytes on an mbarrier. Both addresses 16-byte
 *  aligned, size a multiple of 16. Local memory only (no multicast). */
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
               "l"(src), "r"(bytes), "r"(bar)
               : "memory");
}

/** Before a warp gives a slot of shared memory back to bulk copies: the loads of every lane have been performed then. Neither the
 *  warp's barrier nor the arrive behind it waits for loads whose values nothing has used yet, and a copy that refills the slot
 *  may overtake them (fp16 GEMM, Q4_0 256 x 24576 x 2880, without a fence: wrong elements in every launch; with this one or
 *  __threadfence_block(): none in 3000). Needless where the values have gone into a store, or into a chain that the next round
 *  continues, before the slot is given back. */
__device__ __forceinline__ void loads_before_refill() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

/** Quotients by a number known at run time only, exact while dividend * n < 2^32: a multiplication instead of the 150 clocks
 *  (64 bits: several hundred) of a division, which a loop with one thread or warp per stage of a ring cannot hide. */
struct FastDiv {
  uint32_t n, m;
  __device__ __forceinline__ explicit FastDiv(uint32_t d) : n(d), m(d > 1 ? 0xffffffffu / d + 1 : 0) {}
  __device__ __forceinline__ int div(int t) const { return n > 1 ? (int)__umulhi((uint32_t)t, m) : t; }
  __device__ __forceinline__ int mod(int t, int q) const { return t - q * (int)n; } // q = div(t)
};

/** 4-way dot product of unsigned bytes (a) with signed bytes (b), accumulated in c */
__device__ __forceinline__ int dp4a_us(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

/* explicit shared-space accesses by 32-bit address */
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ uint4 lds128(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t v) {
  asm volatile("st.shared.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
  asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(v0), "r"(v1), "r"(v2), "r"(v3) : "memory");
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t v0, uint32_t v1) {
  asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(a), "r"(v0), "r"(v1) : "memory");
}

} // namespace nntr
