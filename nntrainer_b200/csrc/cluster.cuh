// SPDX-License-Identifier: Apache-2.0
/**
 * @file  cluster.cuh
 * @brief One-dimensional clusters of CTAs that share a tile of a GEMM: each takes a part of K, and the sums meet through
 *        distributed shared memory.
 */
#ifndef NNTR_CLUSTER_CUH_
#define NNTR_CLUSTER_CUH_

#include <atomic>

#include "common.cuh"

namespace nntr {

/* the size is 1 without the launch attribute */
__device__ __forceinline__ int cluster_size() {
  uint32_t n;
  asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
  return (int)n;
}
__device__ __forceinline__ int cluster_rank() {
  uint32_t n;
  asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(n));
  return (int)n;
}
/** four floats at a shared address (of this CTA's window) in the CTA of the given rank */
__device__ __forceinline__ float4 ld_cluster4(uint32_t addr, int rank) {
  uint32_t remote;
  float4 v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(remote)
               : "memory");
  return v;
}

/** the same for a store */
__device__ __forceinline__ void st_cluster4(uint32_t addr, int rank, const float4 &v) {
  uint32_t remote;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(addr), "r"(rank));
  asm volatile("st.shared::cluster.v4.f32 [%0], {%1,%2,%3,%4};" ::"r"(remote), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_sync() {
  cluster_arrive();
  cluster_wait();
}

/* A wait that ran out in one CTA of a cluster leaves its neighbours' results without its part, so they have to know before they
 * store anything. flag: shared address of the word in which a CTA notes that it gave up, the same in every CTA. */
/** Every thread that knows that its CTA gave up raises the neighbours' flags, before the barrier behind which the parts are used
 *  and behind one that says that all have started. */
__device__ __forceinline__ void raise_in_cluster(uint32_t flag) {
  for (int r = 0; r < cluster_size(); ++r) {
    uint32_t remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(flag), "r"(r));
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote), "r"(1) : "memory");
  }
}
/** Where there is no such barrier (it would be one more per call): the flag of the CTA whose rank is the lane's number, 0 in
 *  the other lanes, for a vote of the warp. Between the barrier behind which the parts are used and the one behind which the CTAs
 *  may leave. */
__device__ __forceinline__ uint32_t neighbour_raised(uint32_t flag, int lane) {
  uint32_t v = 0;
  if (lane < cluster_size()) {
    uint32_t remote;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(flag), "r"(lane));
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(remote) : "memory");
  }
  return v;
}

/** Launch of a grid of grid.x * parts by grid.y CTAs in clusters of `parts` CTAs along x. The grid may start before its
 *  predecessor is done: the kernel calls pdl_wait() before it touches what that wrote. */
template <typename... P, typename... A>
cudaError_t launch_in_clusters(void (*kernel)(P...), dim3 grid, int parts, int threads, int smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = parts;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid.x * parts, grid.y);
  cfg.blockDim = threads;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = parts > 1 ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kernel, (P)args...);
}

/** Clusters of 2, 4 or 8 CTAs of one kernel that run at the same time, per device, asked for once. */
struct ClusterFit {
  std::atomic<int> n[64][3];

  template <typename... P> int operator()(void (*kernel)(P...), int parts, int threads, int smem) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64)
      return 0;
    std::atomic<int> &slot = n[dev][parts == 2 ? 0 : parts == 4 ? 1 : 2];
    int v = slot.load(std::memory_order_relaxed);
    if (v == 0) {
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = parts;
      attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(parts);
      cfg.blockDim = threads;
      cfg.dynamicSmemBytes = smem;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&v, kernel, &cfg) != cudaSuccess || v <= 0) {
        (void)cudaGetLastError();
        v = -1;
      }
      slot.store(v, std::memory_order_relaxed);
    }
    return v;
  }
};

} // namespace nntr
#endif
