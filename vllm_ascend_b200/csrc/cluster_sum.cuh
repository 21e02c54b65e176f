// Split-K over a thread-block cluster: the blocks of a cluster keep fp32 partial tiles [token][128 weight rows] in shared
// memory and add them in block order (gemm_small.cu, gemm_small_fp8.cu).
#pragma once
#include "common.cuh"

namespace b200 {

constexpr int SG_ROWS = 128;       // weight rows per tile

__device__ __forceinline__ uint32_t sg_map(uint32_t saddr, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(saddr), "r"(rank));
  return a;
}
__device__ __forceinline__ float4 sg_ld(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr)
               : "memory");
  return v;
}
__device__ __forceinline__ void sg_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// Sum of four neighbouring rows of one token over the blocks of the cluster, in block order.
__device__ __forceinline__ float4 sg_sum(const uint32_t part, int splits, uint32_t off) {
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (int r = 0; r < splits; r++) {
    const float4 v = sg_ld(sg_map(part + off, r));
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  return s;
}

// How many clusters of `blocks` blocks the GPU runs at once with `per_sm` (1 or 2) blocks on an SM.  A cluster lies within one group of SMs,
// and groups leave SMs over that no cluster fits into: one block per SM, 45 clusters of three, where 148 SMs give 49.  A grid that
// counted SMs ran in two waves (64 rows of 6144 x 4096 in six parts 27 us, in five 21 us).  The driver is asked once per size, about
// one block per SM, as its answer does not double where two fit.  With two, a group of n SMs holds as many clusters of six or eight as
// with one of three or four (33 of eight, where twice the answer for eight says 30 and 32 tiles of 4096 x 12288 took 26.2 us in six
// parts, 25.0 us in eight; 45 of six).  Four do not come to that (74 tiles of 9472 x 2048, 128 rows: 24.2 us, the general kernel 18.2), and
// odd sizes have no half: twice the answer is what surely fits.
using sg_fit_t = std::atomic<int>;
template <auto Kernel>
inline int sg_clusters_at_once(sg_fit_t* known, int blocks, int threads, int per_sm) {
  if (per_sm == 2 && (blocks == 6 || blocks == 8)) {
    blocks /= 2;
    per_sm = 1;
  }
  int n = known[blocks].load(std::memory_order_relaxed);
  if (n > 0) return n * per_sm;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(blocks, 1);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = 160 * 1024;             // an SM to itself
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = blocks;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  if (cudaOccupancyMaxActiveClusters(&n, Kernel, &cfg) != cudaSuccess || n < 1) {
    cudaGetLastError();
    return 0;
  }
  known[blocks].store(n, std::memory_order_relaxed);
  return n * per_sm;
}

}  // namespace b200
