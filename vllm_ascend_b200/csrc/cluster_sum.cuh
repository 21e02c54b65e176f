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

}  // namespace b200
