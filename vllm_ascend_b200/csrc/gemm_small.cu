// Few-row bf16 GEMM for sm_100a:  C[M,N] = A[M,K] * W[N,K]^T  with M <= 256 (decode batches, short prompts).
//
// Bound: the weights have to cross HBM once and everything else is small, so what counts is that all SMs
// stream weights from the first microsecond to the last.  Tiles of 128 x 128 or more give N / 128 blocks (32 for a
// 4096-wide layer) that each walk all of K; here the roles of the operands are swapped and K is split:
//   * 128 weight rows are the MMA's M axis, the (few) tokens its N axis in steps of 16, so that a stage holds 16 KB
//     of weights and only as many activation rows as there are;
//   * a cluster of `splits` blocks shares one 128-row tile, each over its part of K; their fp32 partial products
//     meet in shared memory (DSMEM), every block adds its share of the tokens in block order and stores it.
//     No workspace, no atomics: results repeat bit for bit;
//   * two blocks share an SM while their stages are small (up to 128 tokens), so that the grid runs in one wave and
//     one block's prologue and reduction hide behind the other's loads;
//   * launched as a programmatic dependent: barriers, TMEM and an L2 prefetch of the block's own weights (L2 is the point
//     of coherence, so the prefetch reads nothing early) are under way while the previous kernel finishes.
// One row, us with cold weights in a captured chain, general kernel -> this one: 4096 x 4096 25 -> 9, 4096 x 12288 62 -> 17,
// 24576 x 4096 (gate / up) 58 -> 36, 32000 x 4096 71 -> 43 (6.2 TB/s).
// Roles: warps 0..3 read the accumulator (one TMEM lane quarter each), warp 4 issues TMA, warp 5 issues
// tcgen05.mma (cta_group::1, M = 128, N = tokens, K = 16, f32 in TMEM); all six reduce and store.
#include "cluster_sum.cuh"
#include "common.cuh"
#include "tmap_cache.cuh"

namespace b200 {

constexpr int SG_BK = 64;          // columns per stage (128 bytes: one swizzle row)
constexpr int SG_THREADS = 192;
constexpr int SG_WBYTES = SG_ROWS * SG_BK * 2;
constexpr int SG_MAX_STAGES = 12;

struct SmallGemmParams {
  int M, N, K, ldc;
  int nt;                          // tokens rounded up to 16: columns of the accumulator
  int stages, stage_bytes, tmem_cols;
  int splits, prefetch_kb;
  int glu;                         // W = [gate (N rows); up (N rows)], C = gate(.) * up
  float glu_alpha, glu_limit;      // alpha > 0: clamped gate instead of SiLU
  const __nv_bfloat16* bias;
  const __nv_bfloat16* residual;
  __nv_bfloat16* C;
  float* ss_out;                   // [tile][ss_stride]: sum of squares of each stored output row within the tile, or null
  long ss_stride;
  int ss_parts_max;                // behind that many parts: how many there are
  int* status;
};

__device__ __forceinline__ float sg_gate(float g, float u, float alpha, float limit) {
  if (alpha > 0.f) {
    g = fminf(g, limit);
    u = fminf(fmaxf(u, -limit), limit) + 1.f;
    return g / (1.f + __expf(-alpha * g)) * u;
  }
  return g / (1.f + __expf(-g)) * u;
}

__global__ void __launch_bounds__(SG_THREADS, 2)
gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                  const SmallGemmParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = (uint64_t*)(smem + p.stages * p.stage_bytes);
  uint64_t* empty_bar = full_bar + SG_MAX_STAGES;
  uint64_t* tmem_full = empty_bar + SG_MAX_STAGES;
  uint32_t* tmem_ptr = (uint32_t*)(tmem_full + 1);
  volatile int* abort_word = (volatile int*)(tmem_ptr + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int split = blockIdx.x, tile = blockIdx.y;       // the cluster is the whole x extent of the grid
  const int num_kb = (p.K + SG_BK - 1) / SG_BK;
  const int kb0 = (int)((long)num_kb * split / p.splits), kb1 = (int)((long)num_kb * (split + 1) / p.splits);
  const int w_row = p.glu ? tile * (SG_ROWS / 2) : tile * SG_ROWS;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(tmem_full, 1);
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 4 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    for (int kb = kb0; kb < min(kb1, kb0 + p.prefetch_kb); kb++) {
      tma_prefetch_l2_2d(&tmap_w, kb * SG_BK, w_row);
      if (p.glu) tma_prefetch_l2_2d(&tmap_w, kb * SG_BK, p.N + w_row);
    }
  }
  if (warp == 5) {
    tmem_alloc(tmem_ptr, p.tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_ptr);
  asm volatile("griddepcontrol.wait;" ::: "memory");     // activations, residual and C belong to earlier kernels until here

  bool ok = true;
  if (warp == 4) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_word)) break;
        uint8_t* sw = smem + stage * p.stage_bytes;
        mbar_expect_tx(&full_bar[stage], SG_WBYTES + p.nt * SG_BK * 2);
        tma_load_2d(sw, &tmap_w, &full_bar[stage], kb * SG_BK, w_row);
        if (p.glu) tma_load_2d(sw + SG_WBYTES / 2, &tmap_w, &full_bar[stage], kb * SG_BK, p.N + w_row);
        tma_load_2d(sw + SG_WBYTES, &tmap_a, &full_bar[stage], kb * SG_BK, 0);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 5) {
    // ------------------------------------------------------------ MMA issuer: one thread walks the loop (see warp_uniform)
    if (elect_one()) {
      const uint32_t idesc = make_idesc_f16(SG_ROWS, p.nt, true, false, false);
      const uint64_t dw0 = make_smem_desc(smem_u32(smem), 16, 1024, kLayoutSw128);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        ok = mbar_wait(&full_bar[stage], phase, abort_word);
        if (!ok) break;
        tc_fence_after();
        const uint64_t dw = dw0 + (uint32_t)(stage * (p.stage_bytes >> 4)), da = dw + (SG_WBYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < SG_BK / 16; kk++) umma_f16_ss(tmem_base, dw + 2 * kk, da + 2 * kk, idesc, (kb > kb0 || kk > 0) ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
      if (ok) umma_commit(tmem_full);
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ accumulator -> shared memory, [token][weight row]
    ok = mbar_wait(tmem_full, 0, abort_word);
    tc_fence_after();
    if (ok) {
      // every stage has been consumed (the last commit covers all products), so its memory is free
      float* part = (float*)smem + warp * 32 + lane;
      const uint32_t t_row = tmem_base + ((uint32_t)(warp * 32) << 16);
      for (int c0 = 0; c0 < p.nt; c0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_row + c0, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; j++) part[(c0 + j) * SG_ROWS] = __uint_as_float(r[j]);
      }
    }
    tc_fence_before();
  }
  if (p.splits > 1) sg_cluster_sync();
  else __syncthreads();

  // ------------------------------------------------------------ sum over the cluster and store: warp (or half) per token
  const uint32_t part = smem_u32(smem);
  const int t0 = p.M * split / p.splits, t1 = p.M * (split + 1) / p.splits;
  if (*abort_word == 0) {
    if (!p.glu) {
      const int col = tile * SG_ROWS + lane * 4;
      if (p.ss_out && tile == 0 && split == 0 && threadIdx.x == 0)
        *reinterpret_cast<int*>(p.ss_out + (long)p.ss_parts_max * p.ss_stride) = gridDim.y;
      for (int t = t0 + warp; t < t1; t += SG_THREADS / 32) {
        float4 v = sg_sum(part, p.splits, (uint32_t)(t * SG_ROWS + lane * 4) * 4);
        if (col < p.N) {                                  // N is a multiple of 8
          if (p.bias) {
            const uint2 b = *reinterpret_cast<const uint2*>(p.bias + col);
            const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y);
            v.x += b0.x; v.y += b0.y; v.z += b1.x; v.w += b1.y;
          }
          if (p.residual) {
            const uint2 b = *reinterpret_cast<const uint2*>(p.residual + (size_t)t * p.ldc + col);
            const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y);
            v.x += b0.x; v.y += b0.y; v.z += b1.x; v.w += b1.y;
          }
          const uint2 o = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
          *reinterpret_cast<uint2*>(p.C + (size_t)t * p.ldc + col) = o;
          const float2 f0 = unpack_bf16x2(o.x), f1 = unpack_bf16x2(o.y);       // of the values as stored
          v = make_float4(f0.x, f0.y, f1.x, f1.y);
        } else {
          v = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (p.ss_out) {
          const float ss = warp_reduce_sum(v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w);
          if (lane == 0) p.ss_out[(long)tile * p.ss_stride + t] = ss;
        }
      }
    } else {
      const int half = lane >> 4, l = lane & 15, col = tile * (SG_ROWS / 2) + l * 4;
      for (int t = t0 + 2 * warp + half; t < t1; t += SG_THREADS / 16) {
        const float4 g = sg_sum(part, p.splits, (uint32_t)(t * SG_ROWS + l * 4) * 4);
        const float4 u = sg_sum(part, p.splits, (uint32_t)(t * SG_ROWS + SG_ROWS / 2 + l * 4) * 4);
        if (col < p.N)
          *reinterpret_cast<uint2*>(p.C + (size_t)t * p.ldc + col) =
              make_uint2(pack_bf16x2(sg_gate(g.x, u.x, p.glu_alpha, p.glu_limit), sg_gate(g.y, u.y, p.glu_alpha, p.glu_limit)),
                         pack_bf16x2(sg_gate(g.z, u.z, p.glu_alpha, p.glu_limit), sg_gate(g.w, u.w, p.glu_alpha, p.glu_limit)));
      }
    }
  }
  if (p.splits > 1) sg_cluster_sync();                    // no block leaves while another reads its sums
  else __syncthreads();
  if (*abort_word != 0) {
    // give copies in flight time to land before the block's memory is handed on
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 50000ull) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, *abort_word);
    __syncthreads();
  }
  if (warp == 5) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.tmem_cols);
  }
}

static int small_smem(const SmallGemmParams& p) {
  return p.stages * p.stage_bytes + (2 * SG_MAX_STAGES + 1) * 8 + 16 + 1024;
}

// Tokens, stages and (where none are asked for) splits of K.  Nonzero: refused.
static int plan_small(SmallGemmParams& p, int splits) {
  const int rows = p.glu ? SG_ROWS / 2 : SG_ROWS;
  const int tiles = (p.N + rows - 1) / rows, num_kb = (p.K + SG_BK - 1) / SG_BK;
  p.nt = (p.M + 15) / 16 * 16;
  p.stage_bytes = SG_WBYTES + (p.nt * SG_BK * 2 + 1023) / 1024 * 1024;
  // two blocks of ~100 KB per SM while a stage is at most 32 KB (128 tokens), one block with all of it beyond
  const bool pair = p.nt <= 128;
  p.stages = (pair ? 100 : 208) * 1024 / p.stage_bytes;
  if (p.stages > SG_MAX_STAGES) p.stages = SG_MAX_STAGES;
  p.tmem_cols = 32;
  while (p.tmem_cols < p.nt) p.tmem_cols *= 2;
  cudaError_t e = allow_smem<gemm_small_kernel>(227 * 1024);
  if (e != cudaSuccess) return (int)e;
  if (splits <= 0) {
    // as many blocks as fit in one wave, at least four stages of K each (shorter parts are all prologue).  K below 2048 is
    // not split: its rows keep the bits they have in the general kernel
    splits = 1;
    if (num_kb >= 32) {
      static sg_fit_t fit[9];
      splits = num_kb / 4 < 8 ? num_kb / 4 : 8;
      while (splits > 1 && tiles > sg_clusters_at_once<gemm_small_kernel>(fit, splits, SG_THREADS, pair ? 2 : 1)) splits--;
    }
  }
  if (splits > 8 || splits > num_kb) return 9100;
  p.splits = splits;
  // weights asked of L2 ahead of the loads: at most 48 MB over the grid
  p.prefetch_kb = (int)(48l * 1024 * 1024 / ((long)tiles * splits * SG_WBYTES));
  return 0;
}

static int launch_small(const void* A, const void* W, SmallGemmParams& p, int lda, int ldw, int splits, cudaStream_t stream) {
  const int rows = p.glu ? SG_ROWS / 2 : SG_ROWS;
  int rc = plan_small(p, splits);
  if (rc) return rc;
  CUtensorMap tw, ta;
  rc = get_tmap_2d_bf16(&tw, W, (uint64_t)p.N * (p.glu ? 2 : 1), (uint64_t)p.K, (uint64_t)ldw, rows);
  if (rc) return rc;
  rc = get_tmap_2d_bf16(&ta, A, (uint64_t)p.M, (uint64_t)p.K, (uint64_t)lda, p.nt);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits, (p.N + rows - 1) / rows);
  cfg.blockDim = dim3(SG_THREADS);
  cfg.dynamicSmemBytes = small_smem(p);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.splits;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return (int)cudaLaunchKernelEx(&cfg, gemm_small_kernel, tw, ta, p);
}

}  // namespace b200

using namespace b200;

// C[M,N] (row stride ldc) = A[M,K] * W[N,K]^T (+ bias[N]) (+ residual, row stride ldc), 1 <= M <= 256.  With glu, W is [gate;
// up] of 2N rows and C = silu(A gate^T) * (A up^T) (alpha > 0: the clamped gate of b200_gemm_glu_bf16; no bias or
// residual).  K, N and the strides are multiples of 8, bases 16-byte aligned.  splits: parts of K per tile, 0 = chosen.
B200_API int b200_gemm_small_bf16(const void* A, const void* W, void* C, const void* bias, const void* residual, int M, int N,
                                  int K, int lda, int ldw, int ldc, int glu, float alpha, float limit, int splits, int* status,
                                  cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 256 || K <= 0 || (K & 7) || (N & 7) || (lda & 7) || (ldw & 7) || (ldc & 7) || (glu && (bias || residual))) return 9100;
  SmallGemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.glu = glu; p.glu_alpha = alpha; p.glu_limit = limit;
  p.bias = (const __nv_bfloat16*)bias;
  p.residual = (const __nv_bfloat16*)residual;
  p.C = (__nv_bfloat16*)C;
  p.status = status;
  return launch_small(A, W, p, lda, ldw, splits, stream);
}

// The same with the row statistics of the output (b200_gemm_bf16_2cta_norm's row_ss_out): ss_out holds ss_parts_max parts of
// ss_stride rows and the part count; one part per 128 columns.
B200_API int b200_gemm_small_stats(const void* A, const void* W, void* C, const void* bias, const void* residual, int M, int N,
                                   int K, int lda, int ldw, int ldc, void* ss_out, long ss_stride, int ss_parts_max, int* status,
                                   cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 256 || K <= 0 || (K & 7) || (N & 7) || (lda & 7) || (ldw & 7) || (ldc & 7)) return 9100;
  if (!ss_out || ss_stride < M || (long)ss_parts_max * SG_ROWS < N) return 9135;
  SmallGemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.bias = (const __nv_bfloat16*)bias;
  p.residual = (const __nv_bfloat16*)residual;
  p.C = (__nv_bfloat16*)C;
  p.ss_out = (float*)ss_out;
  p.ss_stride = ss_stride;
  p.ss_parts_max = ss_parts_max;
  p.status = status;
  return launch_small(A, W, p, lda, ldw, 0, stream);
}

// Parts of K that a product of these sizes is split into where none are asked for (rules that choose between kernels); negative:
// refused.
B200_API int b200_gemm_small_splits(int M, int N, int K, int glu) {
  if (M <= 0 || N <= 0 || M > 256 || K <= 0) return -1;
  SmallGemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K;
  p.glu = glu;
  return plan_small(p, 0) ? -1 : p.splits;
}
