// Few-row block-scaled fp8 GEMM for sm_100a (at most 128 rows):
//   C[M,N] (bf16) = sum_kb  a_scale[m, kb] * w_scale[n/128, kb] * (A8[m, kb] . W8[n, kb]^T)  (+ bias)
//
// The form of gemm_small.cu (weights on the MMA's M axis, K split over a cluster, sums in shared memory in block order, launched as
// a programmatic dependent) with the two-level accumulation of gemm_fp8_block.cu: the product of one 128-column block goes to
// one of NB accumulators in tensor memory, eight warps scale it and add it to fp32 registers.  Tokens are columns here, so a
// thread (one weight row) needs the scales of all its tokens: they are staged per 32 K blocks as [block][token] products
// a_scale * w_scale, read back four at a time.
// Bound: one pass over the weights.  33 rows of a 70B-shaped layer (four products, 856 MB) 287 -> 180 us.
//   warps 0..7   promotion (two halves of the tokens), then all sums and stores;  warp 8  TMA producer;  warp 9  MMA issuer
#include "cluster_sum.cuh"
#include "common.cuh"

#include <mutex>
#include <unordered_map>

namespace b200 {

constexpr int SF_THREADS = 320;
constexpr int SF_WBYTES = SG_ROWS * 128;
constexpr int SF_MAX_STAGES = 12;
constexpr int SF_SCALE_KB = 32;

struct SmallFp8Params {
  int M, N, ldc, num_kb;
  int stages, stage_bytes, splits, prefetch_kb;
  const float* a_scale;            // [M, num_kb]
  const float* w_scale;            // [ceil(N / 128), num_kb]
  const __nv_bfloat16* bias;
  __nv_bfloat16* C;
  int* status;
};

// NT tokens: half of them per promotion warpgroup
template <int NT>
struct SfCfg {
  static constexpr int CPW = NT / 2;
  static constexpr int BLOCKS = NT <= 64 ? 2 : 1;            // per SM
  static constexpr int NB = 4;                               // accumulators in tensor memory
  static constexpr int TMEM_COLS = NB * NT < 32 ? 32 : NB * NT;      // 128, 256, 512
};

template <int NT>
__global__ void __launch_bounds__(SF_THREADS, SfCfg<NT>::BLOCKS)
gemm_small_fp8_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_a,
                      const SmallFp8Params p) {
  using Cfg = SfCfg<NT>;
  constexpr int NB = Cfg::NB, CPW = Cfg::CPW;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* scales = (float*)(smem + p.stages * p.stage_bytes);          // [SF_SCALE_KB][NT]
  uint64_t* full_bar = (uint64_t*)(scales + SF_SCALE_KB * NT);
  uint64_t* empty_bar = full_bar + SF_MAX_STAGES;
  uint64_t* part_full = empty_bar + SF_MAX_STAGES;
  uint64_t* part_empty = part_full + NB;
  uint32_t* tmem_ptr = (uint32_t*)(part_empty + NB);
  volatile int* abort_word = (volatile int*)(tmem_ptr + 1);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int split = blockIdx.x, tile = blockIdx.y;
  const int kb0 = (int)((long)p.num_kb * split / p.splits), kb1 = (int)((long)p.num_kb * (split + 1) / p.splits);
  const int w_row = tile * SG_ROWS;

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < NB; b++) {
      mbar_init(&part_full[b], 1);
      mbar_init(&part_empty[b], 8);
    }
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tmap_w);
    tma_prefetch_desc(&tmap_a);
    for (int kb = kb0; kb < min(kb1, kb0 + p.prefetch_kb); kb++) tma_prefetch_l2_2d(&tmap_w, kb * 128, w_row);
  }
  if (warp == 9) {
    tmem_alloc(tmem_ptr, Cfg::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_ptr);
  asm volatile("griddepcontrol.wait;" ::: "memory");

  bool ok = true;
  if (warp == 8) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0; kb < kb1; kb++) {
        if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_word)) break;
        uint8_t* sw = smem + stage * p.stage_bytes;
        mbar_expect_tx(&full_bar[stage], SF_WBYTES + NT * 128);
        tma_load_2d(sw, &tmap_w, &full_bar[stage], kb * 128, w_row);
        tma_load_2d(sw + SF_WBYTES, &tmap_a, &full_bar[stage], kb * 128, 0);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else if (warp == 9) {
    // ------------------------------------------------------------ MMA issuer: one thread walks the loop (see warp_uniform)
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_e4m3(SG_ROWS, NT);
      const uint64_t dw0 = make_smem_desc(smem_u32(smem), 16, 1024, kLayoutSw128);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = kb0, it = 0; kb < kb1; kb++, it++) {
        const int b = it % NB;
        if (!mbar_wait(&part_empty[b], ((uint32_t)(it / NB) & 1u) ^ 1u, abort_word) ||
            !mbar_wait(&full_bar[stage], phase, abort_word))
          break;
        tc_fence_after();
        const uint64_t dw = dw0 + (uint32_t)(stage * (p.stage_bytes >> 4)), da = dw + (SF_WBYTES >> 4);
#pragma unroll
        for (int kk = 0; kk < 4; kk++) umma_f8_ss(tmem_base + b * NT, dw + 2 * kk, da + 2 * kk, idesc, kk > 0 ? 1u : 0u);
        umma_commit(&empty_bar[stage]);
        umma_commit(&part_full[b]);
        if (++stage == p.stages) { stage = 0; phase ^= 1; }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------ promotion
    const int half = warp >> 2;
    const uint32_t t_row = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + half * CPW;
    float acc[CPW];
#pragma unroll
    for (int i = 0; i < CPW; i++) acc[i] = 0.f;
    const float* ws = p.w_scale + (size_t)tile * p.num_kb;
    for (int c0 = kb0, it = 0; c0 < kb1; c0 += SF_SCALE_KB) {
      const int n = min(SF_SCALE_KB, kb1 - c0);
      asm volatile("bar.sync 1, 256;" ::: "memory");          // the previous scales have been read
      for (int t = warp; t < NT; t += 8)                      // lane = K block: rows of a_scale are read along
        scales[lane * NT + t] = lane < n && t < p.M ? p.a_scale[(size_t)t * p.num_kb + c0 + lane] * ws[c0 + lane] : 0.f;
      asm volatile("bar.sync 1, 256;" ::: "memory");
      for (int k = 0; k < n; k++, it++) {
        const int b = it % NB;
        ok = ok && mbar_wait(&part_full[b], (uint32_t)(it / NB) & 1u, abort_word);
        if (!ok) break;                                       // the barriers above are still met by every warp
        tc_fence_after();
        uint32_t r[CPW];
#pragma unroll
        for (int c = 0; c < CPW; c += 16) tmem_ld_32x32b_x16(t_row + b * NT + c, r + c);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&part_empty[b]);
        const float4* sc = reinterpret_cast<const float4*>(scales + k * NT + half * CPW);
#pragma unroll
        for (int c = 0; c < CPW / 4; c++) {
          const float4 f = sc[c];
          acc[4 * c] = fmaf(__uint_as_float(r[4 * c]), f.x, acc[4 * c]);
          acc[4 * c + 1] = fmaf(__uint_as_float(r[4 * c + 1]), f.y, acc[4 * c + 1]);
          acc[4 * c + 2] = fmaf(__uint_as_float(r[4 * c + 2]), f.z, acc[4 * c + 2]);
          acc[4 * c + 3] = fmaf(__uint_as_float(r[4 * c + 3]), f.w, acc[4 * c + 3]);
        }
      }
    }
    // every stage has been consumed: the last product is in registers
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if (ok) {
      float* part = (float*)smem + (size_t)half * CPW * SG_ROWS + (warp & 3) * 32 + lane;
#pragma unroll
      for (int i = 0; i < CPW; i++) part[i * SG_ROWS] = acc[i];
    }
  }
  if (p.splits > 1) sg_cluster_sync();
  else __syncthreads();

  const uint32_t part = smem_u32(smem);
  const int t0 = p.M * split / p.splits, t1 = p.M * (split + 1) / p.splits;
  if (*abort_word == 0) {
    const int col = tile * SG_ROWS + lane * 4;
    for (int t = t0 + warp; t < t1; t += SF_THREADS / 32) {
      float4 v = sg_sum(part, p.splits, (uint32_t)(t * SG_ROWS + lane * 4) * 4);
      if (col < p.N) {                                        // N is a multiple of 8
        if (p.bias) {
          const uint2 b = *reinterpret_cast<const uint2*>(p.bias + col);
          const float2 b0 = unpack_bf16x2(b.x), b1 = unpack_bf16x2(b.y);
          v.x += b0.x; v.y += b0.y; v.z += b1.x; v.w += b1.y;
        }
        *reinterpret_cast<uint2*>(p.C + (size_t)t * p.ldc + col) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
      }
    }
  }
  if (p.splits > 1) sg_cluster_sync();                        // no block leaves while another reads its sums
  else __syncthreads();
  if (*abort_word != 0) {
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 50000ull) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, *abort_word);
    __syncthreads();
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// row-major 8-bit matrix, box of box_rows x 128 bytes, 128-byte swizzle; maps are kept by what they encode
static int sf_tmap(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_rows) {
  struct Key {
    const void* ptr;
    uint64_t rows, cols, ld, box;
    bool operator==(const Key& o) const { return ptr == o.ptr && rows == o.rows && cols == o.cols && ld == o.ld && box == o.box; }
  };
  struct Hash {
    size_t operator()(const Key& k) const {
      size_t h = (size_t)k.ptr;
      for (uint64_t v : {k.rows, k.cols, k.ld, k.box}) h = h * 1000003u ^ v;
      return h;
    }
  };
  static std::unordered_map<Key, CUtensorMap, Hash> cache;
  static std::mutex mu;
  const Key key{ptr, rows, cols, ld, box_rows};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  uint64_t dims[2] = {cols, rows}, strides[1] = {ld};
  uint32_t box[2] = {128, box_rows};
  const int rc = make_tmap(out, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  if (cache.size() > 8192) cache.clear();
  cache.emplace(key, *out);
  return 0;
}

template <int NT>
static int sf_smem(const SmallFp8Params& p) {
  return p.stages * p.stage_bytes + SF_SCALE_KB * NT * 4 + (2 * SF_MAX_STAGES + 2 * SfCfg<NT>::NB) * 8 + 16 + 1024;
}

// Stages and (where none are asked for) splits of K.  Nonzero: refused.
template <int NT>
static int plan_sf(SmallFp8Params& p, int splits) {
  using Cfg = SfCfg<NT>;
  const int tiles = (p.N + SG_ROWS - 1) / SG_ROWS;
  p.stage_bytes = SF_WBYTES + NT * 128;
  p.stages = 0;
  p.stages = ((Cfg::BLOCKS == 2 ? 112 : 224) * 1024 - sf_smem<NT>(p)) / p.stage_bytes;
  if (p.stages > SF_MAX_STAGES) p.stages = SF_MAX_STAGES;
  cudaError_t e = allow_smem<gemm_small_fp8_kernel<NT>>(227 * 1024);
  if (e != cudaSuccess) return (int)e;
  if (splits <= 0) {
    // one wave of blocks, at least four K blocks each; K below 2048 is not split (rows keep the general kernel's bits)
    splits = 1;
    if (p.num_kb >= 16) {
      static sg_fit_t fit[9];
      splits = p.num_kb / 4 < 8 ? p.num_kb / 4 : 8;
      while (splits > 1 && tiles > sg_clusters_at_once<gemm_small_fp8_kernel<NT>>(fit, splits, SF_THREADS, Cfg::BLOCKS)) splits--;
    }
  }
  if (splits > 8 || splits > p.num_kb) return 9100;
  p.splits = splits;
  p.prefetch_kb = (int)(48l * 1024 * 1024 / ((long)tiles * splits * SF_WBYTES));      // at most 48 MB over the grid
  return 0;
}

template <int NT>
static int launch_sf(const void* A, const void* W, SmallFp8Params& p, int lda, int ldw, int splits, cudaStream_t stream) {
  int rc = plan_sf<NT>(p, splits);
  if (rc) return rc;
  CUtensorMap tw, ta;
  rc = sf_tmap(&tw, W, (uint64_t)p.N, (uint64_t)p.num_kb * 128, (uint64_t)ldw, SG_ROWS);
  if (rc) return rc;
  rc = sf_tmap(&ta, A, (uint64_t)p.M, (uint64_t)p.num_kb * 128, (uint64_t)lda, NT);
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.splits, (p.N + SG_ROWS - 1) / SG_ROWS);
  cfg.blockDim = dim3(SF_THREADS);
  cfg.dynamicSmemBytes = sf_smem<NT>(p);
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
  return (int)cudaLaunchKernelEx(&cfg, gemm_small_fp8_kernel<NT>, tw, ta, p);
}

}  // namespace b200

using namespace b200;

// As b200_gemm_fp8_block, 1 <= M <= 128.  splits: parts of K per tile, 0 = chosen.
B200_API int b200_gemm_small_fp8(const void* A8, const void* a_scale, const void* W8, const void* w_scale, void* C, const void* bias,
                                 int M, int N, int K, int lda, int ldw, int ldc, int splits, int* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (M > 128 || K <= 0 || (K % 128) || (N & 7) || (lda & 15) || (ldw & 15) || (ldc & 7)) return 9100;
  SmallFp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.ldc = ldc; p.num_kb = K / 128;
  p.a_scale = (const float*)a_scale;
  p.w_scale = (const float*)w_scale;
  p.bias = (const __nv_bfloat16*)bias;
  p.C = (__nv_bfloat16*)C;
  p.status = status;
  if (M <= 32) return launch_sf<32>(A8, W8, p, lda, ldw, splits, stream);
  if (M <= 64) return launch_sf<64>(A8, W8, p, lda, ldw, splits, stream);
  return launch_sf<128>(A8, W8, p, lda, ldw, splits, stream);
}

// Parts of K that a product of these sizes is split into where none are asked for; negative: refused.
B200_API int b200_gemm_small_fp8_splits(int M, int N, int K) {
  if (M <= 0 || N <= 0 || M > 128 || K < 128) return -1;
  SmallFp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.num_kb = K / 128;
  const int rc = M <= 32 ? plan_sf<32>(p, 0) : M <= 64 ? plan_sf<64>(p, 0) : plan_sf<128>(p, 0);
  return rc ? -1 : p.splits;
}
