// Block-scaled FP8 GEMM for sm_100a (the W8A8 serving format of DeepSeek-V3 style
// checkpoints):
//   C[M,N] (bf16) = sum_kb  a_scale[m, kb] * w_scale[n/128, kb] * (A8[m, kb] . W8[n, kb]^T)
// A8 [M,K] e4m3 with one fp32 scale per (row, 128 columns); W8 [N,K] e4m3 with one
// fp32 scale per 128 x 128 block.  Reference scheme: vllm_ascend/quantization/methods/fp8.py
// (block-scaled weights) + w8a8_dynamic.py (per-token activation scales).
//
// The scales change every 128 columns of K, so products of different K blocks cannot
// be summed inside the tensor core.  Two-level accumulation:
//   warp 0      TMA producer: 128 x 128 e4m3 tiles of A, BN x 128 of W (one 128-byte swizzle row each)
//   warp 1      tcgen05.mma kind::f8f6f4 (M=128, N=BN, K=32 x 4) per K block into one of two
//               TMEM partial buffers (fresh accumulator every block)
//   warps 2..   read the partial with tcgen05.ld, scale it by a_scale * w_scale and add it to
//               fp32 accumulators held in registers; store bf16 at the end.  A warpgroup per 64
//               columns of the tile (64 accumulators per thread): the promotion of a block has to keep up
//               with its MMA, which four warps with 128 accumulators each did not
//   last two    multiply the scales of rows and columns and put them into shared memory, eight K blocks ahead
// Tiles are 128 x 256 where they fill the GPU as well as 128 x 128 do: a K block of the small tile brings 32 KB for
// 4.2 MFLOP, of the wide one 24 KB for the same.  4096^3: 1509 TFLOP/s (1130 before the scales lay in shared memory and the issue
// loops were one thread's); what bounds a block is the promotion, not the MMA, whose peak is three times that.
// The MMA of block kb+1 overlaps the promotion of block kb.  Grouped mode (MoE experts)
// uses per-group row offsets and per-expert weight / scale matrices.  Bounded waits.
#include "common.cuh"

#include <mutex>
#include <unordered_map>

namespace b200 {

constexpr int F8_BM = 128, F8_BK = 128;
constexpr int F8_BLOCK = 128;              // rows of W that share a scale
constexpr int F8_COLS = 64;                // columns per promotion warpgroup
constexpr int F8_TILE_BYTES = 128 * 128;                 // 16 KB per 128 operand rows
constexpr int F8_MAX_GROUPS = 512;
// K blocks whose scales (row times block of columns) lie in shared memory together, twice: loads of a scale per row and block by the
// promotion itself, a line of memory per lane, took 210 of the 1140 clocks of a block
constexpr int F8_SCALE_KB = 8;

template <int BN>
struct F8Cfg {
  static constexpr int kThreads = 128 + 2 * BN;          // producer, MMA issuer, BN / 64 promotion warpgroups, two warps for scales
  static constexpr int kStages = BN == 256 ? 4 : 6;
  static constexpr int kStageBytes = F8_TILE_BYTES * (1 + BN / 128);
  static constexpr int kScaleBytes = 2 * F8_SCALE_KB * (BN / 128) * F8_BM * 4;
  static constexpr int kSmemBytes = kStages * kStageBytes + kScaleBytes + 1024 + 256 + (F8_MAX_GROUPS + 1) * 4;
};

struct Fp8Params {
  int M, N, K, ldc;
  const float* a_scale;     // [M, K/128]
  const float* w_scale;     // [groups][ceil(N/128), K/128]
  __nv_bfloat16* C;
  const __nv_bfloat16* bias;
  int* status;
  int tiles_m, tiles_n;
  int num_kb;
  // per-channel mode (dynamic per-token x per-output-channel scales, constant along K):
  // row_scale [M], col_scale [groups][N]; the K blocks are summed unscaled and the product of
  // the two scales is applied once in the epilogue
  const float* row_scale;
  const float* col_scale;
  // grouped
  const int* group_offsets;
  int num_groups;
  int w_rows_per_group;
};

struct F8Tile {
  int row0, row_end, tn, w_row0, group;
};

template <int BN>
__device__ __forceinline__ void f8_tile(const Fp8Params& p, const int* grp_tiles, int t, F8Tile& c) {
  if (p.num_groups > 0) {
    const int total_m = grp_tiles[p.num_groups];
    const int tm_global = t % total_m;
    const int tn = t / total_m;
    int lo = 0, hi = p.num_groups;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (grp_tiles[mid] <= tm_global) lo = mid; else hi = mid;
    }
    c.group = lo;
    c.row0 = p.group_offsets[lo] + (tm_global - grp_tiles[lo]) * F8_BM;
    c.row_end = p.group_offsets[lo + 1];
    c.tn = tn;
    c.w_row0 = lo * p.w_rows_per_group + tn * BN;
  } else {
    c.group = 0;
    c.row0 = (t % p.tiles_m) * F8_BM;
    c.row_end = p.M;
    c.tn = t / p.tiles_m;
    c.w_row0 = c.tn * BN;
  }
}

template <int BN>
__global__ void __launch_bounds__(F8Cfg<BN>::kThreads, 1)
gemm_fp8_block_kernel(const __grid_constant__ CUtensorMap tmap_a,
                      const __grid_constant__ CUtensorMap tmap_b, const Fp8Params p) {
  constexpr int F8_STAGES = F8Cfg<BN>::kStages, F8_STAGE_BYTES = F8Cfg<BN>::kStageBytes;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* tiles = smem;
  constexpr int NB = BN / 128;                    // scale blocks of a tile's columns
  float* scales = (float*)(smem + F8_STAGES * F8_STAGE_BYTES);        // [2][F8_SCALE_KB][NB][rows]
  uint64_t* full_bar = (uint64_t*)(smem + F8_STAGES * F8_STAGE_BYTES + F8Cfg<BN>::kScaleBytes);
  uint64_t* empty_bar = full_bar + F8_STAGES;
  uint64_t* part_full = empty_bar + F8_STAGES;    // [2]
  uint64_t* part_empty = part_full + 2;           // [2]
  uint64_t* sc_full = part_empty + 2;             // [2]
  uint64_t* sc_empty = sc_full + 2;               // [2]
  uint32_t* tmem_ptr = (uint32_t*)(sc_empty + 2);
  volatile int* abort_word = (volatile int*)(tmem_ptr + 1);
  int* grp_tiles = (int*)(tmem_ptr + 2);

  const int warp = warp_index(), lane = threadIdx.x & 31;
  const int num_kb = p.num_kb;

  if (threadIdx.x == 0) {
    for (int s = 0; s < F8_STAGES; s++) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; b++) {
      mbar_init(&part_full[b], 1);
      mbar_init(&part_empty[b], 4 * (BN / F8_COLS));
      mbar_init(&sc_full[b], 2);
      mbar_init(&sc_empty[b], 4 * (BN / F8_COLS));
    }
    *abort_word = 0;
    mbar_fence_init();
    if (p.num_groups > 0) {
      // a table that is not ascending inside [0, M] is reported and yields no tiles
      int acc = 0;
      bool ok = p.group_offsets[0] >= 0;
      for (int e = 0; e < p.num_groups; e++) {
        grp_tiles[e] = acc;
        const int g0 = p.group_offsets[e], g1 = p.group_offsets[e + 1];
        if (g1 < g0 || g1 > p.M) ok = false;
        acc += ok ? (g1 - g0 + F8_BM - 1) / F8_BM : 0;
      }
      if (!ok) {
        for (int e = 0; e <= p.num_groups; e++) grp_tiles[e] = 0;
        acc = 0;
        if (p.status) atomicCAS(p.status, 0, B200_BAD_INDEX);
      }
      grp_tiles[p.num_groups] = acc;
    }
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, 2 * BN);
    tmem_relinquish();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmap_a);
    tma_prefetch_desc(&tmap_b);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_ptr);
  const int num_tiles = (p.num_groups > 0 ? grp_tiles[p.num_groups] : p.tiles_m) * p.tiles_n;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        F8Tile c;
        f8_tile<BN>(p, grp_tiles, t, c);
        for (int kb = 0; kb < num_kb; kb++) {
          if (!mbar_wait(&empty_bar[stage], phase ^ 1, abort_word)) goto done;
          uint8_t* sa = tiles + stage * F8_STAGE_BYTES;
          mbar_expect_tx(&full_bar[stage], F8_STAGE_BYTES);
          tma_load_2d(sa, &tmap_a, &full_bar[stage], kb * F8_BK, c.row0);
#pragma unroll
          for (int h = 0; h < BN / 128; h++)
            tma_load_2d(sa + (1 + h) * F8_TILE_BYTES, &tmap_b, &full_bar[stage], kb * F8_BK, c.w_row0 + h * 128);
          if (++stage == F8_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer: one thread walks the loop (see warp_uniform)
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_e4m3(F8_BM, BN);
      const uint64_t da0 = make_smem_desc(smem_u32(tiles), 16, 1024, kLayoutSw128);
      int stage = 0;
      uint32_t phase = 0;
      uint32_t it = 0;          // K blocks issued so far (selects the partial buffer)
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        for (int kb = 0; kb < num_kb; kb++, it++) {
          const int b = it & 1;
          if (!mbar_wait(&part_empty[b], ((it >> 1) & 1u) ^ 1u, abort_word)) goto done;
          if (!mbar_wait(&full_bar[stage], phase, abort_word)) goto done;
          tc_fence_after();
          const uint64_t da = da0 + (uint32_t)(stage * (F8_STAGE_BYTES >> 4)), db = da + (F8_TILE_BYTES >> 4);
#pragma unroll
          for (int kk = 0; kk < F8_BK / 32; kk++)         // 32 e4m3 = 32 bytes per MMA
            umma_f8_ss(tmem_base + b * BN, da + 2 * kk, db + 2 * kk, idesc, kk > 0 ? 1u : 0u);
          umma_commit(&empty_bar[stage]);
          umma_commit(&part_full[b]);
          if (++stage == F8_STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp >= 2 + BN / 16) {
    // ------------------------------------------------------------ scales (two warps, two rows per thread)
    if (p.row_scale == nullptr) {
      const int t64 = threadIdx.x - (64 + 2 * BN), kblocks = p.K / F8_BK, n_blocks = (p.N + F8_BLOCK - 1) / F8_BLOCK;
      uint32_t grp = 0;
      for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
        F8Tile c;
        f8_tile<BN>(p, grp_tiles, t, c);
        const float* ws[NB];
#pragma unroll
        for (int h = 0; h < NB; h++)                       // columns beyond N have no scale
          ws[h] = p.w_scale + ((size_t)c.group * n_blocks + min(c.tn * NB + h, n_blocks - 1)) * kblocks;
        for (int k0 = 0; k0 < num_kb; k0 += F8_SCALE_KB, grp++) {
          const int b = grp & 1, n = min(F8_SCALE_KB, num_kb - k0);
          if (!mbar_wait(&sc_empty[b], ((grp >> 1) & 1u) ^ 1u, abort_word)) goto done;
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const int r = t64 + 64 * i, row = c.row0 + r;
            const float* as = p.a_scale + (size_t)(row < c.row_end ? row : c.row0) * kblocks + k0;
            float a[F8_SCALE_KB];
            if ((kblocks & 3) == 0 && (reinterpret_cast<uintptr_t>(p.a_scale) & 15) == 0 && n == F8_SCALE_KB) {
#pragma unroll
              for (int k = 0; k < F8_SCALE_KB; k += 4) {
                const float4 v = *reinterpret_cast<const float4*>(as + k);
                a[k] = v.x; a[k + 1] = v.y; a[k + 2] = v.z; a[k + 3] = v.w;
              }
            } else {
#pragma unroll
              for (int k = 0; k < F8_SCALE_KB; k++) a[k] = k < n ? as[k] : 0.f;
            }
#pragma unroll
            for (int k = 0; k < F8_SCALE_KB; k++)
#pragma unroll
              for (int h = 0; h < NB; h++)
                if (k < n) scales[((b * F8_SCALE_KB + k) * NB + h) * F8_BM + r] = a[k] * ws[h][k0 + k];
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sc_full[b]);
        }
      }
    }
  } else {
    // ------------------------------------------------------------ promotion + epilogue
    const int q = warp & 3;                              // TMEM lane quarter this warp may read
    const int wg = (warp - 2) >> 2;                      // which 64 columns of the tile
    uint32_t grp = 0;                                    // groups of scales so far
    uint32_t it = 0;
    for (int t = blockIdx.x; t < num_tiles; t += gridDim.x) {
      F8Tile c;
      f8_tile<BN>(p, grp_tiles, t, c);
      const int row = c.row0 + q * 32 + lane;
      const bool row_ok = row < c.row_end;
      const bool per_channel = p.row_scale != nullptr;
      float acc[F8_COLS];
#pragma unroll
      for (int i = 0; i < F8_COLS; i++) acc[i] = 0.f;
      for (int kb = 0; kb < num_kb; kb++, it++) {
        const int b = it & 1;
        float sc = 1.f;
        if (!per_channel) {
          const int k = kb % F8_SCALE_KB, sb = grp & 1;
          if (k == 0 && !mbar_wait(&sc_full[sb], (grp >> 1) & 1u, abort_word)) goto done;
          sc = scales[((sb * F8_SCALE_KB + k) * NB + wg * F8_COLS / F8_BLOCK) * F8_BM + q * 32 + lane];
          if (k == F8_SCALE_KB - 1 || kb + 1 == num_kb) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&sc_empty[sb]);
            grp++;
          }
        }
        if (!mbar_wait(&part_full[b], (it >> 1) & 1u, abort_word)) goto done;
        tc_fence_after();
        const uint32_t t_row = tmem_base + ((uint32_t)(q * 32) << 16) + b * BN + wg * F8_COLS;
        if constexpr (BN == 128) {
          uint32_t r0[32], r1[32];
          tmem_ld_32x32b_x32(t_row, r0);
          tmem_ld_32x32b_x32(t_row + 32, r1);
          tmem_ld_wait();
          // the partial is in registers: the MMA warp may overwrite the buffer
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&part_empty[b]);
#pragma unroll
          for (int i = 0; i < 32; i++) acc[i] = fmaf(__uint_as_float(r0[i]), sc, acc[i]);
#pragma unroll
          for (int i = 0; i < 32; i++) acc[32 + i] = fmaf(__uint_as_float(r1[i]), sc, acc[32 + i]);
        } else {
          // 640 threads have 96 registers: eight columns at a time leave the accumulators and the loop their own (2048 x 57344 x 8192 by itself:
          // 1074 us with sixteen and a load of scales in every thread, 937 to 960 so; sixteen with scales from shared memory were no gain, for what
          // was then spilled around the loop)
#pragma unroll
          for (int c0 = 0; c0 < F8_COLS; c0 += 8) {
            uint32_t r[8];
            tmem_ld_32x32b_x8(t_row + c0, r);
            tmem_ld_wait();
            if (c0 + 8 == F8_COLS) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&part_empty[b]);
            }
#pragma unroll
            for (int i = 0; i < 8; i++) acc[c0 + i] = fmaf(__uint_as_float(r[i]), sc, acc[c0 + i]);
          }
        }
      }
      if (row_ok) {
        __nv_bfloat16* crow = p.C + (size_t)row * p.ldc;
        const float rs = per_channel ? p.row_scale[row] : 1.f;
        const float* cs = per_channel ? p.col_scale + (size_t)c.group * p.N : nullptr;
#pragma unroll
        for (int g = 0; g < F8_COLS / 8; g++) {
          const int col = c.tn * BN + wg * F8_COLS + g * 8;
          if (col < p.N) {
            float v[8];
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = acc[g * 8 + j];
            if (per_channel) {
              const float4 c0 = *reinterpret_cast<const float4*>(cs + col);
              const float4 c1 = *reinterpret_cast<const float4*>(cs + col + 4);
              const float cv[8] = {c0.x, c0.y, c0.z, c0.w, c1.x, c1.y, c1.z, c1.w};
#pragma unroll
              for (int j = 0; j < 8; j++) v[j] *= rs * cv[j];
            }
            if (p.bias) {
              const uint4 bv = *reinterpret_cast<const uint4*>(p.bias + col);
              const uint32_t bw[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
              for (int j = 0; j < 4; j++) {
                const float2 f = unpack_bf16x2(bw[j]);
                v[2 * j] += f.x;
                v[2 * j + 1] += f.y;
              }
            }
            *reinterpret_cast<uint4*>(crow + col) =
                make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]),
                           pack_bf16x2(v[4], v[5]), pack_bf16x2(v[6], v[7]));
          }
        }
      }
    }
  }
done:
  __syncwarp();             // the elected threads come back to their warps
  tc_fence_before();
  __syncthreads();
  if (*abort_word != 0) {
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 50000ull) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, *abort_word);
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

// ---------------------------------------------------------------- host
struct F8Key {
  const void* ptr;
  uint64_t rows, cols, ld;
  bool operator==(const F8Key& o) const {
    return ptr == o.ptr && rows == o.rows && cols == o.cols && ld == o.ld;
  }
};
struct F8Hash {
  size_t operator()(const F8Key& k) const {
    size_t h = (size_t)k.ptr;
    h = h * 1000003u ^ k.rows;
    h = h * 1000003u ^ k.cols;
    h = h * 1000003u ^ k.ld;
    return h;
  }
};

// row-major 8-bit [rows, cols] (row stride ld bytes), box 128 rows x 128 bytes, 128B swizzle
static int get_tmap_u8(CUtensorMap* out, const void* ptr, uint64_t rows, uint64_t cols,
                       uint64_t ld) {
  static std::unordered_map<F8Key, CUtensorMap, F8Hash> cache;
  static std::mutex mu;
  F8Key key{ptr, rows, cols, ld};
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(key);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  uint64_t dims[2] = {cols, rows};
  uint64_t strides[1] = {ld};
  uint32_t box[2] = {128, 128};
  int rc = make_tmap(out, ptr, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, dims, strides, box,
                     CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  if (cache.size() > 8192) cache.clear();
  cache.emplace(key, *out);
  return 0;
}

template <int BN>
static int launch_fp8_bn(const CUtensorMap& ta, const CUtensorMap& tb, Fp8Params& p, cudaStream_t stream) {
  using Cfg = F8Cfg<BN>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(gemm_fp8_block_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::kSmemBytes);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  p.tiles_n = (p.N + BN - 1) / BN;
  int grid = num_sms();
  if (p.num_groups == 0 && p.tiles_m * p.tiles_n < grid) grid = p.tiles_m * p.tiles_n;
  gemm_fp8_block_kernel<BN><<<grid, Cfg::kThreads, Cfg::kSmemBytes, stream>>>(ta, tb, p);
  return B200_CHECK_LAUNCH();
}

static int launch_fp8(const void* A, const void* W, Fp8Params& p, int lda, int ldw, long a_rows,
                      long w_rows, cudaStream_t stream) {
  CUtensorMap ta, tb;
  int rc = get_tmap_u8(&ta, A, (uint64_t)a_rows, (uint64_t)p.K, (uint64_t)lda);
  if (rc) return rc;
  rc = get_tmap_u8(&tb, W, (uint64_t)w_rows, (uint64_t)p.K, (uint64_t)ldw);
  if (rc) return rc;
  p.tiles_m = (p.M + F8_BM - 1) / F8_BM;
  p.num_kb = p.K / F8_BK;
  // waves times width: a wide tile counts 1.6 narrow ones.  Groups keep the narrow tile (their rows are not known here).
  const long sms = num_sms();
  auto waves = [&](int bn) { return ((long)p.tiles_m * ((p.N + bn - 1) / bn) + sms - 1) / sms; };
  if (p.num_groups == 0 && waves(256) * 16 < waves(128) * 10) return launch_fp8_bn<256>(ta, tb, p, stream);
  return launch_fp8_bn<128>(ta, tb, p, stream);
}

}  // namespace b200

using namespace b200;

// C[M,N] bf16 = block-scaled product of A8 [M,K] e4m3 (a_scale [M, K/128] fp32) and
// W8 [N,K] e4m3 (w_scale [ceil(N/128), K/128] fp32).  K multiple of 128, N multiple of 8.
B200_API int b200_gemm_fp8_block(const void* A8, const void* a_scale, const void* W8,
                                 const void* w_scale, void* C, const void* bias, int M, int N,
                                 int K, int lda, int ldw, int ldc, int* status,
                                 cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if ((K % 128) || (N & 7) || (lda & 15) || (ldw & 15) || (ldc & 7)) return 9100;
  Fp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.a_scale = (const float*)a_scale;
  p.w_scale = (const float*)w_scale;
  p.C = (__nv_bfloat16*)C;
  p.bias = (const __nv_bfloat16*)bias;
  p.status = status;
  return launch_fp8(A8, W8, p, lda, ldw, M, N, stream);
}

// Grouped variant: rows [offsets[e], offsets[e+1]) of A8 use expert e's W8[e] ([N,K]) and
// w_scale[e] ([ceil(N/128), K/128]).
B200_API int b200_grouped_gemm_fp8_block(const void* A8, const void* a_scale, const void* W8,
                                         const void* w_scale, void* C, const void* offsets,
                                         int num_groups, long total_rows, int N, int K, int lda,
                                         int ldw, int ldc, int* status, cudaStream_t stream) {
  if (total_rows <= 0 || N <= 0 || num_groups <= 0) return 0;
  if ((K % 128) || (N & 7) || (lda & 15) || (ldw & 15) || (ldc & 7)) return 9100;
  if (num_groups > F8_MAX_GROUPS) return 9131;
  Fp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = (int)total_rows; p.N = N; p.K = K; p.ldc = ldc;
  p.a_scale = (const float*)a_scale;
  p.w_scale = (const float*)w_scale;
  p.C = (__nv_bfloat16*)C;
  p.status = status;
  p.group_offsets = (const int*)offsets;
  p.num_groups = num_groups;
  p.w_rows_per_group = N;
  return launch_fp8(A8, W8, p, lda, ldw, total_rows, (long)num_groups * N, stream);
}

// Per-token x per-channel form (dynamic W8A8 in e4m3): C = row_scale[m] * col_scale[n] * (A8 . W8^T).
// row_scale [M] fp32, col_scale [N] fp32 (16-byte aligned, N multiple of 8).
B200_API int b200_gemm_fp8_channel(const void* A8, const void* row_scale, const void* W8,
                                   const void* col_scale, void* C, const void* bias, int M, int N,
                                   int K, int lda, int ldw, int ldc, int* status,
                                   cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if ((K % 128) || (N & 7) || (lda & 15) || (ldw & 15) || (ldc & 7) || ((uintptr_t)col_scale & 15))
    return 9100;
  Fp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = M; p.N = N; p.K = K; p.ldc = ldc;
  p.row_scale = (const float*)row_scale;
  p.col_scale = (const float*)col_scale;
  p.C = (__nv_bfloat16*)C;
  p.bias = (const __nv_bfloat16*)bias;
  p.status = status;
  return launch_fp8(A8, W8, p, lda, ldw, M, N, stream);
}

// Grouped per-channel form: expert e's W8[e] [N,K] with col_scale[e] [N].
B200_API int b200_grouped_gemm_fp8_channel(const void* A8, const void* row_scale, const void* W8,
                                           const void* col_scale, void* C, const void* offsets,
                                           int num_groups, long total_rows, int N, int K, int lda,
                                           int ldw, int ldc, int* status, cudaStream_t stream) {
  if (total_rows <= 0 || N <= 0 || num_groups <= 0) return 0;
  if ((K % 128) || (N & 7) || (lda & 15) || (ldw & 15) || (ldc & 7) || ((uintptr_t)col_scale & 15))
    return 9100;
  if (num_groups > F8_MAX_GROUPS) return 9131;
  Fp8Params p;
  memset(&p, 0, sizeof(p));
  p.M = (int)total_rows; p.N = N; p.K = K; p.ldc = ldc;
  p.row_scale = (const float*)row_scale;
  p.col_scale = (const float*)col_scale;
  p.C = (__nv_bfloat16*)C;
  p.status = status;
  p.group_offsets = (const int*)offsets;
  p.num_groups = num_groups;
  p.w_rows_per_group = N;
  return launch_fp8(A8, W8, p, lda, ldw, total_rows, (long)num_groups * N, stream);
}
