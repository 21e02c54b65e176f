// Gated delta rule over prompts in chunks of 64 tokens, on tcgen05 (key dimension 128).
//
//     S <- S e^{g_t};  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t
//
// With gamma_j the running sum of g inside a chunk entered with S0, and e_jm = e^{gamma_j - gamma_m}:
//     u_j + sum_{m<j} beta_j e_jm (k_j . k_m) u_m = beta_j (v_j - e^{gamma_j} S0^T k_j)        (a triangular solve)
//     o_j = e^{gamma_j} S0^T q_j + sum_{m<=j} e_jm (q_j . k_m) u_m
//     S   = e^{gamma_C} S0 + sum_j k_j (e^{gamma_C - gamma_j} u_j)^T
// (the UT form of DeltaNet, Yang et al. 2024; counterpart of vllm_ascend/ops/triton/fla/chunk.py).
//
// Bound: the token-serial kernel (linear_attention.cu) spends 0.7 us per token of a sequence whatever the batch.  Here a chunk of 64
// takes 36,900 clocks (19 us) one after the other: 11,800 are the solve and 8,800 the new state and its parts (CUDA cores, bound by
// what shared memory returns), the rest staging, products and factors.  6000 tokens in three prompts, 32 heads: 1603 -> about 780 us.
//
// 32 bits stay 32 bits.  q and k are bf16 as they come, so k . k and q . k are exact products summed in fp32; their norms
// are factors of rows.  The state and u are fp32: as MMA operands they are three bf16 parts (8 + 8 + 8 bits), which times
// an exact bf16 operand is the fp32 product.  gamma is summed in fp64 and kept in two floats; the solve and the sum over m
// are fp32 FMAs.
//
// One block per (sequence, value head, COLS value columns); the state lives in tensor memory (lane = key row).  Per chunk:
//   all          k, q, v of the chunk -> shared memory (loaded a chunk ahead), norms, gamma
//   MMA          [K; Q] K^T  and  [K; Q] S0 (three parts)
//   warps 0..3   products -> A^T, P^T (factors e_jm, beta, norms);    warps 4..7   S0 products -> right-hand sides, read-outs
//   warps 0..3   solve
//   warps 0..3   u -> three bf16 parts, S0 decayed in place, MMA K^T u;     warps 4..7   outputs
//   warps 0..3   the new state -> three bf16 parts
#include "common.cuh"
#include "delta_chunk.h"
#include "dtypes.cuh"

namespace b200 {

constexpr int DC_C = 64, DC_K = 128, DC_THREADS = 256;
constexpr int DC_PITCH = 68;            // floats per row of A^T / P^T: 16-byte rows, staggered banks

template <int COLS>
struct DcCfg {
  static constexpr int NS = COLS / 64;                               // 64-column slabs of value columns
  static constexpr int UP = COLS + 4;                                // floats per row of u and the read-outs
  static constexpr int S_PART = NS * 128 * 128, U_PART = NS * DC_C * 128;      // bytes of one bf16 part of S, of u
  static constexpr int KQ_OFF = 0;                                   // [2 slabs of 64 dims][K rows, Q rows] swizzled: 32 KB
  static constexpr int S_OFF = 32768;                                // S parts; between MMA and MMA: u and the read-outs
  static constexpr int U_OFF = S_OFF + 3 * S_PART;                   // u parts; before the solve: v
  static constexpr int AT_OFF = U_OFF + 3 * U_PART;
  static constexpr int PT_OFF = AT_OFF + DC_C * DC_PITCH * 4;
  static constexpr int SC_OFF = PT_OFF + DC_C * DC_PITCH * 4;        // scalars
  static constexpr int SMEM = SC_OFF + 2048 + 1024;
  static constexpr int S_COL = 0, D1_COL = 128, D2_COL = 256;        // tensor memory
};
static_assert(2 * DC_C * DcCfg<128>::UP * 4 <= 3 * DcCfg<128>::S_PART && 2 * DC_C * DcCfg<64>::UP * 4 <= 3 * DcCfg<64>::S_PART, "u and read-outs fit");
static_assert(DcCfg<128>::SMEM <= 227 * 1024, "shared memory");

struct DcScalars {
  float2 gam[DC_C];                     // gamma as high + low
  float beta[DC_C], ik[DC_C], iq[DC_C];
  float2 gam_end;
  uint64_t bar1, bar3;
  uint32_t tmem;
  int abort;
};
static_assert(sizeof(DcScalars) <= 2048, "scalars");

__device__ __forceinline__ float dc_decay(float2 a, float2 b) { return expf((a.x - b.x) + (a.y - b.y)); }

// eight fp32 values as three rows of eight bf16, part p at dst + p * stride
__device__ __forceinline__ void dc_split8(const float* x, uint8_t* dst, int stride) {
  uint32_t part[3][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    float a = x[2 * i], b = x[2 * i + 1];
#pragma unroll
    for (int p = 0; p < 3; p++) {
      const uint32_t w = pack_bf16x2(a, b);
      part[p][i] = w;
      const float2 f = unpack_bf16x2(w);
      a -= f.x;
      b -= f.y;
    }
  }
#pragma unroll
  for (int p = 0; p < 3; p++) *reinterpret_cast<uint4*>(dst + p * stride) = make_uint4(part[p][0], part[p][1], part[p][2], part[p][3]);
}

// acc[pair of rows][column] += sum over m in [m0, m1) of coef[m][row] u[m][column]: 2 PAIRS rows from coef, COLUMNS columns from u.
// What bounds these sums is the 128 bytes a clock that shared memory returns, broadcast or not, so a thread takes a tile: a
// column by itself needs nine values for eight products, 8 x 8 outputs sixteen for 64.
// The operands of the next BATCH steps are on their way while BATCH steps are summed; m1 - m0 is a multiple of 2 BATCH.
template <int PAIRS, int COLUMNS, int UP, int BATCH>
__device__ __forceinline__ void dc_tile(f32x2 (*acc)[COLUMNS], const float* coef, const float* u, int m0, int m1) {
  f32x2 a[2][BATCH][PAIRS];
  float um[2][BATCH][COLUMNS];
  auto load = [&](int s, int m) {
#pragma unroll
    for (int k = 0; k < BATCH; k++) {
#pragma unroll
      for (int i = 0; i < PAIRS; i += 2) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(coef + (m + k) * DC_PITCH + 2 * i);
        a[s][k][i] = v.x;
        a[s][k][i + 1] = v.y;
      }
      constexpr int V = COLUMNS < 4 ? COLUMNS : 4;
#pragma unroll
      for (int c = 0; c < COLUMNS; c += V) load_vec<float, V>(u + (m + k) * UP + c, um[s][k] + c);
    }
  };
  auto sum = [&](int s) {
#pragma unroll
    for (int k = 0; k < BATCH; k++)
#pragma unroll
      for (int c = 0; c < COLUMNS; c++) {
        const f32x2 u2 = pack2(um[s][k][c], um[s][k][c]);
#pragma unroll
        for (int i = 0; i < PAIRS; i++) acc[i][c] = fma2(a[s][k][i], u2, acc[i][c]);
      }
  };
  load(0, m0);
#pragma unroll 1
  for (int m = m0; m < m1; m += 2 * BATCH) {
    load(1, m + BATCH);
    sum(0);
    if (m + 2 * BATCH < m1) load(0, m + 2 * BATCH);
    sum(1);
  }
}

template <int COLS>
__global__ void __launch_bounds__(DC_THREADS, 1) delta_chunk_kernel(const DeltaChunkArgs p) {
  using Cfg = DcCfg<COLS>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* kq = smem + Cfg::KQ_OFF;
  uint8_t* s_parts = smem + Cfg::S_OFF;
  uint8_t* u_parts = smem + Cfg::U_OFF;
  constexpr int UP = Cfg::UP;
  float* us = (float*)s_parts;                             // [DC_C][UP] right-hand sides, then u
  float* ro = us + DC_C * UP;                              // [DC_C][UP] read-outs of S0
  __nv_bfloat16* vs = (__nv_bfloat16*)u_parts;             // [DC_C][COLS], 16-byte chunks swizzled by row
  float* at = (float*)(smem + Cfg::AT_OFF);
  float* pt = (float*)(smem + Cfg::PT_OFF);
  DcScalars* sc = (DcScalars*)(smem + Cfg::SC_OFF);

  const int b = blockIdx.x, hv = blockIdx.y, j0 = blockIdx.z * COLS, hk = hv / (p.Hv / p.Hk);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int t0 = p.cu[b], t1 = p.cu[b + 1], slot = p.slots[b];
  if (t1 - t0 < p.min_len) return;                         // short portions run in the token-serial kernel
  if (slot < 0 || slot >= p.num_slots) {
    if (tid == 0 && p.status) atomicExch(p.status, B200_BAD_INDEX);
    return;
  }
  const bool init = p.has_init[b] != 0;
  float* state = p.state + ((long)slot * p.Hv + hv) * DC_K * p.DV + j0;

  if (tid == 0) {
    mbar_init(&sc->bar1, 1);
    mbar_init(&sc->bar3, 1);
    sc->abort = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&sc->tmem, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = sc->tmem;
  volatile int* abort_word = &sc->abort;
  const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const int row = (warp & 3) * 32 + lane;                  // key row of the state, or row of [K; Q]

  // the state's three parts, from registers (32 columns from c)
  auto store_state_parts = [&](const float* v, int c) {
    for (int g = 0; g < 4; g++) {
      const int ch = c / 8 + g;
      dc_split8(v + 8 * g, s_parts + (ch >> 3) * (128 * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4), Cfg::S_PART);
    }
  };
  if (warp < 4) {
    for (int c = 0; c < COLS; c += 32) {
      float v[32];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const float4 f = init ? *reinterpret_cast<const float4*>(state + (long)row * p.DV + c + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
      }
      tmem_st_32x32b_x32(t_lane + Cfg::S_COL + c, reinterpret_cast<const uint32_t*>(v));
      store_state_parts(v, c);
    }
    tmem_st_wait();
  }

  // ---- staging: thread -> 16-byte chunk `ch` of rows tid / 16 + 16 i (i < 4: k, else q); v by 16-byte chunks as well
  constexpr int VCH = COLS / 8, VPER = DC_C * VCH / DC_THREADS;
  const int ch = tid & 15, r0 = tid >> 4;
  const __nv_bfloat16* kp = (const __nv_bfloat16*)p.k + (long)hk * DC_K + ch * 8;
  const __nv_bfloat16* qp = (const __nv_bfloat16*)p.q + (long)hk * DC_K + ch * 8;
  const __nv_bfloat16* vp = (const __nv_bfloat16*)p.v + (long)hv * p.DV + j0;
  uint4 raw[8], rawv[VPER];
  float rg = 0.f, rb = 0.f;
  const uint4 zero4 = make_uint4(0, 0, 0, 0);
  auto fetch = [&](int tc) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int t = tc + r0 + 16 * (i & 3);
      raw[i] = t < t1 ? *reinterpret_cast<const uint4*>((i < 4 ? kp : qp) + (long)t * p.qk_stride) : zero4;
    }
#pragma unroll
    for (int i = 0; i < VPER; i++) {
      const int e = tid + i * DC_THREADS, t = tc + e / VCH;
      rawv[i] = t < t1 ? *reinterpret_cast<const uint4*>(vp + (long)t * p.v_stride + (e % VCH) * 8) : zero4;
    }
    if (tid >= 64 && tid < 128) {
      const int t = tc + tid - 64;
      rg = t < t1 ? p.g[(long)t * p.Hv + hv] : 0.f;
      if (rg < -200.f) rg = -200.f;                        // e^-200 is 0 in 32 bits, and the running sum keeps its low digits
      rb = t < t1 ? p.beta[(long)t * p.Hv + hv] : 0.f;
    }
  };
  fetch(t0);

  uint32_t ph = 0;
  for (int tc = t0; tc < t1; tc += DC_C, ph ^= 1) {
    const int n = min(DC_C, t1 - tc);
    // ---- k, q, v, norms
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int r = r0 + 16 * i;                           // 0..63: k, 64..127: q
      *reinterpret_cast<uint4*>(kq + (ch >> 3) * 16384 + r * 128 + (((ch & 7) ^ (r & 7)) << 4)) = raw[i];
      const uint32_t w[4] = {raw[i].x, raw[i].y, raw[i].z, raw[i].w};
      float ss = 0.f;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const float2 f = unpack_bf16x2(w[j]);
        ss = fmaf(f.x, f.x, fmaf(f.y, f.y, ss));
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      if (ch == 0) {
        const float inv = p.l2norm ? rsqrtf(ss + 1e-6f) : 1.f;
        if (i < 4) sc->ik[r] = inv;
        else sc->iq[r - 64] = inv * p.scale;
      }
    }
#pragma unroll
    for (int i = 0; i < VPER; i++) {
      const int e = tid + i * DC_THREADS, r = e / VCH, c = e % VCH;
      *reinterpret_cast<uint4*>(vs + r * COLS + ((c ^ (r & 7)) << 3)) = rawv[i];
    }
    if (tid >= 64 && tid < 128) {
      sc->beta[tid - 64] = rb;
      // running sum over the 64 tokens: two warps, the second adds the first one's total
      double s = rg;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, s, o);
        if (lane >= o) s += up;
      }
      sc->gam[tid - 64] = make_float2((float)s, (float)(s - (double)(float)s));
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (*abort_word != 0) break;
    if (tid == 0) {
      tc_fence_after();
      const uint32_t a = smem_u32(kq), sb = smem_u32(s_parts);
      constexpr uint32_t id2 = make_idesc_f16(128, DC_C, true, false, false), id1 = make_idesc_f16(128, COLS, true, false, true);
#pragma unroll
      for (int kk = 0; kk < 8; kk++) {
        const uint64_t da = make_smem_desc(a + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024, kLayoutSw128);
        umma_f16_ss(tmem + Cfg::D2_COL, da, da, id2, kk > 0 ? 1u : 0u);
      }
#pragma unroll 1
      for (int part = 2; part >= 0; part--)                // smallest first
#pragma unroll
        for (int kk = 0; kk < 8; kk++)
          umma_f16_ss(tmem + Cfg::D1_COL, make_smem_desc(a + (kk >> 2) * 16384 + (kk & 3) * 32, 16, 1024, kLayoutSw128),
                      make_smem_desc(sb + part * Cfg::S_PART + kk * 2048, 16384, 1024, kLayoutSw128), id1, (part < 2 || kk > 0) ? 1u : 0u);
      umma_commit(&sc->bar1);
    }
    __syncwarp();
    if (tid >= 96 && tid < 128) {                          // second half of gamma: add the first half's total
      const float2 h = sc->gam[31], v = sc->gam[tid - 64];
      const double s = ((double)h.x + (double)h.y) + ((double)v.x + (double)v.y);
      sc->gam[tid - 64] = make_float2((float)s, (float)(s - (double)(float)s));
    }
    if (tc + DC_C < t1) fetch(tc + DC_C);
    __syncthreads();
    mbar_wait(&sc->bar1, ph, abort_word);
    tc_fence_after();
    if (warp < 4) {
      // ---- A^T[m][j] (rows of k), P^T[m][j] (rows of q)
      const bool is_q = row >= DC_C;
      const int j = row & 63;
      float* dst = (is_q ? pt : at) + j;
      const float2 gj = sc->gam[j];
      const float f = is_q ? sc->iq[j] : sc->beta[j] * sc->ik[j];
      const int m_end = (j | 31) + 1;                      // rows of this warp see no later tokens
      for (int m0 = m_end; m0 < DC_C; m0++) dst[m0 * DC_PITCH] = 0.f;
#pragma unroll 1
      for (int m0 = 0; m0 < m_end; m0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_lane + Cfg::D2_COL + m0, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const int m = m0 + i;
          dst[m * DC_PITCH] = m <= j ? __uint_as_float(r[i]) * (f * sc->ik[m]) * dc_decay(gj, sc->gam[m]) : 0.f;
        }
      }
    } else {
      // ---- right-hand sides beta (v - e^gamma S0^T k), read-outs e^gamma S0^T q
      const bool is_q = row >= DC_C;
      const int j = row & 63;
      const float d = dc_decay(sc->gam[j], make_float2(0.f, 0.f));
      const float f = is_q ? d * sc->iq[j] : -sc->beta[j] * d * sc->ik[j], bj = sc->beta[j];
#pragma unroll 1
      for (int c = 0; c < COLS; c += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(t_lane + Cfg::D1_COL + c, r);
        tmem_ld_wait();
        float x[16];
        if (is_q) {
#pragma unroll
          for (int i = 0; i < 16; i++) x[i] = __uint_as_float(r[i]) * f;
        } else {
          const uint4 v0 = *reinterpret_cast<const uint4*>(vs + j * COLS + (((c / 8) ^ (j & 7)) << 3));
          const uint4 v1 = *reinterpret_cast<const uint4*>(vs + j * COLS + (((c / 8 + 1) ^ (j & 7)) << 3));
          const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
          for (int i = 0; i < 8; i++) {
            const float2 vv = unpack_bf16x2(w[i]);
            x[2 * i] = fmaf(__uint_as_float(r[2 * i]), f, bj * vv.x);
            x[2 * i + 1] = fmaf(__uint_as_float(r[2 * i + 1]), f, bj * vv.y);
          }
        }
#pragma unroll
        for (int i = 0; i < 16; i += 4) store_vec<float, 4>((is_q ? ro : us) + j * UP + c + i, x + i);
      }
    }
    tc_fence_before();
    __syncthreads();
    // ---- solve, sixteen rows at a time: what the rows above contribute (tiles of four rows over all threads), then the block's own
    // triangle (thread = value column)
#pragma unroll 1
    for (int jb = 0; jb < DC_C; jb += 16) {
      if (jb > 0) {
        constexpr int CW = COLS / 64;
        const int rr = jb + (tid >> 6) * 4, c = (tid & 63) * CW;
        f32x2 acc[2][CW];
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int k = 0; k < CW; k++) acc[i][k] = 0;
        dc_tile<2, CW, UP, 4>(acc, at + rr, us + c, 0, jb);
#pragma unroll
        for (int i = 0; i < 2; i++)
#pragma unroll
          for (int k = 0; k < CW; k++) {
            const float2 f = unpack2(acc[i][k]);
            us[(rr + 2 * i) * UP + c + k] -= f.x;
            us[(rr + 2 * i + 1) * UP + c + k] -= f.y;
          }
        __syncthreads();
      }
      if (tid < COLS) {
        float* u = us + jb * UP + tid;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; i++) x[i] = u[i * UP];
        float a[2][16];                    // a row ahead
        auto load = [&](int i) {
#pragma unroll
          for (int k0 = (i + 1) / 4 * 4; k0 < 16; k0 += 4) load_vec<float, 4>(at + (jb + i) * DC_PITCH + jb + k0, a[i & 1] + k0);
        };
        load(0);
#pragma unroll
        for (int i = 0; i < 15; i++) {
          if (i < 14) load(i + 1);
#pragma unroll
          for (int k = i + 1; k < 16; k++) x[k] = fmaf(-a[i & 1][k], x[i], x[k]);
        }
#pragma unroll
        for (int i = 1; i < 16; i++) u[i * UP] = x[i];
      }
      __syncthreads();
    }
    if (warp < 4) {
      // ---- e^{gamma_C - gamma_j} |k_j|^-1 u_j in three parts; S0 e^{gamma_C}; S += K^T u
      const float2 ge = sc->gam[DC_C - 1];
      const int j = tid & 63;
      const float f = dc_decay(ge, sc->gam[j]) * sc->ik[j];
#pragma unroll 2
      for (int c = tid >> 6; c < VCH; c += 2) {
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; i += 4) load_vec<float, 4>(us + j * UP + c * 8 + i, x + i);
#pragma unroll
        for (int i = 0; i < 8; i++) x[i] *= f;
        dc_split8(x, u_parts + (c >> 3) * (DC_C * 128) + j * 128 + (((c & 7) ^ (j & 7)) << 4), Cfg::U_PART);
      }
      const float d = dc_decay(ge, make_float2(0.f, 0.f));
#pragma unroll 1
      for (int c = 0; c < COLS; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_lane + Cfg::S_COL + c, r);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 32; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * d);
        tmem_st_32x32b_x32(t_lane + Cfg::S_COL + c, r);
      }
      tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before();
      asm volatile("bar.sync 1, 128;" ::: "memory");
      if (tid == 0) {
        tc_fence_after();
        const uint32_t a = smem_u32(kq), ub = smem_u32(u_parts);
        constexpr uint32_t id3 = make_idesc_f16(128, COLS, true, true, true);
#pragma unroll 1
        for (int part = 2; part >= 0; part--)
#pragma unroll
          for (int kk = 0; kk < DC_C / 16; kk++)
            umma_f16_ss(tmem + Cfg::S_COL, make_smem_desc(a + kk * 2048, 16384, 1024, kLayoutSw128),
                        make_smem_desc(ub + part * Cfg::U_PART + kk * 2048, DC_C * 128, 1024, kLayoutSw128), id3, 1u);
        umma_commit(&sc->bar3);
      }
      __syncwarp();
    } else {
      // ---- o_j = read-out + sum_{m <= j} P_jm u_m: tiles of eight rows, sixteen threads to a row of tiles; a warp has an early
      // and a late one
      constexpr int CW = COLS / 16;
      const int tt = tid - 128, w = tt >> 5, jb = ((tt >> 4) & 1 ? 7 - w : w) * 8, c = (tt & 15) * CW;
      f32x2 acc[4][CW];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float x[CW], y[CW];
#pragma unroll
        for (int k = 0; k < CW; k += 4) {
          load_vec<float, 4>(ro + (jb + 2 * i) * UP + c + k, x + k);
          load_vec<float, 4>(ro + (jb + 2 * i + 1) * UP + c + k, y + k);
        }
#pragma unroll
        for (int k = 0; k < CW; k++) acc[i][k] = pack2(x[k], y[k]);
      }
      if (jb < n) {
        dc_tile<4, CW, UP, 1>(acc, pt + jb, us + c, 0, jb);
        // the tile's own triangle: rows take nothing of later tokens, not even zero times (a NaN there is not theirs)
#pragma unroll
        for (int m = 0; m < 8; m++) {
          float um[CW];
#pragma unroll
          for (int k = 0; k < CW; k += 4) load_vec<float, 4>(us + (jb + m) * UP + c + k, um + k);
          const float* coef = pt + (jb + m) * DC_PITCH + jb;
#pragma unroll
          for (int i = m / 2; i < 4; i++) {
            const float2 a = *reinterpret_cast<const float2*>(coef + 2 * i);
#pragma unroll
            for (int k = 0; k < CW; k++) {
              const float2 f = unpack2(acc[i][k]);
              acc[i][k] = 2 * i >= m ? fma2(pack2(a.x, a.y), pack2(um[k], um[k]), acc[i][k]) : pack2(f.x, fmaf(a.y, um[k], f.y));
            }
          }
        }
      }
      __nv_bfloat16* op = (__nv_bfloat16*)p.out + (long)(tc + jb) * p.out_stride + (long)hv * p.DV + j0 + c;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        float x[CW], y[CW];
#pragma unroll
        for (int k = 0; k < CW; k++) {
          const float2 f = unpack2(acc[i][k]);
          x[k] = f.x;
          y[k] = f.y;
        }
        if (jb + 2 * i < n) store_vec<__nv_bfloat16, CW>(op + (long)(2 * i) * p.out_stride, x);
        if (jb + 2 * i + 1 < n) store_vec<__nv_bfloat16, CW>(op + (long)(2 * i + 1) * p.out_stride, y);
      }
    }
    mbar_wait(&sc->bar3, ph, abort_word);
    __syncthreads();                                       // outputs have read u and the read-outs, K^T u is summed
    tc_fence_after();
    if (warp < 4) {
#pragma unroll 1
      for (int c = 0; c < COLS; c += 32) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_lane + Cfg::S_COL + c, r);
        tmem_ld_wait();
        if (tc + DC_C < t1) store_state_parts(reinterpret_cast<const float*>(r), c);
        else if (*abort_word == 0)
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<uint4*>(state + (long)row * p.DV + c + i) = make_uint4(r[i], r[i + 1], r[i + 2], r[i + 3]);
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_word != 0 && p.status) atomicExch(p.status, *abort_word);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

template <int COLS>
static int launch_dc(const DeltaChunkArgs& p, int B, cudaStream_t stream) {
  const cudaError_t e = allow_smem<delta_chunk_kernel<COLS>>(DcCfg<COLS>::SMEM);
  if (e != cudaSuccess) return (int)e;
  delta_chunk_kernel<COLS><<<dim3((unsigned)B, (unsigned)p.Hv, (unsigned)(p.DV / COLS)), DC_THREADS, DcCfg<COLS>::SMEM, stream>>>(p);
  return B200_CHECK_LAUNCH();
}

// true (with rc set) when the chunked kernel takes these sizes; sequences shorter than p.min_len are left alone
bool launch_delta_chunk(const DeltaChunkArgs& p, int B, int DK, cudaStream_t stream, int* rc) {
  if (DK != DC_K || p.DV % 64 || p.qk_stride % 8 || p.v_stride % 8 || !aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) ||
      !aligned16(p.state) || p.out_stride % 8 || !aligned16(p.out))
    return false;
  // a block keeps an SM to itself: 128 columns a block, 64 while that leaves every block its own SM
  if (p.DV % 128 || (long)B * p.Hv * (p.DV / 64) <= num_sms()) *rc = launch_dc<64>(p, B, stream);
  else *rc = launch_dc<128>(p, B, stream);
  return true;
}

}  // namespace b200
