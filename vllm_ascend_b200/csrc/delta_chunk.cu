// Gated delta rule over prompts in chunks of 64 tokens, on tcgen05 (key dimension 128).
//
//     S <- S e^{g_t};  u = beta_t (v_t - S^T k_t);  S <- S + k_t u^T;  o_t = S^T q_t
//
// With gamma_j the running sum of g inside a chunk entered with S0, and e_jm = e^{gamma_j - gamma_m}:
//     u_j + sum_{m<j} beta_j e_jm (k_j . k_m) u_m = beta_j (v_j - e^{gamma_j} S0^T k_j) =: r_j        (a triangular system I + A)
//     o_j = e^{gamma_j} S0^T q_j + sum_{m<=j} e_jm (q_j . k_m) u_m
//     S   = e^{gamma_C} S0 + sum_j k_j (e^{gamma_C - gamma_j} u_j)^T
// (the UT form of DeltaNet, Yang et al. 2024; counterpart of vllm_ascend/ops/triton/fla/chunk.py).
//
// What does not need S0 is done for all chunks at once: T = (I + A)^-1 and P T, P the matrix of the read-outs, are 64 x 64 triangles
// per chunk and head (delta_prep_kernel, fp32 on CUDA cores).  What is left of a chunk is a chain of three products,
//     [K; Q] S0   ->   r   ->   [T - 1; P T] r = [u - r; o - read-out of S0]   ->   S = e^{gamma_C} S0 + K^T u
// with rows turned into operands in between (delta_chain_kernel).  A block has one sequence, one head and 64 value columns, and two blocks
// fit an SM.  Bound: the chain, chunk after chunk of a sequence: 8,100 clocks a chunk, 10,200 with a second block on the SM, of which the
// three products are 3,400 (60 MMAs of 64 columns: 55 clocks each, 40 with an operand in tensor memory).  Preparing takes 0.047 us a chunk and
// head, three blocks on an SM, issue and shared-memory latency.  6000 tokens in three prompts, 32 heads, us: both together 350 (chain 200,
// preparation 150); the solve, the state's products and their conversions one after the other in one block per head 785; token by token 1603.
//
// 32 bits stay 32 bits.  q and k are bf16 as they come, so k . k and q . k are exact products summed in fp32; their norms
// are factors of rows.  The state, u, r and T are fp32: as MMA operands they are three bf16 parts (8 + 8 + 8 bits), which times an exact
// bf16 operand is the fp32 product, and of two such operands the six products above 2^-24.  T's diagonal of ones stays out of that product, and
// r is added by itself: the tensor cores' sums truncate, which with the diagonal made the state's error 1.2 times that of a solve in fp32
// where decays are strong.  gamma is summed in fp64 and kept in two floats.
//
// A matrix product would carry a NaN or infinity of r to earlier tokens (zero times NaN).  A chunk whose r has one takes that product
// row by row on CUDA cores, without the zeros.
#include "common.cuh"
#include "delta_chunk.h"
#include "dtypes.cuh"

namespace b200 {

constexpr int DC_C = 64, DC_K = 128, DC_COLS = 64, DC_THREADS = 256, DC_CHAIN_THREADS = 288;
constexpr int DC_PITCH = 68;            // floats per row of A^T / P^T / T: 16-byte rows, staggered banks
// what delta_prep_kernel leaves of a chunk and head: T and P T as packed triangles, four factors per row, the chunk's decay.  A triangle
// is kept in groups of four columns, the rows of a group (from the one of its block of sixteen on) one after the other, as the threads
// of the other kernel read them
constexpr int DC_TRI = 2560, DC_WS = 2 * DC_TRI + 4 * DC_C + 16;

struct DcPrepSmem {
  static constexpr int KQ_OFF = 0;                                   // [2 slabs of 64 dims][K rows, Q rows] swizzled: 32 KB; then T
  static constexpr int AT_OFF = 32768, PT_OFF = AT_OFF + DC_C * DC_PITCH * 4;
  static constexpr int E_OFF = PT_OFF + DC_C * DC_PITCH * 4;         // [m][j mod 16]: e_jm of tokens in one block of sixteen
  static constexpr int SC_OFF = E_OFF + DC_C * 16 * 4;
  static constexpr int BYTES = SC_OFF + 2048 + 1024;
};
static_assert(3 * (DcPrepSmem::BYTES + 1024) <= 228 * 1024, "three blocks per SM");
struct DcChainSmem {
  static constexpr int S_PART = DC_K * 128, R_PART = DC_C * 128;     // bytes of one bf16 part of S, of r and u
  static constexpr int KQ_BYTES = 32768;                             // K and Q of a chunk, of two chunks; Q's place holds the next chunk's v and outputs
  static constexpr int S_OFF = 2 * KQ_BYTES;                         // parts of S; from product to product of r, then of u
  static constexpr int SC_OFF = S_OFF + 3 * S_PART;
  static constexpr int BYTES = SC_OFF + 64;
  static constexpr int S_COL = 0, D_COL = 64, T_COL = 128, TMEM = 256;        // tensor memory: 64, 64, 3 x 32 columns
};
static_assert(2 * (DcChainSmem::BYTES + 1024) <= 228 * 1024, "two blocks per SM");

struct DcScalars {
  float2 gam[DC_C];                     // gamma as high + low
  float beta[DC_C], ik[DC_C], iq[DC_C];
  float w[DC_C];                        // |k_m|^-1 times the decay from m to the last token of its sixteen
  uint64_t bar;
  uint32_t tmem;
  int abort;
};
static_assert(sizeof(DcScalars) <= 2048, "scalars");

__device__ __forceinline__ float dc_decay(float2 a, float2 b) { return expf((a.x - b.x) + (a.y - b.y)); }
__device__ __forceinline__ int dc_tri(int g, int j) {      // float of a triangle where columns 4 g .. 4 g + 3 of row j start
  const int b = g >> 2;
  return 4 * (b * (288 - 32 * b) + (g & 3) * (64 - 16 * b) + j - 16 * b);
}
// place of chunk c of sequence b in the workspace
__device__ __forceinline__ long dc_place(const DeltaChunkArgs& p, int b, int c, int t0) {
  return p.per_seq ? (long)b * p.per_seq + (c - p.c0) : (long)(t0 / DC_C + b) + c;
}

// A pair of fp32 values as three pairs of bf16 that sum to it: the parts are rounded (half up) by integer additions, which are full-rate
// where conversions are not, and what is left of 24 bits after two of them fits the third.  A NaN is one in the last part.
__device__ __forceinline__ void dc_split2(float a, float b, uint32_t* part) {
#pragma unroll
  for (int p = 0; p < 2; p++) {
    const uint32_t u = __float_as_uint(a) + 0x8000u, v = __float_as_uint(b) + 0x8000u;
    part[p] = __byte_perm(u, v, 0x7632);
    a -= __uint_as_float(u & 0xffff0000u);
    b -= __uint_as_float(v & 0xffff0000u);
  }
  part[2] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
}
// eight fp32 values as three rows of eight bf16, part p at dst + p * stride
__device__ __forceinline__ void dc_split8(const float* x, uint8_t* dst, int stride) {
  uint32_t part[4][3];
#pragma unroll
  for (int i = 0; i < 4; i++) dc_split2(x[2 * i], x[2 * i + 1], part[i]);
#pragma unroll
  for (int p = 0; p < 3; p++) *reinterpret_cast<uint4*>(dst + p * stride) = make_uint4(part[0][p], part[1][p], part[2][p], part[3][p]);
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

// Grid: places of the workspace, heads.
__global__ void __launch_bounds__(DC_THREADS, 3) delta_prep_kernel(const DeltaChunkArgs p) {
  using Cfg = DcPrepSmem;
  constexpr int UP = DC_PITCH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* kq = smem + Cfg::KQ_OFF;
  float* us = (float*)kq;                                  // T, once the products have read K and Q
  float* at = (float*)(smem + Cfg::AT_OFF);
  float* pt = (float*)(smem + Cfg::PT_OFF);
  float* decay = (float*)(smem + Cfg::E_OFF);
  DcScalars* sc = (DcScalars*)(smem + Cfg::SC_OFF);

  int b, c;
  if (p.per_seq) {
    b = blockIdx.x / p.per_seq;
    c = p.c0 + blockIdx.x % p.per_seq;
  } else {       // sequence b owns the places from cu[b] / 64 + b on
    int lo = 0, hi = p.B - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (p.cu[mid] / DC_C + mid <= (int)blockIdx.x) lo = mid; else hi = mid - 1;
    }
    b = lo;
    c = blockIdx.x - (p.cu[b] / DC_C + b);
  }
  const int hv = blockIdx.y, hk = hv / (p.Hv / p.Hk);
  const int t0 = p.cu[b], t1 = p.cu[b + 1], tc = t0 + c * DC_C;
  if (t1 - t0 < p.min_len || tc >= t1) return;
  float* ws = p.ws + (dc_place(p, b, c, t0) * p.Hv + hv) * DC_WS;
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  if (tid == 0) {
    mbar_init(&sc->bar, 1);
    sc->abort = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(&sc->tmem, 64);
    tmem_relinquish();
  }
  // ---- k, q, norms: thread -> 16-byte chunk `ch` of rows tid / 16 + 16 i (i < 4: k, else q)
  const int ch = tid & 15, r0 = tid >> 4;
  const __nv_bfloat16* kp = (const __nv_bfloat16*)p.k + (long)hk * DC_K + ch * 8;
  const __nv_bfloat16* qp = (const __nv_bfloat16*)p.q + (long)hk * DC_K + ch * 8;
  uint4 raw[8];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int t = tc + r0 + 16 * (i & 3);
    raw[i] = t < t1 ? *reinterpret_cast<const uint4*>((i < 4 ? kp : qp) + (long)t * p.qk_stride) : make_uint4(0, 0, 0, 0);
  }
  if (tid >= 64 && tid < 128) {
    const int t = tc + tid - 64;
    float rg = t < t1 ? p.g[(long)t * p.Hv + hv] : 0.f;
    if (rg < -200.f) rg = -200.f;                          // e^-200 is 0 in 32 bits, and the running sum keeps its low digits
    sc->beta[tid - 64] = t < t1 ? p.beta[(long)t * p.Hv + hv] : 0.f;
    // running sum over the 64 tokens: two warps, the second adds the first one's total
    double s = rg;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += up;
    }
    sc->gam[tid - 64] = make_float2((float)s, (float)(s - (double)(float)s));
  }
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int r = r0 + 16 * i;                             // 0..63: k, 64..127: q
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
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(sc->tmem);
  volatile int* abort_word = &sc->abort;
  if (warp == 0 && elect_one()) {
    const uint64_t d = make_smem_desc(smem_u32(kq), 16, 1024, kLayoutSw128);
    constexpr uint32_t id = make_idesc_f16(128, DC_C, true, false, false);
#pragma unroll
    for (int kk = 0; kk < 8; kk++) {
      const uint64_t dk = d + (uint32_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4);
      umma_f16_ss(tmem, dk, dk, id, kk > 0 ? 1u : 0u);
    }
    umma_commit(&sc->bar);
  }
  __syncwarp();
  if (tid >= 96 && tid < 128) {                            // second half of gamma: add the first half's total
    const float2 h = sc->gam[31], v = sc->gam[tid - 64];
    const double s = ((double)h.x + (double)h.y) + ((double)v.x + (double)v.y);
    sc->gam[tid - 64] = make_float2((float)s, (float)(s - (double)(float)s));
  }
  __syncthreads();
  if (tid < DC_C) sc->w[tid] = sc->ik[tid] * dc_decay(sc->gam[tid | 15], sc->gam[tid]);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int m = (tid >> 4) + 16 * i, j = (m & ~15) + (tid & 15);
    decay[m * 16 + (tid & 15)] = m <= j ? sc->ik[m] * dc_decay(sc->gam[j], sc->gam[m]) : 0.f;
  }
  __syncthreads();
  if (mbar_wait(&sc->bar, 0, abort_word)) {
    tc_fence_after();
    // ---- A^T[m][j] (rows of k), P^T[m][j] (rows of q): warps 0..3 the earlier half of the tokens m, warps 4..7 the later one.  e_jm of
    // tokens in different blocks of sixteen is the decay to the end of m's block times the one from there: both are at most 1
    const int row = (warp & 3) * 32 + lane, j = row & 63, mh = (warp >> 2) * 32;
    const bool is_q = row >= DC_C;
    float* dst = (is_q ? pt : at) + j;
    if (mh > j) {
#pragma unroll
      for (int m = 0; m < 32; m++) dst[(mh + m) * DC_PITCH] = 0.f;
    }
    if (mh <= (j | 31)) {                                  // rows of one warp: all or none
      const float2 gj = sc->gam[j];
      const float f = is_q ? sc->iq[j] : sc->beta[j] * sc->ik[j];
#pragma unroll 1
      for (int m0 = mh; m0 < mh + 32; m0 += 16) {
        uint32_t r[16];
        tmem_ld_32x32b_x16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + m0, r);
        tmem_ld_wait();
        if (m0 >> 4 < j >> 4) {
          const float fd = f * dc_decay(gj, sc->gam[m0 + 15]);
#pragma unroll
          for (int i = 0; i < 16; i++) dst[(m0 + i) * DC_PITCH] = __uint_as_float(r[i]) * (fd * sc->w[m0 + i]);
        } else {
          const int last = m0 >> 4 == j >> 4 ? j & 15 : -1;
#pragma unroll
          for (int i = 0; i < 16; i++)
            dst[(m0 + i) * DC_PITCH] = i <= last ? __uint_as_float(r[i]) * (f * decay[(m0 + i) * 16 + (j & 15)]) : 0.f;
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  // ---- T = (I + A)^-1 by halves: the inverses of the four diagonal blocks of sixteen (thread = column), then twice
  // [a 0; c b]^-1 = [a' 0; -b' c a'  b'].  A product's rows stop at the diagonal (a NaN of a later row is not theirs); c a' waits in the
  // block above the diagonal that mirrors c.
  if (tid < DC_C) {
    const int jb = tid & ~15, col = tid & 15;
    float x[16];
#pragma unroll
    for (int i = 0; i < 16; i++) x[i] = i == col ? 1.f : 0.f;
    float a[2][16];                        // a row ahead
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
    for (int i = 0; i < 16; i++) us[(jb + i) * UP + jb + col] = x[i];
  }
  __syncthreads();
  {
    const int o = (tid >> 7) * 32, i = (tid >> 3) & 15, col = (tid & 7) * 2;
    float x = 0.f, y = 0.f;
#pragma unroll
    for (int k = 0; k < 16; k++) {
      const float a = at[(o + k) * DC_PITCH + o + 16 + i];
      const float2 u = *reinterpret_cast<const float2*>(us + (o + k) * UP + o + col);
      x = fmaf(a, u.x, x);
      y = fmaf(a, u.y, y);
    }
    *reinterpret_cast<float2*>(us + (o + i) * UP + o + 16 + col) = make_float2(x, y);
    __syncthreads();
    x = y = 0.f;
    for (int k = 0; k <= i; k++) {
      const float a = us[(o + 16 + i) * UP + o + 16 + k];
      const float2 u = *reinterpret_cast<const float2*>(us + (o + k) * UP + o + 16 + col);
      x = fmaf(-a, u.x, x);
      y = fmaf(-a, u.y, y);
    }
    *reinterpret_cast<float2*>(us + (o + 16 + i) * UP + o + col) = make_float2(x, y);
  }
  __syncthreads();
  {
    const int i = tid >> 3, col = (tid & 7) * 4;
    float x[4] = {}, u[4];
#pragma unroll 8
    for (int k = col & 16; k < 32; k++) {
      const float a = at[k * DC_PITCH + 32 + i];
      load_vec<float, 4>(us + k * UP + col, u);
#pragma unroll
      for (int e = 0; e < 4; e++) x[e] = fmaf(a, u[e], x[e]);
    }
    store_vec<float, 4>(us + i * UP + 32 + col, x);
    __syncthreads();
#pragma unroll
    for (int e = 0; e < 4; e++) x[e] = 0.f;
    int k = 0;
#pragma unroll 2
    for (; k + 4 <= i + 1; k += 4) {
      float a[4];
      load_vec<float, 4>(us + (32 + i) * UP + 32 + k, a);
#pragma unroll
      for (int q = 0; q < 4; q++) {
        load_vec<float, 4>(us + (k + q) * UP + 32 + col, u);
#pragma unroll
        for (int e = 0; e < 4; e++) x[e] = fmaf(-a[q], u[e], x[e]);
      }
    }
    for (; k <= i; k++) {
      const float a = us[(32 + i) * UP + 32 + k];
      load_vec<float, 4>(us + k * UP + 32 + col, u);
#pragma unroll
      for (int e = 0; e < 4; e++) x[e] = fmaf(-a, u[e], x[e]);
    }
    store_vec<float, 4>(us + (32 + i) * UP + col, x);
    __syncthreads();
    const float zero[4] = {};
    store_vec<float, 4>(us + i * UP + 32 + col, zero);
    if (tid < 128) store_vec<float, 4>(us + ((tid >> 6) * 32 + ((tid >> 2) & 15)) * UP + (tid >> 6) * 32 + 16 + (tid & 3) * 4, zero);
  }
  __syncthreads();
  // ---- T without its diagonal of ones, and the factors of rows
  for (int e = tid; e < DC_C * 16; e += DC_THREADS) {
    const int g = e >> 6, j = e & 63;
    if (g >> 2 <= j >> 4) {
      float x[4];
      load_vec<float, 4>(us + j * UP + 4 * g, x);
#pragma unroll
      for (int i = 0; i < 4; i++) if (4 * g + i == j) x[i] = 0.f;
      store_vec<float, 4>(ws + dc_tri(g, j), x);
    }
  }
  const float2 ge = sc->gam[DC_C - 1], zero2 = make_float2(0.f, 0.f);
  if (tid < DC_C) {
    const float2 gj = sc->gam[tid];
    const float d = dc_decay(gj, zero2), bj = sc->beta[tid];
    *reinterpret_cast<float4*>(ws + 2 * DC_TRI + 4 * tid) =
        make_float4(-bj * d * sc->ik[tid], d * sc->iq[tid], bj, dc_decay(ge, gj) * sc->ik[tid]);
  }
  if (tid == 0) ws[2 * DC_TRI + 4 * DC_C] = *abort_word == 0 ? dc_decay(ge, zero2) : nanf("");
  // ---- P T: tiles of four rows, sixteen threads to a row of tiles
  {
    const int jb = (tid >> 4) * 4, col = (tid & 15) * 4;
    f32x2 acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int k = 0; k < 4; k++) acc[i][k] = 0;
    dc_tile<2, 4, UP, 2>(acc, pt + jb, us + col, 0, jb);
    // the tile's own triangle: rows take nothing of later tokens, not even zero times (a NaN there is not theirs)
#pragma unroll
    for (int m = 0; m < 4; m++) {
      float um[4];
      load_vec<float, 4>(us + (jb + m) * UP + col, um);
      const float* coef = pt + (jb + m) * DC_PITCH + jb;
#pragma unroll
      for (int i = m / 2; i < 2; i++) {
        const float2 a = *reinterpret_cast<const float2*>(coef + 2 * i);
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float2 f = unpack2(acc[i][k]);
          acc[i][k] = 2 * i >= m ? fma2(pack2(a.x, a.y), pack2(um[k], um[k]), acc[i][k]) : pack2(f.x, fmaf(a.y, um[k], f.y));
        }
      }
    }
    if (col >> 4 <= jb >> 4) {
#pragma unroll
      for (int i = 0; i < 2; i++) {
        float x[4], y[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float2 f = unpack2(acc[i][k]);
          x[k] = f.x;
          y[k] = f.y;
        }
        store_vec<float, 4>(ws + DC_TRI + dc_tri(col >> 2, jb + 2 * i), x);
        store_vec<float, 4>(ws + DC_TRI + dc_tri(col >> 2, jb + 2 * i + 1), y);
      }
    }
  }
  __syncthreads();
  if (tid == 0 && *abort_word != 0 && p.status) atomicExch(p.status, *abort_word);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 64);
  }
}

// Threads of warps 0..7: row `row` of [K; Q], [T; P T] or of the state (the lane of tensor memory), 32 of the block's 64 columns.  Warp 8
// issues the products: 24 of them keep a thread busy for 1400 clocks, which is how long a row of T takes to arrive and be split.
__global__ void __launch_bounds__(DC_CHAIN_THREADS, 2) delta_chain_kernel(const DeltaChunkArgs p) {
  using Cfg = DcChainSmem;
  extern __shared__ __align__(1024) uint8_t dc_smem[];     // no room for alignment by hand beside a second block
  uint8_t* smem = dc_smem;
  uint8_t* s_parts = smem + Cfg::S_OFF;
  uint8_t* r_parts = s_parts;
  uint64_t* bars = (uint64_t*)(smem + Cfg::SC_OFF);        // [K; Q] S0, [T; P T] r, K^T u
  uint32_t* tmem_ptr = (uint32_t*)(bars + 3);
  volatile int* abort_word = (volatile int*)(tmem_ptr + 1);

  const int b = blockIdx.x, hv = blockIdx.y, j0 = blockIdx.z * DC_COLS, hk = hv / (p.Hv / p.Hk);
  const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
  const int t0 = p.cu[b], t1 = p.cu[b + 1], slot = p.slots[b];
  if (t1 - t0 < p.min_len) return;                         // short portions run in the token-serial kernel
  if (slot < 0 || slot >= p.num_slots || (smem_u32(smem) & 1023)) {
    if (tid == 0 && p.status) atomicExch(p.status, B200_BAD_INDEX);
    return;
  }
  const int chunks = (t1 - t0 + DC_C - 1) / DC_C, c_end = p.per_seq ? min(chunks, p.c0 + p.per_seq) : chunks;
  if (p.c0 >= c_end) return;
  const bool init = p.c0 > 0 || p.has_init[b] != 0;
  const int row = (warp & 3) * 32 + lane, j = row & 63, col0 = (warp >> 2 & 1) * 32;
  const bool is_q = row >= DC_C;
  float* state = p.state + ((long)slot * p.Hv + hv) * DC_K * p.DV + (long)row * p.DV + j0 + col0;

  if (tid == 0) {
    for (int i = 0; i < 3; i++) mbar_init(&bars[i], 1);
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 0) {
    tmem_alloc(tmem_ptr, Cfg::TMEM);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = warp_uniform(*tmem_ptr);
  const uint32_t t_lane = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  const uint64_t d_s = make_smem_desc(smem_u32(s_parts), 16384, 1024, kLayoutSw128), d_r = make_smem_desc(smem_u32(r_parts), Cfg::R_PART, 1024, kLayoutSw128);

  auto store_parts = [&](const float* v, uint8_t* dst, int r, int stride) {      // columns col0 .. col0 + 31 of row r
#pragma unroll
    for (int g = 0; g < 4; g++) dc_split8(v + 8 * g, dst + r * 128 + ((((col0 >> 3) + g) ^ (r & 7)) << 4), stride);
  };
  if (warp == 8) {
    for (int c = p.c0; c < c_end; c++) {
      const uint32_t kq = smem_u32(smem) + ((c - p.c0) & 1) * Cfg::KQ_BYTES;
      const uint64_t d_kq = make_smem_desc(kq, 16, 1024, kLayoutSw128), d_kt = make_smem_desc(kq, 16384, 1024, kLayoutSw128);
      __syncthreads();
      if (*abort_word != 0) break;
      if (elect_one()) {
        tc_fence_after();
        constexpr uint32_t id = make_idesc_f16(128, DC_COLS, true, false, true);
#pragma unroll
        for (int part = 2; part >= 0; part--)                // smallest first
#pragma unroll
          for (int kk = 0; kk < 8; kk++)
            umma_f16_ss(tmem + Cfg::D_COL, d_kq + (uint32_t)(((kk >> 2) * 16384 + (kk & 3) * 32) >> 4),
                        d_s + (uint32_t)((part * Cfg::S_PART + kk * 2048) >> 4), id, (part < 2 || kk > 0) ? 1u : 0u);
        umma_commit(&bars[0]);
      }
      __syncwarp();
      const int odd = __syncthreads_or(0);
      if (!odd && elect_one()) {
        tc_fence_after();
        constexpr uint32_t id = make_idesc_f16(128, DC_COLS, true, false, true);
        auto product = [&](int pt, int pr) {
#pragma unroll
          for (int kk = 0; kk < DC_C / 16; kk++)
            umma_f16_ts(tmem + Cfg::D_COL, tmem + Cfg::T_COL + pt * 32 + kk * 8, d_r + (uint32_t)((pr * Cfg::R_PART + kk * 2048) >> 4), id, 1u);
        };
        product(0, 2);                                       // smallest first
        product(2, 0);
        product(1, 1);
        product(0, 1);
        product(1, 0);
        product(0, 0);
        umma_commit(&bars[1]);
      }
      __syncwarp();
      if (odd) __syncthreads();
      __syncthreads();
      if (elect_one()) {
        tc_fence_after();
        constexpr uint32_t id = make_idesc_f16(128, DC_COLS, true, true, true);
#pragma unroll
        for (int part = 2; part >= 0; part--)
#pragma unroll
          for (int kk = 0; kk < DC_C / 16; kk++)
            umma_f16_ss(tmem + Cfg::S_COL, d_kt + (uint32_t)((kk * 2048) >> 4), d_r + (uint32_t)((part * Cfg::R_PART + kk * 2048) >> 4), id, 1u);
        umma_commit(&bars[2]);
      }
      __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    return;
  }
  {
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
      const float4 f = init ? *reinterpret_cast<const float4*>(state + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      v[i] = f.x; v[i + 1] = f.y; v[i + 2] = f.z; v[i + 3] = f.w;
    }
    tmem_st_32x32b_x32(t_lane + Cfg::S_COL + col0, reinterpret_cast<const uint32_t*>(v));
    store_parts(v, s_parts, row, Cfg::S_PART);
    tmem_st_wait();
  }
  // ---- k and q of a chunk: thread -> 16-byte chunk `ch` of rows tid / 16 + 16 i (i < 4: k, else q)
  const int ch = tid & 15, r0 = tid >> 4;
  const __nv_bfloat16* kp = (const __nv_bfloat16*)p.k + (long)hk * DC_K + ch * 8;
  const __nv_bfloat16* qp = (const __nv_bfloat16*)p.q + (long)hk * DC_K + ch * 8;
  const __nv_bfloat16* vp = (const __nv_bfloat16*)p.v + (long)hv * p.DV + j0 + (tid & 7) * 8;
  auto copy = [&](uint8_t* dst, const __nv_bfloat16* src, long stride, int t) {      // 16 bytes, zeros behind the sequence's end
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src + (long)(t < t1 ? t : t0) * stride),
                 "r"(t < t1 ? 16 : 0) : "memory");
  };
  auto fetch = [&](int c, bool q) {
    uint8_t* dst = smem + ((c - p.c0) & 1) * Cfg::KQ_BYTES + (ch >> 3) * 16384 + (q ? 8192 : 0);
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const int r = r0 + 16 * i;
      copy(dst + r * 128 + (((ch & 7) ^ (r & 7)) << 4), q ? qp : kp, p.qk_stride, t0 + c * DC_C + r);
    }
  };
  // v of chunk c lies where Q of chunk c - 1 was and Q of chunk c + 1 will be
  auto v_tile = [&](int c) { return smem + ((c - p.c0 + 1) & 1) * Cfg::KQ_BYTES + 8192; };
  auto fetch_v = [&](int c) {
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int r = (tid >> 3) + 32 * i;
      copy(v_tile(c) + r * 128 + (((tid & 7) ^ (r & 7)) << 4), vp, p.v_stride, t0 + c * DC_C + r);
    }
  };
  fetch(p.c0, false);
  fetch(p.c0, true);
  fetch_v(p.c0);

  uint32_t ph = 0, ph_r = 0;
  for (int c = p.c0; c < c_end; c++, ph ^= 1) {
    const int tc = t0 + c * DC_C;
    // the chunk's outputs, on their way to whole rows: the half of Q's place that v leaves, free until Q of the chunk after the next.  (Not
    // beside u: a thread ahead of others writes parts of S there.)
    uint8_t* o_tile = smem + ((c - p.c0) & 1) * Cfg::KQ_BYTES + 24576;
    const float* ws = p.ws + (dc_place(p, b, c, t0) * p.Hv + hv) * DC_WS;
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
    if (*abort_word != 0) break;
    if (c + 1 < c_end) fetch(c + 1, false);                // the other K's last reader was K^T u of the chunk before
    // ---- meanwhile this row of [T; P T] -> three parts in tensor memory (tokens m = col0 .. col0 + 31)
    const float* tri = ws + (is_q ? DC_TRI : 0);
    const float4 fac = *reinterpret_cast<const float4*>(ws + 2 * DC_TRI + 4 * j);      // of S0^T k, of S0^T q, beta, of u
    const float d_end = ws[2 * DC_TRI + 4 * DC_C];
    {
      float x[32];
#pragma unroll
      for (int i = 0; i < 32; i += 4) {
        const int g = (col0 + i) >> 2;
        const float4 f = g >> 2 <= j >> 4 ? *reinterpret_cast<const float4*>(tri + dc_tri(g, j)) : make_float4(0.f, 0.f, 0.f, 0.f);
        x[i] = f.x; x[i + 1] = f.y; x[i + 2] = f.z; x[i + 3] = f.w;
      }
      uint32_t part[3][16];
#pragma unroll
      for (int i = 0; i < 16; i++) {
        uint32_t w[3];
        dc_split2(x[2 * i], x[2 * i + 1], w);
        part[0][i] = w[0]; part[1][i] = w[1]; part[2][i] = w[2];
      }
#pragma unroll
      for (int q = 0; q < 3; q++) tmem_st_32x32b_x16(t_lane + Cfg::T_COL + q * 32 + (col0 >> 1), part[q]);
    }
    mbar_wait(&bars[0], ph, abort_word);
    tc_fence_after();
    // ---- r = beta (v - e^gamma S0^T k) -> parts, its accumulator cleared; e^gamma S0^T q stays in the accumulator
    int odd = 0;
    float x[32];                                           // r, then u (0, then o)
    {
      uint32_t d[32];
      tmem_ld_32x32b_x32(t_lane + Cfg::D_COL + col0, d);
      tmem_ld_wait();
      if (is_q) {
#pragma unroll
        for (int i = 0; i < 32; i++) {
          d[i] = __float_as_uint(__uint_as_float(d[i]) * fac.y);
          x[i] = 0.f;
        }
      } else {
#pragma unroll
        for (int i = 0; i < 4; i++) {
          const uint4 rv = *reinterpret_cast<const uint4*>(v_tile(c) + j * 128 + ((((col0 >> 3) + i) ^ (j & 7)) << 4));
          const uint32_t w[4] = {rv.x, rv.y, rv.z, rv.w};
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const float2 vv = unpack_bf16x2(w[q]);
            x[8 * i + 2 * q] = fmaf(__uint_as_float(d[8 * i + 2 * q]), fac.x, fac.z * vv.x);
            x[8 * i + 2 * q + 1] = fmaf(__uint_as_float(d[8 * i + 2 * q + 1]), fac.x, fac.z * vv.y);
          }
        }
#pragma unroll
        for (int i = 0; i < 32; i++) {
          odd |= !(fabsf(x[i]) < 3.38e38f);                // NaN, infinity, or what would be one in 16 bits
          d[i] = 0;
        }
        store_parts(x, r_parts, j, Cfg::R_PART);
      }
      tmem_st_32x32b_x32(t_lane + Cfg::D_COL + col0, d);
    }
    tmem_st_wait();
    fence_proxy_async_smem();
    tc_fence_before();
    odd = __syncthreads_or(odd);
    // ---- meanwhile the next chunk's q and v are on their way (v and q of this one have been read), and S0 e^{gamma_C} in place
    if (c + 1 < c_end) {
      fetch(c + 1, true);
      fetch_v(c + 1);
    }
    {
      uint32_t s[32];
      tmem_ld_32x32b_x32(t_lane + Cfg::S_COL + col0, s);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 32; i++) s[i] = __float_as_uint(__uint_as_float(s[i]) * d_end);
      tmem_st_32x32b_x32(t_lane + Cfg::S_COL + col0, s);
    }
    tmem_st_wait();
    if (!odd) {
      mbar_wait(&bars[1], ph_r, abort_word);
      ph_r ^= 1;
      tc_fence_after();
    }
#pragma unroll
    for (int h = 0; h < 32; h += 16) {
      uint32_t d[16];
      tmem_ld_32x32b_x16(t_lane + Cfg::D_COL + col0 + h, d);
      tmem_ld_wait();
#pragma unroll
      for (int i = 0; i < 16; i++) x[h + i] += __uint_as_float(d[i]);
    }
    if (odd) {
#pragma unroll 1
      for (int m = 0; m <= j; m++) {
        const float a = tri[dc_tri(m >> 2, j) + (m & 3)];
#pragma unroll
        for (int i = 0; i < 32; i++) {
          const uint8_t* e = r_parts + m * 128 + ((((col0 >> 3) + (i >> 3)) ^ (m & 7)) << 4) + (i & 7) * 2;
          float r = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(e));
          if (fabsf(r) < INFINITY)
            r += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(e + Cfg::R_PART)) +
                 __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(e + 2 * Cfg::R_PART));
          x[i] = fmaf(a, r, x[i]);
        }
      }
      __syncthreads();                                     // r has been read
    }
    if (is_q) {
#pragma unroll
      for (int g = 0; g < 4; g++)
        store_vec<__nv_bfloat16, 8>((__nv_bfloat16*)(o_tile + j * 128 + ((((col0 >> 3) + g) ^ (j & 7)) << 4)), x + 8 * g);
    } else {
#pragma unroll
      for (int i = 0; i < 32; i++) x[i] *= fac.w;
      store_parts(x, r_parts, j, Cfg::R_PART);             // e^{gamma_C - gamma_j} |k_j|^-1 u_j
    }
    fence_proxy_async_smem();
    tc_fence_before();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int r = (tid >> 3) + 32 * i;
      if (tc + r < t1)
        *reinterpret_cast<uint4*>((__nv_bfloat16*)p.out + (long)(tc + r) * p.out_stride + (long)hv * p.DV + j0 + (tid & 7) * 8) =
            *reinterpret_cast<const uint4*>(o_tile + r * 128 + (((tid & 7) ^ (r & 7)) << 4));
    }
    mbar_wait(&bars[2], ph, abort_word);
    tc_fence_after();
    tmem_ld_32x32b_x32(t_lane + Cfg::S_COL + col0, reinterpret_cast<uint32_t*>(x));
    tmem_ld_wait();
    if (c + 1 < c_end) {
      store_parts(x, s_parts, row, Cfg::S_PART);
    } else if (*abort_word == 0) {
#pragma unroll
      for (int i = 0; i < 32; i += 4) *reinterpret_cast<float4*>(state + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *abort_word != 0 && p.status) atomicExch(p.status, *abort_word);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, Cfg::TMEM);
  }
}

// bytes of workspace that a place of one head takes
long delta_chunk_place_bytes() { return DC_WS * sizeof(float); }

// true (with rc set) when the chunked kernels take these sizes; sequences shorter than p.min_len are left alone.  The workspace
// holds all chunks of the step (tokens / 64 + B places of every head), or else slices of as many chunks per sequence as it has room for
bool launch_delta_chunk(DeltaChunkArgs p, long tokens, int max_len, long ws_bytes, int DK, cudaStream_t stream, int* rc) {
  if (DK != DC_K || p.DV % DC_COLS || p.qk_stride % 8 || p.v_stride % 8 || !aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) ||
      !aligned16(p.state) || p.out_stride % 8 || !aligned16(p.out) || p.ws == nullptr || !aligned16(p.ws))
    return false;
  const long places = ws_bytes / (delta_chunk_place_bytes() * p.Hv), all = tokens / DC_C + p.B;
  const int chunks = (max_len + DC_C - 1) / DC_C;
  if (places < p.B) return false;
  cudaError_t e = allow_smem<delta_prep_kernel>(DcPrepSmem::BYTES);
  if (e == cudaSuccess) e = allow_smem<delta_chain_kernel>(DcChainSmem::BYTES);
  if (e != cudaSuccess) {
    *rc = (int)e;
    return true;
  }
  p.per_seq = places >= all ? 0 : (int)(places / p.B);
  const int step = p.per_seq ? p.per_seq : chunks;
  for (p.c0 = 0, *rc = 0; p.c0 < chunks && *rc == 0; p.c0 += step) {
    const long n = p.per_seq ? (long)p.B * p.per_seq : all;
    delta_prep_kernel<<<dim3((unsigned)n, (unsigned)p.Hv), DC_THREADS, DcPrepSmem::BYTES, stream>>>(p);
    delta_chain_kernel<<<dim3((unsigned)p.B, (unsigned)p.Hv, (unsigned)(p.DV / DC_COLS)), DC_CHAIN_THREADS, DcChainSmem::BYTES, stream>>>(p);
    *rc = B200_CHECK_LAUNCH();
  }
  return true;
}

}  // namespace b200
