// Prompt attention on tcgen05: two query tiles per block, probabilities in tensor memory.
//
// Two forms of one kernel:
//   paged GQA, head size 128   keys and values from the paged cache, the G = Hq / Hkv heads that share a KV head packed into
//                              the rows of a tile (row = token * G + head)
//   latent, dn + dr / dv       keys and values of every head in rows of their own (up-projected latents [keys][heads][dn + dv])
//                              with one rotary part [keys][dr] that all heads share: 3 slabs of 64 columns per key
// (counterparts: the prefill paths of vllm_ascend/attention/attention_v1.py:1341-1472 and of mla_v1.py:1373-1577, which
// also attends prompts over up-projected keys and values rather than in the latent space.)
//
// Bound: a tile of 128 x 128 scores is 0.6 to 0.7 us of MMA, and 128 x 128 exponentials with their loads, maxima and conversions
// take one warpgroup about 1.5 us.  One tile at a time (attention_tc.cu) leaves the tensor pipe idle two thirds of the time;
// here two query tiles share every K / V tile and a warpgroup each, and the MMA warp serves one while the other one's
// softmax runs.  Scores S0, S1 and outputs O0, O1 fill the 512 columns of tensor memory; probabilities replace the scores they
// came from (two bf16 to a column) and are the A operand of P V from there, so shared memory holds operands only.
// Because S(j + 1) of a tile is issued behind its P V(j), a softmax that sees S(j + 1) may also rescale O.
// 4096 tokens in two sequences, 32 heads of 128 + 64 / 128: 2687 us in the latent space, 156 us here (0.55 PFLOP/s) and 22 us of
// up-projection; 2048 tokens of 64 / 8 heads of 128 122 -> 103 us, 8000 tokens in eight prompts of 32 / 8 heads 217 -> 178 us.
//   warps 0..3, 4..7   softmax and epilogue of query tile 0, 1 (one thread per row)
//   warp 8             TMA producer;  warp 9  MMA issuer
// All waits are bounded.
#include "common.cuh"

#include <mutex>
#include <string>
#include <unordered_map>

namespace b200 {

constexpr int PF_THREADS = 320;
constexpr int PF_HALF = 128 * 128;          // 128 rows x 64 bf16
constexpr int PF_V_BYTES = 2 * PF_HALF;

struct PrefillParams {
  const int* cu;               // [num_seqs + 1] first query row of each sequence
  const int* kv_start;         // latent: [num_seqs + 1] first key row of each sequence
  const int* seq_lens;         // [num_seqs] keys of each sequence, its new tokens included
  const int* block_table;      // paged
  int num_seqs, max_blocks, block_size, rows_per_load;
  int G, tok_per_tile, dv;
  float scale_log2, rescale_threshold;
  int causal, window;
  __nv_bfloat16* out;
  long out_stride;
  long num_blocks_total;
  int* status;
};

__device__ __forceinline__ float pf_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <bool LATENT>
struct PrefillCfg {
  static constexpr int NK = LATENT ? 3 : 2;            // 64-column slabs of a query / key row
  static constexpr int VST = LATENT ? 1 : 2;           // value stages: what 227 KB leave beside two key stages
  static constexpr int Q_BYTES = NK * PF_HALF;
  static constexpr int K_BYTES = NK * PF_HALF;
  static constexpr int SMEM_BYTES = 2 * Q_BYTES + 2 * K_BYTES + VST * PF_V_BYTES + 1024 + 256;
};

template <bool LATENT>
__global__ void __launch_bounds__(PF_THREADS, 1)
attn_prefill_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                    const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_pe,
                    const PrefillParams p) {
  using Cfg = PrefillCfg<LATENT>;
  constexpr int NK = Cfg::NK, VST = Cfg::VST;
  constexpr int O_COL = 256;

  // ---------------- work item: a pair of query tiles; late pairs see more keys and come first
  const int h = blockIdx.x;
  const int wi = gridDim.y - 1 - blockIdx.y, pair = 2 * p.tok_per_tile, base = p.cu[0];
  int lo = 0, hi = p.num_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((p.cu[mid] - base) / pair + mid <= wi) lo = mid; else hi = mid - 1;
  }
  const int seq = lo;
  const int tok0 = (wi - ((p.cu[seq] - base) / pair + seq)) * pair;
  const int q_start = p.cu[seq], q_len = p.cu[seq + 1] - q_start, seq_len = p.seq_lens[seq], ctx = seq_len - q_len;
  if (tok0 >= q_len) return;
  int ntok[2], t_hi[2];
#pragma unroll
  for (int w = 0; w < 2; w++) {
    ntok[w] = max(0, min(p.tok_per_tile, q_len - tok0 - w * p.tok_per_tile));
    const int end = p.causal ? min(seq_len, ctx + tok0 + w * p.tok_per_tile + ntok[w]) : seq_len;
    t_hi[w] = ntok[w] > 0 ? (end + 127) >> 7 : 0;
  }
  const int t_lo = (p.window > 0 ? max(0, ctx + tok0 - p.window + 1) : 0) >> 7;
  const int n0 = t_hi[0] - t_lo, n = max(t_hi[0], t_hi[1]) - t_lo, n1 = ntok[1] > 0 ? n : 0;    // key tiles of each query tile
  if (n <= 0) return;                        // no keys: nothing would arrive that the roles below wait for; rows stay as they are

  const int warp = warp_index(), lane = threadIdx.x & 31;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint8_t* Qs = smem;
  uint8_t* Ks = Qs + 2 * Cfg::Q_BYTES;
  uint8_t* Vs = Ks + 2 * Cfg::K_BYTES;
  uint64_t* bars = (uint64_t*)(Vs + VST * PF_V_BYTES);
  uint64_t* q_full = bars;             // 2
  uint64_t* k_full = bars + 2;         // 2
  uint64_t* k_empty = bars + 4;        // 2
  uint64_t* v_full = bars + 6;         // 2
  uint64_t* v_empty = bars + 8;        // 2
  uint64_t* s_full = bars + 10;        // 2: scores of query tile w
  uint64_t* p_full = bars + 12;        // 2: probabilities of query tile w
  uint64_t* o_full = bars + 14;        // 2: last product of query tile w
  uint32_t* tmem_ptr = (uint32_t*)(bars + 16);
  volatile int* abort_word = (volatile int*)(tmem_ptr + 1);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; b++) {
      mbar_init(&q_full[b], 1);
      mbar_init(&k_full[b], 1);
      mbar_init(&k_empty[b], 1);
      mbar_init(&v_full[b], 1);
      mbar_init(&v_empty[b], 1);
      mbar_init(&s_full[b], 1);
      mbar_init(&p_full[b], 4);
      mbar_init(&o_full[b], 1);
    }
    *abort_word = 0;
    mbar_fence_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  if (warp == 8 && lane == 0) {
    tma_prefetch_desc(&tmap_q);
    tma_prefetch_desc(&tmap_k);
    tma_prefetch_desc(&tmap_v);
    if (LATENT) tma_prefetch_desc(&tmap_pe);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = warp_uniform(*tmem_ptr);

  if (warp == 8) {
    // ------------------------------------------------------------ producer
    if (lane == 0) {
      for (int w = 0; w < (ntok[1] > 0 ? 2 : 1); w++) {
        mbar_expect_tx(&q_full[w], Cfg::Q_BYTES);
        const int row = q_start + tok0 + w * p.tok_per_tile;
        for (int s = 0; s < NK; s++) {
          uint8_t* dst = Qs + w * Cfg::Q_BYTES + s * PF_HALF;
          if (LATENT) tma_load_3d(dst, &tmap_q, &q_full[w], s * 64, h, row);
          else tma_load_4d(dst, &tmap_q, &q_full[w], s * 64, 0, h, row);
        }
      }
    }
    const int parts = LATENT ? 1 : 128 / p.rows_per_load;
    const int* bt = LATENT ? nullptr : p.block_table + (long)seq * p.max_blocks;
    const int k_row0 = LATENT ? p.kv_start[seq] : 0;
    auto load_blk = [&](int j) -> int {        // lane i: page of part i, one tile ahead of its use
      if (LATENT || j >= n || lane >= parts) return 0;
      return bt[min(((t_lo + j) << 7) + lane * p.rows_per_load, seq_len - 1) / p.block_size];
    };
    int blk_cur = load_blk(0);
    for (int j = 0; j < n; j++) {
      const int key0 = (t_lo + j) << 7;
      const int blk_next = load_blk(j + 1);
      bool bad = !LATENT && (blk_cur < 0 || blk_cur >= p.num_blocks_total);
      bad = __any_sync(0xffffffffu, bad && lane < parts);
      for (int kv = 0; kv < 2; kv++) {
        const int st = kv == 0 ? j & 1 : j % VST;
        const uint32_t ph = (uint32_t)(kv == 0 ? j >> 1 : j / VST) & 1u;
        uint64_t* fullb = kv == 0 ? &k_full[st] : &v_full[st];
        if (!mbar_wait(kv == 0 ? &k_empty[st] : &v_empty[st], ph ^ 1u, abort_word)) goto done;
        if (bad) {
          *abort_word = B200_BAD_INDEX;
          goto done;
        }
        uint8_t* dst = kv == 0 ? Ks + st * Cfg::K_BYTES : Vs + st * PF_V_BYTES;
        if (elect_one()) mbar_expect_tx(fullb, kv == 0 ? Cfg::K_BYTES : PF_V_BYTES);
        if (LATENT) {
          if (elect_one()) {
            for (int s = 0; s < 2; s++)
              tma_load_3d(dst + s * PF_HALF, kv == 0 ? &tmap_k : &tmap_v, fullb, s * 64, h, k_row0 + key0);
            if (kv == 0) tma_load_2d(dst + 2 * PF_HALF, &tmap_pe, fullb, 0, k_row0 + key0);
          }
        } else {
          for (int part = 0; part < parts; part++) {
            const int blk = __shfl_sync(0xffffffffu, blk_cur, part);
            const int off = (key0 + part * p.rows_per_load) % p.block_size;
            if (elect_one())
              for (int s = 0; s < 2; s++)
                tma_load_4d(dst + s * PF_HALF + part * p.rows_per_load * 128, kv == 0 ? &tmap_k : &tmap_v, fullb, s * 64, h, off, blk);
          }
        }
        __syncwarp();
      }
      blk_cur = blk_next;
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------ MMA issuer: one thread walks the loop (see warp_uniform)
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_idesc_f16(128, 128, true, false, false);
      constexpr uint32_t idesc_o = make_idesc_f16(128, 128, true, false, true);
      const uint64_t dq0 = make_smem_desc(smem_u32(Qs), 16, 1024, kLayoutSw128), dk0 = make_smem_desc(smem_u32(Ks), 16, 1024, kLayoutSw128);
      const uint64_t dv0 = make_smem_desc(smem_u32(Vs), PF_HALF, 1024, kLayoutSw128);
      auto issue_s = [&](int w, int j) {
        const uint64_t dq = dq0 + (uint32_t)(w * (Cfg::Q_BYTES >> 4)), dk = dk0 + (uint32_t)((j & 1) * (Cfg::K_BYTES >> 4));
#pragma unroll
        for (int kk = 0; kk < NK * 4; kk++) {
          const uint32_t o = ((kk >> 2) * PF_HALF + (kk & 3) * 32) >> 4;
          umma_f16_ss(tmem_base + w * 128, dq + o, dk + o, idesc_s, kk > 0 ? 1u : 0u);
        }
        umma_commit(&s_full[w]);
      };
      if (!mbar_wait(&q_full[0], 0, abort_word)) goto done;
      if (n1 > 0 && !mbar_wait(&q_full[1], 0, abort_word)) goto done;
      if (!mbar_wait(&k_full[0], 0, abort_word)) goto done;
      tc_fence_after();
      issue_s(0, 0);
      if (n1 > 0) issue_s(1, 0);
      umma_commit(&k_empty[0]);
      for (int j = 0; j < n; j++) {
        const int vs = j % VST;
        if (!mbar_wait(&v_full[vs], (uint32_t)(j / VST) & 1u, abort_word)) goto done;
        if (j + 1 < n && !mbar_wait(&k_full[(j + 1) & 1], (uint32_t)((j + 1) >> 1) & 1u, abort_word)) goto done;
        const uint64_t dv = dv0 + (uint32_t)(vs * (PF_V_BYTES >> 4));
#pragma unroll 1
        for (int w = 0; w < 2; w++) {
          const int nw = w == 0 ? n0 : n1;
          if (j < nw) {
            if (!mbar_wait(&p_full[w], (uint32_t)j & 1u, abort_word)) goto done;
            tc_fence_after();
#pragma unroll
            for (int kk = 0; kk < 8; kk++)
              umma_f16_ts(tmem_base + O_COL + w * 128, tmem_base + w * 128 + kk * 8, dv + kk * 128, idesc_o, (j > 0 || kk > 0) ? 1u : 0u);
            if (j == nw - 1) umma_commit(&o_full[w]);
            if (j + 1 < nw) issue_s(w, j + 1);
          }
        }
        umma_commit(&v_empty[vs]);
        if (j + 1 < n) umma_commit(&k_empty[(j + 1) & 1]);
      }
    }
  } else {
    // ------------------------------------------------------------ softmax / epilogue of query tile w
    const int w = warp >> 2;
    const int nw = w == 0 ? n0 : n1;
    if (nw > 0) {
      const int row = (warp & 3) * 32 + lane, G = p.G;
      const int tok = row / G, g = row - tok * G;
      const int t_first = tok0 + w * p.tok_per_tile, nt = w == 0 ? ntok[0] : ntok[1];
      const bool row_valid = tok < nt;
      const int q_pos = ctx + t_first + tok;
      const uint32_t t_lane = tmem_base + ((uint32_t)((warp & 3) * 32) << 16);
      const uint32_t t_s = t_lane + w * 128, t_o = t_lane + O_COL + w * 128;
      const float sl2 = p.scale_log2;
      int k_hi = seq_len;                      // keys [k_lo, k_hi) are visible to this row
      if (p.causal) k_hi = min(k_hi, q_pos + 1);
      const int k_lo = p.window > 0 ? max(0, q_pos - p.window + 1) : 0;
      const int all_hi = p.causal ? min(seq_len, ctx + t_first + 1) : seq_len;      // seen by every row of the tile
      float m = -INFINITY, l = 0.f;
      for (int j = 0; j < nw; j++) {
        if (!mbar_wait(&s_full[w], (uint32_t)j & 1u, abort_word)) goto done;
        tc_fence_after();
        uint32_t sreg[128];
        tmem_ld_32x32b_x32(t_s, sreg);
        tmem_ld_32x32b_x32(t_s + 32, sreg + 32);
        tmem_ld_32x32b_x32(t_s + 64, sreg + 64);
        tmem_ld_32x32b_x32(t_s + 96, sreg + 96);
        tmem_ld_wait();
        const int key0 = (t_lo + j) << 7;
        if (key0 + 128 > all_hi || p.window > 0) {
#pragma unroll
          for (int i = 0; i < 128; i++) {
            const int key = key0 + i;
            if (key < k_lo || key >= k_hi) sreg[i] = 0xff800000u;   // -inf
          }
        }
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 8)
#pragma unroll
          for (int q = 0; q < 4; q++)
            mx[q] = fmaxf(mx[q], fmaxf(__uint_as_float(sreg[i + 2 * q]), __uint_as_float(sreg[i + 2 * q + 1])));
        const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
        // O is rescaled only when the running maximum moved by more than a threshold (powers of two: exact)
        float alpha = 1.f;
        bool need = false;
        if (mt > m && (m == -INFINITY || (mt - m) * sl2 > p.rescale_threshold)) {
          alpha = m == -INFINITY ? 0.f : pf_exp2((m - mt) * sl2);
          need = m != -INFINITY;               // an all-masked row has accumulated zeros only
          m = mt;
        }
        l *= alpha;
        if (j > 0 && __any_sync(0xffffffffu, need && row_valid)) {
          const float a = need ? alpha : 1.f;
#pragma unroll 1
          for (int c = 0; c < 4; c++) {
            uint32_t r[32];
            tmem_ld_32x32b_x32(t_o + c * 32, r);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * a);
            tmem_st_32x32b_x32(t_o + c * 32, r);
          }
        }
        const float nmb = m == -INFINITY ? 0.f : -m * sl2;
        float rs[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int c = 0; c < 4; c++) {
          uint32_t pk[16];
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const float p0 = pf_exp2(fmaf(__uint_as_float(sreg[c * 32 + 2 * i]), sl2, nmb));
            const float p1 = pf_exp2(fmaf(__uint_as_float(sreg[c * 32 + 2 * i + 1]), sl2, nmb));
            rs[(i & 1) * 2] += p0;
            rs[(i & 1) * 2 + 1] += p1;
            pk[i] = pack_bf16x2(p0, p1);
          }
          tmem_st_32x32b_x16(t_s + c * 16, pk);
        }
        l += (rs[0] + rs[1]) + (rs[2] + rs[3]);
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p_full[w]);
      }
      if (!mbar_wait(&o_full[w], 0, abort_word)) goto done;
      tc_fence_after();
      const float inv = l > 0.f ? 1.f / l : 0.f;
      __nv_bfloat16* dst = p.out + (long)(q_start + t_first + tok) * p.out_stride + (long)(h * G + g) * p.dv;
#pragma unroll 1
      for (int c = 0; c < 4; c++) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(t_o + c * 32, r);
        tmem_ld_wait();
        if (row_valid) {
#pragma unroll
          for (int q4 = 0; q4 < 4; q4++) {
            if (c * 32 + q4 * 8 >= p.dv) break;
            uint4 o;
            o.x = pack_bf16x2(__uint_as_float(r[q4 * 8 + 0]) * inv, __uint_as_float(r[q4 * 8 + 1]) * inv);
            o.y = pack_bf16x2(__uint_as_float(r[q4 * 8 + 2]) * inv, __uint_as_float(r[q4 * 8 + 3]) * inv);
            o.z = pack_bf16x2(__uint_as_float(r[q4 * 8 + 4]) * inv, __uint_as_float(r[q4 * 8 + 5]) * inv);
            o.w = pack_bf16x2(__uint_as_float(r[q4 * 8 + 6]) * inv, __uint_as_float(r[q4 * 8 + 7]) * inv);
            *reinterpret_cast<uint4*>(dst + c * 32 + q4 * 8) = o;
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
    // let copies still in flight land before the block's shared memory is released
    const uint64_t t_start = globaltimer_ns();
    while (globaltimer_ns() - t_start < 50000ull) __nanosleep(1000);
    if (threadIdx.x == 0 && p.status) atomicExch(p.status, *abort_word);
    __syncthreads();
  }
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// Dense row each sequence's keys begin at: out[0] = 0, out[i + 1] = out[i] + lens[i].
__global__ void __launch_bounds__(1024) key_starts_kernel(const int* __restrict__ lens, int n, int* __restrict__ out) {
  __shared__ int part[32];
  int carry = 0;
  if (threadIdx.x == 0) out[0] = 0;
  for (int i0 = 0; i0 < n; i0 += 1024) {
    const int i = i0 + threadIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int v = i < n ? lens[i] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += t;
    }
    if (lane == 31) part[warp] = v;
    __syncthreads();
    int before = carry, all = 0;
    for (int w = 0; w < 32; w++) {
      if (w < warp) before += part[w];
      all += part[w];
    }
    if (i < n) out[i + 1] = before + v;
    carry += all;
    __syncthreads();
  }
}

// Latents and rotary keys of listed sequences out of their pages into dense rows: lat [rows, dc], pe [rows, dr].
// One block per key row; kv_start [num_seqs + 1] is the dense row each sequence begins at.
__global__ void __launch_bounds__(128)
gather_latents_kernel(const __nv_bfloat16* __restrict__ lat_cache, const __nv_bfloat16* __restrict__ pe_cache, int dc, int dr,
                      int block_size, long num_blocks, const int* __restrict__ kv_start, const int* __restrict__ block_table,
                      int max_blocks, int num_seqs, __nv_bfloat16* __restrict__ lat, __nv_bfloat16* __restrict__ pe, int* status) {
  const int row = blockIdx.x;
  int lo = 0, hi = num_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (kv_start[mid] <= row) lo = mid; else hi = mid - 1;
  }
  const int pos = row - kv_start[lo], col = pos / block_size;
  const int blk = col < max_blocks ? block_table[(long)lo * max_blocks + col] : -1;
  if (blk < 0 || blk >= num_blocks) {
    if (threadIdx.x == 0 && status) atomicExch(status, B200_BAD_INDEX);
    return;
  }
  const long src = (long)blk * block_size + pos % block_size;
  const int nl = dc >> 3, np = dr >> 3;
  for (int v = threadIdx.x; v < nl + np; v += blockDim.x) {
    if (v < nl) reinterpret_cast<uint4*>(lat + (long)row * dc)[v] = reinterpret_cast<const uint4*>(lat_cache + src * dc)[v];
    else reinterpret_cast<uint4*>(pe + (long)row * dr)[v - nl] = reinterpret_cast<const uint4*>(pe_cache + src * dr)[v - nl];
  }
}

// ---------------------------------------------------------------- host
static int pf_tmap(CUtensorMap* out, const void* base, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box) {
  // encoding costs a few us; a map is a function of these values alone
  static std::unordered_map<std::string, CUtensorMap> cache;
  static std::mutex mu;
  char key[128];
  memset(key, 0, sizeof(key));
  memcpy(key, &base, 8);
  memcpy(key + 8, dims, 8 * rank);
  memcpy(key + 48, strides, 8 * (rank - 1));
  memcpy(key + 88, box, 4 * rank);
  key[120] = (char)rank;
  const std::string k(key, 128);
  std::lock_guard<std::mutex> g(mu);
  auto it = cache.find(k);
  if (it != cache.end()) {
    *out = it->second;
    return 0;
  }
  const int rc = make_tmap(out, base, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc) return rc;
  if (cache.size() > 4096) cache.clear();
  cache.emplace(k, *out);
  return 0;
}

template <bool LATENT>
static int launch_prefill(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const CUtensorMap& tpe,
                          const PrefillParams& p, int heads, long tokens, cudaStream_t stream) {
  using Cfg = PrefillCfg<LATENT>;
  static bool attr_set = false;
  if (!attr_set) {
    cudaError_t e = cudaFuncSetAttribute(attn_prefill_kernel<LATENT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES);
    if (e != cudaSuccess) return (int)e;
    attr_set = true;
  }
  const long pairs = tokens / (2 * p.tok_per_tile) + p.num_seqs;
  if (pairs > 65535) return 9875;
  attn_prefill_kernel<LATENT><<<dim3((unsigned)heads, (unsigned)pairs), PF_THREADS, Cfg::SMEM_BYTES, stream>>>(tq, tk, tv, tpe, p);
  return B200_CHECK_LAUNCH();
}

}  // namespace b200

using namespace b200;

// Causal (or full) attention of the new tokens of num_seqs sequences over their paged keys.  q [*, Hq, 128] and out rows have
// the token strides given; cu [num_seqs + 1] are row numbers of q / out, tokens = cu[num_seqs] - cu[0]; q_rows bounds q's rows.
B200_API int b200_attn_prefill(const void* q, long q_stride, long q_rows, const void* k_cache, const void* v_cache, long num_blocks,
                               int block_size, const void* cu, const void* seq_lens, const void* block_table, int max_blocks,
                               int num_seqs, long tokens, int Hq, int Hkv, float scale, int causal, int window, void* out,
                               long out_stride, int kv_layout, int* status, cudaStream_t stream) {
  if (num_seqs <= 0 || tokens <= 0) return 0;
  const int G = Hkv > 0 ? Hq / Hkv : 0, D = 128;
  if (G < 1 || G * Hkv != Hq || 128 % G) return 9870;
  if (block_size < 8 || (block_size < 128 && 128 % block_size) || (block_size > 128 && block_size % 128)) return 9871;
  if ((q_stride & 7) || (out_stride & 7)) return 9872;
  const int tpt = 128 / G, rpl = block_size < 128 ? block_size : 128;
  CUtensorMap tq, tk, tv;
  {
    uint64_t dims[4] = {(uint64_t)D, (uint64_t)G, (uint64_t)Hkv, (uint64_t)q_rows};
    uint64_t str[3] = {(uint64_t)D * 2, (uint64_t)G * D * 2, (uint64_t)q_stride * 2};
    uint32_t box[4] = {64, (uint32_t)G, 1, (uint32_t)tpt};
    int rc = pf_tmap(&tq, q, 4, dims, str, box);
    if (rc) return rc;
  }
  for (int kv = 0; kv < 2; kv++) {
    uint64_t dims[4] = {(uint64_t)D, (uint64_t)Hkv, (uint64_t)block_size, (uint64_t)num_blocks};
    uint64_t str[3] = {(uint64_t)D * 2, (uint64_t)Hkv * D * 2, (uint64_t)block_size * Hkv * D * 2};
    if (kv_layout == 1) {   // [blocks, heads, tokens, D]
      str[0] = (uint64_t)block_size * D * 2;
      str[1] = (uint64_t)D * 2;
    }
    uint32_t box[4] = {64, 1, (uint32_t)rpl, 1};
    int rc = pf_tmap(kv ? &tv : &tk, kv ? v_cache : k_cache, 4, dims, str, box);
    if (rc) return rc;
  }
  PrefillParams p = {};
  p.cu = (const int*)cu;
  p.seq_lens = (const int*)seq_lens;
  p.block_table = (const int*)block_table;
  p.num_seqs = num_seqs; p.max_blocks = max_blocks; p.block_size = block_size; p.rows_per_load = rpl;
  p.G = G; p.tok_per_tile = tpt; p.dv = D;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.rescale_threshold = 8.f;
  p.causal = causal; p.window = window;
  p.out = (__nv_bfloat16*)out;
  p.out_stride = out_stride;
  p.num_blocks_total = num_blocks;
  p.status = status;
  return launch_prefill<false>(tq, tk, tv, tk, p, Hkv, tokens, stream);
}

// Causal attention over up-projected latents: q [*, H, dn + dr] (token stride q_stride), kv [keys, H, dn + dv] dense, pe [keys, dr]
// dense, out [*, H, dv] dense.  cu [num_seqs + 1] rows of q / out, kv_start [num_seqs + 1] rows of kv / pe, seq_lens the keys of
// each sequence.  dn = 128, dv a multiple of 8 up to 128, dr a multiple of 8 up to 64.
B200_API int b200_attn_prefill_latent(const void* q, long q_stride, long q_rows, const void* kv, const void* pe, long keys,
                                      const void* cu, const void* kv_start, const void* seq_lens, int num_seqs, long tokens,
                                      int H, int dn, int dr, int dv, float scale, void* out, int* status, cudaStream_t stream) {
  if (num_seqs <= 0 || tokens <= 0) return 0;
  if (dn != 128 || dv < 8 || dv > 128 || dv % 8 || dr < 8 || dr > 64 || dr % 8 || H < 1 || (q_stride & 7)) return 9873;
  CUtensorMap tq, tk, tv, tpe;
  {
    uint64_t dims[3] = {(uint64_t)(dn + dr), (uint64_t)H, (uint64_t)q_rows};
    uint64_t str[2] = {(uint64_t)(dn + dr) * 2, (uint64_t)q_stride * 2};
    uint32_t box[3] = {64, 1, 128};
    int rc = pf_tmap(&tq, q, 3, dims, str, box);
    if (rc) return rc;
  }
  for (int v = 0; v < 2; v++) {
    uint64_t dims[3] = {(uint64_t)(v ? dv : dn), (uint64_t)H, (uint64_t)keys};
    uint64_t str[2] = {(uint64_t)(dn + dv) * 2, (uint64_t)H * (dn + dv) * 2};
    uint32_t box[3] = {64, 1, 128};
    int rc = pf_tmap(v ? &tv : &tk, (const __nv_bfloat16*)kv + (v ? dn : 0), 3, dims, str, box);
    if (rc) return rc;
  }
  {
    uint64_t dims[2] = {(uint64_t)dr, (uint64_t)keys};
    uint64_t str[1] = {(uint64_t)dr * 2};
    uint32_t box[2] = {64, 128};
    int rc = pf_tmap(&tpe, pe, 2, dims, str, box);
    if (rc) return rc;
  }
  PrefillParams p = {};
  p.cu = (const int*)cu;
  p.kv_start = (const int*)kv_start;
  p.seq_lens = (const int*)seq_lens;
  p.num_seqs = num_seqs;
  p.G = 1; p.tok_per_tile = 128; p.dv = dv;
  p.scale_log2 = scale * 1.4426950408889634f;
  p.rescale_threshold = 8.f;
  p.causal = 1;
  p.out = (__nv_bfloat16*)out;
  p.out_stride = (long)H * dv;
  p.status = status;
  return launch_prefill<true>(tq, tk, tv, tpe, p, H, tokens, stream);
}

// The keys of num_seqs sequences as dense rows: kv_start [num_seqs + 1] (written), lat [keys, dc], pe [keys, dr]; keys is the
// sum of seq_lens.
B200_API int b200_gather_latents(const void* lat_cache, const void* pe_cache, int dc, int dr, int block_size, long num_blocks,
                                 const void* seq_lens, const void* block_table, int max_blocks, int num_seqs, long keys,
                                 void* kv_start, void* lat, void* pe, int* status, cudaStream_t stream) {
  if (num_seqs <= 0 || keys <= 0) return 0;
  if (dc % 8 || dr % 8) return 9874;
  key_starts_kernel<<<1, 1024, 0, stream>>>((const int*)seq_lens, num_seqs, (int*)kv_start);
  gather_latents_kernel<<<(unsigned)keys, 128, 0, stream>>>(
      (const __nv_bfloat16*)lat_cache, (const __nv_bfloat16*)pe_cache, dc, dr, block_size, num_blocks, (const int*)kv_start,
      (const int*)block_table, max_blocks, num_seqs, (__nv_bfloat16*)lat, (__nv_bfloat16*)pe, status);
  return B200_CHECK_LAUNCH();
}
