// Sampling kernels.  Semantics follow the reference sampler
// (vllm_ascend/sample/sampler.py:20-271): penalties -> temperature -> top-k ->
// top-p (-> min-p) -> exponential-race sampling argmax(p / Exp(1)); greedy rows
// take argmax of the raw logits.  Instead of the reference's full sort, the
// top-k and top-p cut-offs are found with a 3-pass radix select over the float
// bit patterns (count histograms for top-k, mass histograms for top-p) on a row
// that stays in the shared memory of a cluster.
#include "common.cuh"

#include <type_traits>

namespace b200 {

constexpr int SAMP_THREADS = 1024;

// ---------------------------------------------------------------- Philox4x32-10
__device__ __forceinline__ uint4 philox4x32(uint4 ctr, uint2 key) {
  const uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u, W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
#pragma unroll
  for (int i = 0; i < 10; i++) {
    const uint32_t hi0 = __umulhi(M0, ctr.x), lo0 = M0 * ctr.x;
    const uint32_t hi1 = __umulhi(M1, ctr.z), lo1 = M1 * ctr.z;
    ctr = make_uint4(hi1 ^ ctr.y ^ key.x, lo1, hi0 ^ ctr.w ^ key.y, lo0);
    key.x += W0;
    key.y += W1;
  }
  return ctr;
}
__device__ __forceinline__ float u32_to_unit(uint32_t x) {  // (0, 1]
  return ((float)(x >> 8) + 1.0f) * (1.0f / 16777216.0f);
}

template <typename T>
__device__ __forceinline__ float ld_logit(const T* p, long i);
template <>
__device__ __forceinline__ float ld_logit<float>(const float* p, long i) { return p[i]; }
template <>
__device__ __forceinline__ float ld_logit<__nv_bfloat16>(const __nv_bfloat16* p, long i) {
  return __bfloat162float(p[i]);
}

// block-wide argmax helper: (value, index) with lowest index on ties
__device__ __forceinline__ void block_argmax(float& v, int& idx, float* sv, int* si) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, o);
    const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
    if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) { sv[warp] = v; si[warp] = idx; }
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    v = lane < nw ? sv[lane] : -INFINITY;
    idx = lane < nw ? si[lane] : 0x7fffffff;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xffffffffu, v, o);
      const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
      if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    if (lane == 0) { sv[0] = v; si[0] = idx; }
  }
  __syncthreads();
  v = sv[0];
  idx = si[0];
  __syncthreads();
}

template <typename T>
__global__ void argmax_kernel(const T* __restrict__ logits, long ld, int V,
                              long* __restrict__ out) {
  __shared__ float sv[32];
  __shared__ int si[32];
  const T* row = logits + (long)blockIdx.x * ld;
  float best = -INFINITY;
  int bi = 0x7fffffff;
  int done = 0;                        // elements [0, done) are covered by the vector loop
  if constexpr (sizeof(T) == 2) {
    // 16-byte loads (8 logits) when the row starts on a 16-byte boundary; a thread walks its
    // chunks in ascending index order, so "first maximum wins" still holds per thread
    if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
      const int nvec = V >> 3;
      const uint4* rv = reinterpret_cast<const uint4*>(row);
      for (int c = threadIdx.x; c < nvec; c += blockDim.x) {
        const uint4 q = rv[c];
        const uint32_t w4[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const float lo = __uint_as_float(w4[k] << 16);
          const float hi = __uint_as_float(w4[k] & 0xffff0000u);
          if (lo > best) { best = lo; bi = c * 8 + 2 * k; }
          if (hi > best) { best = hi; bi = c * 8 + 2 * k + 1; }
        }
      }
      done = nvec << 3;
    }
  }
  for (int i = done + threadIdx.x; i < V; i += blockDim.x) {
    const float v = ld_logit<T>(row, i);
    if (v > best || (v == best && i < bi)) { best = v; bi = i; }
  }
  block_argmax(best, bi, sv, si);
  if (threadIdx.x == 0) out[blockIdx.x] = bi;
}

// ---------------------------------------------------------------- penalties
// logits fp32 [B, V] in place. prompt_ids [B, Lp], output_ids [B, Lo] int64, padded with
// values >= V. rep/freq/pres: [B].  Dynamic smem: 2 bitmaps of ceil(V/32) words.
__global__ void penalties_kernel(float* logits, long ld, int V, const long* prompt_ids, int Lp,
                                 const long* output_ids, int Lo, const float* rep,
                                 const float* freq, const float* pres) {
  extern __shared__ uint32_t bm[];
  const int words = (V + 31) / 32;
  uint32_t* seen_all = bm;
  uint32_t* seen_out = bm + words;
  const int b = blockIdx.x;
  float* row = logits + (long)b * ld;
  const float rp = rep ? rep[b] : 1.f, fp = freq ? freq[b] : 0.f, pp = pres ? pres[b] : 0.f;
  if (rp == 1.f && fp == 0.f && pp == 0.f) return;
  for (int i = threadIdx.x; i < 2 * words; i += blockDim.x) bm[i] = 0;
  __syncthreads();
  if (rp != 1.f) {
    for (int i = threadIdx.x; i < Lp + Lo; i += blockDim.x) {
      const long id = i < Lp ? prompt_ids[(long)b * Lp + i] : output_ids[(long)b * Lo + (i - Lp)];
      if (id < 0 || id >= V) continue;
      const uint32_t bit = 1u << (id & 31);
      const uint32_t old = atomicOr(&seen_all[id >> 5], bit);
      if (!(old & bit)) {
        const float x = row[id];
        row[id] = x > 0.f ? x / rp : x * rp;
      }
    }
  }
  __syncthreads();
  if (fp != 0.f || pp != 0.f) {
    for (int i = threadIdx.x; i < Lo; i += blockDim.x) {
      const long id = output_ids[(long)b * Lo + i];
      if (id < 0 || id >= V) continue;
      const uint32_t bit = 1u << (id & 31);
      const uint32_t old = atomicOr(&seen_out[id >> 5], bit);
      float d = -fp;
      if (!(old & bit)) d -= pp;
      atomicAdd(&row[id], d);
    }
  }
}

// ---------------------------------------------------------------- top-k/top-p sampling
// A row of 150k fp32 logits is walked about ten times (maximum, exponentials, three digits of a radix select for
// top-k and three for top-p, the race), so the row is spread over a cluster of up to eight blocks and stays in their shared memory
// after one read of HBM.  What bounds it then is instructions and the cluster's meetings, so a walk touches as little as it can:
//   * the select passes only look at elements above a cut that already holds enough of them (2^-6 to 2^-24 of the
//     maximum, counted while the exponentials are taken): with peaked rows that leaves a few thousand shared-memory
//     atomics where there were V per pass.  Rows without top-k and top-p skip sums, cuts and their meeting;
//   * bins are integers (mass in units of 2^-40: shared memory adds 64-bit integers by itself, floats in a loop, and the
//     sum has no order), added and searched in parallel;
//   * where the cut leaves at most 2048 elements (top-k, peaked top-p), one block sorts them and ends the row by itself;
//   * rows with a small top-k need neither exponentials nor cuts of the whole row: the k-th largest of the threads' own maxima is a
//     bound that k elements of the block's slice reach, so no smaller one is among the row's k largest.  What reaches it, little more than
//     k a block, is all that the rest looks at;
//   * a slice comes in by bulk copies, all of it in flight at once;
//   * random numbers are drawn only for groups of four that hold a kept element;
//   * what the other blocks of the cluster say is read once per block: read by every thread, 192 x 32000 without top-k and top-p
//     took 115 us of which 88 reads per thread were most, 56 us so (37 us with two blocks a row, 66 us one block with the row in L2).
//   * top-p without top-k: one histogram of fine bins between the cut and the maximum, and the elements of the bin in question to rank 0.
// 192 rows of 151936, cold, us: greedy 44 (58 with plain loads), top-k 50 78 (135 with exponentials and cuts of the whole row, 849 with one block
// per row and thread-serial bins), top-p 0.8 144 (172), 0.95 at temperature 0.8 233 (278) and 1 272 (366; three digits and remote additions
// per warp), nothing cut 122 (135).
constexpr int SAMP_T = 512;
constexpr int SAMP_BINS = 2048;
constexpr int SAMP_MAX_SLICE = 50 * 1024;        // elements of a row that a block keeps in shared memory
constexpr int SAMP_PAIR_SLICE = 23000;           // ... while an SM holds two such blocks
constexpr int SAMP_TWO_HIST_SLICE = 47000;       // ... beside a second histogram (256 flat rows of 262144, top-p: 4294 -> 2960 us)
constexpr int SAMP_CUTS = 5;
constexpr int SAMP_SMALL_K = 1024;               // blocks of a row (four or more) times k, up to which top-k takes what threads' maxima bound
constexpr int SAMP_BULK = 4;                     // bulk copies of a slice
using samp_n = unsigned long long;     // elements, or mass in units of 2^-40 (e <= 1, so a row's mass fits)
constexpr float SAMP_UNIT = 1099511627776.f;

struct SampXch { float v[1 + SAMP_CUTS]; uint32_t n[SAMP_CUTS]; int i; };

// C: blocks per row (a cluster), K: histograms per block (a lane adds to its own, so that fewer lanes meet in a bin)
template <int C, int K>
struct SampSmem {
  samp_n hist[K * SAMP_BINS];
  static constexpr int OWN = C > 1 ? SAMP_BINS / C : 512;
  samp_n own[OWN];                     // this block's bins, summed over the cluster; top-k: its candidates (logit, index)
  samp_n tot[6];                       // sum of `own`, one slot per select pass
  samp_n remaining;
  SampXch xch[4];                      // what a block tells the others: one slot per meeting
  SampXch all[4];                      // the same over the cluster
  float red[SAMP_T / 32][1 + 2 * SAMP_CUTS];
  float sv[32];
  int si[32];
  samp_n sn[SAMP_T / 32];
  uint64_t bar[SAMP_BULK];
  uint32_t prefix;
  uint32_t listed;                     // candidates in hist (rank 0)
  uint32_t found, odd;                 // top-k: candidates in `own`, whether one is a NaN
  int abort;
};

template <int C>
__device__ __forceinline__ void samp_meet() {
  if constexpr (C == 1) __syncthreads();
  else asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// the value at `p` (shared memory of this block) in block r of the cluster
template <int C, typename U>
__device__ __forceinline__ U samp_peek(const U* p, int r) {
  if constexpr (C == 1) return *(const volatile U*)p;
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(r));
  U out;
  if constexpr (sizeof(U) == 8) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    memcpy(&out, &v, 8);
  } else {
    uint32_t v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
    memcpy(&out, &v, 4);
  }
  return out;
}
// sum of v over the block, in every thread
__device__ __forceinline__ float samp_block_sum(float v, float* red) {
  v = warp_reduce_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = threadIdx.x % 32 < SAMP_T / 32 ? red[threadIdx.x % 32] : 0.f;
  v = warp_reduce_sum(v);
  __syncthreads();
  return v;
}
__device__ __forceinline__ samp_n samp_warp_sum(samp_n v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ void samp_better(float& v, int& i, float ov, int oi) {
  if (ov > v || (ov == v && oi < i)) { v = ov; i = oi; }
}
// argmax over the cluster, lowest index on ties; `found`: all blocks' numbers of candidates (SAMP_NONE: one has none to offer), in
// all[slot].n[0] the sum and in n[1] what blocks before this one have
constexpr uint32_t SAMP_NONE = 1u << 20;
template <int C, int K>
__device__ void samp_cluster_argmax(float& v, int& idx, SampSmem<C, K>* s, int slot, uint32_t found = 0, int rank = 0) {
  block_argmax(v, idx, s->sv, s->si);
  if constexpr (C == 1) {
    if (threadIdx.x == 0) { s->all[slot].n[0] = found; s->all[slot].n[1] = 0; }
    __syncthreads();
  } else {
    if (threadIdx.x == 0) { s->xch[slot].v[0] = v; s->xch[slot].i = idx; s->xch[slot].n[0] = found; }
    samp_meet<C>();
    if (threadIdx.x < 32) {
      v = samp_peek<C>(&s->xch[slot].v[0], threadIdx.x % C);
      idx = samp_peek<C>(&s->xch[slot].i, threadIdx.x % C);
      const uint32_t f = threadIdx.x < C ? samp_peek<C>(&s->xch[slot].n[0], threadIdx.x) : 0;
      const uint32_t sum = __reduce_add_sync(0xffffffffu, f), before = __reduce_add_sync(0xffffffffu, (int)threadIdx.x < rank ? f : 0);
      if (threadIdx.x == 0) { s->all[slot].n[0] = sum; s->all[slot].n[1] = before; }
#pragma unroll
      for (int o = C / 2; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        samp_better(v, idx, ov, oi);
      }
      if (threadIdx.x == 0) { s->all[slot].v[0] = v; s->all[slot].i = idx; }
    }
    __syncthreads();
    v = s->all[slot].v[0];
    idx = s->all[slot].i;
  }
}

// One digit of the select: histogram (elements or their mass) of the `bits`-wide digit at `shift` of the key less `base` over the
// elements whose higher bits equal the prefix and whose key reaches floor_key, then the bin, walking down from the top, at which the
// running sum reaches `remaining`.  Every block of the cluster ends with the same prefix and remaining.
template <bool MASS, int C, int K>
__device__ void samp_pass(const float* e, int n, SampSmem<C, K>* s, int pass, int shift, int bits, uint32_t hi_mask, uint32_t floor_key, int rank,
                          uint32_t base = 0) {
  const int nb = 1 << bits;
  for (int i = threadIdx.x; i < K * nb; i += SAMP_T) s->hist[i] = 0;
  samp_n* hist = s->hist + (threadIdx.x & (K - 1)) * nb;
  __syncthreads();
  const uint32_t prefix = s->prefix;
  const samp_n rem0 = s->remaining;
  for (int i = threadIdx.x; i < n; i += SAMP_T) {
    const float v = e[i];
    const uint32_t k = __float_as_uint(v);
    if (k < floor_key || (k & hi_mask) != prefix) continue;
    atomicAdd(&hist[((k - base) >> shift) & (nb - 1)], MASS ? __float2ull_rn(v * SAMP_UNIT) : 1ull);
  }
  samp_meet<C>();
  if constexpr (C == 1) {
    // thread t owns bins [top - w (t + 1), top - w t)
    constexpr int W = SAMP_BINS / SAMP_T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, w = nb / SAMP_T;
    samp_n mine[W], sum = 0;
#pragma unroll
    for (int j = 0; j < W; j++) {
      mine[j] = 0;
      for (int h = 0; h < K; h++) mine[j] += j < w ? s->hist[h * nb + nb - 1 - ((int)threadIdx.x * w + j)] : 0;
      sum += mine[j];
    }
    samp_n upto = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const samp_n t = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += t;
    }
    if (lane == 31) s->sn[warp] = upto;
    __syncthreads();
    samp_n before = upto - sum, all = 0;
    for (int v = 0; v < SAMP_T / 32; v++) {
      if (v < warp) before += s->sn[v];
      all += s->sn[v];
    }
    // rounding can leave the whole sum below rem0: the lowest bin
    if (rem0 == 0 ? threadIdx.x == 0 : all < rem0 ? threadIdx.x == SAMP_T - 1 : before < rem0 && before + sum >= rem0) {
      samp_n rem = rem0 - before;
      int sel = w - 1;
#pragma unroll
      for (int j = 0; j < W; j++)
        if (j < w - 1 && sel == w - 1) {
          if (mine[j] >= rem) sel = j;
          else rem -= mine[j];
        }
      s->prefix = prefix | ((uint32_t)(nb - 1 - ((int)threadIdx.x * w + sel)) << shift);
      s->remaining = rem;
    }
  } else {
    const int per = nb / C;
    samp_n b = 0;
    for (int i = threadIdx.x; i < per; i += SAMP_T) {
      samp_n t = 0;
#pragma unroll
      for (int r = 0; r < C * K; r++) t += samp_peek<C>(&s->hist[r / C * nb + rank * per + i], r % C);
      s->own[i] = t;
      b += t;
    }
    b = samp_warp_sum(b);
    if ((threadIdx.x & 31) == 0) s->sn[threadIdx.x >> 5] = b;
    __syncthreads();
    if (threadIdx.x < 32) {
      b = samp_warp_sum(threadIdx.x < SAMP_T / 32 ? s->sn[threadIdx.x] : 0);
      if (threadIdx.x == 0) s->tot[pass] = b;
    }
    samp_meet<C>();
    if (threadIdx.x < 32) {
      const int lane = threadIdx.x;
      const samp_n t_lane = samp_peek<C>(&s->tot[pass], lane % C);
      samp_n rem = rem0;
      int r = C - 1;
      for (; r > 0; r--) {
        const samp_n t = __shfl_sync(0xffffffffu, t_lane, r);
        if (t >= rem) break;
        rem -= t;
      }
      // lane l owns bins [top - w (l + 1), top - w l) of block r
      constexpr int W = SAMP_BINS / C / 32;
      const int w = per / 32;
      samp_n mine[W], sum = 0;
#pragma unroll
      for (int j = 0; j < W; j++) {
        mine[j] = j < w ? samp_peek<C>(&s->own[per - 1 - (lane * w + j)], r) : 0;
        sum += mine[j];
      }
      samp_n upto = sum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const samp_n t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
      }
      const uint32_t hit = __ballot_sync(0xffffffffu, upto >= rem);
      const int who = hit ? __ffs(hit) - 1 : 31;                     // rounding can leave every sum below rem: the lowest bin
      if (lane == who) {
        rem -= upto - sum;
        int sel = w - 1;
#pragma unroll
        for (int j = 0; j < W; j++)
          if (j < w - 1 && sel == w - 1) {
            if (mine[j] >= rem) sel = j;
            else rem -= mine[j];
          }
        s->prefix = prefix | ((uint32_t)(r * per + per - 1 - (lane * w + sel)) << shift);
        s->remaining = rem;
      }
    }
  }
  __syncthreads();
}

// Elements above the cut (and no higher than `top`), gathered from the whole cluster into rank 0's `hist` as (key, inverted index): value
// descending, index ascending is then one 64-bit order.  A block counts before it writes, so that it asks rank 0 for room once: with a
// remote addition per warp and hit, 2000 candidates of a row took 10 us, one after the other.
template <int C, int K>
__device__ void samp_gather(const float* e, int n, int first, uint32_t cut, SampSmem<C, K>* s, uint32_t top = 0xffffffffu) {
  uint32_t list, count;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(list) : "r"(smem_u32(s->hist)));
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(count) : "r"(smem_u32(&s->listed)));
  const bool whole = (reinterpret_cast<uintptr_t>(e) & 15) == 0;
  const int nv = whole ? n >> 2 : 0, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto in = [&](float v) { const uint32_t k = __float_as_uint(v); return k >= cut && k <= top; };
  auto each = [&](auto f) {
    for (int c = threadIdx.x; c < nv; c += SAMP_T) {
      const float4 q = reinterpret_cast<const float4*>(e)[c];
      if (in(q.x)) f(q.x, 4 * c);
      if (in(q.y)) f(q.y, 4 * c + 1);
      if (in(q.z)) f(q.z, 4 * c + 2);
      if (in(q.w)) f(q.w, 4 * c + 3);
    }
    for (int i = 4 * nv + threadIdx.x; i < n; i += SAMP_T)
      if (in(e[i])) f(e[i], i);
  };
  uint32_t mine = 0;
  each([&](float, int) { mine++; });
  uint32_t upto = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  __syncthreads();
  if (lane == 31) s->sn[warp] = upto;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (int w = 0; w < SAMP_T / 32; w++) {
    if (w < warp) before += (uint32_t)s->sn[w];
    all += (uint32_t)s->sn[w];
  }
  if (threadIdx.x == 0) {
    uint32_t at = 0;
    if (all) asm volatile("atom.relaxed.cluster.shared::cluster.add.u32 %0, [%1], %2;" : "=r"(at) : "r"(count), "r"(all) : "memory");
    s->found = at;
  }
  __syncthreads();
  uint32_t at = s->found + before + upto - mine;
  if (mine)
    each([&](float v, int i) {
      const samp_n w = (samp_n)__float_as_uint(v) << 32 | (uint32_t)~(first + i);
      if (at < SAMP_BINS) asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(list + at * 8), "l"(w) : "memory");
      at++;
    });
}

// Rank 0 alone: the n gathered candidates in descending order
template <int C, int K>
__device__ void samp_sort(SampSmem<C, K>* s, int n) {
  samp_n* c = s->hist;
  int size = 32;
  while (size < n) size *= 2;
  for (int i = n + threadIdx.x; i < size; i += SAMP_T) c[i] = 0;
  __syncthreads();
  for (int len = 2; len <= size; len *= 2)
    for (int step = len / 2; step > 0; step /= 2) {
      for (int t = threadIdx.x; t < size / 2; t += SAMP_T) {
        const int i = 2 * t - (t & (step - 1)), j = i + step;
        const samp_n a = c[i], b = c[j];
        if ((a < b) == ((i & len) == 0)) { c[i] = b; c[j] = a; }       // descending
      }
      __syncthreads();
    }
}
// Rank 0 alone: running mass over the n sorted candidates that reach thr, in units of 2^-40 (a thread sums its run of neighbours, then
// their sums are scanned); s->prefix becomes the value of the first at which it reaches want(total).  Returns want.
template <int C, int K, typename F>
__device__ samp_n samp_reach(SampSmem<C, K>* s, int n, uint32_t thr, F want_of) {
  const samp_n* c = s->hist;
  auto value = [&](int i) { return (uint32_t)(c[i] >> 32); };
  constexpr int PER = SAMP_BINS / SAMP_T;
  samp_n run[PER], sum = 0;
#pragma unroll
  for (int j = 0; j < PER; j++) {
    const int i = threadIdx.x * PER + j;
    if (i < n && value(i) >= thr) sum += __float2ull_rn(__uint_as_float(value(i)) * SAMP_UNIT);
    run[j] = sum;
  }
  samp_n upto = sum;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const samp_n t = __shfl_up_sync(0xffffffffu, upto, o);
    if (lane >= o) upto += t;
  }
  if (lane == 31) s->sn[warp] = upto;
  if (threadIdx.x == 0) s->prefix = 0;
  __syncthreads();
  samp_n before = upto - sum, all = 0;
  for (int w = 0; w < SAMP_T / 32; w++) {
    if (w < warp) before += s->sn[w];
    all += s->sn[w];
  }
  const samp_n want = want_of(all);
#pragma unroll
  for (int j = 0; j < PER; j++) {                        // the first element at which the sum reaches what is wanted
    const int i = threadIdx.x * PER + j;
    const samp_n prev = before + (j ? run[j - 1] : 0);
    if (i < n && before + run[j] >= want && (prev < want || i == 0)) s->prefix = value(i);
  }
  __syncthreads();
  return want;
}

// Rank 0 alone: orders the n gathered candidates, cuts them by rank and by mass, and runs the race.  `mass` is what top-p is a
// share of where top-k is off.
template <int C, int K>
__device__ int samp_finish(SampSmem<C, K>* s, int n, int k, float pth, float mp, float mass, uint2 key, long offset, int fallback) {
  samp_n* c = s->hist;
  samp_sort(s, n);
  auto value = [&](int i) { return (uint32_t)(c[i] >> 32); };
  uint32_t thr = k > 0 ? value(k - 1) : 0;
  if (pth < 1.f && value(0) <= 0x7F800000u) {              // a row with a NaN has no mass to take a share of
    const samp_n want = samp_reach(s, n, thr, [&](samp_n all) {
      return __float2ull_rn(pth * (k > 0 ? (float)all / SAMP_UNIT : mass) * SAMP_UNIT);
    });
    if (want == 0) thr = 0xffffffffu;                      // a share of nothing: the largest element
    else if (s->prefix > thr) thr = s->prefix;
  }
  if (mp > 0.f && __float_as_uint(mp) > thr) thr = __float_as_uint(mp);
  float bestv = -INFINITY;
  int besti = fallback;
  for (int i = threadIdx.x; i < n; i += SAMP_T) {
    const float v = __uint_as_float(value(i));
    if (value(i) < thr) break;
    if (!(v > 0.f)) continue;
    const int idx = (int)~(uint32_t)c[i];
    const uint4 rnd = philox4x32(make_uint4((uint32_t)(idx & ~3), (uint32_t)offset, (uint32_t)((unsigned long long)offset >> 32), 0u), key);
    const uint32_t r = (idx & 2) ? ((idx & 1) ? rnd.w : rnd.z) : ((idx & 1) ? rnd.y : rnd.x);
    const float ex = -__logf(u32_to_unit(r));  // Exp(1)
    samp_better(bestv, besti, v / fmaxf(ex, 1e-20f), idx);
  }
  block_argmax(bestv, besti, s->sv, s->si);
  return besti;
}

// logits: fp32 [B, V] (already penalised); overwritten where a row does not fit the cluster's shared memory.
// temperature/top_k/top_p/min_p: per row (top_k <= 0 or >= V: off; top_p >= 1: off).
// seeds: per-row uint64 seed, offsets: per-row counter (e.g. number of tokens generated).
template <int C, int K>
__global__ void __launch_bounds__(SAMP_T, 2)
sample_kernel(float* logits, long ld, int V, int slice, int resident, const float* __restrict__ temperature,
              const int* __restrict__ top_k, const float* __restrict__ top_p,
              const float* __restrict__ min_p, const unsigned long long* __restrict__ seeds,
              const long* __restrict__ offsets, long* __restrict__ out) {
  __shared__ SampSmem<C, K> s;
  extern __shared__ __align__(16) float kept_row[];
  const int rank = blockIdx.x, b = blockIdx.y;
  const int first = rank * slice, n = max(0, min(V - first, slice));
  float* row = logits + (long)b * ld + first;
  float* e = resident ? kept_row : row;
  const float temp = temperature ? temperature[b] : 1.f;
  const int k = top_k ? top_k[b] : 0;
  const float pth = top_p ? top_p[b] : 1.f, mp = min_p ? min_p[b] : 0.f;
  const bool greedy = temp < 1e-5f, by_rank = k > 0 && k < V;
  // ---- the row comes in; its maximum (also the greedy answer)
  float best = -INFINITY;
  int bi = 0x7fffffff;
  const bool keep = resident && !greedy;
  int done = 0;
  auto look = [&](const float4& q, int c) {
    if (q.x > best) { best = q.x; bi = first + 4 * c; }
    if (q.y > best) { best = q.y; bi = first + 4 * c + 1; }
    if (q.z > best) { best = q.z; bi = first + 4 * c + 2; }
    if (q.w > best) { best = q.w; bi = first + 4 * c + 3; }
  };
  if (threadIdx.x == 0) { s.listed = 0; s.found = 0; s.odd = 0; s.abort = 0; }
  if ((reinterpret_cast<uintptr_t>(row) & 15) == 0) {
    const int nv = n >> 2;
    bool here = false;                   // the slice is in shared memory
    if (resident) {
      if (threadIdx.x == 0) {
        for (int i = 0; i < SAMP_BULK; i++) mbar_init(&s.bar[i], 1);
        mbar_fence_init();
        for (int i = 0; i < SAMP_BULK; i++) {
          const int c0 = nv * i / SAMP_BULK, bytes = (nv * (i + 1) / SAMP_BULK - c0) * 16;
          mbar_expect_tx(&s.bar[i], bytes);
          if (bytes)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             smem_u32(e + 4 * c0)), "l"(row + 4 * c0), "r"(bytes), "r"(smem_u32(&s.bar[i])) : "memory");
        }
      }
      __syncthreads();
      here = true;
      for (int i = 0; i < SAMP_BULK && here; i++) {
        here = mbar_wait(&s.bar[i], 0, &s.abort);
        const int c1 = nv * (i + 1) / SAMP_BULK;
        if (here)
#pragma unroll 4
          for (int c = nv * i / SAMP_BULK + threadIdx.x; c < c1; c += SAMP_T) look(reinterpret_cast<const float4*>(e)[c], c);
      }
      here = __syncthreads_and(here);
    }
    if (!here) {                         // not resident, or a copy that did not arrive
#pragma unroll 4
      for (int c = threadIdx.x; c < nv; c += SAMP_T) {
        const float4 q = reinterpret_cast<const float4*>(row)[c];
        if (keep) reinterpret_cast<float4*>(e)[c] = q;
        look(q, c);
      }
    }
    done = 4 * nv;
  }
#pragma unroll 4
  for (int i = done + threadIdx.x; i < n; i += SAMP_T) {
    const float v = row[i];
    if (keep) e[i] = v;
    if (v > best) { best = v; bi = first + i; }
  }
  // ---- a small top-k: what reaches the k-th largest of the threads' maxima (its upper sixteen bits, in an order of integers)
  uint32_t found = SAMP_NONE;
  if (by_rank && keep && k <= SAMP_SMALL_K / (C > 4 ? C : 4)) {
    uint32_t key = __float_as_uint(best);
    key ^= (uint32_t)((int)key >> 31) | 0x80000000u;
    uint32_t t = 0;
#pragma unroll 1
    for (int bit = 31; bit >= 16; bit--)
      if (__syncthreads_count(key >= (t | 1u << bit)) >= k) t |= 1u << bit;
    const float bound = __uint_as_float(t & 0x80000000u ? t ^ 0x80000000u : ~t);
    auto offer = [&](float v, int i) {
      if (v < bound) return;             // a NaN is offered, and told
      if (v != v) s.odd = 1;
      const uint32_t at = atomicAdd(&s.found, 1u);
      if (at < s.OWN) s.own[at] = (samp_n)__float_as_uint(v) << 32 | (uint32_t)i;
    };
    for (int c = threadIdx.x; c < n >> 2; c += SAMP_T) {
      const float4 q = reinterpret_cast<const float4*>(e)[c];
      if (q.x < bound && q.y < bound && q.z < bound && q.w < bound) continue;
      offer(q.x, 4 * c); offer(q.y, 4 * c + 1); offer(q.z, 4 * c + 2); offer(q.w, 4 * c + 3);
    }
    for (int i = (n & ~3) + threadIdx.x; i < n; i += SAMP_T) offer(e[i], i);
    __syncthreads();
    if (!s.odd && s.found <= s.OWN) found = s.found;
  }
  samp_cluster_argmax(best, bi, &s, 0, found, rank);
  if (greedy) {
    if (rank == 0 && threadIdx.x == 0) out[b] = bi;
    samp_meet<C>();                    // nobody leaves while another reads its memory
    return;
  }
  const float invT = 1.f / temp;
  const unsigned long long seed = seeds ? seeds[b] : 0ull;
  const long offset = offsets ? offsets[b] : 0;
  const uint2 key = make_uint2((uint32_t)seed, (uint32_t)(seed >> 32));
  const uint32_t offered = s.all[0].n[0];
  if (offered < SAMP_NONE && fabsf(best) < INFINITY) {               // every block has offered: the same in all of them
    uint32_t list;
    if constexpr (C > 1) asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(list) : "r"(smem_u32(s.hist)));
    else list = smem_u32(s.hist);
    list += s.all[0].n[1] * 8;
    for (uint32_t i = threadIdx.x; i < found; i += SAMP_T) {
      const float v = __uint_as_float((uint32_t)(s.own[i] >> 32));
      const samp_n w = (samp_n)__float_as_uint(__expf((v - best) * invT)) << 32 | (uint32_t)~(first + (uint32_t)s.own[i]);
      if constexpr (C > 1) asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(list + i * 8), "l"(w) : "memory");
      else s.hist[i] = w;
    }
    samp_meet<C>();
    if (rank != 0) return;
    const int win = samp_finish(&s, (int)offered, k, pth, mp, 0.f, key, offset, bi);
    if (threadIdx.x == 0) out[b] = win;
    return;
  }
  // ---- e = exp((x - max)/T); where something is cut by rank or mass, their sum and how much lies above each cut
  const uint32_t cuts[SAMP_CUTS] = {0x3C800000u, 0x3A800000u, 0x38800000u, 0x36800000u, 0x33800000u};   // 2^-6, -10, -14, -18, -24
  float z = 0.f, zc[SAMP_CUTS];
  uint32_t nc[SAMP_CUTS];
  if (by_rank || pth < 1.f) {
    float part[1 + 2 * SAMP_CUTS];     // sum, sum and number above each cut
#pragma unroll
    for (int j = 0; j < 1 + 2 * SAMP_CUTS; j++) part[j] = 0.f;
    for (int i = threadIdx.x; i < n; i += SAMP_T) {
      const float ev = __expf((e[i] - best) * invT);
      e[i] = ev;
      part[0] += ev;
#pragma unroll
      for (int j = 0; j < SAMP_CUTS; j++)
        if (__float_as_uint(ev) >= cuts[j]) { part[1 + j] += ev; part[1 + SAMP_CUTS + j] += 1.f; }
    }
#pragma unroll
    for (int j = 0; j < 1 + 2 * SAMP_CUTS; j++) {
      part[j] = warp_reduce_sum(part[j]);
      if ((threadIdx.x & 31) == 0) s.red[threadIdx.x >> 5][j] = part[j];
    }
    __syncthreads();
    if (threadIdx.x < 1 + 2 * SAMP_CUTS) {
      float t = 0.f;
      for (int w = 0; w < SAMP_T / 32; w++) t += s.red[w][threadIdx.x];
      if (threadIdx.x <= SAMP_CUTS) s.xch[1].v[threadIdx.x] = t;
      else s.xch[1].n[threadIdx.x - 1 - SAMP_CUTS] = (uint32_t)t;
    }
    samp_meet<C>();
    if (threadIdx.x <= SAMP_CUTS) {
      float t = 0.f;
#pragma unroll
      for (int r = 0; r < C; r++) t += samp_peek<C>(&s.xch[1].v[threadIdx.x], r);
      s.all[1].v[threadIdx.x] = t;
    } else if (threadIdx.x < 1 + 2 * SAMP_CUTS) {
      uint32_t t = 0;
#pragma unroll
      for (int r = 0; r < C; r++) t += samp_peek<C>(&s.xch[1].n[threadIdx.x - 1 - SAMP_CUTS], r);
      s.all[1].n[threadIdx.x - 1 - SAMP_CUTS] = t;
    }
    __syncthreads();
    z = s.all[1].v[0];
#pragma unroll
    for (int j = 0; j < SAMP_CUTS; j++) { zc[j] = s.all[1].v[1 + j]; nc[j] = s.all[1].n[j]; }
  } else {
    for (int i = threadIdx.x; i < n; i += SAMP_T) e[i] = __expf((e[i] - best) * invT);
#pragma unroll
    for (int j = 0; j < SAMP_CUTS; j++) { zc[j] = 0.f; nc[j] = 0; }
    __syncthreads();
  }
  float mass = z;
  uint32_t thr_key = 0;                // keep elements with key >= thr_key

  uint32_t cut = 0, above = 0;         // the highest cut that holds enough, and how many elements reach it
#pragma unroll
  for (int j = SAMP_CUTS - 1; j >= 0; j--)
    if (by_rank ? nc[j] >= (uint32_t)k : pth < 1.f && zc[j] >= pth * mass * 1.001f) { cut = cuts[j]; above = nc[j]; }
  if (cut != 0 && above <= SAMP_BINS) {
    // everything that can be kept fits one block: no more meetings of the cluster
    samp_gather(e, n, first, cut, &s);
    samp_meet<C>();
    if (rank != 0) return;
    const int win = samp_finish(&s, (int)above, by_rank ? k : 0, pth, mp, mass, key, offset, bi);
    if (threadIdx.x == 0) out[b] = win;
    return;
  }
  if (by_rank) {
    if (threadIdx.x == 0) { s.prefix = 0; s.remaining = (samp_n)k; }
    __syncthreads();
    samp_pass<false, C, K>(e, n, &s, 0, 21, 11, 0x00000000u, cut, rank);
    samp_pass<false, C, K>(e, n, &s, 1, 10, 11, 0xFFE00000u, cut, rank);
    samp_pass<false, C, K>(e, n, &s, 2, 0, 10, 0xFFFFFC00u, cut, rank);
    thr_key = s.prefix;
    // mass of the kept set
    float mk = 0.f;
    for (int i = threadIdx.x; i < n; i += SAMP_T) {
      const float v = e[i];
      if (__float_as_uint(v) >= thr_key) mk += v;
    }
    mk = samp_block_sum(mk, s.sv);
    if (threadIdx.x == 0) s.xch[2].v[0] = mk;
    samp_meet<C>();
    if (threadIdx.x == 0) {
      mk = 0.f;
      for (int r = 0; r < C; r++) mk += samp_peek<C>(&s.xch[2].v[0], r);
      s.all[2].v[0] = mk;
    }
    __syncthreads();
    mass = s.all[2].v[0];
  }
  if (pth < 1.f && mass == mass) {
    cut = 0;                           // a margin for the order of the sums
#pragma unroll
    for (int j = SAMP_CUTS - 1; j >= 0; j--) if (zc[j] >= pth * mass * 1.001f) cut = cuts[j];
    if (thr_key > cut) cut = thr_key;
    if (threadIdx.x == 0) { s.prefix = 0; s.remaining = __float2ull_rn(pth * mass * SAMP_UNIT); }
    __syncthreads();
    bool found_it = false;
    if (cut != 0) {
      // between the cut and the maximum there are few enough values for bins of 64 or more to a factor of two: the one in question
      // holds so little that rank 0 sorts it
      constexpr uint32_t ONE = 0x3F800000u;
      int shift = 0;
      while ((ONE - cut) >> shift >= SAMP_BINS) shift++;
      samp_pass<true, C, K>(e, n, &s, 3, shift, 11, 0x00000000u, cut, rank, cut);
      const uint32_t low = cut + s.prefix;
      const samp_n rem = s.remaining;
      samp_gather(e, n, first, low, &s, low + (1u << shift) - 1);      // over rank 0's bins, which nobody reads any more
      samp_meet<C>();
      if (threadIdx.x == 0) s.all[3].n[0] = samp_peek<C>(&s.listed, 0);
      __syncthreads();
      const int listed = (int)s.all[3].n[0];
      if (listed > 0 && listed <= SAMP_BINS) {
        if (rank == 0) {
          samp_sort(&s, listed);
          samp_reach(&s, listed, 0u, [&](samp_n) { return rem; });
          // rounding can leave the bin's sum below what remains: its lowest element
          if (threadIdx.x == 0 && s.prefix == 0) s.prefix = (uint32_t)(s.hist[listed - 1] >> 32);
        }
        samp_meet<C>();
        if (threadIdx.x == 0) s.all[3].n[1] = samp_peek<C>(&s.prefix, 0);
        __syncthreads();
        if (s.all[3].n[1] > thr_key) thr_key = s.all[3].n[1];
        found_it = true;
      } else {
        if (threadIdx.x == 0) { s.prefix = 0; s.remaining = __float2ull_rn(pth * mass * SAMP_UNIT); }
        samp_meet<C>();                  // the number has been read
      }
    }
    if (!found_it) {
      samp_pass<true, C, K>(e, n, &s, 3, 21, 11, 0x00000000u, cut, rank);
      samp_pass<true, C, K>(e, n, &s, 4, 10, 11, 0xFFE00000u, cut, rank);
      samp_pass<true, C, K>(e, n, &s, 5, 0, 10, 0xFFFFFC00u, cut, rank);
      if (s.prefix > thr_key) thr_key = s.prefix;
    }
  }
  if (mp > 0.f) {
    const uint32_t tm = __float_as_uint(mp);  // max e is exactly 1
    if (tm > thr_key) thr_key = tm;
  }
  // ---- exponential race over the kept set
  float bestv = -INFINITY;
  int besti = bi;
  for (int i0 = threadIdx.x * 4; i0 < n; i0 += SAMP_T * 4) {     // slices start at multiples of four
    float v[4];
    bool any = false;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      v[j] = i0 + j < n ? e[i0 + j] : 0.f;
      any |= __float_as_uint(v[j]) >= thr_key && v[j] > 0.f;
    }
    if (!any) continue;
    const uint4 rnd = philox4x32(
        make_uint4((uint32_t)(first + i0), (uint32_t)offset, (uint32_t)((unsigned long long)offset >> 32), 0u), key);
    const uint32_t rr[4] = {rnd.x, rnd.y, rnd.z, rnd.w};
#pragma unroll
    for (int j = 0; j < 4; j++)
      if (__float_as_uint(v[j]) >= thr_key && v[j] > 0.f) {
        const float ex = -__logf(u32_to_unit(rr[j]));  // Exp(1)
        samp_better(bestv, besti, v[j] / fmaxf(ex, 1e-20f), first + i0 + j);
      }
  }
  samp_cluster_argmax(bestv, besti, &s, 3);
  if (rank == 0 && threadIdx.x == 0) out[b] = besti;
  samp_meet<C>();
}

// Rows of 16-byte aligned storage go eight elements at a time: 192 x 151936 81 us with single elements, 33 us so.
__global__ void __launch_bounds__(256) cast_bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ in, long ld_in,
                                                               float* __restrict__ out, long ld_out, int V) {
  const __nv_bfloat16* r = in + (long)blockIdx.y * ld_in;
  float* o = out + (long)blockIdx.y * ld_out;
  const int step = gridDim.x * blockDim.x, i0 = blockIdx.x * blockDim.x + threadIdx.x;
  int done = 0;
  if (((reinterpret_cast<uintptr_t>(r) | reinterpret_cast<uintptr_t>(o)) & 15) == 0) {
    for (int c = i0; c < V >> 3; c += step) {
      const uint4 q = reinterpret_cast<const uint4*>(r)[c];
      const float2 f0 = unpack_bf16x2(q.x), f1 = unpack_bf16x2(q.y), f2 = unpack_bf16x2(q.z), f3 = unpack_bf16x2(q.w);
      reinterpret_cast<float4*>(o)[2 * c] = make_float4(f0.x, f0.y, f1.x, f1.y);
      reinterpret_cast<float4*>(o)[2 * c + 1] = make_float4(f2.x, f2.y, f3.x, f3.y);
    }
    done = V & ~7;
  }
  for (int i = done + i0; i < V; i += step) o[i] = __bfloat162float(r[i]);
}

}  // namespace b200

using namespace b200;

// dtype: 0 = bf16, 1 = fp32.  out: int64 [B]
B200_API int b200_argmax(const void* logits, int dtype, long ld, int B, int V, void* out,
                         cudaStream_t stream) {
  if (B <= 0) return 0;
  if (dtype == 0)
    argmax_kernel<__nv_bfloat16><<<B, SAMP_THREADS, 0, stream>>>((const __nv_bfloat16*)logits, ld,
                                                                  V, (long*)out);
  else
    argmax_kernel<float><<<B, SAMP_THREADS, 0, stream>>>((const float*)logits, ld, V, (long*)out);
  return B200_CHECK_LAUNCH();
}

B200_API int b200_cast_bf16_f32(const void* in, long ld_in, void* out, long ld_out, int B, int V,
                                cudaStream_t stream) {
  if (B <= 0 || V <= 0) return 0;
  const unsigned blocks = (unsigned)((V + 8191) / 8192);             // 32 elements a thread
  for (int b0 = 0; b0 < B; b0 += 65535)                              // rows are the grid's y
    cast_bf16_to_f32_kernel<<<dim3(blocks, (unsigned)(B - b0 < 65535 ? B - b0 : 65535)), 256, 0, stream>>>(
        (const __nv_bfloat16*)in + (long)b0 * ld_in, ld_in, (float*)out + (long)b0 * ld_out, ld_out, V);
  return B200_CHECK_LAUNCH();
}

B200_API int b200_apply_penalties(void* logits, long ld, int B, int V, const void* prompt_ids,
                                  int Lp, const void* output_ids, int Lo, const void* rep,
                                  const void* freq, const void* pres, cudaStream_t stream) {
  if (B <= 0) return 0;
  const int words = (V + 31) / 32;
  const size_t smem = (size_t)2 * words * 4;
  static size_t smem_set = 0;
  if (smem > 48 * 1024 && smem > smem_set) {
    cudaError_t e = cudaFuncSetAttribute(penalties_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    smem_set = smem;
  }
  penalties_kernel<<<B, 512, smem, stream>>>((float*)logits, ld, V, (const long*)prompt_ids, Lp,
                                             (const long*)output_ids, Lo, (const float*)rep,
                                             (const float*)freq, (const float*)pres);
  return B200_CHECK_LAUNCH();
}

template <int C, int K>
static int launch_sample(float* logits, long ld, int B, int V, int slice, const float* temperature, const int* top_k,
                         const float* top_p, const float* min_p, const unsigned long long* seeds, const long* offsets,
                         long* out, cudaStream_t stream) {
  const int resident = slice <= SAMP_MAX_SLICE;
  cudaError_t e = allow_smem<sample_kernel<C, K>>((K == 1 ? SAMP_MAX_SLICE : SAMP_TWO_HIST_SLICE) * 4);
  if (e != cudaSuccess) return (int)e;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(SAMP_T);
  cfg.dynamicSmemBytes = resident ? (size_t)slice * 4 : 0;
  cfg.stream = stream;
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = C;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  for (int b0 = 0; b0 < B; b0 += 65535) {
    const int nb = B - b0 < 65535 ? B - b0 : 65535;
    cfg.gridDim = dim3(C, (unsigned)nb);
    e = cudaLaunchKernelEx(&cfg, sample_kernel<C, K>, logits + (long)b0 * ld, ld, V, slice, resident,
                           temperature ? temperature + b0 : nullptr, top_k ? top_k + b0 : nullptr, top_p ? top_p + b0 : nullptr,
                           min_p ? min_p + b0 : nullptr, seeds ? seeds + b0 : nullptr, offsets ? offsets + b0 : nullptr, out + b0);
    if (e != cudaSuccess) return (int)e;
  }
  return 0;
}

B200_API int b200_sample(void* logits_f32, long ld, int B, int V, const void* temperature,
                         const void* top_k, const void* top_p, const void* min_p,
                         const void* seeds, const void* offsets, void* out,
                         cudaStream_t stream) {
  if (B <= 0) return 0;
  // Blocks per row: as many as two per SM give every row (a row of 32000 on eight blocks, 192 rows: plain 56 us, top-p 72; on
  // two 37 and 49), but so few elements to a block that an SM holds two of them (on one 50 and 58); rows too long for that share
  // an SM with nobody, and clusters of four then leave no SM out (256 rows of 200000, eight blocks 1.2 times as long).
  auto slice = [&](int c) { return ((V + c - 1) / c + 3) / 4 * 4; };
  int c = 8;
  while (c > 1 && (long)B * c > 2l * num_sms() && slice(c / 2) <= SAMP_PAIR_SLICE) c /= 2;
  if (slice(8) > SAMP_PAIR_SLICE && slice(4) <= SAMP_MAX_SLICE && B * 8l > num_sms()) c = 4;
  auto* launch = c == 1 ? launch_sample<1, 1> : c == 2 ? launch_sample<2, 1> : c == 4 ? launch_sample<4, 1>
                 : slice(8) > SAMP_PAIR_SLICE && slice(8) <= SAMP_TWO_HIST_SLICE ? launch_sample<8, 2> : launch_sample<8, 1>;
  return launch((float*)logits_f32, ld, B, V, slice(c), (const float*)temperature, (const int*)top_k, (const float*)top_p,
                (const float*)min_p, (const unsigned long long*)seeds, (const long*)offsets, (long*)out, stream);
}
