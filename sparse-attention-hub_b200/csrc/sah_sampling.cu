// Sampling maskers (maskers/sampling/implementations/adaptive_sampling.py,
// utils/mask_attention_utils.py:105-184):
//   sah_adaptive_budget   per-row sample budget of the adaptive (epsilon, delta) masker
//   sah_sample_scatter    budgeted uniform draws scattered into a bitmap
//
// Random draws are a pure function of (seed, draw index): Philox4x32-10 with the
// counter (index, 0, 0, 0) and key (seed_lo, seed_hi); the first output word u gives the
// column  start + floor(u * n / 2^32).  A caller that wants the very same sample from
// another implementation regenerates or hands in the same draws.
#include "sah_common.cuh"

__host__ __device__ __forceinline__ uint32_t sah_mulhi32(uint32_t a, uint32_t b) {
  return (uint32_t)(((uint64_t)a * (uint64_t)b) >> 32);
}

__host__ __device__ __forceinline__ uint32_t sah_philox_u32(uint64_t seed, uint64_t index) {
  uint32_t c0 = (uint32_t)index, c1 = (uint32_t)(index >> 32), c2 = 0u, c3 = 0u;
  uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint32_t hi0 = sah_mulhi32(0xD2511F53u, c0), lo0 = 0xD2511F53u * c0;
    const uint32_t hi1 = sah_mulhi32(0xCD9E8D57u, c2), lo1 = 0xCD9E8D57u * c2;
    const uint32_t n0 = hi1 ^ c1 ^ k0, n1 = lo1, n2 = hi0 ^ c3 ^ k1, n3 = lo0;
    c0 = n0; c1 = n1; c2 = n2; c3 = n3;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
  return c0;
}

__device__ __forceinline__ int64_t sah_draw_column(uint64_t seed, uint64_t index, int64_t start,
                                                   int64_t n) {
  return start + (int64_t)sah_mulhi32(sah_philox_u32(seed, index), (uint32_t)n);
}

// Sum over the CTA in a fixed order: each thread already holds the sequential sum of its
// strided elements; lanes combine by xor shuffles (16, 8, 4, 2, 1), then the 32 warp sums
// combine the same way.  Every thread returns the same value.  blockDim.x must be 1024.
__device__ __forceinline__ float sah_block_sum_fixed(float v, float* scratch32) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch32[threadIdx.x >> 5] = v;
  __syncthreads();
  float w = scratch32[threadIdx.x & 31];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = __fadd_rn(w, __shfl_xor_sync(0xffffffffu, w, o));
  return w;
}

__device__ __forceinline__ float sah_block_max(float v, float* scratch32) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch32[threadIdx.x >> 5] = v;
  __syncthreads();
  float w = scratch32[threadIdx.x & 31];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
  return w;
}

template <typename T>
__device__ __forceinline__ float ad_exp(float x, const uint16_t* table);
template <>
__device__ __forceinline__ float ad_exp<__nv_bfloat16>(float x, const uint16_t* table) {
  return __uint_as_float(((uint32_t)table[__float_as_uint(x) >> 16]) << 16);
}
template <>
// fp32: the double-precision exponential rounded once, so that a CPU restatement using the
// same recipe reproduces the value (expf differs between libraries in the last place)
__device__ __forceinline__ float ad_exp<float>(float x, const uint16_t*) { return (float)exp((double)x); }

// Calls f(j) for the set bits j = threadIdx.x, threadIdx.x + 1024, ... below S of a bitmap, in that
// order (1024 threads).  A thread's bits are the same bit of every 32nd word, so 32 words of a warp
// are turned over (a 32 x 32 bit transposition, five exchanges) and each lane walks its own bits:
// testing word after word, every warp went through the body for nearly all of them.
#define AD_FEW 2  // words per warp up to which the bits are picked one by one
template <typename F>
__device__ __forceinline__ void ad_own_columns(const uint32_t* bits, int64_t S, F f) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = (S + 31) / 32;
  for (int64_t n0 = 0; n0 * 32 < words; n0 += 32) {  // words warp + 32 (n0 + lane)
    uint32_t m = 0u;
    if (words <= 32 * AD_FEW) {  // a few words per warp: every lane reads its own bit of each
#pragma unroll
      for (int i = 0; i < AD_FEW; ++i) {
        const int64_t w = warp + 32 * i;
        if (w * 32 + lane < S) m |= ((bits[w] >> lane) & 1u) << i;
      }
    } else {
      const int64_t w = warp + 32 * (n0 + lane);
      m = w < words ? bits[w] : 0u;
      if (w == words - 1 && (S & 31)) m &= (1u << (int)(S & 31)) - 1u;
#pragma unroll
      for (int o = 16, keep = 0x0000FFFF; o > 0; o >>= 1, keep ^= keep << o) {
        // exchange the off-diagonal blocks of size o
        const uint32_t other = __shfl_xor_sync(0xffffffffu, m, o);
        m = (lane & o) ? ((m & ~(uint32_t)keep) | ((other >> o) & (uint32_t)keep))
                       : ((m & (uint32_t)keep) | ((other << o) & ~(uint32_t)keep));
      }
    }
    while (m) {  // bit i: column lane of word warp + 32 (n0 + i)
      const int i = __ffs(m) - 1;
      m &= m - 1u;
      f((warp + 32 * (n0 + i)) * 32 + lane);
    }
  }
}

struct AdaptiveArgs {
  const void* scores;      // [rows][S] unscaled q.k in dtype
  float scaling;
  const void* bias;
  int64_t bias_s_b, bias_s_h, bias_s_q;
  const uint32_t* prev_bits;  // null: previous mask empty or full (plain sum over all keys)
  const void* prev_data;
  const int32_t* wpre;
  const int64_t* ptr;
  int Hq, Sq;
  int64_t S, W, start, end, nb;
  uint64_t seed;
  const int64_t* base_draws;  // optional [rows][nb] columns; null: Philox(seed, row * nb + i)
  const uint16_t* exp_table;
  float delta_ppf, epsilon;
  int64_t* budget;
  void* prob;
  float* stats;  // optional [rows][4]: static denominator, std, estimated denominator, budget^2
};

// bfloat16 weights: exp rounds to 1 for |d| < 2^-10 and to 0 from |d| = 128 on; the part of the
// table between (d negative) is kept in shared memory.
#define AD_D0 0xBA80  // bf16 bits of -2^-10
#define AD_D1 0xC300  // -128
#define AD_SMEM (200 * 1024)       // the base sample's bitmap, or that and the row
#define AD_ROW_BYTES (160 * 1024)  // logits of a bfloat16 row in shared memory: 81920 keys

// One CTA (1024 threads) per mask row.  Every tensor operation of the reference is one
// rounding to the dtype here; reductions use the fixed order above.
// RESIDENT (bfloat16): the scaled logits of the row are formed once, eight at a time, and stay in
// shared memory beside the table, because the sums visit scattered keys (the previous mask's, the
// sample's) one after the other: with a load of the score and a gather of the weight from global
// memory for each of them 128 rows x 65536 keys took 44.6 us, all of it latency; 19.3 us now.
// KEEP: draws per thread whose weights stay in registers between the two sums over the sample.
template <typename T, bool RESIDENT, int KEEP>
__global__ void __launch_bounds__(1024, RESIDENT ? 1 : 2)
adaptive_budget_kernel(AdaptiveArgs a) {
  sah_pdl_entry();
  extern __shared__ __align__(16) uint32_t ad_base_bits[];  // W words: distinct base-sample columns
  __shared__ float scratch[32];
  __shared__ uint16_t table_sm[RESIDENT ? AD_D1 - AD_D0 : 1];
  T* row_sm = reinterpret_cast<T*>(ad_base_bits + (a.W + 3) / 4 * 4);  // [W * 32] logits
  const int tid = threadIdx.x;
  const int64_t row = blockIdx.x;
  const int qi = (int)(row % a.Sq);
  const int64_t bh = row / a.Sq;
  const int h = (int)(bh % a.Hq);
  const int64_t b = bh / a.Hq;
  const T* s = reinterpret_cast<const T*>(a.scores) + row * a.S;
  const T* bias = a.bias ? reinterpret_cast<const T*>(a.bias) + b * a.bias_s_b + h * a.bias_s_h +
                               qi * a.bias_s_q
                         : nullptr;
  const int64_t n = a.end - a.start;

  auto make_logit = [&](int64_t j) {
    float t = sah_round_to<T>(__fmul_rn(sah_to_float<T>(s[j]), a.scaling));
    if (bias) t = sah_round_to<T>(__fadd_rn(t, sah_to_float<T>(bias[j])));
    return t;
  };
  for (int64_t w = tid; w < a.W; w += 1024) ad_base_bits[w] = 0u;

  // 1. row maximum over all keys
  float mx = -INFINITY;
  if constexpr (RESIDENT) {
    for (int i = tid; i < AD_D1 - AD_D0; i += 1024) table_sm[i] = a.exp_table[AD_D0 + i];
    const bool vec = (reinterpret_cast<uintptr_t>(s) & 15) == 0;
    const bool bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
    for (int64_t c0 = (int64_t)tid * 8; c0 < a.S; c0 += 1024 * 8) {
      if (vec && (bias == nullptr || bias_vec) && c0 + 8 <= a.S) {
        float f[8], bv[8];
        sah_load8<T>(s + c0, f);
        if (bias) sah_load8<T>(bias + c0, bv);
        __align__(16) T out[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          float t = sah_round_to<T>(__fmul_rn(f[i], a.scaling));
          if (bias) t = sah_round_to<T>(__fadd_rn(t, bv[i]));
          mx = fmaxf(mx, t);
          out[i] = sah_from_float<T>(t);
        }
        *reinterpret_cast<uint4*>(row_sm + c0) = *reinterpret_cast<const uint4*>(out);
      } else {
        for (int64_t j = c0; j < c0 + 8 && j < a.S; ++j) {
          const float t = make_logit(j);
          mx = fmaxf(mx, t);
          row_sm[j] = sah_from_float<T>(t);
        }
      }
    }
  } else {
    for (int64_t j = tid; j < a.S; j += 1024) mx = fmaxf(mx, make_logit(j));
  }
  mx = sah_block_max(mx, scratch);  // (its barriers also publish the logits and the table)
  auto expw = [&](int64_t j) {
    if constexpr (RESIDENT) {
      const float d = sah_round_to<T>(__fsub_rn(sah_to_float<T>(row_sm[j]), mx));
      const uint32_t b = __float_as_uint(d) >> 16;
      const uint32_t e = b - AD_D0 < AD_D1 - AD_D0 ? table_sm[b - AD_D0] : a.exp_table[b];
      return __uint_as_float(e << 16);
    } else {
      return ad_exp<T>(sah_round_to<T>(__fsub_rn(make_logit(j), mx)), a.exp_table);
    }
  };

  // 2. static denominator: exp weights of the previous mask under its inverse weights
  float part = 0.f;
  const float unit_w = sah_inv_weight<T>(1.f);
  const uint32_t* pb = a.prev_bits ? a.prev_bits + row * a.W : nullptr;
  if (pb == nullptr) {
    for (int64_t j = tid; j < a.S; j += 1024) part = __fadd_rn(part, expw(j));
  } else {
    // (the keys outside the mask would add +0)
    ad_own_columns(pb, a.S, [&](int64_t j) {
      float w = unit_w;  // unit weights still pass through 1 / (1 + 1e-6)
      if (a.prev_data != nullptr) {
        const uint32_t word = pb[j >> 5];
        const int bit = (int)(j & 31);
        const int64_t pos = a.ptr[row] + a.wpre[row * a.W + (j >> 5)] + __popc(word & ((1u << bit) - 1u));
        w = sah_inv_weight<T>(sah_to_float<T>(reinterpret_cast<const T*>(a.prev_data)[pos]));
      }
      part = __fadd_rn(part, sah_round_to<T>(__fmul_rn(expw(j), w)));
    });
  }
  const float static_den = sah_round_to<T>(sah_block_sum_fixed(part, scratch));

  // 3. base sample: unbiased standard deviation of the sampled exp weights
  auto base_col = [&](int64_t i) {
    return a.base_draws ? a.base_draws[row * a.nb + i]
                        : sah_draw_column(a.seed, (uint64_t)(row * a.nb + i), a.start, n);
  };
  // the weights of a thread's first draws are kept for the second sum
  float drawn[KEEP];
  part = 0.f;
#pragma unroll
  for (int n = 0; n < KEEP; ++n) {
    const int64_t i = tid + n * 1024;
    drawn[n] = 0.f;
    if (i < a.nb) {
      const int64_t c = base_col(i);
      atomicOr(&ad_base_bits[c >> 5], 1u << (c & 31));
      drawn[n] = expw(c);
      part = __fadd_rn(part, drawn[n]);
    }
  }
  for (int64_t i = tid + KEEP * 1024; i < a.nb; i += 1024) {
    const int64_t c = base_col(i);
    atomicOr(&ad_base_bits[c >> 5], 1u << (c & 31));
    part = __fadd_rn(part, expw(c));
  }
  const float mean = __fdiv_rn(sah_block_sum_fixed(part, scratch), (float)a.nb);
  part = 0.f;
#pragma unroll
  for (int n = 0; n < KEEP; ++n)
    if (tid + n * 1024 < a.nb) {
      const float d = __fsub_rn(drawn[n], mean);
      part = __fadd_rn(part, __fmul_rn(d, d));
    }
  for (int64_t i = tid + KEEP * 1024; i < a.nb; i += 1024) {
    const float d = __fsub_rn(expw(base_col(i)), mean);
    part = __fadd_rn(part, __fmul_rn(d, d));
  }
  const float var = __fdiv_rn(sah_block_sum_fixed(part, scratch), (float)(a.nb - 1));
  float sd = sah_round_to<T>(sqrtf(var));
  sd = fmaxf(sd, sah_round_to<T>(1e-8f));

  // 4. denominator estimate from the distinct base positions, weight 1 / (nb / n)
  const float p_base = sah_round_to<T>((float)((double)a.nb / (double)n));
  const float w_base = sah_inv_weight<T>(p_base);
  __syncthreads();
  part = 0.f;
  ad_own_columns(ad_base_bits, a.S,
                 [&](int64_t j) { part = __fadd_rn(part, sah_round_to<T>(__fmul_rn(expw(j), w_base))); });
  const float sampled_den = sah_round_to<T>(sah_block_sum_fixed(part, scratch));
  const float est_den = sah_round_to<T>(__fadd_rn(static_den, sampled_den));

  // 5. budget (adaptive_sampling.py:282-302, :394-397)
  if (tid == 0) {
    const float err = fmaxf(sah_round_to<T>(__fmul_rn(a.epsilon, est_den)), sah_round_to<T>(1e-8f));
    float num = sah_round_to<T>(__fmul_rn(a.delta_ppf, sd));
    num = sah_round_to<T>(__fmul_rn(num, (float)n));
    const float ratio = sah_round_to<T>(__fdiv_rn(num, err));
    float b2 = sah_round_to<T>(__fmul_rn(ratio, ratio));
    float clamped = fminf(fmaxf(b2, 1.0f), sah_round_to<T>((float)n));
    if (!(b2 == b2)) clamped = b2;  // NaN propagates as in the reference
    long long bud = (long long)clamped;  // truncation, as .long()
    if (bud < a.nb) bud = a.nb;
    if (bud > n) bud = n;
    a.budget[row] = bud;
    reinterpret_cast<T*>(a.prob)[row] = sah_from_float<T>(__fdiv_rn((float)bud, (float)n));
    if (a.stats) {
      a.stats[row * 4 + 0] = static_den;
      a.stats[row * 4 + 1] = sd;
      a.stats[row * 4 + 2] = est_den;
      a.stats[row * 4 + 3] = b2;
    }
  }
}

extern "C" int sah_adaptive_budget(const void* scores, int dtype, float scaling, const void* bias,
                                   int64_t bias_s_b, int64_t bias_s_h, int64_t bias_s_q,
                                   const uint32_t* prev_bits, const void* prev_data,
                                   const int32_t* wpre, const int64_t* ptr, int B, int Hq, int Sq,
                                   int64_t S, int64_t W, int64_t start, int64_t end, int64_t nb,
                                   uint64_t seed, const int64_t* base_draws,
                                   const uint16_t* exp_table, float delta_ppf, float epsilon,
                                   int64_t* budget, void* prob, float* stats, void* stream) {
  SAH_REQUIRE(scores && budget && prob, "adaptive_budget: null pointer");
  SAH_REQUIRE(B > 0 && Hq > 0 && Sq > 0 && S > 0 && W * 32 >= S, "adaptive_budget: bad extents");
  SAH_REQUIRE(0 <= start && start < end && end <= S && end - start >= 2 && nb >= 2,
              "adaptive_budget: bad sampling range");
  SAH_REQUIRE(end - start < (1ll << 32), "adaptive_budget: range too long");
  SAH_REQUIRE(prev_data == nullptr || (prev_bits && wpre && ptr), "adaptive_budget: data needs bits, wpre, ptr");
  SAH_REQUIRE(dtype != SAH_BF16 || exp_table != nullptr, "adaptive_budget: bf16 needs the exp table");
  AdaptiveArgs a;
  a.scores = scores; a.scaling = scaling; a.bias = bias;
  a.bias_s_b = bias_s_b; a.bias_s_h = bias_s_h; a.bias_s_q = bias_s_q;
  a.prev_bits = prev_bits; a.prev_data = prev_data; a.wpre = wpre; a.ptr = ptr;
  a.Hq = Hq; a.Sq = Sq; a.S = S; a.W = W; a.start = start; a.end = end; a.nb = nb;
  a.seed = seed; a.base_draws = base_draws; a.exp_table = exp_table;
  a.delta_ppf = delta_ppf; a.epsilon = epsilon; a.budget = budget; a.prob = prob; a.stats = stats;
  const size_t smem = (size_t)W * sizeof(uint32_t);
  if (smem > AD_SMEM)
    return sah_fail(SAH_ERR_UNSUPPORTED, "adaptive_budget: %lld keys per row exceed the base-sample bitmap",
                    (long long)S);
  const int64_t rows = (int64_t)B * Hq * Sq;
  cudaStream_t st = (cudaStream_t)stream;
  sah_prof_begin(SAH_PROF_ADAPTIVE, st);
#define AD_LAUNCH(RESIDENT, KEEP)                                                                           \
  do {                                                                                                      \
    if (bytes > 40 * 1024) {                                                                                \
      const cudaError_t e = cudaFuncSetAttribute(adaptive_budget_kernel<T, RESIDENT, KEEP>,                 \
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, AD_SMEM);     \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "adaptive_budget attr: %s", cudaGetErrorString(e)); \
    }                                                                                                       \
    sah_launch_chain(adaptive_budget_kernel<T, RESIDENT, KEEP>, (unsigned)rows, 1024, bytes, st, a);        \
  } while (0)
  SAH_DISPATCH_DTYPE(dtype, T, {
    // Bfloat16 rows that fit stay in shared memory, unless several of them can share an SM that would
    // hold one (from 149 rows on, up to 65536 keys: 256 x 8192 15.0 us resident, 12.9 us not; 256 x
    // 65536 even) or the table takes longer to copy than the row to read (below 2048 keys).  float32
    // weights come from a double-precision exponential, not from a table, and longer rows are read
    // again.
    const size_t row_bytes = (size_t)W * 32 * sizeof(T);
    const bool resident = sizeof(T) == 2 && row_bytes <= AD_ROW_BYTES && S >= 2048 && (rows <= 148 || S > 65536);
    constexpr bool RES = sizeof(T) == 2;
    const size_t bytes = resident ? (size_t)(W + 3) / 4 * 16 + row_bytes : smem;
    // one draw per thread (5 % of 20480 keys), or up to four kept (of 81920) and the others made again
    if (resident && nb <= 1024) AD_LAUNCH(RES, 1);
    else if (resident) AD_LAUNCH(RES, 4);
    else if (nb <= 1024) AD_LAUNCH(false, 1);
    else AD_LAUNCH(false, 4);
  });
#undef AD_LAUNCH
  SAH_LAUNCH_CHECK("adaptive_budget");
  sah_prof_end(SAH_PROF_ADAPTIVE, st);
  return SAH_OK;
}

// sample j (0 <= j < sptr[rows]) belongs to the row r with sptr[r] <= j < sptr[r+1] and is
// the column pool[j], or start + floor(philox(seed, j) * n / 2^32) without a pool
// (create_sampling_mask_with_per_head_budget, utils/mask_attention_utils.py:145-173).
__global__ void sample_scatter_kernel(const int64_t* __restrict__ sptr, int64_t rows,
                                      const int64_t* __restrict__ pool, uint64_t seed,
                                      int64_t start, int64_t n, int64_t S, int64_t W,
                                      uint32_t* __restrict__ bits) {
  sah_pdl_entry_early();
  const int64_t total = sptr[rows];
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total;
       j += (int64_t)gridDim.x * blockDim.x) {
    int64_t lo = 0, hi = rows;  // invariant: sptr[lo] <= j < sptr[hi]
    while (hi - lo > 1) {
      const int64_t mid = (lo + hi) >> 1;
      if (sptr[mid] <= j) lo = mid; else hi = mid;
    }
    const int64_t c = pool ? pool[j] : sah_draw_column(seed, (uint64_t)j, start, n);
    if (c >= 0 && c < S) atomicOr(bits + lo * W + (c >> 5), 1u << (c & 31));
  }
}

extern "C" int sah_sample_scatter(const int64_t* sptr, int64_t rows, const int64_t* pool,
                                  uint64_t seed, int64_t start, int64_t n, int64_t S, int64_t W,
                                  int sm_count, uint32_t* bits, void* stream) {
  SAH_REQUIRE(sptr && bits, "sample_scatter: null pointer");
  SAH_REQUIRE(rows >= 0 && n > 0 && n < (1ll << 32) && W * 32 >= S, "sample_scatter: bad extents");
  if (rows == 0) return SAH_OK;
  if (sm_count <= 0) sm_count = 148;
  sah_launch_chain(sample_scatter_kernel, (unsigned)(sm_count * 8), 256, 0, (cudaStream_t)stream, sptr, rows,
      pool, seed, start, n, S, W, bits);
  SAH_LAUNCH_CHECK("sample_scatter");
  return SAH_OK;
}
