// MagicPig: SimHash (LSH) sampling of keys (maskers/sampling/implementations/magic_pig.py).
//
//   sah_lsh_key_sums      per (batch, KV head, channel) sum of the keys in float64 (key mean, :152-183)
//   sah_lsh_key_stats     norm of every centred key and the running maximum norm (:348-353)
//   sah_lsh_key_sign      MIPS transform + random-hyperplane signatures of keys, packed per table (:332-372, :120-150)
//   sah_lsh_query         centred, normalised query, its signatures and its unit vector (:152-183, :332-403)
//   sah_lsh_match         keys that share at least one table code with the query (:455-463)
//   sah_lsh_prob          collision probability of every matched key (:374-403)
//
// Signatures are stored key-major: the L table codes of a key (uint8 for lsh_k <= 8, uint16 for
// lsh_k <= 16) sit side by side in a row padded to a multiple of 16 bytes, rows in key order,
// so that the match kernel reads one contiguous stream per (batch, KV head).  The reference
// repeats keys over the query heads of a group and uses one projection per layer, so the
// signatures of a group's heads are identical and are stored once per KV head.
//
// Reductions over the head dimension use one fixed order ("lane order"): lane t of a warp
// owns the D/32 consecutive channels starting at t*D/32 and sums them in ascending order,
// then the 32 lane sums combine by xor shuffles 16, 8, 4, 2, 1.  Every tensor operation of
// the reference is one rounding to the dtype here.
#include "sah_common.cuh"

#define LSH_MAX_PER_LANE 8  // D <= 256

// codes per signature row: L rounded up so that a row is a multiple of 16 bytes
template <typename CodeT>
__host__ __device__ __forceinline__ int lsh_row_pitch(int L) {
  const int per16 = 16 / (int)sizeof(CodeT);
  return (L + per16 - 1) / per16 * per16;
}

__device__ __forceinline__ float lsh_warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = __fadd_rn(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------------------
// key sums
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void lsh_key_sums_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h,
                                    int64_t ks_s, int Hkv, int64_t s0, int64_t s1, int D,
                                    int64_t chunk, double* __restrict__ sums) {
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / Hkv, h = bh % Hkv;
  const int64_t lo = s0 + (int64_t)blockIdx.x * chunk;
  const int64_t hi = lo + chunk < s1 ? lo + chunk : s1;
  const T* base = k + b * ks_b + h * ks_h;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    double acc = 0.0;
    int64_t s = lo;
    for (; s + 16 <= hi; s += 16) {  // sixteen rows in flight; one at a time took 111 us for 8 x 65500 keys
      T x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) x[i] = base[(s + i) * ks_s + d];
#pragma unroll
      for (int i = 0; i < 16; ++i) acc += (double)sah_to_float<T>(x[i]);
    }
    for (; s < hi; ++s) acc += (double)sah_to_float<T>(base[s * ks_s + d]);
    atomicAdd(&sums[bh * D + d], acc);
  }
}

extern "C" int sah_lsh_key_sums(const void* keys, int dtype, int64_t ks_b, int64_t ks_h,
                                int64_t ks_s, int B, int Hkv, int64_t s0, int64_t s1, int D,
                                double* sums, void* stream) {
  SAH_REQUIRE(keys && sums, "lsh_key_sums: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && D > 0 && s0 >= 0 && s1 >= s0, "lsh_key_sums: bad extents");
  if (s1 == s0) return SAH_OK;
  const int64_t chunk = 256;
  dim3 grid((unsigned)((s1 - s0 + chunk - 1) / chunk), (unsigned)(B * Hkv));
  SAH_DISPATCH_DTYPE(dtype, T, {
    lsh_key_sums_kernel<T><<<grid, 128, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hkv, s0, s1, D, chunk, sums);
  });
  SAH_LAUNCH_CHECK("lsh_key_sums");
  return SAH_OK;
}

// ---------------------------------------------------------------------------------------
// key statistics: norm of the centred key, running maximum
// ---------------------------------------------------------------------------------------
// lane `lane` loads its `per` consecutive channels of a row (one vector load when the row
// address allows it: rows of the usual 64 / 128 / 256 channels always do)
template <typename T>
__device__ __forceinline__ void lsh_load_lane(const T* row, int per, int lane, float* x) {
  const T* p = row + lane * per;
  const uintptr_t a = reinterpret_cast<uintptr_t>(p);
  if (sizeof(T) == 2 && per == 4 && (a & 7) == 0) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    x[0] = __uint_as_float(v.x << 16);
    x[1] = __uint_as_float(v.x & 0xffff0000u);
    x[2] = __uint_as_float(v.y << 16);
    x[3] = __uint_as_float(v.y & 0xffff0000u);
  } else if (sizeof(T) == 2 && per == 2 && (a & 3) == 0) {
    const uint32_t v = *reinterpret_cast<const uint32_t*>(p);
    x[0] = __uint_as_float(v << 16);
    x[1] = __uint_as_float(v & 0xffff0000u);
  } else if (sizeof(T) == 2 && per == 8 && (a & 15) == 0) {
    sah_unpack8(*reinterpret_cast<const uint4*>(p), x);
  } else if (sizeof(T) == 4 && per == 4 && (a & 15) == 0) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else {
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) x[t] = sah_to_float<T>(p[t]);
  }
}

template <typename T>
__global__ void lsh_key_stats_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h,
                                     int64_t ks_s, int Hkv, int64_t s0, int64_t s1, int D,
                                     const T* __restrict__ mean, int64_t cap,
                                     float* __restrict__ norms, unsigned int* __restrict__ max_bits) {
  sah_pdl_entry_early();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / Hkv, h = bh % Hkv;
  const int per = D / 32;
  float m[LSH_MAX_PER_LANE];
  if (mean) lsh_load_lane<T>(mean + bh * D, per, lane, m);
  float local_max = 0.f;
  for (int64_t s = s0 + (int64_t)blockIdx.x * nwarp + warp; s < s1; s += (int64_t)gridDim.x * nwarp) {
    float x[LSH_MAX_PER_LANE];
    lsh_load_lane<T>(k + b * ks_b + h * ks_h + s * ks_s, per, lane, x);
    float acc = 0.f;
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        const float c = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
        acc = __fadd_rn(acc, __fmul_rn(c, c));
      }
    const float nk = sah_round_to<T>(sqrtf(lsh_warp_sum(acc)));
    if (lane == 0) norms[bh * cap + s] = nk;
    local_max = fmaxf(local_max, nk);
  }
  if (lane == 0 && local_max > 0.f) atomicMax(max_bits, __float_as_uint(local_max));
}

// augmentation column of the MIPS transform: sqrt(M^2 - |k|^2) / M, rounded per operation
template <typename T>
__device__ __forceinline__ float lsh_augment(float nk, float M) {
  const float m2 = sah_round_to<T>(__fmul_rn(M, M));
  const float n2 = sah_round_to<T>(__fmul_rn(nk, nk));
  const float d = sah_round_to<T>(__fsub_rn(m2, n2));
  return sah_round_to<T>(__fdiv_rn(sah_round_to<T>(sqrtf(d)), M));
}

// ---------------------------------------------------------------------------------------
// key signatures
// ---------------------------------------------------------------------------------------
#define LSH_KT 64  // keys per CTA tile

// Hyperplane columns [c0, c0 + nc) of all Dp channels into shared memory [Dp][LSH_COLS], every
// copy requested before the first is waited for (no wait in here).
#define LSH_COLS 64
#define LSH_COLS_THREADS 128
#define LSH_QUERY_FOUR (4 * 148)
// the hyperplanes, a row of head dim + 1 and the signs: at most, for head dim 256
#define LSH_COLS_SMEM(T) (257 * (LSH_COLS * (int)sizeof(T) + 4) + LSH_COLS)
// Tables per CTA: as many as fit, but if rows of hyperplanes start on 16 bytes no more than leave
// every CTA's columns starting there too (10 bits per table in bfloat16: four tables, not six).
template <typename T>
static int lsh_cta_tables(int K, int L) {
  constexpr int PER = 16 / (int)sizeof(T);
  const int most = LSH_COLS / K;
  if ((L * K) % PER == 0)
    for (int t = most; t > 0; --t)
      if (t * K % PER == 0) return t;
  return most;
}
template <typename T>
__device__ __forceinline__ void lsh_stage_columns(const T* __restrict__ proj, int nbits, int Dp, int c0, int nc,
                                                  T* __restrict__ sm) {
  constexpr int PER = 16 / (int)sizeof(T);
  if ((reinterpret_cast<uintptr_t>(proj) & 15) == 0 && nbits % PER == 0 && c0 % PER == 0 && nc % PER == 0) {
    const int cpr = nc / PER;
    for (int i = threadIdx.x; i < Dp * cpr; i += LSH_COLS_THREADS) {
      const int ch = i / cpr, c = (i - ch * cpr) * PER;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                       (uint32_t)__cvta_generic_to_shared(sm + ch * LSH_COLS + c)),
                   "l"(proj + (int64_t)ch * nbits + c0 + c)
                   : "memory");
    }
  } else {
#pragma unroll 8
    for (int i = threadIdx.x; i < Dp * nc; i += LSH_COLS_THREADS) {
      const int ch = i / nc, c = i - ch * nc;
      sm[ch * LSH_COLS + c] = proj[(int64_t)ch * nbits + c0 + c];
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// The keys that a decode step appends: a CTA takes one key and LSH_COLS / K tables, so that the
// hyperplanes (155 KB for 75 tables of 8 bits) are fetched by many SMs at once and every value is
// on its way before the first is used; then one thread per column adds up the channels in order.
// Latency is all there is: 8 heads x 1 key took 25 us with one CTA per head, 4.5 us now.
#define LSH_FEW_KEYS 4
template <typename T, typename CodeT>
__global__ void __launch_bounds__(LSH_COLS_THREADS)
lsh_key_sign_few_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv,
                        int64_t s0, int D, const T* __restrict__ mean, const float* __restrict__ norms,
                        const unsigned int* __restrict__ max_bits, const T* __restrict__ proj, int L, int K,
                        int tables, int64_t cap, CodeT* __restrict__ codes) {
  sah_pdl_entry_early();
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  const int nbits = L * K, Dp = D + 1;
  T* pr = reinterpret_cast<T*>(lsh_smem);                                         // [Dp][LSH_COLS]
  float* xt = reinterpret_cast<float*>(lsh_smem + (size_t)Dp * LSH_COLS * sizeof(T));  // [Dp]
  unsigned char* sb = reinterpret_cast<unsigned char*>(xt + Dp);                  // [LSH_COLS]
  const int l0 = blockIdx.x * tables;
  const int lt = L - l0 < tables ? L - l0 : tables;
  lsh_stage_columns<T>(proj, nbits, Dp, l0 * K, lt * K, pr);
  const int64_t bh = blockIdx.y, s = s0 + blockIdx.z;
  const T* kr = k + bh / Hkv * ks_b + bh % Hkv * ks_h + s * ks_s;
  const float M = __uint_as_float(*max_bits);
  for (int c = threadIdx.x; c < D; c += LSH_COLS_THREADS) {
    const float x = sah_to_float<T>(kr[c]);
    const float cx = mean ? sah_round_to<T>(__fsub_rn(x, sah_to_float<T>(mean[bh * D + c]))) : x;
    xt[c] = sah_round_to<T>(__fdiv_rn(cx, M));
  }
  if (threadIdx.x == 0) xt[D] = lsh_augment<T>(norms[bh * cap + s], M);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  if (threadIdx.x < lt * K) {
    float acc = 0.f;
#pragma unroll 8
    for (int c = 0; c < Dp; ++c)
      acc = __fadd_rn(acc, __fmul_rn(xt[c], sah_to_float<T>(pr[c * LSH_COLS + threadIdx.x])));
    sb[threadIdx.x] = acc > 0.f ? 1 : 0;
  }
  __syncthreads();
  // bit j of table l is column l * K + j; the last CTA also writes the zero padding of the row
  const int LP = lsh_row_pitch<CodeT>(L);
  const int end = blockIdx.x == gridDim.x - 1 ? LP : l0 + lt;
  for (int l = l0 + threadIdx.x; l < end; l += LSH_COLS_THREADS) {
    unsigned int code = 0;
    if (l < L)
      for (int j = 0; j < K; ++j) code |= (unsigned int)sb[(l - l0) * K + j] << j;
    codes[(bh * cap + s) * LP + l] = (CodeT)code;
  }
}

template <typename T, typename CodeT>
__global__ void __launch_bounds__(256)
lsh_key_sign_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv,
                    int64_t s0, int64_t s1, int D, const T* __restrict__ mean,
                    const float* __restrict__ norms, const unsigned int* __restrict__ max_bits,
                    const T* __restrict__ proj, int L, int K, int64_t cap,
                    CodeT* __restrict__ codes) {
  sah_pdl_entry_early();
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  const int nbits = L * K;
  const int Dp = D + 1;
  float* xt = reinterpret_cast<float*>(lsh_smem);                       // [Dp][LSH_KT] transformed keys
  unsigned char* sb = lsh_smem + (size_t)Dp * LSH_KT * sizeof(float);   // [LSH_KT][nbits] sign bits
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / Hkv, h = bh % Hkv;
  const int64_t t0 = s0 + (int64_t)blockIdx.x * LSH_KT;
  const int per = D / 32;
  const float M = __uint_as_float(*max_bits);

  float m[LSH_MAX_PER_LANE];
  if (mean) lsh_load_lane<T>(mean + bh * D, per, lane, m);
  for (int kk = warp; kk < LSH_KT; kk += 8) {
    const int64_t s = t0 + kk;
    float x[LSH_MAX_PER_LANE];
    if (s < s1) lsh_load_lane<T>(k + b * ks_b + h * ks_h + s * ks_s, per, lane, x);
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        float v = 0.f;
        if (s < s1) {
          const float c = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
          v = sah_round_to<T>(__fdiv_rn(c, M));
        }
        xt[(lane * per + t) * LSH_KT + kk] = v;
      }
    if (lane == 0) xt[D * LSH_KT + kk] = s < s1 ? lsh_augment<T>(norms[bh * cap + s], M) : 0.f;
  }
  __syncthreads();

  // one output column per thread, 8 keys at a time; single accumulator per (key, column),
  // channels ascending (products of dtype values, added in float)
  // keys of this tile that exist
  const int kt_used = (int)((s1 - t0 < LSH_KT ? s1 - t0 : LSH_KT) + 7) & ~7;
  for (int o = threadIdx.x; o < nbits; o += 256) {
    for (int k8 = 0; k8 < kt_used; k8 += 8) {
      float acc[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[j] = 0.f;
      // unrolled by eight, the loads of as many channels are on their way (left to itself the loop
      // took 416 us for 64 heads x 4096 keys of 16 tables of 2 bits, 352 us this way)
#pragma unroll 8
      for (int c = 0; c < Dp; ++c) {
        const float p = sah_to_float<T>(proj[(int64_t)c * nbits + o]);
        const float4 a = *reinterpret_cast<const float4*>(xt + c * LSH_KT + k8);
        const float4 bq = *reinterpret_cast<const float4*>(xt + c * LSH_KT + k8 + 4);
        acc[0] = __fadd_rn(acc[0], __fmul_rn(a.x, p));
        acc[1] = __fadd_rn(acc[1], __fmul_rn(a.y, p));
        acc[2] = __fadd_rn(acc[2], __fmul_rn(a.z, p));
        acc[3] = __fadd_rn(acc[3], __fmul_rn(a.w, p));
        acc[4] = __fadd_rn(acc[4], __fmul_rn(bq.x, p));
        acc[5] = __fadd_rn(acc[5], __fmul_rn(bq.y, p));
        acc[6] = __fadd_rn(acc[6], __fmul_rn(bq.z, p));
        acc[7] = __fadd_rn(acc[7], __fmul_rn(bq.w, p));
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) sb[(k8 + j) * nbits + o] = acc[j] > 0.f ? 1 : 0;
    }
  }
  __syncthreads();
  // pack: bit j of table l is column l*K + j (magic_pig.py:120-150); the row of a key holds
  // its L codes and zero padding up to the row pitch
  const int LP = lsh_row_pitch<CodeT>(L);
  for (int i = threadIdx.x; i < LP * kt_used; i += 256) {
    const int kk = i / LP, l = i % LP;
    const int64_t s = t0 + kk;
    if (s >= s1) continue;
    unsigned int code = 0;
    if (l < L)
      for (int j = 0; j < K; ++j) code |= (unsigned int)sb[kk * nbits + l * K + j] << j;
    codes[(bh * cap + s) * LP + l] = (CodeT)code;
  }
}

extern "C" int sah_lsh_key_sign(const void* keys, int dtype, int64_t ks_b, int64_t ks_h,
                                int64_t ks_s, int B, int Hkv, int64_t s0, int64_t s1, int D,
                                const void* mean, const float* norms,
                                const unsigned int* max_norm_bits, const void* proj, int L, int K,
                                int64_t cap, void* codes, void* stream) {
  SAH_REQUIRE(keys && norms && max_norm_bits && proj && codes, "lsh_key_sign: null pointer");
  SAH_REQUIRE(D % 32 == 0 && D <= 32 * LSH_MAX_PER_LANE, "lsh_key_sign: head_dim must be a multiple of 32, <= 256");
  SAH_REQUIRE(L > 0 && K > 0, "lsh_key_sign: bad table shape");
  if (K > 16) return sah_fail(SAH_ERR_UNSUPPORTED, "lsh: lsh_k = %d > 16 bits per table is not built", K);
  SAH_REQUIRE(s0 >= 0 && s1 >= s0 && s1 <= cap, "lsh_key_sign: bad key range");
  if (s1 == s0) return SAH_OK;
  const size_t smem = (size_t)(D + 1) * LSH_KT * sizeof(float) + (size_t)LSH_KT * L * K;
  if (smem > 200 * 1024)
    return sah_fail(SAH_ERR_UNSUPPORTED, "lsh_key_sign: %d x %d signature bits exceed shared memory", L, K);
  dim3 grid((unsigned)((s1 - s0 + LSH_KT - 1) / LSH_KT), (unsigned)(B * Hkv));
  cudaStream_t st = (cudaStream_t)stream;
  if (s1 - s0 <= LSH_FEW_KEYS) {
#define LSH_FEW_LAUNCH(T, CodeT)                                                                   \
  do {                                                                                             \
    const int tables = lsh_cta_tables<T>(K, L);                                                    \
    const dim3 fgrid((unsigned)((L + tables - 1) / tables), (unsigned)(B * Hkv), (unsigned)(s1 - s0)); \
    const int bytes = (D + 1) * (LSH_COLS * (int)sizeof(T) + 4) + LSH_COLS;                        \
    if (bytes > 48 * 1024) {                                                                       \
      cudaError_t e = cudaFuncSetAttribute(lsh_key_sign_few_kernel<T, CodeT>,                      \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, LSH_COLS_SMEM(T)); \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_key_sign attr: %s", cudaGetErrorString(e)); \
    }                                                                                              \
    sah_launch_chain(lsh_key_sign_few_kernel<T, CodeT>, fgrid, LSH_COLS_THREADS, bytes, st, \
        reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hkv, s0, D,                            \
        reinterpret_cast<const T*>(mean), norms, max_norm_bits, reinterpret_cast<const T*>(proj),  \
        L, K, tables, cap, reinterpret_cast<CodeT*>(codes));                                       \
  } while (0)
    SAH_DISPATCH_DTYPE(dtype, T, {
      if (K <= 8) LSH_FEW_LAUNCH(T, uint8_t); else LSH_FEW_LAUNCH(T, uint16_t);
    });
#undef LSH_FEW_LAUNCH
    SAH_LAUNCH_CHECK("lsh_key_sign_few");
    return SAH_OK;
  }
#define LSH_SIGN_LAUNCH(T, CodeT)                                                                  \
  do {                                                                                             \
    cudaError_t e = cudaFuncSetAttribute(lsh_key_sign_kernel<T, CodeT>,                            \
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); \
    if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_key_sign attr: %s", cudaGetErrorString(e)); \
    sah_launch_chain(lsh_key_sign_kernel<T, CodeT>, grid, 256, smem, st, \
        reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hkv, s0, s1, D,                        \
        reinterpret_cast<const T*>(mean), norms, max_norm_bits, reinterpret_cast<const T*>(proj),  \
        L, K, cap, reinterpret_cast<CodeT*>(codes));                                               \
  } while (0)
  SAH_DISPATCH_DTYPE(dtype, T, {
    if (K <= 8) LSH_SIGN_LAUNCH(T, uint8_t); else LSH_SIGN_LAUNCH(T, uint16_t);
  });
  SAH_LAUNCH_CHECK("lsh_key_sign");
  return SAH_OK;
}

#include "sah_lsh_tc.cuh"

// Workspace of sah_lsh_key_sign_tc: two status words (entries appended to the list; error word
// of the bounded waits), padding to 16 bytes, then the list of 32-column groups to redo.
extern "C" int64_t sah_lsh_key_sign_tc_ws_bytes(int B, int Hkv, int64_t n_keys) {
  if (B <= 0 || Hkv <= 0 || n_keys <= 0) return 0;
  const int64_t rows = (int64_t)B * Hkv * n_keys;
  return 16 + (rows / 4 + 4096) * (int64_t)sizeof(LtcUncertain);
}

extern "C" int sah_lsh_key_sign_tc(const void* keys, int64_t ks_b, int64_t ks_h, int64_t ks_s, int B,
                                   int Hkv, int64_t s0, int64_t s1, int D, const void* mean,
                                   const float* norms, const unsigned int* max_norm_bits,
                                   const void* proj, int L, int K, int64_t cap, void* codes,
                                   void* workspace, int64_t workspace_bytes, int sm_count, void* stream) {
  SAH_REQUIRE(keys && norms && max_norm_bits && proj && codes && workspace, "lsh_key_sign_tc: null pointer");
  if (D != 128 || K != 8)
    return sah_fail(SAH_ERR_UNSUPPORTED, "lsh_key_sign_tc: head dim 128 and 8 bits per table (got %d, %d)", D, K);
  SAH_REQUIRE(L > 0 && s0 >= 0 && s1 >= s0 && s1 <= cap, "lsh_key_sign_tc: bad extents");
  SAH_REQUIRE((ks_s * 2) % 16 == 0 && (ks_h * 2) % 16 == 0 && (ks_b * 2) % 16 == 0 && ((uintptr_t)keys % 16) == 0 &&
                  (mean == nullptr || ((uintptr_t)mean % 16) == 0) && ((uintptr_t)codes % 16) == 0 &&
                  ((uintptr_t)workspace % 16) == 0,
              "lsh_key_sign_tc: rows must be 16-byte aligned");
  if (s1 == s0) return SAH_OK;
  const int64_t need = sah_lsh_key_sign_tc_ws_bytes(B, Hkv, s1 - s0);
  if (workspace_bytes < need)
    return sah_fail(SAH_ERR_WORKSPACE, "lsh_key_sign_tc: workspace of %lld bytes, need %lld",
                    (long long)workspace_bytes, (long long)need);
  cudaStream_t st = (cudaStream_t)stream;
  int* status = reinterpret_cast<int*>(workspace);
  LtcUncertain* list = reinterpret_cast<LtcUncertain*>(reinterpret_cast<unsigned char*>(workspace) + 16);
  int64_t entries = (workspace_bytes - 16) / (int64_t)sizeof(LtcUncertain);
  if (entries > (1ll << 30)) entries = 1ll << 30;
  // A long list leaves its end to the hyperplanes, one by one: a column of `proj` is a sector per
  // channel (88 thousand entries 102 -> 51 us).  It holds a quarter of the keys and takes up to a sixth.
  const int64_t plane_entries = (int64_t)L * 8 * LTC_PLANE * 2 / (int64_t)sizeof(LtcUncertain);
  __nv_bfloat16* planes = nullptr;
  if (entries >= 8 * plane_entries) {
    entries -= plane_entries;
    planes = reinterpret_cast<__nv_bfloat16*>(list + entries);
  }
  const int list_cap = (int)entries;
  cudaError_t e = cudaMemsetAsync(status, 0, 16, st);
  if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_key_sign_tc memset: %s", cudaGetErrorString(e));
  static bool allowed[2][64] = {};
  e = sah_allow_smem(lsh_key_sign_tc_kernel, LtcCfg::SMEM, allowed[0]);
  if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_key_sign_tc attr: %s", cudaGetErrorString(e));
  e = sah_allow_smem(lsh_sign_recheck_kernel, LTC_RC_SMEM, allowed[1]);
  if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_sign_recheck attr: %s", cudaGetErrorString(e));
  if (sm_count <= 0) sm_count = 148;
  // chunks of equal width: every CTA transforms as many keys and reads as many columns
  int chunks = (L * 8 + LTC_NCHUNK - 1) / LTC_NCHUNK;
  const int chunk_cols = ((L * 8 + chunks - 1) / chunks + 31) / 32 * 32;
  chunks = (L * 8 + chunk_cols - 1) / chunk_cols;
  const int64_t BH = (int64_t)B * Hkv;
  const int64_t tiles = BH * ((s1 - s0 + LTC_TILE - 1) / LTC_TILE);
  int64_t workers = sm_count / chunks;
  if (workers < 1) workers = 1;
  if (workers > tiles) workers = tiles;
  dim3 grid((unsigned)workers, (unsigned)chunks);
  lsh_key_sign_tc_kernel<<<grid, LTC_THREADS, LtcCfg::SMEM, st>>>(
      reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hkv, BH, s0, s1,
      reinterpret_cast<const __nv_bfloat16*>(mean), norms, max_norm_bits, reinterpret_cast<const __nv_bfloat16*>(proj),
      L, chunk_cols, cap, reinterpret_cast<uint8_t*>(codes), list, list_cap, status, status + 1, planes);
  SAH_LAUNCH_CHECK("lsh_key_sign_tc");
  lsh_sign_recheck_kernel<<<(unsigned)(sm_count * 3), LTC_RC_WARPS * 32, LTC_RC_SMEM, st>>>(
      reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hkv, reinterpret_cast<const __nv_bfloat16*>(mean),
      norms, max_norm_bits, reinterpret_cast<const __nv_bfloat16*>(proj), L, cap, reinterpret_cast<uint8_t*>(codes),
      list, list_cap, status, planes);
  SAH_LAUNCH_CHECK("lsh_sign_recheck");
  return SAH_OK;
}

// ---------------------------------------------------------------------------------------
// query: centre, normalise, signatures, unit vector
// ---------------------------------------------------------------------------------------
// A CTA takes one query row and up to LSH_COLS / K tables: the hyperplanes are requested at once, the
// first warp normalises the query meanwhile (every CTA of the row does; the first one writes it
// out), then one thread per column adds up the channels in order.  This kernel sits on the
// critical path of every decode step and is all latency: 32 rows took 12.5 us with one CTA per
// row, 7.7 us now.  Where that makes more CTAs than an SM holds at once, the hyperplanes' way from L2
// takes the time, and a CTA takes four rows, a warp normalising each: 512 rows x 75 tables of 8 bits
// in float32 22.0 us with one CTA per row, 30.6 us with ROWS = 1, 14.4 us with 4 (bfloat16 25.2, 22.3,
// 13.3).
template <typename T, typename CodeT, int ROWS>
__global__ void __launch_bounds__(LSH_COLS_THREADS)
lsh_query_kernel(const T* __restrict__ q, int64_t qs_b, int64_t qs_h, int64_t qs_q, int Hq, int Sq,
                 int G, int D, const T* __restrict__ mean, const T* __restrict__ proj, int L, int K,
                 int tables, int64_t rows, CodeT* __restrict__ qcodes, float* __restrict__ qunit, T* __restrict__ qhat,
                 float* __restrict__ qmu) {
  sah_pdl_entry_early();
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  const int nbits = L * K, Dp = D + 1;
  T* pr = reinterpret_cast<T*>(lsh_smem);                                         // [Dp][LSH_COLS]
  float* qn_sm = reinterpret_cast<float*>(lsh_smem + (size_t)Dp * LSH_COLS * sizeof(T));  // [ROWS][D] normalised
  unsigned char* sb = reinterpret_cast<unsigned char*>(qn_sm + ROWS * D);         // [ROWS][LSH_COLS]
  const int l0 = blockIdx.y * tables;
  const int lt = L - l0 < tables ? L - l0 : tables;
  lsh_stage_columns<T>(proj, nbits, Dp, l0 * K, lt * K, pr);
  const bool writer = blockIdx.y == 0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t row0 = (int64_t)blockIdx.x * ROWS, row = row0 + warp;  // the row of this warp, if it has one
  const int per = D / 32;
  if (warp < ROWS && row < rows) {
    const int qi = (int)(row % Sq);
    const int64_t bh = row / Sq;
    const int h = (int)(bh % Hq);
    const int64_t b = bh / Hq;
    float* qn = qn_sm + warp * D;
    float x[LSH_MAX_PER_LANE], m[LSH_MAX_PER_LANE], c[LSH_MAX_PER_LANE];
    lsh_load_lane<T>(q + b * qs_b + h * qs_h + qi * qs_q, per, lane, x);
    if (mean) lsh_load_lane<T>(mean + (b * (Hq / G) + h / G) * D, per, lane, m);
    float acc = 0.f;
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        c[t] = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
        acc = __fadd_rn(acc, __fmul_rn(c[t], c[t]));
      }
    // q / (|q| + 1e-8)
    const float nq = sah_round_to<T>(sqrtf(lsh_warp_sum(acc)));
    const float den = sah_round_to<T>(__fadd_rn(nq, 1e-8f));
    acc = 0.f;
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        c[t] = sah_round_to<T>(__fdiv_rn(c[t], den));
        qn[lane * per + t] = c[t];
        acc = __fadd_rn(acc, __fmul_rn(c[t], c[t]));
      }
    // unit vector of the transformed query (its extra column is zero): qn / (|qn| + 1e-8)
    const float n2 = sah_round_to<T>(sqrtf(lsh_warp_sum(acc)));
    const float den2 = sah_round_to<T>(__fadd_rn(n2, 1e-8f));
    float mu = 0.f;
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        const float u = sah_round_to<T>(__fdiv_rn(c[t], den2));
        if (writer) qunit[row * D + lane * per + t] = u;
        if (writer && qhat != nullptr) qhat[row * D + lane * per + t] = sah_from_float<T>(u);  // exact
        if (mean) mu = __fmaf_rn(u, m[t], mu);
      }
    // unit query . key mean, the query-side constant of the centred cosine
    mu = lsh_warp_sum(mu);
    if (writer && qmu != nullptr && lane == 0) qmu[row] = mu;
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  // one accumulator per row and column, channels ascending, as everywhere; with four rows, two each
  constexpr int PER = ROWS == 1 ? 1 : ROWS * LSH_COLS / LSH_COLS_THREADS;
  const int col = ROWS == 1 ? threadIdx.x : threadIdx.x % LSH_COLS;
  const int r0 = ROWS == 1 ? 0 : threadIdx.x / LSH_COLS * PER;
  if (col < lt * K) {
    float acc[PER];
#pragma unroll
    for (int r = 0; r < PER; ++r) acc[r] = 0.f;
#pragma unroll 8
    for (int c = 0; c < D; ++c) {
      const float p = sah_to_float<T>(pr[c * LSH_COLS + col]);
#pragma unroll
      for (int r = 0; r < PER; ++r) acc[r] = __fadd_rn(acc[r], __fmul_rn(qn_sm[(r0 + r) * D + c], p));
    }
    const float last = __fmul_rn(0.f, sah_to_float<T>(pr[D * LSH_COLS + col]));
#pragma unroll
    for (int r = 0; r < PER; ++r) sb[(r0 + r) * LSH_COLS + col] = __fadd_rn(acc[r], last) > 0.f ? 1 : 0;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ROWS * lt; i += LSH_COLS_THREADS) {
    const int r = ROWS == 1 ? 0 : i / lt, l = i - r * lt;
    if (row0 + r >= rows) break;
    unsigned int code = 0;
    for (int j = 0; j < K; ++j) code |= (unsigned int)sb[r * LSH_COLS + l * K + j] << j;
    qcodes[(row0 + r) * L + l0 + l] = (CodeT)code;
  }
}

extern "C" int sah_lsh_query(const void* q, int dtype, int64_t qs_b, int64_t qs_h, int64_t qs_q,
                             int B, int Hq, int Sq, int G, int D, const void* mean,
                             const void* proj, int L, int K, void* qcodes, float* qunit,
                             void* qhat, float* qmu, void* stream) {
  SAH_REQUIRE(q && proj && qcodes && qunit, "lsh_query: null pointer");
  SAH_REQUIRE(D % 32 == 0 && D <= 32 * LSH_MAX_PER_LANE, "lsh_query: head_dim must be a multiple of 32, <= 256");
  SAH_REQUIRE(G > 0 && Hq % G == 0 && L > 0 && K > 0, "lsh_query: bad shape");
  if (K > 16) return sah_fail(SAH_ERR_UNSUPPORTED, "lsh: lsh_k = %d > 16 bits per table is not built", K);
  const size_t smem = (size_t)D * sizeof(float) + (size_t)L * K;
  if (smem > 48 * 1024)
    return sah_fail(SAH_ERR_UNSUPPORTED, "lsh_query: %d x %d signature bits exceed shared memory", L, K);
  const int64_t rows = (int64_t)B * Hq * Sq;
  cudaStream_t st = (cudaStream_t)stream;
#define LSH_QUERY_LAUNCH(T, CodeT, ROWS)                                                           \
  do {                                                                                             \
    const dim3 grid((unsigned)((rows + ROWS - 1) / ROWS), (unsigned)chunks);                       \
    const int bytes = (D + 1) * LSH_COLS * (int)sizeof(T) + ROWS * (D * 4 + LSH_COLS);             \
    if (bytes > 48 * 1024) {                                                                       \
      cudaError_t e = cudaFuncSetAttribute(lsh_query_kernel<T, CodeT, ROWS>,                             \
                                           cudaFuncAttributeMaxDynamicSharedMemorySize, LSH_COLS_SMEM(T) + ROWS * (256 * 4 + LSH_COLS)); \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_query attr: %s", cudaGetErrorString(e)); \
    }                                                                                              \
    sah_launch_chain(lsh_query_kernel<T, CodeT, ROWS>, grid, LSH_COLS_THREADS, bytes, st, \
        reinterpret_cast<const T*>(q), qs_b, qs_h, qs_q, Hq, Sq, G, D,                             \
        reinterpret_cast<const T*>(mean), reinterpret_cast<const T*>(proj), L, K, tables, rows,    \
        reinterpret_cast<CodeT*>(qcodes), qunit, reinterpret_cast<T*>(qhat), qmu);                 \
  } while (0)
  SAH_DISPATCH_DTYPE(dtype, T, {
    const int tables = lsh_cta_tables<T>(K, L), chunks = (L + tables - 1) / tables;
    // four rows per CTA from four CTAs per SM on
    const bool four = rows * chunks > LSH_QUERY_FOUR;
    if (K <= 8 && four) LSH_QUERY_LAUNCH(T, uint8_t, 4);
    else if (K <= 8) LSH_QUERY_LAUNCH(T, uint8_t, 1);
    else if (four) LSH_QUERY_LAUNCH(T, uint16_t, 4);
    else LSH_QUERY_LAUNCH(T, uint16_t, 1);
  });
#undef LSH_QUERY_LAUNCH
  SAH_LAUNCH_CHECK("lsh_query");
  return SAH_OK;
}

// ---------------------------------------------------------------------------------------
// match: any table code equal
// ---------------------------------------------------------------------------------------
// One thread per key: it loads the key's signature row (a few 16-byte loads, all requested
// before the first compare) and tests it against the signature rows of the group's queries,
// which sit in shared memory padded with a value no key row holds in its padding.  "Some
// table code equal" is "some byte (halfword) of key XOR query is zero": with x = key ^ query,
// (x - 0x01..01) & ~x & 0x80..80 is non-zero exactly when x has a zero byte (a borrow can only
// start at a zero byte, so the test of the whole word is exact even though single positions
// above a zero byte are not), three integer instructions per word and query row.  A warp
// covers 32 consecutive keys, so a ballot of the result is the bitmap word of those keys;
// every warp does four such words and writes them side by side.
#define LSH_MATCH_WARPS 8
#define LSH_MATCH_WORDS 4

// One word of key XOR query: the high bits of its zero codes join `acc`.  The other bits of acc
// carry rubbish until lsh_matched() looks at the high bits, which saves the mask per word.
template <typename CodeT>
__device__ __forceinline__ void lsh_match_word(uint32_t x, uint32_t& acc) {
  acc |= (x - (sizeof(CodeT) == 1 ? 0x01010101u : 0x00010001u)) & ~x;
}
template <typename CodeT>
__device__ __forceinline__ bool lsh_matched(uint32_t acc) {
  return (acc & (sizeof(CodeT) == 1 ? 0x80808080u : 0x80008000u)) != 0u;
}
#define LSH_MAX_CHUNKS 16  // 16-byte chunks per signature row (256 byte codes, 128 halfword codes)

template <typename CodeT, int NC>
__global__ void __launch_bounds__(LSH_MATCH_WARPS * 32)
lsh_match_kernel(const CodeT* __restrict__ codes, int64_t cap, const CodeT* __restrict__ qcodes,
                 int Hq, int Sq, int G, int L, int64_t S, int64_t W,
                 const uint32_t* __restrict__ prev_bits, uint32_t* __restrict__ out_bits) {
  sah_pdl_entry();
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  uint4* qs = reinterpret_cast<uint4*>(lsh_smem);  // [R][NC]
  const int R = G * Sq;
  constexpr int PER16 = 16 / (int)sizeof(CodeT);
  constexpr int LP = NC * PER16;
  const int64_t bh = blockIdx.y;           // b * Hkv + hkv
  const int Hkv = Hq / G;
  const int64_t b = bh / Hkv, hkv = bh % Hkv;
  {
    CodeT* qflat = reinterpret_cast<CodeT*>(lsh_smem);
    for (int i = threadIdx.x; i < R * LP; i += blockDim.x) {
      const int r = i / LP, l = i % LP;
      const int g = r / Sq, qi = r % Sq;
      // padding: all ones, which the zero padding of a key row never equals
      qflat[i] = l < L ? qcodes[(((b * Hq) + hkv * G + g) * Sq + qi) * L + l] : (CodeT)~(CodeT)0;
    }
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t word0 = ((int64_t)blockIdx.x * LSH_MATCH_WARPS + warp) * LSH_MATCH_WORDS;
  if (word0 * 32 >= S) return;
  const uint4* base = reinterpret_cast<const uint4*>(codes + bh * cap * LP);
  const int64_t words = (S + 31) / 32;
  // the four words of a mask row as one 16-byte access
  const bool quad = W % 4 == 0 && word0 + LSH_MATCH_WORDS <= words && (reinterpret_cast<uintptr_t>(out_bits) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(prev_bits) & 15) == 0;
  // A key's row is read once for 64 query rows (once per four of them, at 16 query positions, took
  // 187 us for 8 x 65500 keys of 75 tables; 165 us now, the integer instructions).  A lane keeps the
  // words of two query rows until all four are there and stores them together.  Of short signatures it
  // reads all four words' keys before it starts on the queries, so that a query row read from shared
  // memory serves four words (16 tables, 8 rows x 65500 keys: 9.6 us reading the keys once per four
  // queries, 12.1 us word by word, 10.2 us this way; 64 rows x 16384 26.4, 26.2 and 17.2).
  for (int rb = 0; rb < R; rb += 64) {
    const int re = R - rb < 64 ? R - rb : 64;
    uint32_t keep[2][LSH_MATCH_WORDS];  // lane l: the words of rows rb + l and rb + 32 + l
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int j = 0; j < LSH_MATCH_WORDS; ++j) keep[n][j] = 0u;
    constexpr int JW = NC <= 2 ? LSH_MATCH_WORDS : 1;  // words whose keys a lane holds at once
#pragma unroll 1
    for (int j0 = 0; j0 < LSH_MATCH_WORDS; j0 += JW) {
      if ((word0 + j0) * 32 >= S) break;
      uint4 v[JW][NC];
      uint32_t mine[JW][2];
#pragma unroll
      for (int j = 0; j < JW; ++j) {
        const int64_t key = (word0 + j0 + j) * 32 + lane;
#pragma unroll
        for (int c = 0; c < NC; ++c) v[j][c] = key < S ? __ldg(base + key * NC + c) : make_uint4(0u, 0u, 0u, 0u);
        mine[j][0] = mine[j][1] = 0u;
      }
      for (int r0 = 0; r0 < re; r0 += 4) {
        uint32_t hit[JW][4];
#pragma unroll
        for (int j = 0; j < JW; ++j)
#pragma unroll
          for (int r = 0; r < 4; ++r) hit[j][r] = 0u;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            if (r0 + r < re) {
              const uint4 q = qs[(rb + r0 + r) * NC + c];
#pragma unroll
              for (int j = 0; j < JW; ++j) {
                lsh_match_word<CodeT>(v[j][c].x ^ q.x, hit[j][r]);
                lsh_match_word<CodeT>(v[j][c].y ^ q.y, hit[j][r]);
                lsh_match_word<CodeT>(v[j][c].z ^ q.z, hit[j][r]);
                lsh_match_word<CodeT>(v[j][c].w ^ q.w, hit[j][r]);
              }
            }
          }
        }
#pragma unroll
        for (int j = 0; j < JW; ++j) {
          const bool live = (word0 + j0 + j) * 32 + lane < S;
#pragma unroll
          for (int r = 0; r < 4; ++r) {
            const uint32_t wbits = __ballot_sync(0xffffffffu, lsh_matched<CodeT>(hit[j][r]) && live);
            if (lane == ((r0 + r) & 31)) {
              if (r0 + r < 32) mine[j][0] = wbits; else mine[j][1] = wbits;
            }
          }
        }
      }
#pragma unroll
      for (int j = 0; j < LSH_MATCH_WORDS; ++j)
        if (JW == LSH_MATCH_WORDS || j == j0) {
          keep[0][j] = mine[j % JW][0];
          keep[1][j] = mine[j % JW][1];
        }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      const int r = rb + n * 32 + lane;
      if (n * 32 + lane < re) {
        const int g = r / Sq, qi = r % Sq;
        const int64_t at = (((b * Hq) + hkv * G + g) * Sq + qi) * W + word0;  // keys past S never set a bit
        if (quad) {
          uint4 bits = make_uint4(keep[n][0], keep[n][1], keep[n][2], keep[n][3]);
          if (prev_bits != nullptr) {
            const uint4 p = *reinterpret_cast<const uint4*>(prev_bits + at);
            bits = make_uint4(bits.x | p.x, bits.y | p.y, bits.z | p.z, bits.w | p.w);
          }
          *reinterpret_cast<uint4*>(out_bits + at) = bits;
        } else {
#pragma unroll
          for (int j = 0; j < LSH_MATCH_WORDS; ++j)
            if (word0 + j < words) out_bits[at + j] = keep[n][j] | (prev_bits != nullptr ? prev_bits[at + j] : 0u);
        }
      }
    }
  }
}

// Decode shapes (at most four query rows per group, signature rows of up to 96 bytes): the
// group's query rows stay in registers (4 x NC 16-byte chunks), so that a (word, row) test is
// three integer instructions with no shared-memory operand, and a warp takes one bitmap word
// (32 consecutive keys) per round, striding over the row with all warps of the group's CTAs:
// the grid is two CTAs per SM whatever the key count, every warp gets the same number of words
// to within one.  The 32 signature rows of a round are contiguous in memory; the warp copies
// them to shared memory with 16-byte asynchronous copies, lane after lane (every copy
// instruction covers 512 contiguous bytes, where a lane loading its own row of 80 bytes makes
// each load instruction touch 20 cache lines), three rounds ahead, and every lane then reads
// its own row from there.  Lane r writes the word of row r.
// Measured at 1M keys (8.4M signature rows of 80 bytes, 671 MB): 139 us, 4.8 TB/s; the
// shared-memory form below 177 us; this form with per-lane 16-byte loads instead of the staged
// copies 164 us; with two of the four query rows read from shared memory and three CTAs per SM
// instead of two 182 us.  ~420 thread instructions per (key, group), 0.58 issue slots busy.
#define LSH_MATCH_REG_MAX_NC 6
#define LSH_MATCH_REG_STAGES 4

template <typename CodeT, int NC>
__global__ void __launch_bounds__(LSH_MATCH_WARPS * 32, 2)
lsh_match_reg_kernel(const CodeT* __restrict__ codes, int64_t cap, const CodeT* __restrict__ qcodes,
                     int Hq, int Sq, int G, int L, int64_t S, int64_t W,
                     const uint32_t* __restrict__ prev_bits, uint32_t* __restrict__ out_bits) {
  sah_pdl_entry();
  extern __shared__ __align__(16) unsigned char mr_smem[];  // [warps][stages][32 rows of NC chunks]
  __shared__ __align__(16) CodeT qflat[4 * NC * (16 / (int)sizeof(CodeT))];
  constexpr int PER16 = 16 / (int)sizeof(CodeT);
  constexpr int LP = NC * PER16;
  constexpr int NST = LSH_MATCH_REG_STAGES;
  constexpr int ROUND_BYTES = 32 * NC * 16;
  const int R = G * Sq;  // <= 4
  const int64_t bh = blockIdx.y;  // b * Hkv + hkv
  const int Hkv = Hq / G;
  const int64_t b = bh / Hkv, hkv = bh % Hkv;
  for (int i = threadIdx.x; i < 4 * LP; i += blockDim.x) {
    const int r = i / LP, l = i % LP;
    CodeT c = (CodeT)~(CodeT)0;  // padding: all ones, which the zero padding of a key row never equals
    if (r < R && l < L) {
      const int g = r / Sq, qi = r % Sq;
      c = qcodes[(((b * Hq) + hkv * G + g) * Sq + qi) * L + l];
    }
    qflat[i] = c;
  }
  __syncthreads();
  uint4 q[4][NC];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < NC; ++c) q[r][c] = reinterpret_cast<const uint4*>(qflat)[r * NC + c];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t words = (S + 31) / 32;
  const uint4* base = reinterpret_cast<const uint4*>(codes + bh * cap * LP);
  const int64_t chunks_end = S * NC;  // 16-byte chunks of this (batch, KV head) that hold keys
  unsigned char* wbuf = mr_smem + (size_t)warp * NST * ROUND_BYTES;
  const uint32_t wbuf_s = (uint32_t)__cvta_generic_to_shared(wbuf);
  int64_t my_row = -1;  // lane r < R writes row r
  if (lane < R) {
    const int g = lane / Sq, qi = lane % Sq;
    my_row = ((b * Hq) + hkv * G + g) * Sq + qi;
  }
  const int64_t stride = (int64_t)gridDim.x * LSH_MATCH_WARPS;
  const int64_t w0 = (int64_t)blockIdx.x * LSH_MATCH_WARPS + warp;
  // copies of round `w` into stage `st`; one commit per call whether or not anything was copied
  auto issue = [&](int64_t w, int st) {
    if (w < words) {
      const int64_t first = w * 32 * NC;
#pragma unroll
      for (int it = 0; it < NC; ++it) {
        const int j = it * 32 + lane;
        if (first + j < chunks_end)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(wbuf_s + st * ROUND_BYTES + j * 16),
                       "l"(base + first + j)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll
  for (int s0 = 0; s0 < NST - 1; ++s0) issue(w0 + s0 * stride, s0);
  int i = 0;
  for (int64_t w = w0; w < words; w += stride, ++i) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NST - 2) : "memory");
    __syncwarp();  // every lane's copies of this round have landed; everyone is done with round i - 1
    issue(w + (NST - 1) * stride, (i + NST - 1) % NST);
    const int64_t key = w * 32 + lane;
    uint32_t hit[4] = {0u, 0u, 0u, 0u};
    if (key < S) {
      const uint4* mine_row = reinterpret_cast<const uint4*>(wbuf + (i % NST) * ROUND_BYTES) + lane * NC;
      uint4 v[NC];
#pragma unroll
      for (int c = 0; c < NC; ++c) v[c] = mine_row[c];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          lsh_match_word<CodeT>(v[c].x ^ q[r][c].x, hit[r]);
          lsh_match_word<CodeT>(v[c].y ^ q[r][c].y, hit[r]);
          lsh_match_word<CodeT>(v[c].z ^ q[r][c].z, hit[r]);
          lsh_match_word<CodeT>(v[c].w ^ q[r][c].w, hit[r]);
        }
      }
    }
    uint32_t mine = 0u;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const uint32_t wbits = __ballot_sync(0xffffffffu, lsh_matched<CodeT>(hit[r]));
      if (lane == r) mine = wbits;
    }
    if (my_row >= 0) {
      if (prev_bits != nullptr) mine |= prev_bits[my_row * W + w];
      out_bits[my_row * W + w] = mine;
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

template <typename CodeT>
static int lsh_match_launch(const void* codes, int64_t cap, const void* qcodes, int Hq, int Sq, int G, int L,
                            int64_t S, int64_t W, const uint32_t* prev_bits, uint32_t* out_bits, dim3 grid,
                            size_t smem, cudaStream_t st) {
  const int nc = lsh_row_pitch<CodeT>(L) / (16 / (int)sizeof(CodeT));
  // SAH_LSH_MATCH_REG=0 in the environment keeps the shared-memory form for every shape
  static int reg_env = -1;
  if (reg_env < 0) {
    const char* e = getenv("SAH_LSH_MATCH_REG");
    reg_env = (e != nullptr && e[0] == '0') ? 0 : 1;
  }
  if (reg_env == 1 && G * Sq <= 4 && nc <= LSH_MATCH_REG_MAX_NC) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) {
      int n = 0;
      if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0) sms = n;
    }
    const int64_t words = (S + 31) / 32;
    int64_t per_group = sah_ceil_div((int64_t)2 * sms, (int64_t)grid.y);
    const int64_t most = sah_ceil_div(words, LSH_MATCH_WARPS);
    if (per_group > most) per_group = most;
    if (per_group < 1) per_group = 1;
    const dim3 rgrid((unsigned)per_group, grid.y);
#define LSH_MATCH_REG_CASE(NC)                                                                      \
  case NC: {                                                                                        \
    constexpr int RSMEM = LSH_MATCH_WARPS * LSH_MATCH_REG_STAGES * 32 * NC * 16;                    \
    static bool allowed[64] = {};                                                                   \
    if (RSMEM + 4 * NC * 16 > 48 * 1024) {  /* beside the four query rows */                        \
      const cudaError_t e = sah_allow_smem(lsh_match_reg_kernel<CodeT, NC>, RSMEM, allowed);        \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "lsh_match attr: %s", cudaGetErrorString(e)); \
    }                                                                                               \
    sah_launch_chain(lsh_match_reg_kernel<CodeT, NC>, rgrid, LSH_MATCH_WARPS * 32, RSMEM, st,       \
        reinterpret_cast<const CodeT*>(codes), cap, reinterpret_cast<const CodeT*>(qcodes), Hq, Sq, \
        G, L, S, W, prev_bits, out_bits);                                                           \
  } break;
    switch (nc) {
      LSH_MATCH_REG_CASE(1) LSH_MATCH_REG_CASE(2) LSH_MATCH_REG_CASE(3) LSH_MATCH_REG_CASE(4)
      LSH_MATCH_REG_CASE(5) LSH_MATCH_REG_CASE(6)
    }
#undef LSH_MATCH_REG_CASE
    return SAH_OK;
  }
#define LSH_MATCH_CASE(NC)                                                                          \
  case NC:                                                                                          \
    sah_launch_chain(lsh_match_kernel<CodeT, NC>, grid, LSH_MATCH_WARPS * 32, smem, st, \
        reinterpret_cast<const CodeT*>(codes), cap, reinterpret_cast<const CodeT*>(qcodes), Hq, Sq, \
        G, L, S, W, prev_bits, out_bits);                                                           \
    break;
  switch (nc) {
    LSH_MATCH_CASE(1) LSH_MATCH_CASE(2) LSH_MATCH_CASE(3) LSH_MATCH_CASE(4) LSH_MATCH_CASE(5)
    LSH_MATCH_CASE(6) LSH_MATCH_CASE(7) LSH_MATCH_CASE(8) LSH_MATCH_CASE(9) LSH_MATCH_CASE(10)
    LSH_MATCH_CASE(11) LSH_MATCH_CASE(12) LSH_MATCH_CASE(13) LSH_MATCH_CASE(14) LSH_MATCH_CASE(15)
    LSH_MATCH_CASE(16)
    default:
      return sah_fail(SAH_ERR_UNSUPPORTED, "lsh_match: %d tables exceed %d bytes per signature row", L,
                      LSH_MAX_CHUNKS * 16);
  }
#undef LSH_MATCH_CASE
  return SAH_OK;
}

extern "C" int sah_lsh_match(const void* codes, int64_t cap, const void* qcodes, int B, int Hq,
                             int Sq, int G, int L, int K, int64_t S, int64_t W,
                             const uint32_t* prev_bits, uint32_t* out_bits, void* stream) {
  SAH_REQUIRE(codes && qcodes && out_bits, "lsh_match: null pointer");
  SAH_REQUIRE(G > 0 && Hq % G == 0 && L > 0 && K > 0 && S > 0 && W * 32 >= S, "lsh_match: bad shape");
  SAH_REQUIRE(cap >= S && (uintptr_t)codes % 16 == 0, "lsh_match: signature rows must be 16-byte aligned");
  if (K > 16) return sah_fail(SAH_ERR_UNSUPPORTED, "lsh: lsh_k = %d > 16 bits per table is not built", K);
  const int csz = K <= 8 ? 1 : 2;
  const int lp = csz == 1 ? lsh_row_pitch<uint8_t>(L) : lsh_row_pitch<uint16_t>(L);
  const size_t smem = (size_t)G * Sq * lp * csz;
  if (smem > 48 * 1024) return sah_fail(SAH_ERR_UNSUPPORTED, "lsh_match: too many query rows per group");
  const int64_t words = (S + 31) / 32;
  dim3 grid((unsigned)sah_ceil_div(words, LSH_MATCH_WARPS * LSH_MATCH_WORDS), (unsigned)(B * (Hq / G)));
  cudaStream_t st = (cudaStream_t)stream;
  sah_prof_begin(SAH_PROF_LSH_MATCH, st);
  const int rc = csz == 1 ? lsh_match_launch<uint8_t>(codes, cap, qcodes, Hq, Sq, G, L, S, W, prev_bits,
                                                      out_bits, grid, smem, st)
                          : lsh_match_launch<uint16_t>(codes, cap, qcodes, Hq, Sq, G, L, S, W, prev_bits,
                                                       out_bits, grid, smem, st);
  if (rc != SAH_OK) return rc;
  SAH_LAUNCH_CHECK("lsh_match");
  sah_prof_end(SAH_PROF_LSH_MATCH, st);
  return SAH_OK;
}

// ---------------------------------------------------------------------------------------
// collision probability of matched keys
// ---------------------------------------------------------------------------------------
// 1 - (1 - (1 - acos(c) / pi)^K)^L with every operation rounded to the dtype (:374-403).
// bf16 goes through a 65536-entry table of the whole chain; fp32 evaluates acos and pow in
// double precision and rounds once, so that a CPU restatement reproduces the bits.
template <typename T>
__device__ __forceinline__ float lsh_collision_prob(float c, int K, int L, const uint16_t* table);
template <>
__device__ __forceinline__ float lsh_collision_prob<__nv_bfloat16>(float c, int, int,
                                                                   const uint16_t* table) {
  return __uint_as_float(((uint32_t)table[__float_as_uint(c) >> 16]) << 16);
}
template <>
__device__ __forceinline__ float lsh_collision_prob<float>(float c, int K, int L, const uint16_t*) {
  const float theta = (float)acos((double)c);
  const float a = __fdiv_rn(theta, 3.14159274101257324f);
  const float s = __fsub_rn(1.0f, a);
  const float st = (float)pow((double)s, (double)K);
  const float u = __fsub_rn(1.0f, st);
  const float ul = (float)pow((double)u, (double)L);
  return __fsub_rn(1.0f, ul);
}

// x / M for a fixed divisor.  bf16: the quotient of two bf16 values rounded to bf16 depends on
// the dividend only through its 7 mantissa bits (a power-of-two factor commutes with both
// roundings), so a 128-entry table of bf16((1 + m/128) / M), built with true divisions,
// replaces the division; dividends with a zero or all-ones exponent field take the division.
// fp32: the IEEE division.
template <typename T>
struct LshDivM;
template <>
struct LshDivM<__nv_bfloat16> {
  static __device__ __forceinline__ void build(float* tab, float M) {
    for (int m = threadIdx.x; m < 128; m += blockDim.x)
      tab[m] = sah_round_to<__nv_bfloat16>(__fdiv_rn(1.0f + (float)m * 0.0078125f, M));
  }
  static __device__ __forceinline__ float div(float c, float M, const float* tab) {
    const uint32_t u = __float_as_uint(c);
    const uint32_t e = (u >> 23) & 0xffu;
    if (e == 0u || e == 255u) return sah_round_to<__nv_bfloat16>(__fdiv_rn(c, M));
    const float r = __fmul_rn(__uint_as_float(u & 0xff800000u), tab[(u >> 16) & 0x7fu]);
    // the product of a power of two and a bf16 value is exact unless it leaves the normal range
    const uint32_t er = (__float_as_uint(r) >> 23) & 0xffu;
    return (er == 0u || er == 255u) ? sah_round_to<__nv_bfloat16>(__fdiv_rn(c, M)) : r;
  }
};
template <>
struct LshDivM<float> {
  static __device__ __forceinline__ void build(float*, float) {}
  static __device__ __forceinline__ float div(float c, float M, const float*) { return __fdiv_rn(c, M); }
};

// x / den for a per-key divisor.  bf16: both operands are bf16 values; with y = RN(1 / den),
// q = RN(x * y), r = x - q * den (exact in one fma), RN(q + r * y) rounded to bf16 equals the
// IEEE quotient rounded to bf16 for every pair of bf16 significands (checked exhaustively on
// the host, tests/test_magicpig.py); operands outside the normal range take the division.
template <typename T>
__device__ __forceinline__ float lsh_div_den(float x, float den, float rcp);
template <>
__device__ __forceinline__ float lsh_div_den<__nv_bfloat16>(float x, float den, float rcp) {
  const float q = __fmul_rn(x, rcp);
  const float r = __fmaf_rn(-q, den, x);
  const float q2 = __fmaf_rn(r, rcp, q);
  const uint32_t e = (__float_as_uint(q2) >> 23) & 0xffu;
  if (e < 2u || e >= 254u) return sah_round_to<__nv_bfloat16>(__fdiv_rn(x, den));
  return sah_round_to<__nv_bfloat16>(q2);
}
template <>
__device__ __forceinline__ float lsh_div_den<float>(float x, float den, float) {
  return __fdiv_rn(x, den);
}

// One CTA per (KV group, chunk of bitmap words); a warp takes a word, forms the union of the
// group's rows for it, transforms each key of the union once (centre, scale, normalise) and
// dots it with the unit query of every row that matched it.
template <typename T>
__global__ void __launch_bounds__(256)
lsh_prob_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hq, int Sq,
                int G, int D, const T* __restrict__ mean, const float* __restrict__ norms,
                int64_t cap, const unsigned int* __restrict__ max_bits,
                const float* __restrict__ qunit, const uint32_t* __restrict__ bits,
                const int32_t* __restrict__ wpre, const int64_t* __restrict__ ptr, int64_t W,
                int K, int L, const uint16_t* __restrict__ table, int q_in_smem,
                T* __restrict__ data) {
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  float* tab = reinterpret_cast<float*>(lsh_smem);  // [128]
  float* qs = tab + 128;                            // [R][D] when q_in_smem
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int Hkv = Hq / G;
  const int64_t kvh = blockIdx.x;  // b * Hkv + hkv
  const int64_t b = kvh / Hkv;
  const int hkv = (int)(kvh % Hkv);
  const int R = G * Sq;
  const int per = D / 32;
  const float M = __uint_as_float(*max_bits);
  const int64_t row0 = (b * Hq + (int64_t)hkv * G) * Sq;  // rows of a group are contiguous
  LshDivM<T>::build(tab, M);
  if (q_in_smem)
    for (int i = threadIdx.x; i < R * D; i += blockDim.x) qs[i] = qunit[row0 * D + i];
  __syncthreads();
  const float* qsrc = q_in_smem ? qs : qunit + row0 * D;
  float m[LSH_MAX_PER_LANE];
  if (mean) lsh_load_lane<T>(mean + kvh * D, per, lane, m);
  const T* kbase = k + b * ks_b + hkv * ks_h;
  for (int64_t w = (int64_t)blockIdx.y * nwarp + warp; w < W; w += (int64_t)gridDim.y * nwarp) {
    // union of the rows' words (lane r holds row r, r + 32, ...)
    uint32_t uni = 0u, myword = 0u;
    for (int r = lane; r < R; r += 32) {
      const uint32_t wd = bits[(row0 + r) * W + w];
      if (r < 32) myword = wd;
      uni |= wd;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) uni |= __shfl_xor_sync(0xffffffffu, uni, o);
    if (!uni) continue;
    // the next key's row is loaded while the current one is worked on
    int nbit = __ffs(uni) - 1;
    float xn[LSH_MAX_PER_LANE];
    lsh_load_lane<T>(kbase + (w * 32 + nbit) * ks_s, per, lane, xn);
    float nkn = norms[kvh * cap + w * 32 + nbit];
    while (uni) {
      const int bit = nbit;
      const float nk = nkn;
      float x[LSH_MAX_PER_LANE];
#pragma unroll
      for (int t = 0; t < LSH_MAX_PER_LANE; ++t) x[t] = xn[t];
      uni &= uni - 1;
      if (uni) {
        nbit = __ffs(uni) - 1;
        lsh_load_lane<T>(kbase + (w * 32 + nbit) * ks_s, per, lane, xn);
        nkn = norms[kvh * cap + w * 32 + nbit];
      }
      float acc = 0.f;
#pragma unroll
      for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
        if (t < per) {
          const float c = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
          x[t] = LshDivM<T>::div(c, M, tab);
          acc = __fadd_rn(acc, __fmul_rn(x[t], x[t]));
        }
      const float aug = lsh_augment<T>(nk, M);
      // |transformed key|, then its unit vector
      const float n2 = __fadd_rn(lsh_warp_sum(acc), __fmul_rn(aug, aug));
      const float den = sah_round_to<T>(__fadd_rn(sah_round_to<T>(sqrtf(n2)), 1e-8f));
      const float rcp = __frcp_rn(den);
#pragma unroll
      for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
        if (t < per) x[t] = lsh_div_den<T>(x[t], den, rcp);
      for (int r = 0; r < R; ++r) {
        // warp-uniform: the first 32 rows' words sit in the lanes, the rest are re-read (L1)
        const uint32_t word = r < 32 ? __shfl_sync(0xffffffffu, myword, r) : bits[(row0 + r) * W + w];
        if (!((word >> bit) & 1u)) continue;
        const float* qu = qsrc + r * D + lane * per;
        acc = 0.f;
#pragma unroll
        for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
          if (t < per) acc = __fadd_rn(acc, __fmul_rn(qu[t], x[t]));
        float c = sah_round_to<T>(lsh_warp_sum(acc));
        c = fminf(fmaxf(c, -1.0f), 1.0f);
        if (lane == 0) {
          const int64_t pos = ptr[row0 + r] + wpre[(row0 + r) * W + w] + __popc(word & ((1u << bit) - 1u));
          data[pos] = sah_from_float<T>(lsh_collision_prob<T>(c, K, L, table));
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------------------
// Cached norm of the transformed key.  |[k_c / M, sqrt(M^2 - |k_c|^2) / M]| + 1e-8 depends on
// the key, the key mean and the maximum norm M only, not on the query, so it is computed when
// keys arrive (and again for every key if M moved) instead of at every decode step.
// dens_max_bits holds the M the cached values were computed with.
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256)
lsh_key_den_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv,
                   int64_t s_new0, int64_t s1, int D, const T* __restrict__ mean,
                   const float* __restrict__ norms, int64_t cap,
                   const unsigned int* __restrict__ max_bits,
                   const unsigned int* __restrict__ dens_max_bits, float* __restrict__ dens) {
  sah_pdl_entry_early();
  __shared__ float tab[128];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int64_t bh = blockIdx.y;
  const int64_t b = bh / Hkv, h = bh % Hkv;
  const int per = D / 32;
  const unsigned int mb = *max_bits;
  const float M = __uint_as_float(mb);
  const int64_t begin = (mb == *dens_max_bits) ? s_new0 : 0;  // M moved: every key again
  if (begin >= s1) return;
  LshDivM<T>::build(tab, M);
  __syncthreads();
  float m[LSH_MAX_PER_LANE];
  if (mean) lsh_load_lane<T>(mean + bh * D, per, lane, m);
  for (int64_t s = begin + (int64_t)blockIdx.x * nwarp + warp; s < s1; s += (int64_t)gridDim.x * nwarp) {
    float x[LSH_MAX_PER_LANE];
    lsh_load_lane<T>(k + b * ks_b + h * ks_h + s * ks_s, per, lane, x);
    float acc = 0.f;
#pragma unroll
    for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
      if (t < per) {
        const float c = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
        const float ks = LshDivM<T>::div(c, M, tab);
        acc = __fadd_rn(acc, __fmul_rn(ks, ks));
      }
    const float aug = lsh_augment<T>(norms[bh * cap + s], M);
    const float n2 = __fadd_rn(lsh_warp_sum(acc), __fmul_rn(aug, aug));
    if (lane == 0) dens[bh * cap + s] = sah_round_to<T>(__fadd_rn(sah_round_to<T>(sqrtf(n2)), 1e-8f));
  }
}

__global__ void lsh_den_commit_kernel(const unsigned int* max_bits, unsigned int* dens_max_bits) {
  sah_pdl_entry_early();
  *dens_max_bits = *max_bits;
}

// The same two passes (norms of the centred keys; norms of the transformed keys) over many bfloat16
// keys of 128 channels, as an index build makes them: a warp takes 32 neighbouring keys, lane by
// lane as lsh_load_lane does, and turns the 32 x 32 partial sums over on the way down the xor tree
// (lane l ends up with key l: 31 exchanges instead of 160, the same pairs added at every level),
// so that the square roots, the augmentation column and the stores are one instruction for 32
// keys.  Bound by the channel arithmetic (20 us to read the keys at the measured copy rate).
// 8 x 65500 keys: 88 us (norms) and 180 us (transformed norms) with a key per warp, 43 us and
// 70 us this way.
template <bool DEN>
__global__ void __launch_bounds__(256)
lsh_key_rows_kernel(const __nv_bfloat16* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv, int64_t s0,
                    int64_t s1, const __nv_bfloat16* __restrict__ mean, int64_t cap, float* __restrict__ norms,
                    unsigned int* __restrict__ max_bits, float* __restrict__ dens) {
  typedef __nv_bfloat16 T;
  constexpr int D = 128;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t bh = blockIdx.y;
  const __nv_bfloat16* kb = k + bh / Hkv * ks_b + bh % Hkv * ks_h + lane * 4;
  // c / M as a product with 1 / M: the same bfloat16 number for a bfloat16 M and operands well
  // inside the range (lsh_key_sign_tc_kernel says why); the others are divided
  const float M = DEN ? __uint_as_float(*max_bits) : 1.f, rM = __frcp_rn(M);
  const bool divide = (__float_as_uint(M) & 0xffffu) != 0u || !(M >= 8.673617e-19f && M <= 1.152921504606847e18f);
  float m[4] = {0.f, 0.f, 0.f, 0.f};
  if (mean) lsh_load_lane<T>(mean + bh * D, 4, lane, m);
  float local_max = 0.f;
  for (int64_t base = s0 + ((int64_t)blockIdx.x * 8 + warp) * 32; base < s1; base += (int64_t)gridDim.x * 8 * 32) {
    float v[32];
#pragma unroll
    for (int j0 = 0; j0 < 32; j0 += 8) {
      uint2 raw[8];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        raw[j] = base + j0 + j < s1 ? *reinterpret_cast<const uint2*>(kb + (base + j0 + j) * ks_s) : make_uint2(0u, 0u);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x[4] = {__uint_as_float(raw[j].x << 16), __uint_as_float(raw[j].x & 0xffff0000u),
                            __uint_as_float(raw[j].y << 16), __uint_as_float(raw[j].y & 0xffff0000u)};
        float acc = 0.f, c[4];
        bool odd = divide;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          c[t] = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
          if (DEN) odd = odd || (fabsf(c[t]) < 8.673617e-19f && c[t] != 0.f);
          const float y = DEN ? sah_round_to<T>(__fmul_rn(c[t], rM)) : c[t];
          acc = __fadd_rn(acc, __fmul_rn(y, y));
        }
        if (DEN && odd) {
          acc = 0.f;
#pragma unroll 1
          for (int t = 0; t < 4; ++t) {
            const float ct = t == 0 ? c[0] : t == 1 ? c[1] : t == 2 ? c[2] : c[3];
            const float y = sah_round_to<T>(__fdiv_rn(ct, M));
            acc = __fadd_rn(acc, __fmul_rn(y, y));
          }
        }
        v[j0 + j] = acc;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const bool upper = lane & o;
#pragma unroll
      for (int j = 0; j < o; ++j) {
        const float other = __shfl_xor_sync(0xffffffffu, upper ? v[j] : v[j + o], o);
        v[j] = __fadd_rn(upper ? v[j + o] : v[j], other);
      }
    }
    const int64_t s = base + lane;
    if (s < s1) {
      if (DEN) {
        const float aug = lsh_augment<T>(norms[bh * cap + s], M);
        const float n2 = __fadd_rn(v[0], __fmul_rn(aug, aug));
        dens[bh * cap + s] = sah_round_to<T>(__fadd_rn(sah_round_to<T>(sqrtf(n2)), 1e-8f));
      } else {
        const float nk = sah_round_to<T>(sqrtf(v[0]));
        norms[bh * cap + s] = nk;
        local_max = fmaxf(local_max, nk);
      }
    }
  }
  if (!DEN) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local_max = fmaxf(local_max, __shfl_xor_sync(0xffffffffu, local_max, o));
    if (lane == 0 && local_max > 0.f) atomicMax(max_bits, __float_as_uint(local_max));
  }
}

// From how many keys on, all heads together, 32 keys per warp are ahead of a key per warp, which
// spreads fewer keys better over the chip.  Norms: 2 x 1024 keys 6.2 against 4.2 us, 2 x 2048 equal,
// 8 x 1024 6.2 against 8.4 us.  Transformed norms (with the clearing of a word, 2 us): 8 x 2048 16.4
// against 14.4 us, 2 x 16384 16.4 against 18.5 us, 8 x 4096 16.4 against 20.5 us.
#define LSH_ROWS_MIN_STATS 4096
#define LSH_ROWS_MIN_DENS 32768
static bool lsh_rows_fits(const void* keys, int dtype, int64_t ks_b, int64_t ks_h, int64_t ks_s, int64_t n,
                          int64_t heads, int64_t least, int D) {
  return dtype == SAH_BF16 && D == 128 && n >= 1024 && n * heads >= least && ((uintptr_t)keys & 7) == 0 &&
         ks_b % 4 == 0 && ks_h % 4 == 0 && ks_s % 4 == 0;
}
static dim3 lsh_rows_grid(int64_t n, int64_t heads, int sm_count) {
  int64_t gx = (n + 255) / 256;
  const int64_t most = ((int64_t)sm_count * 8 + heads - 1) / heads;
  return dim3((unsigned)(gx < most ? gx : most), (unsigned)heads);
}

extern "C" int sah_lsh_key_stats(const void* keys, int dtype, int64_t ks_b, int64_t ks_h,
                                 int64_t ks_s, int B, int Hkv, int64_t s0, int64_t s1, int D,
                                 const void* mean, int64_t cap, float* norms,
                                 unsigned int* max_norm_bits, int sm_count, void* stream) {
  SAH_REQUIRE(keys && norms && max_norm_bits, "lsh_key_stats: null pointer");
  SAH_REQUIRE(D % 32 == 0 && D <= 32 * LSH_MAX_PER_LANE, "lsh_key_stats: head_dim must be a multiple of 32, <= 256");
  SAH_REQUIRE(s0 >= 0 && s1 >= s0 && s1 <= cap, "lsh_key_stats: bad key range");
  if (s1 == s0) return SAH_OK;
  if (sm_count <= 0) sm_count = 148;
  if (lsh_rows_fits(keys, dtype, ks_b, ks_h, ks_s, s1 - s0, (int64_t)B * Hkv, LSH_ROWS_MIN_STATS, D)) {
    lsh_key_rows_kernel<false><<<lsh_rows_grid(s1 - s0, (int64_t)B * Hkv, sm_count), 256, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hkv, s0, s1,
        reinterpret_cast<const __nv_bfloat16*>(mean), cap, norms, max_norm_bits, nullptr);
    SAH_LAUNCH_CHECK("lsh_key_rows");
    return SAH_OK;
  }
  int64_t gx = (s1 - s0 + 7) / 8;
  const int64_t cap_x = ((int64_t)sm_count * 16 + (int64_t)B * Hkv - 1) / ((int64_t)B * Hkv);
  if (gx > cap_x) gx = cap_x;
  dim3 grid((unsigned)gx, (unsigned)(B * Hkv));
  SAH_DISPATCH_DTYPE(dtype, T, {
    sah_launch_chain(lsh_key_stats_kernel<T>, grid, 256, 0, (cudaStream_t)stream,
        reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hkv, s0, s1, D,
        reinterpret_cast<const T*>(mean), cap, norms, max_norm_bits);
  });
  SAH_LAUNCH_CHECK("lsh_key_stats");
  return SAH_OK;
}

extern "C" int sah_lsh_key_den(const void* keys, int dtype, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                               int B, int Hkv, int64_t s_new0, int64_t s1, int D, const void* mean,
                               const float* norms, int64_t cap, const unsigned int* max_norm_bits,
                               unsigned int* dens_max_bits, float* dens, int sm_count, void* stream) {
  SAH_REQUIRE(keys && norms && max_norm_bits && dens_max_bits && dens, "lsh_key_den: null pointer");
  SAH_REQUIRE(D % 32 == 0 && D <= 32 * LSH_MAX_PER_LANE, "lsh_key_den: head_dim must be a multiple of 32, <= 256");
  SAH_REQUIRE(s_new0 >= 0 && s_new0 <= s1 && s1 <= cap, "lsh_key_den: bad key range");
  if (s1 == 0) return SAH_OK;
  if (sm_count <= 0) sm_count = 148;
  cudaStream_t st = (cudaStream_t)stream;
  // An index build: every key is new (whether M moved or not), so the first key is known here.
  if (s_new0 == 0 && lsh_rows_fits(keys, dtype, ks_b, ks_h, ks_s, s1, (int64_t)B * Hkv, LSH_ROWS_MIN_DENS, D)) {
    lsh_key_rows_kernel<true><<<lsh_rows_grid(s1, (int64_t)B * Hkv, sm_count), 256, 0, st>>>(
        reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hkv, 0, s1,
        reinterpret_cast<const __nv_bfloat16*>(mean), cap, const_cast<float*>(norms),
        const_cast<unsigned int*>(max_norm_bits), dens);
    SAH_LAUNCH_CHECK("lsh_key_rows");
    sah_launch_chain(lsh_den_commit_kernel, 1, 1, 0, st, max_norm_bits, dens_max_bits);
    SAH_LAUNCH_CHECK("lsh_den_commit");
    return SAH_OK;
  }
  int64_t gx = (s1 + 7) / 8;
  const int64_t cap_x = ((int64_t)sm_count * 8 + (int64_t)B * Hkv - 1) / ((int64_t)B * Hkv);
  if (gx > cap_x) gx = cap_x;
  dim3 grid((unsigned)gx, (unsigned)(B * Hkv));
  SAH_DISPATCH_DTYPE(dtype, T, {
    sah_launch_chain(lsh_key_den_kernel<T>, grid, 256, 0, st, reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hkv,
                                                s_new0, s1, D, reinterpret_cast<const T*>(mean), norms,
                                                cap, max_norm_bits, dens_max_bits, dens);
  });
  SAH_LAUNCH_CHECK("lsh_key_den");
  sah_launch_chain(lsh_den_commit_kernel, 1, 1, 0, st, max_norm_bits, dens_max_bits);
  SAH_LAUNCH_CHECK("lsh_den_commit");
  return SAH_OK;
}

// bf16 with cached norms: the two divisions collapse into one table.  A centred key channel c
// (a bf16 value) times 1 / M rounded to bf16, times 1 / den rounded to bf16, equals
// 2^exponent(c) * U[den][mantissa(c)] with U = bf16(bf16((1 + m/128) / M) / den), because a
// power-of-two factor commutes with both roundings while everything stays in the normal
// range.  den is the norm of an (almost) unit vector: the 32 bf16 values from 0.9375 up
// cover it; other dens, and channels whose exponent could leave the normal range, take the
// two IEEE divisions.
#define LSH_DEN_BASE 0x3F70u
#define LSH_DEN_TABLES 32

__global__ void __launch_bounds__(256)
lsh_prob_fast_kernel(const __nv_bfloat16* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                     int Hq, int Sq, int G, int D, const __nv_bfloat16* __restrict__ mean,
                     const float* __restrict__ dens, int64_t cap,
                     const unsigned int* __restrict__ max_bits, const float* __restrict__ qunit,
                     const uint32_t* __restrict__ bits, const int32_t* __restrict__ wpre,
                     const int64_t* __restrict__ ptr, int64_t W, const uint16_t* __restrict__ table,
                     int q_in_smem, __nv_bfloat16* __restrict__ data) {
  typedef __nv_bfloat16 T;
  extern __shared__ __align__(16) unsigned char lsh_smem[];
  float* U = reinterpret_cast<float*>(lsh_smem);  // [LSH_DEN_TABLES][128]
  float* qs = U + LSH_DEN_TABLES * 128;           // [R][D] when q_in_smem
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int Hkv = Hq / G;
  const int64_t kvh = blockIdx.x;
  const int64_t b = kvh / Hkv;
  const int hkv = (int)(kvh % Hkv);
  const int R = G * Sq;
  const int per = D / 32;
  const unsigned int mbits = *max_bits;
  const float M = __uint_as_float(mbits);
  const int64_t row0 = (b * Hq + (int64_t)hkv * G) * Sq;
  for (int i = threadIdx.x; i < LSH_DEN_TABLES * 128; i += blockDim.x) {
    const int di = i >> 7, m = i & 127;
    const float t = sah_round_to<T>(__fdiv_rn(1.0f + (float)m * 0.0078125f, M));
    const float d = __uint_as_float((LSH_DEN_BASE + (unsigned)di) << 16);
    U[i] = sah_round_to<T>(__fdiv_rn(t, d));
  }
  if (q_in_smem)
    for (int i = threadIdx.x; i < R * D; i += blockDim.x) qs[i] = qunit[row0 * D + i];
  __syncthreads();
  // exponent fields of c for which c / M / den surely stays normal (den is within [0.9375, 1.12])
  const int shift = 127 - (int)((mbits >> 23) & 0xffu);
  const int elo = max(1, 4 - shift), ehi = min(254, 250 - shift);
  const float* qsrc = q_in_smem ? qs : qunit + row0 * D;
  float m[LSH_MAX_PER_LANE];
  if (mean) lsh_load_lane<T>(mean + kvh * D, per, lane, m);
  const T* kbase = k + b * ks_b + hkv * ks_h;
  for (int64_t w = (int64_t)blockIdx.y * nwarp + warp; w < W; w += (int64_t)gridDim.y * nwarp) {
    uint32_t uni = 0u, myword = 0u;
    for (int r = lane; r < R; r += 32) {
      const uint32_t wd = bits[(row0 + r) * W + w];
      if (r < 32) myword = wd;
      uni |= wd;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) uni |= __shfl_xor_sync(0xffffffffu, uni, o);
    if (!uni) continue;
    int nbit = __ffs(uni) - 1;
    float xn[LSH_MAX_PER_LANE];
    lsh_load_lane<T>(kbase + (w * 32 + nbit) * ks_s, per, lane, xn);
    float dn = dens[kvh * cap + w * 32 + nbit];
    while (uni) {
      const int bit = nbit;
      const float den = dn;
      float x[LSH_MAX_PER_LANE];
#pragma unroll
      for (int t = 0; t < LSH_MAX_PER_LANE; ++t) x[t] = xn[t];
      uni &= uni - 1;
      if (uni) {
        nbit = __ffs(uni) - 1;
        lsh_load_lane<T>(kbase + (w * 32 + nbit) * ks_s, per, lane, xn);
        dn = dens[kvh * cap + w * 32 + nbit];
      }
      const unsigned int di = (__float_as_uint(den) >> 16) - LSH_DEN_BASE;
      const float* Ud = U + (di < LSH_DEN_TABLES ? di : 0u) * 128;
#pragma unroll
      for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
        if (t < per) {
          const float c = mean ? sah_round_to<T>(__fsub_rn(x[t], m[t])) : x[t];
          const uint32_t u = __float_as_uint(c);
          const int e = (int)((u >> 23) & 0xffu);
          if (di < LSH_DEN_TABLES && e >= elo && e <= ehi) {
            x[t] = __fmul_rn(__uint_as_float(u & 0xff800000u), Ud[(u >> 16) & 0x7fu]);
          } else {
            const float ks = sah_round_to<T>(__fdiv_rn(c, M));
            x[t] = sah_round_to<T>(__fdiv_rn(ks, den));
          }
        }
      for (int r = 0; r < R; ++r) {
        const uint32_t word = r < 32 ? __shfl_sync(0xffffffffu, myword, r) : bits[(row0 + r) * W + w];
        if (!((word >> bit) & 1u)) continue;
        const float* qu = qsrc + r * D + lane * per;
        float acc = 0.f;
#pragma unroll
        for (int t = 0; t < LSH_MAX_PER_LANE; ++t)
          if (t < per) acc = __fadd_rn(acc, __fmul_rn(qu[t], x[t]));
        float c = sah_round_to<T>(lsh_warp_sum(acc));
        c = fminf(fmaxf(c, -1.0f), 1.0f);
        if (lane == 0) {
          const int64_t pos = ptr[row0 + r] + wpre[(row0 + r) * W + w] + __popc(word & ((1u << bit) - 1u));
          data[pos] = __ushort_as_bfloat16(table[__float_as_uint(c) >> 16]);
        }
      }
    }
  }
}

// The decode shape of the same kernel: at most 4 rows per KV group (GQA 4, one query), head
// dim 32 * PER known at compile time, keys 8-byte aligned.  Row words, CSR bases and the unit
// queries sit in registers / shared memory for a whole bitmap word; the rows' results are
// written by lanes 0..3 side by side.
template <int PER>
__global__ void __launch_bounds__(256, 4)
lsh_prob_decode_kernel(const __nv_bfloat16* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                       int Hq, int Sq, int G, const __nv_bfloat16* __restrict__ mean,
                       const float* __restrict__ dens, int64_t cap,
                       const unsigned int* __restrict__ max_bits, const float* __restrict__ qunit,
                       const uint32_t* __restrict__ bits, const int32_t* __restrict__ wpre,
                       const int64_t* __restrict__ ptr, int64_t W, const uint16_t* __restrict__ table,
                       __nv_bfloat16* __restrict__ data) {
  typedef __nv_bfloat16 T;
  constexpr int D = 32 * PER;
  __shared__ float U[LSH_DEN_TABLES * 128];
  __shared__ float qs[4 * D];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int Hkv = Hq / G;
  const int64_t kvh = blockIdx.x;
  const int64_t b = kvh / Hkv;
  const int hkv = (int)(kvh % Hkv);
  const int R = G * Sq;  // <= 4
  const unsigned int mbits = *max_bits;
  const float M = __uint_as_float(mbits);
  const int64_t row0 = (b * Hq + (int64_t)hkv * G) * Sq;
  for (int i = threadIdx.x; i < LSH_DEN_TABLES * 128; i += blockDim.x) {
    const int di = i >> 7, m = i & 127;
    const float t = sah_round_to<T>(__fdiv_rn(1.0f + (float)m * 0.0078125f, M));
    const float d = __uint_as_float((LSH_DEN_BASE + (unsigned)di) << 16);
    U[i] = sah_round_to<T>(__fdiv_rn(t, d));
  }
  for (int i = threadIdx.x; i < 4 * D; i += blockDim.x) qs[i] = i < R * D ? qunit[row0 * D + i] : 0.f;
  __syncthreads();
  const int shift = 127 - (int)((mbits >> 23) & 0xffu);
  const int elo = max(1, 4 - shift), ehi = min(254, 250 - shift);
  float m[PER];
#pragma unroll
  for (int t = 0; t < PER; ++t) m[t] = mean ? __bfloat162float(mean[kvh * D + lane * PER + t]) : 0.f;
  // this lane's slice of the (up to) four unit queries
  float qu[4][PER];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int t = 0; t < PER; ++t) qu[r][t] = qs[r * D + lane * PER + t];
  const T* kbase = k + b * ks_b + hkv * ks_h;
  const float* dbase = dens + kvh * cap;
  for (int64_t w = (int64_t)blockIdx.y * nwarp + warp; w < W; w += (int64_t)gridDim.y * nwarp) {
    // lane 8r (r < R): word of row r and the CSR position of its first bit; the reduction
    // below leaves row r's cosine in lanes 8r .. 8r+7
    uint32_t myword = 0u;
    int64_t mypos = 0;
    if ((lane & 7) == 0 && (lane >> 3) < R) {
      const int r = lane >> 3;
      myword = bits[(row0 + r) * W + w];
      mypos = ptr[row0 + r] + wpre[(row0 + r) * W + w];
    }
    uint32_t uni = myword;
#pragma unroll
    for (int o = 16; o >= 8; o >>= 1) uni |= __shfl_xor_sync(0xffffffffu, uni, o);
    uni = __shfl_sync(0xffffffffu, uni, 0);
    if (!uni) continue;
    // Keys are taken four at a time: their rows are requested together, so that a warp has
    // four independent row loads in flight, then worked on one after the other.
    while (uni) {
      int kb[4];
      float xs[4][PER], dn[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        kb[j] = uni ? __ffs(uni) - 1 : -1;
        uni &= uni - 1;  // 0 stays 0
        if (kb[j] >= 0) {
          lsh_load_lane<T>(kbase + (w * 32 + kb[j]) * ks_s, PER, lane, xs[j]);
          dn[j] = dbase[w * 32 + kb[j]];
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (kb[j] < 0) break;
        const int bit = kb[j];
        const float den = dn[j];
        float x[PER];
        const unsigned int di = (__float_as_uint(den) >> 16) - LSH_DEN_BASE;
        const float* Ud = U + (di < LSH_DEN_TABLES ? di : 0u) * 128;
        float cc[PER];
        bool slow = di >= LSH_DEN_TABLES;
#pragma unroll
        for (int t = 0; t < PER; ++t) {
          cc[t] = mean ? sah_round_to<T>(__fsub_rn(xs[j][t], m[t])) : xs[j][t];
          const uint32_t u = __float_as_uint(cc[t]);
          const unsigned int e = (u >> 23) & 0xffu;
          slow |= (e - (unsigned)elo) > (unsigned)(ehi - elo);
          x[t] = __fmul_rn(__uint_as_float(u & 0xff800000u), Ud[(u >> 16) & 0x7fu]);
        }
        if (__any_sync(0xffffffffu, slow)) {  // rare: zero channels, denormals, an unusual norm
          if (slow) {
#pragma unroll
            for (int t = 0; t < PER; ++t) {
              const unsigned int e = (__float_as_uint(cc[t]) >> 23) & 0xffu;
              if (di >= LSH_DEN_TABLES || (e - (unsigned)elo) > (unsigned)(ehi - elo))
                x[t] = sah_round_to<T>(__fdiv_rn(sah_round_to<T>(__fdiv_rn(cc[t], M)), den));
            }
          }
        }
        // Four dot products at once.  Each row's 32 lane partials combine in the fixed tree
        // (xor 16, 8, 4, 2, 1); the first two levels also sort the rows onto lane groups, so
        // six shuffles serve all four rows and every sum is associated exactly as in a
        // per-row tree.
        float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f;
#pragma unroll
        for (int t = 0; t < PER; ++t) {
          a0 = __fadd_rn(a0, __fmul_rn(qu[0][t], x[t]));
          a1 = __fadd_rn(a1, __fmul_rn(qu[1][t], x[t]));
          a2 = __fadd_rn(a2, __fmul_rn(qu[2][t], x[t]));
          a3 = __fadd_rn(a3, __fmul_rn(qu[3][t], x[t]));
        }
        const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
        const float r0 = __shfl_xor_sync(0xffffffffu, hi16 ? a0 : a2, 16);
        const float r1 = __shfl_xor_sync(0xffffffffu, hi16 ? a1 : a3, 16);
        const float k0 = __fadd_rn(hi16 ? a2 : a0, r0);  // rows 0 / 2
        const float k1 = __fadd_rn(hi16 ? a3 : a1, r1);  // rows 1 / 3
        const float r2 = __shfl_xor_sync(0xffffffffu, hi8 ? k0 : k1, 8);
        float cosv = __fadd_rn(hi8 ? k1 : k0, r2);       // row 2 * bit4 + bit3
        cosv = __fadd_rn(cosv, __shfl_xor_sync(0xffffffffu, cosv, 4));
        cosv = __fadd_rn(cosv, __shfl_xor_sync(0xffffffffu, cosv, 2));
        cosv = __fadd_rn(cosv, __shfl_xor_sync(0xffffffffu, cosv, 1));
        if ((myword >> bit) & 1u) {  // only lanes 8r hold a word
          float c = sah_round_to<T>(cosv);
          c = fminf(fmaxf(c, -1.0f), 1.0f);
          data[mypos + __popc(myword & ((1u << bit) - 1u))] =
              __ushort_as_bfloat16(table[__float_as_uint(c) >> 16]);
        }
      }
    }
  }
}

extern "C" int sah_lsh_prob(const void* keys, int dtype, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                            int B, int Hq, int Sq, int G, int D, const void* mean,
                            const float* norms, const float* dens, int64_t cap,
                            const unsigned int* max_norm_bits, const float* qunit,
                            const uint32_t* bits, const int32_t* wpre, const int64_t* ptr, int64_t W,
                            int K, int L, const uint16_t* table, void* data, int sm_count,
                            void* stream) {
  SAH_REQUIRE(keys && norms && max_norm_bits && qunit && bits && wpre && ptr && data,
              "lsh_prob: null pointer");
  SAH_REQUIRE(D % 32 == 0 && D <= 32 * LSH_MAX_PER_LANE, "lsh_prob: head_dim must be a multiple of 32, <= 256");
  SAH_REQUIRE(G > 0 && Hq % G == 0, "lsh_prob: bad head grouping");
  SAH_REQUIRE(dtype != SAH_BF16 || table != nullptr, "lsh_prob: bf16 needs the probability table");
  const int64_t groups = (int64_t)B * (Hq / G);
  const int R = G * Sq;
  if (sm_count <= 0) sm_count = 148;
  int64_t gy = (W + 7) / 8;
  const int64_t cap_y = ((int64_t)sm_count * 8 + groups - 1) / groups;
  if (gy > cap_y) gy = cap_y;
  if (gy < 1) gy = 1;
  if (gy > 65535) gy = 65535;
  const int q_in_smem = (size_t)R * D * sizeof(float) <= 24 * 1024;
  dim3 grid((unsigned)groups, (unsigned)gy);
  sah_prof_begin(SAH_PROF_LSH_PROB, (cudaStream_t)stream);
  if (dtype == SAH_BF16 && dens != nullptr) {
    // cached key norms (sah_lsh_key_den): one table lookup per channel
    if (R <= 4 && (D == 64 || D == 128 || D == 256)) {
#define LSH_DECODE_LAUNCH(PER)                                                                       \
  lsh_prob_decode_kernel<PER><<<grid, 256, 0, (cudaStream_t)stream>>>(                               \
      reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hq, Sq, G,                     \
      reinterpret_cast<const __nv_bfloat16*>(mean), dens, cap, max_norm_bits, qunit, bits, wpre, ptr, \
      W, table, reinterpret_cast<__nv_bfloat16*>(data))
      if (D == 64) LSH_DECODE_LAUNCH(2);
      else if (D == 128) LSH_DECODE_LAUNCH(4);
      else LSH_DECODE_LAUNCH(8);
      SAH_LAUNCH_CHECK("lsh_prob");
      sah_prof_end(SAH_PROF_LSH_PROB, (cudaStream_t)stream);
      return SAH_OK;
    }
    size_t fsmem = (size_t)LSH_DEN_TABLES * 128 * sizeof(float);
    if (q_in_smem) fsmem += (size_t)R * D * sizeof(float);
    lsh_prob_fast_kernel<<<grid, 256, fsmem, (cudaStream_t)stream>>>(
        reinterpret_cast<const __nv_bfloat16*>(keys), ks_b, ks_h, ks_s, Hq, Sq, G, D,
        reinterpret_cast<const __nv_bfloat16*>(mean), dens, cap, max_norm_bits, qunit, bits, wpre, ptr,
        W, table, q_in_smem, reinterpret_cast<__nv_bfloat16*>(data));
    SAH_LAUNCH_CHECK("lsh_prob");
    sah_prof_end(SAH_PROF_LSH_PROB, (cudaStream_t)stream);
    return SAH_OK;
  }
  size_t smem = 128 * sizeof(float);
  if (q_in_smem) smem += (size_t)R * D * sizeof(float);
  SAH_DISPATCH_DTYPE(dtype, T, {
    lsh_prob_kernel<T><<<grid, 256, smem, (cudaStream_t)stream>>>(
        reinterpret_cast<const T*>(keys), ks_b, ks_h, ks_s, Hq, Sq, G, D,
        reinterpret_cast<const T*>(mean), norms, cap, max_norm_bits, qunit, bits, wpre, ptr, W, K, L,
        table, q_in_smem, reinterpret_cast<T*>(data));
  });
  SAH_LAUNCH_CHECK("lsh_prob");
  sah_prof_end(SAH_PROF_LSH_PROB, (cudaStream_t)stream);
  return SAH_OK;
}
