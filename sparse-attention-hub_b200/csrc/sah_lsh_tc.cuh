// SimHash key signatures on the fifth-generation tensor cores (bfloat16, head dim 128, 8 bits
// per table): the projection of the transformed keys onto the L * 8 hyperplanes
// (magic_pig.py:120-150, :332-372) as a tcgen05 GEMM, with every sign that the tensor core's
// summation order could have changed redone in the fixed order of lsh_key_sign_kernel.
//
//   A  = transformed keys, 128 per tile, [128][144] bf16 (129 channels, zero padded), built by
//        the producer warps from K, the key mean, the key norms and the maximum norm exactly as
//        the fixed-order kernel builds them (every operation rounded to bfloat16), stored
//        K-major in the 128-byte swizzled layout;
//   B  = a chunk of up to 256 hyperplanes, [256][144] bf16, K-major, same layout, resident in
//        shared memory for the life of the CTA (gridDim.y chunks of equal width cover the L * 8
//        columns);
//   D  = A . B^T, [128 keys][256 columns] fp32 in tensor memory, two accumulators so that the
//        epilogue of a tile overlaps the products of the next.
//
// The products are exact in float32 (bf16 x bf16); only the order of the 129 additions differs
// from the fixed-order kernel.  Both sums are within 129 * 2^-24 * sum|x_c p_c| of the exact
// value (the tensor core at least as close), and sum|x_c p_c| <= |x| |p| with |x| <= 1.01 for a
// transformed key, so a projection whose magnitude exceeds tau = 2^-15 * |p| has the same sign in
// both.  The epilogue (one thread per key) shifts the 32 sign
// bits of a group into a word of the key's signature row, takes the smallest magnitude of the
// group, and only where that is within the group's largest tau looks at the columns one by one;
// groups that hold a projection within tau go through a small queue per warp (one global counter
// addition per 64 of them) to a list, and lsh_sign_recheck_kernel recomputes exactly those in the
// fixed order and corrects the bits.  A list that overflows sets a flag, and the caller redoes
// the range with the fixed-order kernel.
//
// What bounds it is the instruction issue of the producers and of the epilogue, not the products
// (51 us of tensor-core time at 8 x 65500 keys x 600 columns).  The producers divide by the
// maximum norm M with one multiplication: for a bfloat16 M and a bfloat16 dividend the quotient
// is never halfway between two bfloat16 numbers (a 9-bit odd significand times that of M would
// have to be an 8-bit one), nor closer than 2^-17 to it, so a float product with 1 / M, 2^-22
// away at most, rounds to the same bfloat16 number; operands near the ends of the range take the
// division (a division per channel, its slow path's branch and the load in front of it in series
// were most of the 1495 us that the kernel took at that size; 629 us with one set of producers that
// branched per row; 546 us with two, which sent every row with a zero to the division -- a few in
// every tile -- and with an epilogue that waited for each group's values in turn; 336 us now, pairs of
// channels in one operation.  The recheck went from 507 over 121 to 51 us).
//
// Every mbarrier wait is bounded (sah_tcgen05.cuh); a wait that runs out sets the error word,
// all roles leave their loops, tensor memory is freed.
#pragma once
#include "sah_tcgen05.cuh"

#define LTC_TILE 128
#define LTC_NCHUNK 256   // hyperplanes per CTA
#define LTC_KSTEPS 9     // 144 = 9 x 16 channels (129 used)
#define LTC_EPI 4        // epilogue warps, one per 32 keys
#define LTC_PROD 8       // producer warps, in two sets that take alternate tiles
#define LTC_THREADS (32 * (LTC_EPI + LTC_PROD + 1))  // and 1 issuing warp
#define LTC_QUEUE 64     // entries of a warp's queue of groups to redo
#define LTC_PLANE 136    // channels of a hyperplane where they are stored one by one
#define LTC_TAU_SCALE 3.0517578125e-05f  // 2^-15

struct LtcCfg {
  static constexpr int A_ATOM = LTC_TILE * 128;    // [128 rows][128 B]: 64 channels
  static constexpr int A_TILE = 3 * A_ATOM;        // channels 0-63, 64-127, 128-191 (128-143 read)
  static constexpr int B_ATOM = LTC_NCHUNK * 128;  // [256 rows][128 B]
  static constexpr int B_OFF = 0;
  static constexpr int A_OFF = 3 * B_ATOM;         // two A tiles
  static constexpr int TAU_OFF = A_OFF + 2 * A_TILE;          // [256] floats
  static constexpr int BAR_OFF = TAU_OFF + LTC_NCHUNK * 4;    // a_full[2] a_empty[2] d_full[2] d_free[2]
  static constexpr int MISC_OFF = BAR_OFF + 64;               // tmem slot, abort word
  static constexpr int GTAU_OFF = MISC_OFF + 16;              // [8] floats: largest tau of a group
  static constexpr int QUEUE_OFF = GTAU_OFF + 32;             // [LTC_EPI][LTC_QUEUE] entries
  static constexpr int SMEM = 1024 + QUEUE_OFF + LTC_EPI * LTC_QUEUE * 16;
};

struct LtcUncertain {
  long long key;      // row of the signature array (bh * cap + s)
  int col0;           // first of the 32 columns of the group
  unsigned int mask;  // columns of the group whose projection was within tau
};

__device__ __forceinline__ void ltc_tmem_ld32(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
      "%29,%30,%31}, [%32];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
// the values of a load may be read after this on the same registers
__device__ __forceinline__ void ltc_tmem_wait(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}

// smallest magnitude of three; NaN if there is one
__device__ __forceinline__ float ltc_minabs3(float a, float b, float c) {
  float d;
  asm("min.NaN.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(fabsf(b)), "f"(fabsf(c)));
  return d;
}

// pairs of floats in one operation, each half rounded as the scalar one is
__device__ __forceinline__ unsigned long long ltc_bits(float2 v) {
  unsigned long long u;
  asm("mov.b64 %0, {%1, %2};" : "=l"(u) : "f"(v.x), "f"(v.y));
  return u;
}
__device__ __forceinline__ float2 ltc_pair(unsigned long long u) {
  float2 v;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(v.x), "=f"(v.y) : "l"(u));
  return v;
}
__device__ __forceinline__ unsigned long long ltc_add2(unsigned long long a, unsigned long long b) {
  unsigned long long c;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}
__device__ __forceinline__ unsigned long long ltc_mul2(unsigned long long a, unsigned long long b) {
  unsigned long long c;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(c) : "l"(a), "l"(b));
  return c;
}

// Grid: (workers, column chunks of `chunk_cols`, a multiple of 32).  Worker w of a chunk takes the tiles w, w + workers, ... of the
// flattened (batch x KV head, key tile) space.
__global__ void __launch_bounds__(LTC_THREADS, 1)
lsh_key_sign_tc_kernel(const __nv_bfloat16* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv,
                       int64_t BH, int64_t s0, int64_t s1, const __nv_bfloat16* __restrict__ mean,
                       const float* __restrict__ norms, const unsigned int* __restrict__ max_bits,
                       const __nv_bfloat16* __restrict__ proj, int L, int chunk_cols, int64_t cap,
                       uint8_t* __restrict__ codes, LtcUncertain* __restrict__ list, int list_cap,
                       int* __restrict__ list_count, int* __restrict__ errflag, __nv_bfloat16* __restrict__ planes) {
  constexpr int D = 128;
  using C = LtcCfg;
  extern __shared__ __align__(1024) unsigned char ltc_raw[];
  const uint32_t raw_s = (uint32_t)__cvta_generic_to_shared(ltc_raw);
  unsigned char* sm = ltc_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
  const uint32_t sm_s = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nbits = L * 8;
  const int LP = lsh_row_pitch<uint8_t>(L);
  const int col_base = blockIdx.y * chunk_cols;
  int ncols = nbits - col_base;               // real columns of this chunk
  if (ncols > chunk_cols) ncols = chunk_cols;
  const uint32_t n_mma = (uint32_t)((ncols + 15) / 16 * 16);
  const int64_t tiles_per_bh = (s1 - s0 + LTC_TILE - 1) / LTC_TILE;
  const int64_t total_tiles = BH * tiles_per_bh;
  const int64_t first = blockIdx.x, stride = gridDim.x;
  const int my_tiles = first < total_tiles ? (int)((total_tiles - first + stride - 1) / stride) : 0;

  const uint32_t bar0 = sm_s + C::BAR_OFF;
  const uint32_t a_full = bar0, a_empty = bar0 + 16, d_full = bar0 + 32, d_free = bar0 + 48;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + C::MISC_OFF);
  volatile int* abort_sm = reinterpret_cast<volatile int*>(sm + C::MISC_OFF + 4);
  float* tau_sm = reinterpret_cast<float*>(sm + C::TAU_OFF);
  float* gtau_sm = reinterpret_cast<float*>(sm + C::GTAU_OFF);

  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      atm_mbar_init(a_full + i * 8, 4);   // one arrival per producer warp
      atm_mbar_init(a_empty + i * 8, 1);  // tcgen05.commit
      atm_mbar_init(d_full + i * 8, 1);   // tcgen05.commit
      atm_mbar_init(d_free + i * 8, LTC_EPI);  // one arrival per epilogue warp
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    *abort_sm = 0;
  }
  if (warp == LTC_EPI + LTC_PROD) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::
                     "r"((uint32_t)__cvta_generic_to_shared(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  // ---- B chunk: row n = hyperplane col_base + n, 144 channels (zero beyond 128 and beyond the
  //      real columns); 16-byte chunk c of row n sits in atom c / 8 at slot (c % 8) ^ (n % 8).
  //      Neighbouring lanes take neighbouring hyperplanes, which adjoin in a row of proj ----
  for (int i = tid; i < LTC_NCHUNK * 24; i += LTC_THREADS) {
    const int n = i % LTC_NCHUNK, c = i / LTC_NCHUNK;  // 24 chunks of 8 channels = 192 channels
    __align__(16) __nv_bfloat16 v[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int ch = c * 8 + e;
      v[e] = (n < ncols && ch <= D) ? proj[(int64_t)ch * nbits + col_base + n] : __float2bfloat16(0.f);
    }
    *reinterpret_cast<uint4*>(sm + C::B_OFF + (c >> 3) * C::B_ATOM + n * 128 + (((c & 7) ^ (n & 7)) << 4)) =
        *reinterpret_cast<const uint4*>(v);
    // the hyperplanes one by one for the kernel behind this one
    if (planes != nullptr && blockIdx.x == 0 && n < ncols && c * 8 < LTC_PLANE)
      *reinterpret_cast<uint4*>(planes + (int64_t)(col_base + n) * LTC_PLANE + c * 8) = *reinterpret_cast<const uint4*>(v);
  }
  // tau of every column: 2^-15 * 1.01 * |p|
  for (int n = tid; n < LTC_NCHUNK; n += LTC_THREADS) {
    float ss = 0.f;
    if (n < ncols) {
#pragma unroll 16
      for (int ch = 0; ch <= D; ++ch) {
        const float p = __bfloat162float(proj[(int64_t)ch * nbits + col_base + n]);
        ss = fmaf(p, p, ss);
      }
    }
    tau_sm[n] = LTC_TAU_SCALE * 1.01f * sqrtf(ss) * 1.0001f;
  }
  // the padding channels of the third atom of both A tiles stay zero for the whole kernel
  for (int i = tid; i < 2 * LTC_TILE * 8; i += LTC_THREADS) {
    const int buf = i / (LTC_TILE * 8), r = (i / 8) % LTC_TILE, c = i % 8;
    *reinterpret_cast<uint4*>(sm + C::A_OFF + buf * C::A_TILE + 2 * C::A_ATOM + r * 128 + (c << 4)) =
        make_uint4(0u, 0u, 0u, 0u);
  }
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  aum_fence_before();
  __syncthreads();
  aum_fence_after();
  const uint32_t tmem = *tmem_slot;
  const float M = __uint_as_float(*max_bits);

  if (warp >= LTC_EPI && warp < LTC_EPI + LTC_PROD) {
    // =========================== producers: transformed keys ===========================
    // 16 lanes cover one key row (8 channels each), two rows per pass, 32 rows per warp.
    // The rows of a set's next tile are requested before its present one is handed over.
    const int pw = (warp - LTC_EPI) & 3, set = (warp - LTC_EPI) >> 2;
    const int my_chunk = lane & 15, my_sub = lane >> 4;
    const float rM = __frcp_rn(M);
    // the multiplication stands for the division only for a bfloat16 M well inside the range
    const bool divide = (__float_as_uint(M) & 0xffffu) != 0u || !(M >= 8.673617e-19f && M <= 1.152921504606847e18f);
    int64_t bh_cur = -1;
    unsigned long long neg_mean[4];
    const unsigned long long rM2 = ltc_bits(make_float2(rM, rM));
    uint4 raw[16];
    auto fetch = [&](int t) {
      const int64_t flat = first + (int64_t)t * stride;
      const int64_t bh = flat / tiles_per_bh;
      const int64_t key0 = s0 + (flat - bh * tiles_per_bh) * LTC_TILE + pw * 32 + my_sub;
      const __nv_bfloat16* kb = k + (bh / Hkv) * ks_b + (bh % Hkv) * ks_h + my_chunk * 8;
#pragma unroll
      for (int it = 0; it < 16; ++it) {
        raw[it] = make_uint4(0u, 0u, 0u, 0u);
        if (key0 + it * 2 < s1) raw[it] = *reinterpret_cast<const uint4*>(kb + (key0 + it * 2) * ks_s);
      }
    };
    if (set < my_tiles) fetch(set);
    for (int t = set; t < my_tiles; t += 2) {
      const int buf = set;
      const int64_t flat = first + (int64_t)t * stride;
      const int64_t bh = flat / tiles_per_bh;
      const int64_t key0 = s0 + (flat - bh * tiles_per_bh) * LTC_TILE;
      if (bh != bh_cur) {
        bh_cur = bh;
        if (mean != nullptr) {
          float m8[8];
          sah_unpack8(*reinterpret_cast<const uint4*>(mean + bh * D + my_chunk * 8), m8);
#pragma unroll
          for (int i = 0; i < 4; ++i) neg_mean[i] = ltc_bits(make_float2(-m8[2 * i], -m8[2 * i + 1]));
        }
      }
      const float nk = key0 + pw * 32 + lane < s1 ? norms[bh * cap + key0 + pw * 32 + lane] : 0.f;
      if (t >= 2 && !aum_wait_warp(a_empty + buf * 8, (uint32_t)(((t >> 1) - 1) & 1), abort_sm, errflag)) break;
      unsigned char* at = sm + C::A_OFF + buf * C::A_TILE;
      auto chunk_at = [&](int r) -> unsigned char* {
        return at + (my_chunk >> 3) * C::A_ATOM + r * 128 + (((my_chunk & 7) ^ (r & 7)) << 4);
      };
      uint32_t slow = 0u;  // rows with an operand that has to be divided
#pragma unroll
      for (int it = 0; it < 16; ++it) {
        const int r = pw * 32 + it * 2 + my_sub;
        uint32_t w[4] = {raw[it].x, raw[it].y, raw[it].z, raw[it].w};
        float smallest = INFINITY;
        float2 x[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
          if (mean != nullptr) {
            x[i] = ltc_pair(ltc_add2(ltc_bits(x[i]), neg_mean[i]));  // x - mean
            const __nv_bfloat162 h = __floats2bfloat162_rn(x[i].x, x[i].y);
            const uint32_t u = *reinterpret_cast<const uint32_t*>(&h);
            x[i] = make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u));
          }
          smallest = ltc_minabs3(smallest, x[i].x, x[i].y);
          const float2 p = ltc_pair(ltc_mul2(ltc_bits(x[i]), rM2));
          const __nv_bfloat162 q = __floats2bfloat162_rn(p.x, p.y);
          w[i] = *reinterpret_cast<const uint32_t*>(&q);
        }
        bool odd = divide;
        if (!(smallest >= 8.673617e-19f)) {  // below 2^-60 the quotient might be denormal; zero stays zero
#pragma unroll
          for (int i = 0; i < 4; ++i)
            odd = odd || !(fabsf(x[i].x) >= 8.673617e-19f || x[i].x == 0.f) ||
                  !(fabsf(x[i].y) >= 8.673617e-19f || x[i].y == 0.f);
        }
        const bool live = key0 + r < s1;
        if (odd && live) slow |= 1u << it;
        *reinterpret_cast<uint4*>(chunk_at(r)) =
            live ? make_uint4(w[0], w[1], w[2], w[3]) : make_uint4(0u, 0u, 0u, 0u);
      }
      if (slow) {  // rare
#pragma unroll 1
        for (int it = 0; it < 16; ++it) {
          if (!((slow >> it) & 1u)) continue;
          const int r = pw * 32 + it * 2 + my_sub;
          const __nv_bfloat16* kr = k + (bh / Hkv) * ks_b + (bh % Hkv) * ks_h + (key0 + r) * ks_s + my_chunk * 8;
          __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(chunk_at(r));
#pragma unroll 1
          for (int e = 0; e < 8; ++e) {
            float x = __bfloat162float(kr[e]);
            if (mean != nullptr)
              x = sah_round_to<__nv_bfloat16>(__fsub_rn(x, __bfloat162float(mean[bh * D + my_chunk * 8 + e])));
            dst[e] = __float2bfloat16_rn(__fdiv_rn(x, M));
          }
        }
      }
      {  // channel 128: the augmentation column (chunk 0 of the third atom), one row per lane
        const int r = pw * 32 + lane;
        const float aug = key0 + r < s1 ? lsh_augment<__nv_bfloat16>(nk, M) : 0.f;
        *reinterpret_cast<__nv_bfloat16*>(at + 2 * C::A_ATOM + r * 128 + ((r & 7) << 4)) = __float2bfloat16_rn(aug);
      }
      if (t + 2 < my_tiles) fetch(t + 2);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      __syncwarp();
      if (lane == 0) aum_arrive(a_full + buf * 8);
    }
  } else if (warp == LTC_EPI + LTC_PROD) {
    // =========================== tensor-core issuer ===========================
    if (lane == 0) {
      const uint32_t idesc = aum_idesc(false, false, n_mma);
      for (int t = 0; t < my_tiles; ++t) {
        const int buf = t & 1;
        if (!aum_wait(a_full + buf * 8, (uint32_t)((t >> 1) & 1), abort_sm, errflag)) break;
        if (t >= 2 && !aum_wait(d_free + buf * 8, (uint32_t)(((t >> 1) - 1) & 1), abort_sm, errflag)) break;
        aum_fence_after();
        const uint32_t a_s = sm_s + C::A_OFF + buf * C::A_TILE, b_s = sm_s + C::B_OFF;
#pragma unroll
        for (int ks = 0; ks < LTC_KSTEPS; ++ks) {
          const uint64_t ad = aum_desc(a_s + (ks >> 2) * C::A_ATOM + (ks & 3) * 32, 0, 1024, 2);
          const uint64_t bd = aum_desc(b_s + (ks >> 2) * C::B_ATOM + (ks & 3) * 32, 0, 1024, 2);
          aum_mma(tmem + buf * LTC_NCHUNK, ad, bd, idesc, ks > 0 ? 1u : 0u);
        }
        aum_commit(d_full + buf * 8);
        aum_commit(a_empty + buf * 8);
      }
    }
    __syncwarp();
  } else {
    // =========================== epilogue: one thread per key ===========================
    const int keyl = tid;  // 0..127
    const uint32_t lane_base = ((uint32_t)(warp * 32)) << 16;
    const int groups = (ncols + 31) / 32;
    LtcUncertain* queue = reinterpret_cast<LtcUncertain*>(sm + C::QUEUE_OFF) + warp * LTC_QUEUE;
    int queued = 0;  // the same in every lane
    auto flush = [&]() {
      if (queued == 0) return;
      int base = 0;
      if (lane == 0) base = atomicAdd(list_count, queued);
      base = __shfl_sync(0xffffffffu, base, 0);
      __syncwarp();
      for (int i = lane; i < queued; i += 32)
        if (base + i < list_cap) list[base + i] = queue[i];
      if (lane == 0 && base + queued > list_cap) atomicExch(errflag, 1);
      __syncwarp();
      queued = 0;
    };
    // largest tau of each of this warp's groups; a group with columns past the end is looked at
    // one by one (a threshold that every magnitude is within)
    for (int gq = 0; gq < groups; ++gq) {
      float g = tau_sm[gq * 32 + lane];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, o));
      if (!(g >= 0.f)) g = INFINITY;  // a NaN among the hyperplanes
      if (lane == 0 && warp == 0) gtau_sm[gq] = gq * 32 + 32 <= ncols ? g : INFINITY;
    }
    asm volatile("bar.sync 1, %0;\n" ::"n"(LTC_EPI * 32) : "memory");
    for (int t = 0; t < my_tiles; ++t) {
      const int buf = t & 1;
      const int64_t flat = first + (int64_t)t * stride;
      const int64_t bh = flat / tiles_per_bh;
      const int64_t s = s0 + (flat - bh * tiles_per_bh) * LTC_TILE + keyl;
      if (!aum_wait_warp(d_full + buf * 8, (uint32_t)((t >> 1) & 1), abort_sm, errflag)) break;
      aum_fence_after();
      const int64_t row = bh * cap + s;
      auto group = [&](int gq, const uint32_t* acc) {
        uint32_t neg[4] = {0u, 0u, 0u, 0u};
        float mn[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) mn[q] = fabsf(__uint_as_float(acc[q]));
#pragma unroll
        for (int i = 7; i >= 0; --i)
#pragma unroll
          for (int q = 0; q < 4; ++q) neg[q] = __funnelshift_l(acc[q * 8 + i], neg[q], 1);
#pragma unroll
        for (int i = 4; i < 32; i += 2)
          mn[(i >> 1) & 3] = ltc_minabs3(mn[(i >> 1) & 3], __uint_as_float(acc[i]), __uint_as_float(acc[i + 1]));
        const float smallest = ltc_minabs3(ltc_minabs3(mn[0], mn[1], mn[2]), mn[3], mn[3]);
        uint32_t bits = ~(neg[0] | (neg[1] << 8) | (neg[2] << 16) | (neg[3] << 24));
        const int c0 = col_base + gq * 32;
        const int valid = nbits - c0;  // real columns in this group
        const uint32_t vm = valid < 32 ? (1u << valid) - 1u : 0xffffffffu;
        bits &= vm;
        if (s < s1) {
          // bit j of table l is column 8 l + j: the 32 columns of the group are 4 code bytes in order
          const int byte0 = c0 >> 3;
          if (byte0 + 4 <= LP) {
            *reinterpret_cast<uint32_t*>(codes + row * LP + byte0) = bits;
          } else {
            for (int bq = 0; bq < 4 && byte0 + bq < LP; ++bq) codes[row * LP + byte0 + bq] = (uint8_t)(bits >> (8 * bq));
          }
        }
        const bool look = !(smallest > gtau_sm[gq]) && s < s1;  // also where there is a NaN
        if (__any_sync(0xffffffffu, look)) {
          uint32_t unsure = 0u;
          if (look) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              unsure |= (fabsf(__uint_as_float(acc[i])) > tau_sm[gq * 32 + i] ? 0u : 1u) << i;
            unsure &= vm;
          }
          const uint32_t who = __ballot_sync(0xffffffffu, unsure != 0u);
          if (who) {
            if (queued + __popc(who) > LTC_QUEUE) flush();
            if (unsure) {
              LtcUncertain u;
              u.key = row; u.col0 = c0; u.mask = unsure;
              queue[queued + __popc(who & ((1u << lane) - 1u))] = u;
            }
            queued += __popc(who);
            __syncwarp();
          }
        }
      };
      // the next group's values are on their way while a group is looked at
      uint32_t va[32], vb[32];
      const uint32_t cols = tmem + lane_base + buf * LTC_NCHUNK;
      ltc_tmem_ld32(cols, va);
#pragma unroll 1
      for (int gq = 0; gq < groups; gq += 2) {
        ltc_tmem_wait(va);
        if (gq + 1 < groups) ltc_tmem_ld32(cols + (gq + 1) * 32, vb);
        group(gq, va);
        if (gq + 1 >= groups) break;
        ltc_tmem_wait(vb);
        if (gq + 2 < groups) ltc_tmem_ld32(cols + (gq + 2) * 32, va);
        group(gq + 1, vb);
      }
      // the row's padding bytes beyond the last table (the last chunk owns them)
      if (blockIdx.y == gridDim.y - 1 && s < s1)
        for (int bq = (col_base >> 3) + groups * 4; bq < LP; bq += 4)
          *reinterpret_cast<uint32_t*>(codes + row * LP + bq) = 0u;
      aum_fence_before();
      __syncwarp();
      if (lane == 0) aum_arrive(d_free + buf * 8);
    }
    flush();
  }
  aum_fence_before();
  __syncthreads();
  if (warp == LTC_EPI + LTC_PROD) {
    aum_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
  }
}

// The flagged columns in the fixed order of lsh_key_sign_kernel (single float32 accumulator,
// channels ascending): sets or clears their bits.  A warp takes up to 32 list entries at a time, fewer
// where that spreads the list over all warps (a list of 2700 entries 48 -> 10 us, 87 thousand 119 -> 102).  It
// forms the 129 products of an entry together (coalesced row reads, four channels per lane) and
// leaves them in shared memory; then lane j adds up those of entry j in order, all 32 chains at
// once (one entry per warp and a chain of dependent global loads before: 507 us for 88 thousand
// entries).  Entries with several flagged columns, a few per thousand, take more rounds.  The
// bits of one signature word may be corrected by several lanes: atomics.
#define LTC_RC_WARPS 4
#define LTC_RC_PITCH 129  // odd: the lanes' rows start in different banks
#define LTC_RC_SMEM (LTC_RC_WARPS * 32 * LTC_RC_PITCH * (int)sizeof(float))
__global__ void __launch_bounds__(LTC_RC_WARPS * 32)
lsh_sign_recheck_kernel(const __nv_bfloat16* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s, int Hkv,
                        const __nv_bfloat16* __restrict__ mean, const float* __restrict__ norms,
                        const unsigned int* __restrict__ max_bits, const __nv_bfloat16* __restrict__ proj, int L,
                        int64_t cap, uint8_t* __restrict__ codes, const LtcUncertain* __restrict__ list,
                        int list_cap, const int* __restrict__ list_count,
                        const __nv_bfloat16* __restrict__ planes) {
  constexpr int D = 128;
  extern __shared__ float ltc_prod[];  // [LTC_RC_WARPS][32][LTC_RC_PITCH]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* prod = ltc_prod + warp * 32 * LTC_RC_PITCH;
  const int64_t wid = (int64_t)blockIdx.x * LTC_RC_WARPS + warp;
  const int64_t nwarps = (int64_t)gridDim.x * LTC_RC_WARPS;
  int n = *list_count;
  if (n > list_cap) n = list_cap;
  const int nbits = L * 8;
  const int LP = lsh_row_pitch<uint8_t>(L);
  const float M = __uint_as_float(*max_bits);
  const int64_t rounds = (n + nwarps * 32 - 1) / (nwarps * 32);
  const int per = n > 0 ? (int)((n + nwarps * rounds - 1) / (nwarps * rounds)) : 32;  // entries at a time
  // as in the kernel above: a product with 1 / M stands for the division of a number that is not tiny
  const float rM = __frcp_rn(M);
  const bool divide = (__float_as_uint(M) & 0xffffu) != 0u || !(M >= 8.673617e-19f && M <= 1.152921504606847e18f);
  for (int64_t e0 = wid * per; e0 < n; e0 += nwarps * per) {
    LtcUncertain u;
    u.key = 0; u.col0 = 0; u.mask = 0u;
    if (lane < per && e0 + lane < n) u = list[e0 + lane];
    const int64_t bh_l = u.key / cap, s_l = u.key - bh_l * cap;
    const float aug_l = u.mask ? lsh_augment<__nv_bfloat16>(norms[u.key], M) : 0.f;
    while (__any_sync(0xffffffffu, u.mask != 0u)) {
      const int col_l = u.mask ? u.col0 + __ffs(u.mask) - 1 : -1;
#pragma unroll 4
      for (int j = 0; j < per; ++j) {
        const int col = __shfl_sync(0xffffffffu, col_l, j);
        const int64_t bh = __shfl_sync(0xffffffffu, bh_l, j), s = __shfl_sync(0xffffffffu, s_l, j);
        if (col >= 0) {
          const uint2 kr = *reinterpret_cast<const uint2*>(k + (bh / Hkv) * ks_b + (bh % Hkv) * ks_h + s * ks_s + lane * 4);
          float x[4] = {__uint_as_float(kr.x << 16), __uint_as_float(kr.x & 0xffff0000u),
                        __uint_as_float(kr.y << 16), __uint_as_float(kr.y & 0xffff0000u)};
          if (mean != nullptr) {
            const uint2 mr = *reinterpret_cast<const uint2*>(mean + bh * D + lane * 4);
            const float m[4] = {__uint_as_float(mr.x << 16), __uint_as_float(mr.x & 0xffff0000u),
                                __uint_as_float(mr.y << 16), __uint_as_float(mr.y & 0xffff0000u)};
#pragma unroll
            for (int c = 0; c < 4; ++c) x[c] = sah_round_to<__nv_bfloat16>(__fsub_rn(x[c], m[c]));
          }
          float p[4];
          if (planes != nullptr) {
            const uint2 pr = *reinterpret_cast<const uint2*>(planes + (int64_t)col * LTC_PLANE + lane * 4);
            p[0] = __uint_as_float(pr.x << 16), p[1] = __uint_as_float(pr.x & 0xffff0000u);
            p[2] = __uint_as_float(pr.y << 16), p[3] = __uint_as_float(pr.y & 0xffff0000u);
          } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) p[c] = __bfloat162float(proj[(int64_t)(lane * 4 + c) * nbits + col]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const float v = sah_round_to<__nv_bfloat16>(
                !divide && (fabsf(x[c]) >= 8.673617e-19f || x[c] == 0.f) ? __fmul_rn(x[c], rM) : __fdiv_rn(x[c], M));
            prod[j * LTC_RC_PITCH + c * 32 + lane] =  // channel ch at (ch % 4) * 32 + ch / 4
                __fmul_rn(v, p[c]);
          }
        }
      }
      if (col_l >= 0)
        prod[lane * LTC_RC_PITCH + D] = __fmul_rn(aug_l, __bfloat162float(proj[(int64_t)D * nbits + col_l]));
      __syncwarp();
      if (col_l >= 0) {
        float acc = 0.f;
#pragma unroll 8
        for (int c = 0; c < D; ++c) acc = __fadd_rn(acc, prod[lane * LTC_RC_PITCH + (c & 3) * 32 + (c >> 2)]);
        acc = __fadd_rn(acc, prod[lane * LTC_RC_PITCH + D]);
        // the code byte of column col is byte col / 8 of the row; its 32-bit word is aligned
        // (rows are multiples of 16 bytes)
        const int64_t byte = u.key * LP + (col_l >> 3);
        unsigned int* word = reinterpret_cast<unsigned int*>(codes + (byte & ~3ll));
        const unsigned int bit = 1u << (((int)(byte & 3) << 3) + (col_l & 7));
        if (acc > 0.f) atomicOr(word, bit);
        else atomicAnd(word, ~bit);
        u.mask &= u.mask - 1u;
      }
      __syncwarp();
    }
  }
}
