// k-means assignment of PQCache on the fifth-generation tensor cores (bfloat16 keys, sub-vectors
// of 8 channels, 16..256 centroids): the distance contraction of kmeans_batched
// (utils/pq_utils.py:220-257) as a tcgen05 product, with the argmin decided by the fixed-order
// distance of pq_assign_kernel among the centroids that the product cannot tell apart.
//
//   Per (batch, KV head, sub-vector) group and tile of 128 keys:
//     A = [128 keys][32]: the key's 8 channels three times, then 1 1 1 0 ...
//     B = [n_cent][32]: the float32 centroid split into three bfloat16 numbers (24 bits, so the
//         split is exact: high, middle and low parts in columns 0-7, 8-15, 16-23), then
//         -|c|^2 / 2 split the same way,
//   so that two tcgen05.mma (K = 16) give a_c = x . c - |c|^2 / 2 = (|x|^2 - distance) / 2 and the
//   nearest centroid is the largest a_c.  One thread per key reads its row of a_c from tensor
//   memory once, as a matrix of 16 columns, and keeps the largest value of every matrix row and of
//   every matrix column: half an instruction per value each (three-operand maximum).  The overall
//   maximum lies where a row's and a column's meet; a centroid within E of it shows in both.  One row
//   and one column within E: that centroid is the answer.  Otherwise the fixed-order float32
//   distance (dimensions ascending, (x - c)^2 rounded, then added) of all centroids where such rows
//   and columns meet, first minimum wins, as torch.argmin does.
//   Equal centroids (of equal keys, of channels that are 0) tie at every key, and their rows and columns meet nearly
//   everywhere: only the lowest of them can be the answer, so the columns of the others are put below every
//   centroid.  8 KV heads x 65472 keys, 16 of them distinct, 5.57 -> 0.25 ms, a fifth of the centroids one bit off
//   5.46 -> 0.38 ms; half of the sub-vectors 0 6.3 -> 0.25 ms; all different 0.25 ms, of which finding that out is 7 us.
//   E = 2^-16 (|x|^2 + max_c |c|^2).  A float32 sum of 27 exact products, in whatever order and
//   even truncated, is within 27 * 2^-23 (|x||c| + |c|^2 / 2) <= 2^-18.2 (|x|^2 + |c|^2) of the
//   exact one; the fixed-order distance is within 10 * 2^-24 * 2 (|x|^2 + |c|^2) <= 2^-19.6 (...)
//   of the exact one and |c|^2 within 2^-21 |c|^2.  Two centroids whose exact distances are
//   ordered the other way round therefore differ by less than 0.6 E in a_c: the fixed-order argmin
//   is always among the candidates, and the codes equal pq_assign_kernel's bit for bit.
//
// Bound: the vector instructions of the epilogue, 1.25 per (key, centroid) on the 16-lane ALU pipe.
// 8 KV heads x 65472 keys x 16 sub-vectors x 256 centroids are 2.1e9 pairs, 0.15 ms at that rate;
// measured 0.24 ms.  With the row read twice (maximum, then the sign of a_c - (max - E) shifted into
// a bit mask, 2.5 instructions per pair) and the product issued by a thread of the epilogue behind
// a barrier of its group it took 0.46 ms.  The product in halves of 128 columns, each handed back by
// itself, takes 0.26 ms, two products under way 0.31 ms: what remains are instructions, not waits.
//
// One CTA of 320 threads per SM holding all of tensor memory: two groups of four warps, each with
// an accumulator of 256 columns and an A tile of its own, and a warp per group that issues its
// products.  A group writes the A rows of its next product as soon as the present one is complete
// and hands the accumulator back when its last columns are in registers, so that the next product
// runs behind the rest of the epilogue and behind the other group's.  A CTA carries NS neighbouring
// sub-vectors (a key's 64 contiguous bytes for NS = 4: whole sectors, and one 4-byte store of codes)
// and a contiguous share of the flattened (sub-vector block, key tile) space, cut evenly over the
// SMs; the B tiles are rebuilt when the share crosses into another block.  The mbarrier waits are
// bounded; when one runs out the error word is set, and the threads walk through their remaining
// tiles without working on them.
#pragma once
#include "sah_tcgen05.cuh"

#define PTC_TILE 128
#define PTC_SLOT_BITS 10
#define PTC_SLOTS (1 << PTC_SLOT_BITS)  // where the lowest of equal centroids is noted
#define PTC_SLOTS2 256                  // ... of those whose slot a lower one of another value has
#define PTC_THREADS 320  // two groups of four warps, and an issuing warp for each

template <int NS>
struct PtcCfg {
  static constexpr int A_OFF = 0;                                // two groups' [128 rows][128 B], first 64 B used
  static constexpr int B_OFF = 2 * PTC_TILE * 128;               // NS x [256 rows][128 B], first 64 B used
  static constexpr int CENT_OFF = B_OFF + NS * 256 * 128;        // NS x float32 [256][8]
  static constexpr int FIRST_OFF = CENT_OFF + NS * 256 * 8 * 4;    // lowest centroids of the slots
  static constexpr int MISC_OFF = FIRST_OFF + NS * (PTC_SLOTS + PTC_SLOTS2) * 4;  // max |c|^2 per sub-vector, mbarriers, slot, abort
  static constexpr int NEED = 1024 + MISC_OFF + 128;
  // never less than half of an SM's shared memory: one CTA per SM, it holds all of tensor memory
  static constexpr int SMEM = NEED > 120 * 1024 ? NEED : 120 * 1024;
};

// 32 consecutive columns of this thread's lane; the values may be read after ptc_tmem_wait on
// the same registers
__device__ __forceinline__ void ptc_tmem_ld32(uint32_t taddr, uint32_t* r) {
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
__device__ __forceinline__ void ptc_tmem_wait(uint32_t* r) {
  asm volatile("tcgen05.wait::ld.sync.aligned;\n"
               : "+r"(r[0]), "+r"(r[1]), "+r"(r[2]), "+r"(r[3]), "+r"(r[4]), "+r"(r[5]), "+r"(r[6]), "+r"(r[7]),
                 "+r"(r[8]), "+r"(r[9]), "+r"(r[10]), "+r"(r[11]), "+r"(r[12]), "+r"(r[13]), "+r"(r[14]),
                 "+r"(r[15]), "+r"(r[16]), "+r"(r[17]), "+r"(r[18]), "+r"(r[19]), "+r"(r[20]), "+r"(r[21]),
                 "+r"(r[22]), "+r"(r[23]), "+r"(r[24]), "+r"(r[25]), "+r"(r[26]), "+r"(r[27]), "+r"(r[28]),
                 "+r"(r[29]), "+r"(r[30]), "+r"(r[31])
               :
               : "memory");
}
// the largest of three (a NaN operand is ignored)
__device__ __forceinline__ float ptc_max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;\n" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
// v as three bfloat16 numbers whose sum is v
__device__ __forceinline__ void ptc_split3(float v, __nv_bfloat16* h, __nv_bfloat16* m, __nv_bfloat16* l) {
  *h = __float2bfloat16_rn(v);
  const float r1 = __fsub_rn(v, __bfloat162float(*h));
  *m = __float2bfloat16_rn(r1);
  *l = __float2bfloat16_rn(__fsub_rn(r1, __bfloat162float(*m)));
}

// by which equal centroids of 8 floats are found (bits 22 to 31, then 7 to 14)
__device__ __forceinline__ unsigned int ptc_hash(const float* c) {
  const uint4 a = reinterpret_cast<const uint4*>(c)[0], b = reinterpret_cast<const uint4*>(c)[1];
  const unsigned int v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
  unsigned int h = 0u;
#pragma unroll
  for (int d = 0; d < 8; ++d) h += v[d] * (0x9e3779b1u + 0x3c6ef372u * d);  // odd factors, terms that do not wait for one another
  return (h ^ (h >> 16)) * 0x85ebca6bu;
}

// 32 columns of an accumulator: two matrix rows of 16
__device__ __forceinline__ void ptc_fold(const uint32_t* v, float* row, float* col) {
  auto f = [&](int i) { return __uint_as_float(v[i]); };
#pragma unroll
  for (int q = 0; q < 16; ++q) col[q] = ptc_max3(col[q], f(q), f(16 + q));
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int o = 16 * h;
    float a = ptc_max3(f(o), f(o + 1), f(o + 2)), b = ptc_max3(f(o + 3), f(o + 4), f(o + 5));
    a = ptc_max3(a, f(o + 6), f(o + 7)), b = ptc_max3(b, f(o + 8), f(o + 9));
    a = ptc_max3(a, f(o + 10), f(o + 11)), b = ptc_max3(b, f(o + 12), f(o + 13));
    row[h] = fmaxf(ptc_max3(a, f(o + 14), f(o + 15)), b);
  }
}
// bit i: value i is not below thr (or one of the two is NaN)
template <int N>
__device__ __forceinline__ uint32_t ptc_near(const float* v, float thr) {
  uint32_t m = 0u;
#pragma unroll
  for (int i = N - 1; i >= 0; --i) m = __funnelshift_l(__float_as_uint(__fsub_rn(v[i], thr)), m, 1);
  return ~m & (N == 32 ? 0xffffffffu : (1u << (N & 31)) - 1u);
}

// NB: blocks of 32 accumulator columns (n_cent <= 32 NB; the columns past n_cent hold -inf)
template <int NS, int NB>
__global__ void __launch_bounds__(PTC_THREADS, 1)
pq_assign_tc_kernel(const __nv_bfloat16* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int Hkv,
                    int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub, int n_cent,
                    int64_t n_blocks, const float* __restrict__ centroids, uint8_t* __restrict__ codes,
                    int64_t cap, int* __restrict__ errflag, const int* __restrict__ done) {
  if (done && *done) return;  // nothing allocated yet
  constexpr int SD = 8, NC = 32 * NB;
  using C = PtcCfg<NS>;
  extern __shared__ __align__(1024) unsigned char ptc_raw[];
  const uint32_t raw_s = (uint32_t)__cvta_generic_to_shared(ptc_raw);
  unsigned char* sm = ptc_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
  const uint32_t sm_s = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool issuer = warp >= 8;
  const int wg = issuer ? warp - 8 : warp >> 2, keyl = tid & 127;  // group of four warps, key of its tile
  float* cent_sm = reinterpret_cast<float*>(sm + C::CENT_OFF);
  unsigned int* first_sm = reinterpret_cast<unsigned int*>(sm + C::FIRST_OFF);
  unsigned int* second_sm = first_sm + NS * PTC_SLOTS;
  unsigned int* cmax_sm = reinterpret_cast<unsigned int*>(sm + C::MISC_OFF);  // [NS], float bits
  const uint32_t full = sm_s + C::MISC_OFF + 32 + wg * 8;   // the group's product is complete
  const uint32_t ready = sm_s + C::MISC_OFF + 48 + wg * 8;  // its A rows are written, its accumulator is read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + C::MISC_OFF + 64);
  volatile int* abort_sm = reinterpret_cast<volatile int*>(sm + C::MISC_OFF + 68);

  if (tid == 0) {
    for (int g = 0; g < 2; ++g) {
      atm_mbar_init(sm_s + C::MISC_OFF + 32 + g * 8, 1);
      atm_mbar_init(sm_s + C::MISC_OFF + 48 + g * 8, 4);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    *abort_sm = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::
                     "r"((uint32_t)__cvta_generic_to_shared(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  unsigned char* arow = sm + C::A_OFF + wg * (PTC_TILE * 128) + keyl * 128;
  if (!issuer) {  // chunk 3 of an A row (the factors of -|c|^2 / 2) never changes
    const uint32_t one2 = 0x3f803f80u;
    *reinterpret_cast<uint4*>(arow + ((3 ^ (keyl & 7)) << 4)) = make_uint4(one2, 0x3f80u, 0u, 0u);
  }
  aum_fence_before();
  __syncthreads();
  aum_fence_after();
  const uint32_t tmem = *tmem_slot + wg * 256;
  const uint32_t tmem_row = tmem + (((uint32_t)((warp & 3) * 32)) << 16);
  const uint32_t idesc = aum_idesc(false, false, (uint32_t)NC);
  const uint32_t a_s = sm_s + C::A_OFF + wg * (PTC_TILE * 128);

  const int64_t n_tiles = (key_end - key_begin + PTC_TILE - 1) / PTC_TILE;
  const int64_t total = n_blocks * n_tiles;
  int64_t it = total * blockIdx.x / gridDim.x;
  const int64_t it_end = total * (blockIdx.x + 1) / gridDim.x;
  uint32_t phase = 0;
  while (it < it_end) {
    // ---- one block of NS sub-vectors: float32 centroids and the B tiles ----
    const int64_t blk = it / n_tiles;
    const int sub0 = (int)(blk % (n_sub / NS)) * NS;
    const int64_t bk = blk / (n_sub / NS);
    const __nv_bfloat16* xb = x + (bk / Hkv) * xs_b + (bk % Hkv) * xs_h + sub0 * SD;
    __syncthreads();  // both groups are done with the previous block
    if (tid < NS) cmax_sm[tid] = 0u;
    for (int i = tid; i < NS * (PTC_SLOTS + PTC_SLOTS2); i += PTC_THREADS) first_sm[i] = 256u;
    __syncthreads();
    for (int i = tid; i < NS * NC; i += PTC_THREADS) {
      const int s = i / NC, c = i - s * NC;
      __align__(16) __nv_bfloat16 hi[8], mi[8], lo[8], nn[8];
      float n2 = 0.f;
#pragma unroll
      for (int d = 0; d < SD; ++d) {
        const float v = c < n_cent ? centroids[((bk * n_sub + sub0 + s) * n_cent + c) * SD + d] : 0.f;
        cent_sm[(s * 256 + c) * SD + d] = v;
        n2 = __fadd_rn(n2, __fmul_rn(v, v));
        ptc_split3(v, hi + d, mi + d, lo + d);
        nn[d] = __float2bfloat16_rn(0.f);
      }
      if (c < n_cent) ptc_split3(-0.5f * n2, nn, nn + 1, nn + 2);
      else nn[0] = __float2bfloat16_rn(-INFINITY);  // below every centroid, however far out those lie
      if (c < n_cent) atomicMin(first_sm + s * PTC_SLOTS + (ptc_hash(cent_sm + (s * 256 + c) * SD) >> (32 - PTC_SLOT_BITS)), (unsigned int)c);
      // a NaN or infinite norm makes the margin NaN or infinite: every centroid is then measured
      if (c < n_cent) atomicMax(cmax_sm + s, __float_as_uint(n2));
      unsigned char* row = sm + C::B_OFF + s * (256 * 128) + c * 128;
      *reinterpret_cast<uint4*>(row + ((0 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(hi);
      *reinterpret_cast<uint4*>(row + ((1 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(mi);
      *reinterpret_cast<uint4*>(row + ((2 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(lo);
      *reinterpret_cast<uint4*>(row + ((3 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(nn);
    }
    __syncthreads();
    // copies of a lower centroid go below every centroid too; the lowest of others that hold their slot are looked up
    // a second time among those
    auto copy_of = [&](int s, int c, int f) {
      if (f >= c) return false;
      const uint4 *own = reinterpret_cast<const uint4*>(cent_sm + (s * 256 + c) * SD),
                  *other = reinterpret_cast<const uint4*>(cent_sm + (s * 256 + f) * SD);
      const uint4 a0 = own[0], a1 = own[1], b0 = other[0], b1 = other[1];
      if (a0.x != b0.x || a0.y != b0.y || a0.z != b0.z || a0.w != b0.w || a1.x != b1.x || a1.y != b1.y || a1.z != b1.z ||
          a1.w != b1.w)
        return false;
      *reinterpret_cast<uint4*>(sm + C::B_OFF + s * (256 * 128) + c * 128 + ((3 ^ (c & 7)) << 4)) = make_uint4(0xff80u, 0u, 0u, 0u);
      return true;
    };
    uint32_t again = 0u;
    int m = 0;
    for (int i = tid; i < NS * NC; i += PTC_THREADS, ++m) {
      const int s = i / NC, c = i - s * NC;
      if (c >= n_cent) continue;
      const unsigned int bits = ptc_hash(cent_sm + (s * 256 + c) * SD);
      const int f = (int)first_sm[s * PTC_SLOTS + (bits >> (32 - PTC_SLOT_BITS))];
      if (f == c || copy_of(s, c, f)) continue;
      again |= 1u << m;
      atomicMin(second_sm + s * PTC_SLOTS2 + ((bits >> 7) & (PTC_SLOTS2 - 1)), (unsigned int)c);
    }
    __syncthreads();
    for (; again; again &= again - 1) {
      const int i = tid + (__ffs(again) - 1) * PTC_THREADS, s = i / NC, c = i - s * NC;
      copy_of(s, c, (int)second_sm[s * PTC_SLOTS2 + ((ptc_hash(cent_sm + (s * 256 + c) * SD) >> 7) & (PTC_SLOTS2 - 1))]);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    const int64_t seg_end = (blk + 1) * n_tiles < it_end ? (blk + 1) * n_tiles : it_end;
    if (issuer) {
      int left = it + wg < seg_end ? (int)((seg_end - it - wg + 1) >> 1) : 0;
      for (; left > 0; --left) {
#pragma unroll 1
        for (int s = 0; s < NS; ++s) {
          const bool ok = aum_wait_warp(ready, phase, abort_sm, errflag);
          phase ^= 1u;
          if (ok && lane == 0) {
            aum_fence_after();
            const uint32_t b_s = sm_s + C::B_OFF + s * (256 * 128);
            aum_mma(tmem, aum_desc(a_s, 0, 1024, 2), aum_desc(b_s, 0, 1024, 2), idesc, 0u);
            aum_mma(tmem, aum_desc(a_s + 32, 0, 1024, 2), aum_desc(b_s + 32, 0, 1024, 2), idesc, 1u);
            aum_commit(full);
          }
          __syncwarp();
        }
      }
      it = seg_end;
      continue;
    }
    const int my_tiles = it + wg < seg_end ? (int)((seg_end - it - wg + 1) >> 1) : 0;
    const int64_t j_first = key_begin + (it + wg - blk * n_tiles) * PTC_TILE + keyl;
    const int64_t keys_left = key_end - j_first;
    // tiles of this thread's share in which its key exists
    const int have = keys_left <= 0 ? 0 : (int)min((int64_t)my_tiles, (keys_left + 2 * PTC_TILE - 1) / (2 * PTC_TILE));
    const __nv_bfloat16* xp = xb + j_first * xs_s;   // its row in the tile that is fetched next
    int ft = 0, fs = 0;
    // the 16 bytes of its next sub-vector; all but the first of a key come out of L1
    auto fetch = [&] {
      const uint4 r = ft < have ? *reinterpret_cast<const uint4*>(xp + fs * SD) : make_uint4(0u, 0u, 0u, 0u);
      if (++fs == NS) {
        fs = 0;
        ++ft;
        xp += 2 * PTC_TILE * xs_s;
      }
      return r;
    };
    uint4 rw = fetch();  // the present product's
    uint4 rn = fetch();  // the next one's
    auto put_a = [&](const uint4& rw) {
      *reinterpret_cast<uint4*>(arow + ((0 ^ (keyl & 7)) << 4)) = rw;
      *reinterpret_cast<uint4*>(arow + ((1 ^ (keyl & 7)) << 4)) = rw;
      *reinterpret_cast<uint4*>(arow + ((2 ^ (keyl & 7)) << 4)) = rw;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    };
    auto hand_over = [&] {
      aum_fence_before();
      __syncwarp();
      if (lane == 0) aum_arrive(ready);
    };
    if (my_tiles > 0) {
      put_a(rw);
      hand_over();
    }
    uint8_t* dst = codes + (bk * cap + (j_first - init_offset)) * n_sub + sub0;
#pragma unroll 1
    for (int t = 0; t < my_tiles; ++t) {
      uint32_t packed = 0u;
#pragma unroll 1
      for (int s = 0; s < NS; ++s) {
        const bool more = s + 1 < NS || t + 1 < my_tiles;
        const uint4 rnn = fetch();
        float x2 = 0.f;
        {
          float xv[SD];
          sah_unpack8(rw, xv);
#pragma unroll
          for (int d = 0; d < SD; ++d) x2 = fmaf(xv[d], xv[d], x2);
        }
        const float margin = 1.52587890625e-05f * (x2 + __uint_as_float(cmax_sm[s]));  // E
        const bool ok = aum_wait_warp(full, phase, abort_sm, errflag);
        phase ^= 1u;
        if (!ok) continue;
        aum_fence_after();
        uint32_t va[32], vb[32];
        float row[2 * NB], col[16];
        ptc_tmem_ld32(tmem_row, va);
        if (more) put_a(rn);  // the product has read the rows before
#pragma unroll
        for (int q = 0; q < 16; ++q) col[q] = -INFINITY;
#pragma unroll
        for (int gq = 0; gq < NB; gq += 2) {
          ptc_tmem_wait(va);
          if (NB > 1) ptc_tmem_ld32(tmem_row + (gq + 1) * 32, vb);
          else if (more) hand_over();
          ptc_fold(va, row + 2 * gq, col);
          if (NB > 1) {
            ptc_tmem_wait(vb);
            if (gq + 2 < NB) ptc_tmem_ld32(tmem_row + (gq + 2) * 32, va);
            else if (more) hand_over();
            ptc_fold(vb, row + 2 * gq + 2, col);
          }
        }
        float top = fmaxf(col[0], col[1]);
#pragma unroll
        for (int q = 2; q < 16; q += 2) top = ptc_max3(top, col[q], col[q + 1]);
        const float thr = __fsub_rn(top, margin);
        uint32_t rows = ptc_near<2 * NB>(row, thr);
        const uint32_t cols = ptc_near<16>(col, thr);
        int arg;
        if (__popc(rows) == 1 && __popc(cols) == 1) {
          arg = (__ffs(rows) - 1) * 16 + __ffs(cols) - 1;
        } else {
          float best = INFINITY;
          arg = 0;
          uint4 r = rw;  // unpacked anew: the channels are not to stay in registers through the fold
          asm volatile("" : "+r"(r.x), "+r"(r.y), "+r"(r.z), "+r"(r.w));
          float xv[SD];
          sah_unpack8(r, xv);
#pragma unroll 1
          for (; rows; rows &= rows - 1) {  // ascending c: the first minimum wins
            const int c0 = (__ffs(rows) - 1) * 16;
#pragma unroll 1
            for (uint32_t w = cols; w; w &= w - 1) {
              const int c = c0 + __ffs(w) - 1;
              if (c < n_cent) {
                const float dist = pq_dist(xv, cent_sm + (s * 256 + c) * SD, SD);
                if (dist < best) { best = dist; arg = c; }
              }
            }
          }
        }
        packed |= (uint32_t)arg << (8 * s);
        rw = rn;
        rn = rnn;
      }
      if (t < have) {
        if (NS == 4) *reinterpret_cast<uint32_t*>(dst) = packed;
        else *dst = (uint8_t)packed;
      }
      dst += (int64_t)(2 * PTC_TILE) * n_sub;
    }
    it = seg_end;
  }
  aum_fence_before();
  __syncthreads();
  if (warp == 0) {
    aum_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(*tmem_slot), "r"(512));
  }
}
