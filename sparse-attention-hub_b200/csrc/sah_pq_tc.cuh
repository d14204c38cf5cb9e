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
//   memory twice: first the maximum (three-operand maximum: half an instruction per value), then
//   the sign of a_c - (max - E) shifted into a bit mask (an addition and a funnel shift per
//   value).  One bit set: that is the answer.  Several: the fixed-order float32 distance
//   (dimensions ascending, (x - c)^2 rounded, then added) of those, first minimum wins, as
//   torch.argmin does.
//   E = 2^-16 (|x|^2 + max_c |c|^2).  A float32 sum of 27 exact products, in whatever order and
//   even truncated, is within 27 * 2^-23 (|x||c| + |c|^2 / 2) <= 2^-18.2 (|x|^2 + |c|^2) of the
//   exact one; the fixed-order distance is within 10 * 2^-24 * 2 (|x|^2 + |c|^2) <= 2^-19.6 (...)
//   of the exact one and |c|^2 within 2^-21 |c|^2.  Two centroids whose exact distances are
//   ordered the other way round therefore differ by less than 0.6 E in a_c: the fixed-order argmin
//   is always among the candidates, and the codes equal pq_assign_kernel's bit for bit.
//
// Bound: the vector instructions of the epilogue, about 2.5 per (key, centroid), half of them on
// the 16-lane ALU pipe; 8 KV heads x 65472 keys x 16 sub-vectors x 256 centroids are 2.1e9 pairs,
// 0.18 ms at that rate; measured 0.45 ms.  The previous form (product and |c|^2 apart, E sixteen
// times wider, a branch per centroid in the second pass) took 5.07 ms for it.
//
// One CTA of 256 threads per SM holding all of tensor memory: two groups of four warps, each with
// an accumulator of 256 columns and an A tile of its own, so that one group's product and waits
// hide behind the other's epilogue.  A CTA carries NS neighbouring sub-vectors (a key's 64
// contiguous bytes for NS = 4: whole sectors, and one 4-byte store of codes) and a contiguous
// share of the flattened (sub-vector block, key tile) space, cut evenly over the SMs; the B tiles
// are rebuilt when the share crosses into another block.  The only mbarrier wait
// (tcgen05.commit) is bounded; when it runs out the error word is set, and the threads walk
// through their remaining tiles without working on them.
#pragma once
#include "sah_tcgen05.cuh"

#define PTC_TILE 128
#define PTC_THREADS 256

template <int NS>
struct PtcCfg {
  static constexpr int A_OFF = 0;                                // two groups' [128 rows][128 B], first 64 B used
  static constexpr int B_OFF = 2 * PTC_TILE * 128;               // NS x [256 rows][128 B], first 64 B used
  static constexpr int CENT_OFF = B_OFF + NS * 256 * 128;        // NS x float32 [256][8]
  static constexpr int CAND_OFF = CENT_OFF + NS * 256 * 8 * 4;   // candidate masks [8][threads]
  static constexpr int MISC_OFF = CAND_OFF + 8 * PTC_THREADS * 4;  // max |c|^2 per sub-vector, mbarriers, slot, abort
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

__device__ __forceinline__ void ptc_max_block(const uint32_t* v, float* mx) {
#pragma unroll
  for (int i = 0; i < 32; i += 2)
    mx[(i >> 1) & 3] = ptc_max3(mx[(i >> 1) & 3], __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
}
// bit 31 - i: value i is not below thr (or is NaN); four short chains of shifts
__device__ __forceinline__ uint32_t ptc_candidates(const uint32_t* v, float thr) {
  uint32_t below[4] = {0u, 0u, 0u, 0u};
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int q = 0; q < 4; ++q)
      below[q] = __funnelshift_l(__float_as_uint(__fsub_rn(__uint_as_float(v[q * 8 + i]), thr)), below[q], 1);
  return ~((below[0] << 24) | (below[1] << 16) | (below[2] << 8) | below[3]);
}

// NB: blocks of 32 accumulator columns (n_cent <= 32 NB; the columns past n_cent hold -inf)
template <int NS, int NB>
__global__ void __launch_bounds__(PTC_THREADS, 1)
pq_assign_tc_kernel(const __nv_bfloat16* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int Hkv,
                    int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub, int n_cent,
                    int64_t n_blocks, const float* __restrict__ centroids, uint8_t* __restrict__ codes,
                    int64_t cap, int* __restrict__ errflag) {
  constexpr int SD = 8, NC = 32 * NB;
  using C = PtcCfg<NS>;
  extern __shared__ __align__(1024) unsigned char ptc_raw[];
  const uint32_t raw_s = (uint32_t)__cvta_generic_to_shared(ptc_raw);
  unsigned char* sm = ptc_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
  const uint32_t sm_s = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wg = tid >> 7, keyl = tid & 127;  // group of four warps, key of its tile
  float* cent_sm = reinterpret_cast<float*>(sm + C::CENT_OFF);
  uint32_t* cand_sm = reinterpret_cast<uint32_t*>(sm + C::CAND_OFF);
  unsigned int* cmax_sm = reinterpret_cast<unsigned int*>(sm + C::MISC_OFF);  // [NS], float bits
  const uint32_t bar = sm_s + C::MISC_OFF + 32 + wg * 8;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + C::MISC_OFF + 48);
  volatile int* abort_sm = reinterpret_cast<volatile int*>(sm + C::MISC_OFF + 52);

  if (keyl == 0) atm_mbar_init(bar, 1);
  if (tid == 0) {
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
  {  // chunk 3 of an A row (the factors of -|c|^2 / 2) never changes
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
      // a NaN or infinite norm makes the margin NaN or infinite: every centroid is then measured
      if (c < n_cent) atomicMax(cmax_sm + s, __float_as_uint(n2));
      unsigned char* row = sm + C::B_OFF + s * (256 * 128) + c * 128;
      *reinterpret_cast<uint4*>(row + ((0 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(hi);
      *reinterpret_cast<uint4*>(row + ((1 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(mi);
      *reinterpret_cast<uint4*>(row + ((2 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(lo);
      *reinterpret_cast<uint4*>(row + ((3 ^ (c & 7)) << 4)) = *reinterpret_cast<const uint4*>(nn);
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    const int64_t seg_end = (blk + 1) * n_tiles < it_end ? (blk + 1) * n_tiles : it_end;
    uint4 raw[NS];
    {
      const int64_t j = key_begin + (it + wg - blk * n_tiles) * PTC_TILE + keyl;
#pragma unroll
      for (int s = 0; s < NS; ++s)
        raw[s] = it + wg < seg_end && j < key_end ? *reinterpret_cast<const uint4*>(xb + j * xs_s + s * SD)
                                                  : make_uint4(0u, 0u, 0u, 0u);
    }
    for (int64_t t = it + wg; t < seg_end; t += 2) {
      const int64_t j = key_begin + (t - blk * n_tiles) * PTC_TILE + keyl;
      uint4 next[NS];
      const int64_t jn = j + 2 * PTC_TILE;
#pragma unroll
      for (int s = 0; s < NS; ++s)
        next[s] = t + 2 < seg_end && jn < key_end ? *reinterpret_cast<const uint4*>(xb + jn * xs_s + s * SD)
                                                  : make_uint4(0u, 0u, 0u, 0u);
      uint32_t packed = 0u;
#pragma unroll 1
      for (int s = 0; s < NS; ++s) {
        uint4 rw = raw[0];
#pragma unroll
        for (int q = 1; q < NS; ++q)
          if (s == q) rw = raw[q];
        *reinterpret_cast<uint4*>(arow + ((0 ^ (keyl & 7)) << 4)) = rw;
        *reinterpret_cast<uint4*>(arow + ((1 ^ (keyl & 7)) << 4)) = rw;
        *reinterpret_cast<uint4*>(arow + ((2 ^ (keyl & 7)) << 4)) = rw;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        aum_fence_before();
        // the group's A rows are written and its reads of the previous accumulator are done
        asm volatile("bar.sync %0, 128;\n" ::"r"(1 + wg) : "memory");
        if (keyl == 0 && !*abort_sm) {
          aum_fence_after();
          const uint32_t b_s = sm_s + C::B_OFF + s * (256 * 128);
          aum_mma(tmem, aum_desc(a_s, 0, 1024, 2), aum_desc(b_s, 0, 1024, 2), idesc, 0u);
          aum_mma(tmem, aum_desc(a_s + 32, 0, 1024, 2), aum_desc(b_s + 32, 0, 1024, 2), idesc, 1u);
          aum_commit(bar);
        }
        float xv[SD];
        sah_unpack8(rw, xv);
        float x2 = 0.f;
#pragma unroll
        for (int d = 0; d < SD; ++d) x2 = fmaf(xv[d], xv[d], x2);
        const float margin = 1.52587890625e-05f * (x2 + __uint_as_float(cmax_sm[s]));  // E
        const bool ok = aum_wait_warp(bar, phase, abort_sm, errflag);
        phase ^= 1u;
        if (!ok) continue;
        aum_fence_after();
        uint32_t va[32], vb[32];
        // ---- the largest a_c; the loops stay rolled over pairs of blocks, which keeps the two
        //      buffers the only long-lived values (unrolled, the kernel spilled) ----
        float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        ptc_tmem_ld32(tmem_row, va);
#pragma unroll 1
        for (int gq = 0; gq < NB; gq += 2) {
          ptc_tmem_wait(va);
          if (NB > 1) ptc_tmem_ld32(tmem_row + (gq + 1) * 32, vb);
          ptc_max_block(va, mx);
          if (NB > 1) {
            ptc_tmem_wait(vb);
            if (gq + 2 < NB) ptc_tmem_ld32(tmem_row + (gq + 2) * 32, va);
            ptc_max_block(vb, mx);
          }
        }
        const float thr = __fsub_rn(fmaxf(ptc_max3(mx[0], mx[1], mx[2]), mx[3]), margin);
        // ---- candidates: bit 31 - i of word gq is centroid 32 gq + i ----
        int n_cand = 0, arg = 0;
        ptc_tmem_ld32(tmem_row, va);
#pragma unroll 1
        for (int gq = 0; gq < NB; gq += 2) {
          ptc_tmem_wait(va);
          if (NB > 1) ptc_tmem_ld32(tmem_row + (gq + 1) * 32, vb);
          uint32_t w = ptc_candidates(va, thr);
          cand_sm[gq * PTC_THREADS + tid] = w;
          n_cand += __popc(w);
          if (w) arg = gq * 32 + __clz(w);
          if (NB > 1) {
            ptc_tmem_wait(vb);
            if (gq + 2 < NB) ptc_tmem_ld32(tmem_row + (gq + 2) * 32, va);
            w = ptc_candidates(vb, thr);
            cand_sm[(gq + 1) * PTC_THREADS + tid] = w;
            n_cand += __popc(w);
            if (w) arg = gq * 32 + 32 + __clz(w);
          }
        }
        if (n_cand != 1) {
          float best = INFINITY;
          arg = 0;
#pragma unroll 1
          for (int gq = 0; gq < NB; ++gq) {
            uint32_t w = cand_sm[gq * PTC_THREADS + tid];
#pragma unroll 1
            while (w) {  // ascending c: the first minimum wins
              const int i = __clz(w);
              w &= ~(0x80000000u >> i);
              const int c = gq * 32 + i;
              if (c < n_cent) {
                const float dist = pq_dist(xv, cent_sm + (s * 256 + c) * SD, SD);
                if (dist < best) { best = dist; arg = c; }
              }
            }
          }
        }
        packed |= (uint32_t)arg << (8 * s);
      }
      if (j < key_end) {
        uint8_t* dst = codes + (bk * cap + (j - init_offset)) * n_sub + sub0;
        if (NS == 4) *reinterpret_cast<uint32_t*>(dst) = packed;
        else *dst = (uint8_t)packed;
      }
#pragma unroll
      for (int s = 0; s < NS; ++s) raw[s] = next[s];
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
