// bf16 attention with MagicPig weights for many query rows per KV head, head dim 128 (tcgen05): all
// keys are streamed once for a block of rows, and a (row, key) pair counts where the row's bitmap
// has the key.
//
// The gather kernels walk the union of at most four rows' matches.  With sixteen query positions
// that is sixteen lists of half the keys and more per KV head; here the K and V rows of a head are
// read once for up to 64 rows (G query heads x Sq positions), contiguously, and there is no plan.
//
//   A CTA takes a contiguous range of tiles of 64 keys of one (batch, KV head, block of rows).  Two
//   producer warps copy the tiles into rings of three K and four V tiles (128-byte swizzle, as in the
//   gather kernel) and leave every key's constant 1 / (M |k~|) beside them.  Per tile
//     S[128 x 64] = Qtile . Ktile^T   and   C[128 x 64] = Qhat tile . Ktile^T      8 tcgen05.mma each
//     O[128 x 128] += P[128 x 64] . Vtile                                          4 tcgen05.mma
//   with the rows on the lanes of tensor memory.  RP = 32 or 64 rows are laid out 128 / RP times: each
//   copy evaluates its own share of a tile's keys, has its own running maximum, and holds zeros
//   in the P columns of the others.  Two threads, in warps that read the same quarter of tensor
//   memory, share a lane's keys (half each) and agree on its maximum through shared memory.  Two
//   groups of eight warps take the even and the odd tiles, each with its own S, C, P and O (all
//   512 columns of tensor memory).  The running maximum is exact: the accumulator is rescaled whenever
//   it grows, so that a row's largest weight enters P as itself.  Everything else -- weights,
//   roundings, who is a member -- is as in the gather kernels.
//
// Partials of the CTAs go to `parts` [nsplit][rows][D + 2]; attn_stream_merge_kernel adds them up.
// Waits are bounded as in the gather kernel: one that runs out sets the abort word and the caller's
// error word, and every role leaves its loop.
//
// Bound: the chain of a tile through a group (scores out of tensor memory, weights from the table, maximum,
// exponentials, rescale, P: 5000 to 9000 cycles, two groups in turn) and the 20 products of a tile, about 90
// cycles each.  8 KV heads x 65500 keys x 64 rows: gather kernel and its plan 708 us, this 144 us; with a tile's
// scores issued only after the products of the tile before the last, 161 us; with one thread per lane, four
// producer warps and a proxy fence behind every tile's copies 196 us.  Reading K and V takes 41 us.
#pragma once

#define AST_TILE 64
#define AST_STAGES 4
#define AST_K_SLOTS 3    // a K tile is done with when the scores of its tile are complete
#define AST_PROD_WARPS 2
#define AST_THREADS ((16 + AST_PROD_WARPS + 1) * 32)  // softmax, producers, issuer

struct AstCfg {
  static constexpr int QT = 128 * 256;              // a query tile: two halves of [128 rows][128 B]
  static constexpr int KT = AST_TILE * 256;         // a K (or V) tile: two halves of [64 rows][128 B]
  static constexpr int Q_OFF = 0, H_OFF = QT;
  static constexpr int K_RING = 2 * QT, V_RING = K_RING + AST_K_SLOTS * KT;
  static constexpr int P_OFF = V_RING + AST_STAGES * KT;    // per group [128 rows][128 B]
  static constexpr int INV_OFF = P_OFF + 2 * 128 * 128;     // per stage 64 key constants
  static constexpr int TOP_OFF = INV_OFF + AST_STAGES * AST_TILE * 4;  // maxima: [tile parity][group][half][128]
  static constexpr int BAR_OFF = TOP_OFF + 2 * 2 * 2 * 128 * 4;
  // full and empty per stage, k_free per K slot, then per group s_full s_free p_full p_free (two of each)
  static constexpr int MISC_OFF = BAR_OFF + (2 * AST_STAGES + AST_K_SLOTS + 9) * 8;
  static constexpr int SMEM = 1024 + MISC_OFF + 16;
  // after the last tile: accumulators [2][128][129]; their factors and maxima [2][128], denominators [2][2][128]
  static constexpr int OB_OFF = K_RING, OB_LD = 129, F_OFF = 0, ML_OFF = 1024;
};
static_assert(AstCfg::OB_OFF + 2 * 128 * AstCfg::OB_LD * 4 <= AstCfg::BAR_OFF, "accumulators overlap the barriers");
static_assert(AstCfg::SMEM <= 227 * 1024, "shared memory");

struct AstArgs {
  const __nv_bfloat16 *q, *k, *v, *qhat, *bias;
  int64_t qs_b, qs_h, qs_q, ks_b, ks_h, ks_s, vs_b, vs_h, vs_s, bias_s_b, bias_s_h, bias_s_q;
  int Hq, Hkv, Sq, G, blocks, bias_bytes;  // blocks: of rows per KV head; bias_bytes: 16, 8, 4 or 2, what its rows are aligned to
  int64_t S, W, dens_cap;
  float scaling;
  const uint32_t *match, *unit;
  const float *dens, *qmu;
  const unsigned int* max_bits;
  const uint16_t* wtable;
  float* parts;
  int* errflag;
};

// 16 or 8 columns; the values may be read after tcgen05.wait::ld and ast_tmem_tie
__device__ __forceinline__ void ast_tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void ast_tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
template <int N>
__device__ __forceinline__ void ast_tmem_tie(uint32_t* r) {
#pragma unroll
  for (int i = 0; i < N; i += 8)
    asm volatile("" : "+r"(r[i]), "+r"(r[i + 1]), "+r"(r[i + 2]), "+r"(r[i + 3]), "+r"(r[i + 4]), "+r"(r[i + 5]),
                      "+r"(r[i + 6]), "+r"(r[i + 7]));
}
__device__ __forceinline__ void ast_tmem_st16(uint32_t taddr, const uint32_t* r) {  // complete after tcgen05.wait::st
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::
          "r"(taddr),
      "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
      "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
      : "memory");
}

// NS additive-mask entries of a row from column j on, two to a word; zeros past `left` of them.  The
// row may start on any element: `bytes` is what the host found all rows aligned to.
template <int NS>
__device__ __forceinline__ void ast_bias(const __nv_bfloat16* p, int left, int bytes, uint32_t* out) {
  if (left >= NS && bytes == 16) {
#pragma unroll
    for (int i = 0; i < NS / 8; ++i) {
      const uint4 v = reinterpret_cast<const uint4*>(p)[i];
      out[4 * i] = v.x, out[4 * i + 1] = v.y, out[4 * i + 2] = v.z, out[4 * i + 3] = v.w;
    }
  } else if (left >= NS && bytes == 8) {
#pragma unroll
    for (int i = 0; i < NS / 4; ++i) {
      const uint2 v = reinterpret_cast<const uint2*>(p)[i];
      out[2 * i] = v.x, out[2 * i + 1] = v.y;
    }
  } else if (left >= NS && bytes == 4) {
#pragma unroll
    for (int i = 0; i < NS / 2; ++i) out[i] = reinterpret_cast<const uint32_t*>(p)[i];
  } else {
    const unsigned short* s = reinterpret_cast<const unsigned short*>(p);
#pragma unroll
    for (int i = 0; i < NS / 2; ++i) {
      const uint32_t lo = 2 * i < left ? s[2 * i] : 0, hi = 2 * i + 1 < left ? s[2 * i + 1] : 0;
      out[i] = lo | (hi << 16);
    }
  }
}

// the table's weight if `take`, else `otherwise`; no branch, so that a thread's loads go out together
__device__ __forceinline__ uint32_t ast_weight(const uint16_t* table, uint32_t bits, uint32_t take, uint32_t otherwise) {
  asm("{\n.reg .pred p;\nsetp.ne.u32 p, %1, 0;\n@p ld.global.nc.u16 %0, [%2];\n}\n"
      : "+r"(otherwise) : "r"(take), "l"(table + bits));
  return otherwise;
}

// RP: rows of a block; a thread evaluates NS = RP / 4 keys of a tile
template <int RP>
__global__ void __launch_bounds__(AST_THREADS, 1)
masked_attention_stream_kernel(AstArgs a) {
  sah_pdl_entry();
  constexpr int D = 128, NS = AST_TILE * RP / 256, NST = AST_STAGES;
  using C = AstCfg;
  extern __shared__ __align__(1024) unsigned char ast_raw[];
  const uint32_t raw_s = (uint32_t)__cvta_generic_to_shared(ast_raw);
  unsigned char* sm = ast_raw + (((raw_s + 1023u) & ~1023u) - raw_s);
  const uint32_t sm_s = (uint32_t)__cvta_generic_to_shared(sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int PROD0 = 16, ISSUER = PROD0 + AST_PROD_WARPS;

  const int split = blockIdx.x, nsplit = gridDim.x;
  const int blk = (int)(blockIdx.y % a.blocks);
  const int64_t bk = blockIdx.y / a.blocks;
  const int kvh = (int)(bk % a.Hkv);
  const int64_t b = bk / a.Hkv;
  const int64_t tiles = (a.S + AST_TILE - 1) / AST_TILE;
  const int64_t t0 = tiles * split / nsplit;
  const int n_tiles = (int)(tiles * (split + 1) / nsplit - t0);
  const int n_rows = a.G * a.Sq - blk * RP < RP ? a.G * a.Sq - blk * RP : RP;
  auto row_of = [&](int r) {  // global row of the block's row r
    const int rr = blk * RP + r, gi = rr / a.Sq;
    return (b * a.Hq + kvh * a.G + gi) * a.Sq + (rr - gi * a.Sq);
  };

  const uint32_t full = sm_s + C::BAR_OFF, empty = full + NST * 8, k_free = empty + NST * 8,
                 s_full = k_free + AST_K_SLOTS * 8, s_free = s_full + 16,
                 p_full = s_full + 32, p_free = s_full + 48;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + C::MISC_OFF);
  volatile int* abort_sm = reinterpret_cast<volatile int*>(sm + C::MISC_OFF + 4);
  if (tid == 0) {
#pragma unroll
    for (int i = 0; i < NST; ++i) {
      atm_mbar_init(full + i * 8, AST_PROD_WARPS * 33);  // the producers' copies, and a warp's own arrival
      atm_mbar_init(empty + i * 8, 1);  // tcgen05.commit behind the tile's second product
    }
#pragma unroll
    for (int i = 0; i < AST_K_SLOTS; ++i) atm_mbar_init(k_free + i * 8, 1);  // ... behind its first
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      atm_mbar_init(s_full + i * 8, 1);
      atm_mbar_init(s_free + i * 8, 8);  // one arrival per warp of the group
      atm_mbar_init(p_full + i * 8, 8);
      atm_mbar_init(p_free + i * 8, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    *abort_sm = 0;
  }
  if (warp == ISSUER) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::
                     "r"((uint32_t)__cvta_generic_to_shared(tmem_slot)),
                 "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
  }
  // the two query tiles (every copy of the rows), and P of zeros
  for (int i = tid; i < 2 * 128 * 16; i += AST_THREADS) {
    const int which = i >> 11, l = (i >> 4) & 127, c = i & 15, r = l % RP;
    uint4 val = make_uint4(0u, 0u, 0u, 0u);
    if (r < n_rows) {
      const int rr = blk * RP + r, gi = rr / a.Sq, h = kvh * a.G + gi, qi = rr - gi * a.Sq;
      const __nv_bfloat16* src = which ? a.qhat + ((b * a.Hq + h) * a.Sq + qi) * D
                                       : a.q + b * a.qs_b + (int64_t)h * a.qs_h + (int64_t)qi * a.qs_q;
      val = *reinterpret_cast<const uint4*>(src + c * 8);
    }
    *reinterpret_cast<uint4*>(sm + (which ? C::H_OFF : C::Q_OFF) + (c >> 3) * 16384 + l * 128 + (((c & 7) ^ (l & 7)) << 4)) = val;
  }
  for (int i = tid; i < 2 * 128 * 8; i += AST_THREADS)
    *reinterpret_cast<uint4*>(sm + C::P_OFF + i * 16) = make_uint4(0u, 0u, 0u, 0u);
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  aum_fence_before();
  __syncthreads();
  aum_fence_after();
  const uint32_t tmem = *tmem_slot;
  // tensor memory columns of group g: S at 128 g, C at 128 g + 64, O at 256 + 128 g

  float m_run = -INFINITY, l_run = 0.f;
  uint32_t orow_base = 0;
  bool have_o = false;
  if (warp >= PROD0 && warp < ISSUER) {
    // =========================== producers: rows PR pw .. PR pw + PR - 1 of every tile ===========================
    constexpr int PR = AST_TILE / AST_PROD_WARPS;
    const int pw = warp - PROD0, chunk = lane & 15, sub = lane >> 4;
    const int64_t first = t0 * AST_TILE + pw * PR;
    const unsigned char* kb = reinterpret_cast<const unsigned char*>(a.k + b * a.ks_b + kvh * a.ks_h + (first + sub) * a.ks_s) + chunk * 16;
    const unsigned char* vb = reinterpret_cast<const unsigned char*>(a.v + b * a.vs_b + kvh * a.vs_h + (first + sub) * a.vs_s) + chunk * 16;
    const int64_t k2 = a.ks_s * 4, v2 = a.vs_s * 4;  // two rows
    const float* gd = a.dens + bk * a.dens_cap;
    const float M = __uint_as_float(*a.max_bits);
    auto load_dens = [&](int t) {
      const int64_t j = first + (int64_t)t * AST_TILE + lane;
      return t < n_tiles && j < a.S && lane < PR ? __ldg(gd + j) : 1.f;
    };
    float dens_next = load_dens(0);
    const uint32_t in = (chunk >> 3) * (AST_TILE * 128) + (pw * PR + sub) * 128;
    const unsigned char *k_row0 = kb - (first + sub) * a.ks_s * 2, *v_row0 = vb - (first + sub) * a.vs_s * 2;
    auto copy = [&](uint32_t dst, const unsigned char*& src, const unsigned char* row0, int64_t step, int64_t left) {
#pragma unroll 8
      for (int it = 0; it < PR / 2; ++it) {  // rows 2 it + sub; zeros past the last key
        atm_cp_async16_zfill(dst + it * 256 + ((uint32_t)((chunk & 7) ^ ((it * 2 + sub) & 7)) << 4),
                             it * 2 < left ? src : row0, it * 2 < left ? 16u : 0u);
        src += step;
      }
      src += step / 2 * (AST_TILE - PR);
    };
    // The copies arrive on the barrier by themselves and the issuer orders them before the tensor core's
    // reads: a fence by a producer would hold up its next copies.
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t % NST, ks = t % AST_K_SLOTS;
      const int64_t left = a.S - (first + (int64_t)t * AST_TILE) - sub;
      if (t >= AST_K_SLOTS && !aum_wait_warp(k_free + ks * 8, (uint32_t)((t / AST_K_SLOTS - 1) & 1), abort_sm, a.errflag)) break;
      copy(sm_s + C::K_RING + ks * C::KT + in, kb, k_row0, k2, left);
      if (t >= NST && !aum_wait_warp(empty + st * 8, (uint32_t)((t / NST - 1) & 1), abort_sm, a.errflag)) break;
      copy(sm_s + C::V_RING + st * C::KT + in, vb, v_row0, v2, left);
      atm_cp_async_arrive(full + st * 8);
      if (lane < PR) *reinterpret_cast<float*>(sm + C::INV_OFF + (st * AST_TILE + pw * PR + lane) * 4) =
          __frcp_rn(__fmul_rn(M, dens_next));
      __syncwarp();
      if (lane == 0) aum_arrive(full + st * 8);
      dens_next = load_dens(t + 1);
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
  } else if (warp == ISSUER) {
    // The whole warp walks the tiles and one lane issues: operands that are the same for all lanes and
    // descriptors that differ by constants cost an addition a product (one lane alone in the loop, every
    // descriptor put together anew: 169 against 161 us).
    const uint32_t idesc_s = aum_idesc(false, false, AST_TILE), idesc_o = aum_idesc(false, true, D);
    const uint64_t dq = aum_desc(sm_s + C::Q_OFF, 0, 1024, 2), dk = aum_desc(sm_s + C::K_RING, 0, 1024, 2),
                   dp = aum_desc(sm_s + C::P_OFF, 0, 1024, 2), dv = aum_desc(sm_s + C::V_RING, AST_TILE * 128, 1024, 2);
    bool ok = true;
    auto pv = [&](int t) {
      const int st = t % NST, gg = t & 1, j = t >> 1;
      if (!aum_wait_warp(p_full + gg * 8, (uint32_t)(j & 1), abort_sm, a.errflag)) return false;
      aum_fence_after();
      if (aum_elect()) {
        const uint64_t p = aum_desc_at(dp, gg * 16384), v = aum_desc_at(dv, st * C::KT);
#pragma unroll
        for (int ks = 0; ks < AST_TILE / 16; ++ks)
          // A: P, K-major, 32 bytes per k-step; B: V, MN-major, 8 keys per 1 KB atom, the second 64 dims one half further
          aum_mma(tmem + 256 + gg * 128, aum_desc_at(p, ks * 32), aum_desc_at(v, ks * 2048), idesc_o,
                  (j > 0 || ks > 0) ? 1u : 0u);
        aum_commit(empty + st * 8);
        aum_commit(p_free + gg * 8);
      }
      __syncwarp();
      return true;
    };
    auto qk = [&](int t) {
      const int gg = t & 1, j = t >> 1;
      if (!aum_wait_warp(full + t % NST * 8, (uint32_t)((t / NST) & 1), abort_sm, a.errflag)) return false;
      if (j >= 1 && !aum_wait_warp(s_free + gg * 8, (uint32_t)((j - 1) & 1), abort_sm, a.errflag)) return false;
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // the producers' copies -> tensor-core reads
      aum_fence_after();
      if (aum_elect()) {
        const uint64_t k = aum_desc_at(dk, t % AST_K_SLOTS * C::KT);
#pragma unroll
        for (int hat = 0; hat < 2; ++hat)
#pragma unroll
          for (int ks = 0; ks < 8; ++ks)
            aum_mma(tmem + gg * 128 + hat * 64, aum_desc_at(dq, hat * (C::H_OFF - C::Q_OFF) + (ks >> 2) * 16384 + (ks & 3) * 32),
                    aum_desc_at(k, (ks >> 2) * (AST_TILE * 128) + (ks & 3) * 32), idesc_s, ks > 0 ? 1u : 0u);
        aum_commit(s_full + gg * 8);
        aum_commit(k_free + t % AST_K_SLOTS * 8);
      }
      __syncwarp();
      return true;
    };
    // A group's next scores run while it still works on the present ones, which it has in registers.
    for (int t = 0; t < 2 && t < n_tiles && ok; ++t) ok = qk(t);
    for (int t = 0; t < n_tiles && ok; ++t) {
      if (t + 2 < n_tiles) ok = qk(t + 2);
      ok = ok && pv(t);
    }
  } else {
    // =========================== softmax: two threads per lane of tensor memory ===========================
    const int gg = warp >> 3, wq = warp & 3, half = (warp >> 2) & 1, l = (wq << 5) | lane;
    const int r = l % RP, key0 = (l / RP * 2 + half) * NS;
    const uint32_t lane_base = ((uint32_t)(wq * 32)) << 16;
    const uint32_t t_s = tmem + lane_base + gg * 128 + key0, t_o = tmem + lane_base + 256 + gg * 128 + half * 64;
    const bool live = r < n_rows;
    const int64_t row = live ? row_of(r) : 0;
    const uint32_t* mrow = a.match + row * a.W;
    const uint32_t* urow = a.unit ? a.unit + row * a.W : nullptr;
    const float mu = live ? a.qmu[row] : 0.f;
    const __nv_bfloat16* brow = nullptr;
    if (a.bias && live) {
      const int64_t h = row / a.Sq % a.Hq, qi = row % a.Sq;
      brow = a.bias + b * a.bias_s_b + h * a.bias_s_h + qi * a.bias_s_q;
    }
    uint32_t mw_next = 0u, uw_next = 0u, bias_next[NS / 2];
    auto load_tile = [&](int t) {  // the row's words and additive mask
      mw_next = uw_next = 0u;
      const int64_t j0 = (t0 + t) * AST_TILE + key0;
      if (t >= n_tiles || !live || j0 >= a.S) return;
      mw_next = mrow[j0 >> 5] >> (j0 & 31);
      if (urow) uw_next = urow[j0 >> 5] >> (j0 & 31);
      const int64_t left = a.S - j0;
      if (left < 32) mw_next &= (1u << left) - 1u, uw_next &= (1u << left) - 1u;
      if (brow) ast_bias<NS>(brow + j0, left < NS ? (int)left : NS, a.bias_bytes, bias_next);
    };
#pragma unroll
    for (int i = 0; i < NS / 2; ++i) bias_next[i] = 0u;
    load_tile(gg);
    unsigned char* prow = sm + C::P_OFF + gg * 16384 + l * 128;
    float* tops = reinterpret_cast<float*>(sm + C::TOP_OFF) + gg * 256 + l;
    // A warp that leaves the loop lets the other half's warp go at the exchange of maxima that it would have
    // come to next.  That warp then gets to a bounded wait that the leaving one did not arrive for, and leaves
    // there: for the next tile's scores if the wait for tile j's ran out (no s_free for j), for tile j's product if
    // the wait for the one before did (no p_full for j; the scores of j + 1 may be there already).  Should both
    // leave, the arrivals complete an exchange that nobody is at, or stay behind.
    auto let_go = [&] { asm volatile("bar.arrive %0, 64;\n" ::"r"(1 + gg * 4 + wq) : "memory"); };
    bool ok = true;
    int j = 0;
    for (int t = gg; t < n_tiles; t += 2, ++j) {
      ok = aum_wait_warp(full + (t % NST) * 8, (uint32_t)((t / NST) & 1), abort_sm, a.errflag) &&  // the key constants
           aum_wait_warp(s_full + gg * 8, (uint32_t)(j & 1), abort_sm, a.errflag);
      if (!ok) {
        let_go();
        break;
      }
      aum_fence_after();
      uint32_t sr[NS], hr[NS], wp[NS / 2];
      if constexpr (NS == 16) {
        ast_tmem_ld16(t_s + 64, hr);
        ast_tmem_ld16(t_s, sr);
      } else {
        ast_tmem_ld8(t_s + 64, hr);
        ast_tmem_ld8(t_s, sr);
      }
      const uint32_t uw = uw_next, drawn = mw_next & ~uw_next;
      float inv[NS];
#pragma unroll
      for (int i = 0; i < NS; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(sm + C::INV_OFF + (t % NST * AST_TILE + key0 + i) * 4);
        inv[i] = v.x, inv[i + 1] = v.y, inv[i + 2] = v.z, inv[i + 3] = v.w;
      }
      asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
      ast_tmem_tie<NS>(hr);
      ast_tmem_tie<NS>(sr);
      aum_fence_before();
      __syncwarp();
      if (lane == 0) aum_arrive(s_free + gg * 8);
      // the weights 1 / (p + 1e-6) as bfloat16 bits; 0 where the probability is, or nothing is selected
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        float c = __fmul_rn(__fsub_rn(__uint_as_float(hr[i]), mu), inv[i]);
        c = fminf(fmaxf(__bfloat162float(__float2bfloat16_rn(c)), -1.0f), 1.0f);
        hr[i] = ast_weight(a.wtable, __float_as_uint(c) >> 16, drawn & (1u << i), uw & (1u << i) ? 0x3f80u : 0u);
      }
      float top = -INFINITY;
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        float x = __uint_as_float(sr[i]) * a.scaling;
        if (brow) x += __uint_as_float(i & 1 ? bias_next[i / 2] & 0xffff0000u : bias_next[i / 2] << 16);
        x = hr[i] != 0u ? x : -INFINITY;
        top = fmaxf(top, x);
        sr[i] = __float_as_uint(x);
        if (i & 1) wp[i / 2] = hr[i - 1] | (hr[i] << 16);
      }
      load_tile(t + 2);
      // the maximum of both halves of the lane
      tops[(j & 1) * 512 + half * 128] = top;
      asm volatile("bar.sync %0, 64;\n" ::"r"(1 + gg * 4 + wq) : "memory");
      top = fmaxf(top, tops[(j & 1) * 512 + (half ^ 1) * 128]);
      const bool grew = top > m_run;
      const float m_new = grew ? top : m_run;
      const float alpha = !grew ? 1.f : m_run == -INFINITY ? 0.f : __expf(m_run - m_new);
      const float m_use = m_new == -INFINITY ? 0.f : m_new;
      m_run = m_new;
      float sum = 0.f;
#pragma unroll
      for (int n = 0; n < NS; n += 2) {
        const float p0 = __expf(__uint_as_float(sr[n]) - m_use) * __uint_as_float(wp[n / 2] << 16);
        const float p1 = __expf(__uint_as_float(sr[n + 1]) - m_use) * __uint_as_float(wp[n / 2] & 0xffff0000u);
        sum += p0 + p1;
        wp[n / 2] = atm_pack_bf16(p0, p1);
      }
      l_run = l_run * alpha + sum;
      if (j >= 1) {
        ok = aum_wait_warp(p_free + gg * 8, (uint32_t)((j - 1) & 1), abort_sm, a.errflag);
        if (!ok) {
          let_go();
          break;
        }
        if (__any_sync(0xffffffffu, grew)) {  // this half's dims of the accumulator
          aum_fence_after();
#pragma unroll
          for (int c = 0; c < 64; c += 32) {
            uint32_t o[32];
            ast_tmem_ld16(t_o + c, o);
            ast_tmem_ld16(t_o + c + 16, o + 16);
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
            ast_tmem_tie<32>(o);
#pragma unroll
            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
            ast_tmem_st16(t_o + c, o);
            ast_tmem_st16(t_o + c + 16, o + 16);
          }
          asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
        }
      }
#pragma unroll
      for (int c = 0; c < NS / 8; ++c)
        *reinterpret_cast<uint4*>(prow + (((key0 / 8 + c) ^ (l & 7)) << 4)) =
            make_uint4(wp[4 * c], wp[4 * c + 1], wp[4 * c + 2], wp[4 * c + 3]);
      asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
      aum_fence_before();
      __syncwarp();
      if (lane == 0) aum_arrive(p_full + gg * 8);
    }
    if (ok && j > 0) ok = aum_wait_warp(p_free + gg * 8, (uint32_t)((j - 1) & 1), abort_sm, a.errflag);
    have_o = ok && j > 0;
    if (!have_o) m_run = -INFINITY, l_run = 0.f;
    orow_base = t_o;
  }
  // ---- the copies and groups of a row are added up in shared memory, whose rings are idle now ----
  aum_fence_before();
  __syncthreads();
  aum_fence_after();
  float* ob = reinterpret_cast<float*>(sm + C::OB_OFF);
  float* fac = reinterpret_cast<float*>(sm + C::F_OFF);  // [2][128]
  float* ml = reinterpret_cast<float*>(sm + C::ML_OFF);  // [3][2][128]
  if (warp < PROD0) {
    const int gg = warp >> 3, half = (warp >> 2) & 1, l = ((warp & 3) << 5) | lane;
    float* mine = ob + (gg * 128 + l) * C::OB_LD + half * 64;
#pragma unroll
    for (int c = 0; c < 64; c += 32) {
      uint32_t o[32];
      if (have_o) {  // the same for the whole warp
        ast_tmem_ld16(orow_base + c, o);
        ast_tmem_ld16(orow_base + c + 16, o + 16);
        asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        ast_tmem_tie<32>(o);
      }
#pragma unroll
      for (int i = 0; i < 32; ++i) mine[c + i] = have_o ? __uint_as_float(o[i]) : 0.f;
    }
    if (half == 0) ml[gg * 128 + l] = m_run;
    ml[256 + half * 256 + gg * 128 + l] = l_run;
  }
  aum_fence_before();
  __syncthreads();
  if (warp == ISSUER) {
    aum_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
  }
  const int64_t all_rows = (int64_t)gridDim.y / a.blocks / a.Hkv * a.Hq * a.Sq;
  if (tid < n_rows) {
    float mx = -INFINITY, L = 0.f;
    for (int c = tid; c < 256; c += RP) mx = fmaxf(mx, ml[c]);
    for (int c = tid; c < 256; c += RP) {
      const float f = ml[c] == -INFINITY ? 0.f : __expf(ml[c] - mx);
      fac[c] = f;
      L += (ml[256 + c] + ml[512 + c]) * f;
    }
    float* out = a.parts + (split * all_rows + row_of(tid)) * (D + 2);
    out[D] = mx;
    out[D + 1] = L;
  }
  __syncthreads();
  for (int i = tid; i < n_rows * D; i += AST_THREADS) {
    const int r = i / D, d = i - r * D;
    float o = 0.f;
#pragma unroll
    for (int c = 0; c < 256; c += RP) o += ob[(c + r) * C::OB_LD + d] * fac[c + r];
    a.parts[(split * all_rows + row_of(r)) * (D + 2) + d] = o;
  }
}

// Adds up the partials of a row, a thread per dim, and writes its output.
//
// The product takes every key's V row, with a probability of 0 where the row does not have the key, and
// 0 times an infinity or a NaN is NaN.  A row whose sum is not finite is therefore added up anew from its own
// keys alone, which is what the gather kernels read: M and L stand, they come from the scores of those keys.
// Plain loads and float32 sums (512 rows x 65500 keys with a NaN in every head 3.6 ms in all; finite values pay for a
// vote alone, 165 us).
__global__ void __launch_bounds__(128)
attn_stream_merge_kernel(AstArgs a, int n_parts, int64_t rows, const float* __restrict__ sinks, __nv_bfloat16* __restrict__ out) {
  sah_pdl_entry_early();
  constexpr int D = 128;
  __shared__ float part[4][D];
  const int64_t row = blockIdx.x;
  const int d = threadIdx.x, lane = d & 31, warp = d >> 5;
  const int qi = (int)(row % a.Sq), h = (int)(row / a.Sq % a.Hq);
  const int64_t b = row / a.Sq / a.Hq, pstride = rows * (D + 2);
  const float* pr = a.parts + row * (D + 2);
  float M = -INFINITY, L = 0.f, o = 0.f;
  for (int p = 0; p < n_parts; ++p) M = fmaxf(M, pr[p * pstride + D]);
  for (int p = 0; p < n_parts; ++p) {
    const float mp = pr[p * pstride + D];
    if (mp != -INFINITY) {
      const float f = expf(mp - M);
      L += pr[p * pstride + D + 1] * f;
      o += pr[p * pstride + d] * f;
    }
  }
  if (__syncthreads_or(!(fabsf(o) < INFINITY))) {
    const int kvh = h / a.G;
    const int64_t bk = b * a.Hkv + kvh;
    float q[4], qh[4], num[4] = {0.f, 0.f, 0.f, 0.f};
    constexpr int AHEAD = 8;
    auto four = [](const uint2& v, float* x) {
      x[0] = __uint_as_float(v.x << 16), x[1] = __uint_as_float(v.x & 0xffff0000u);
      x[2] = __uint_as_float(v.y << 16), x[3] = __uint_as_float(v.y & 0xffff0000u);
    };
    four(*reinterpret_cast<const uint2*>(a.q + b * a.qs_b + (int64_t)h * a.qs_h + (int64_t)qi * a.qs_q + lane * 4), q);
    four(*reinterpret_cast<const uint2*>(a.qhat + row * D + lane * 4), qh);
    const __nv_bfloat16 *kb = a.k + b * a.ks_b + kvh * a.ks_h, *vb = a.v + b * a.vs_b + kvh * a.vs_h;
    const __nv_bfloat16* brow = a.bias ? a.bias + b * a.bias_s_b + h * a.bias_s_h + qi * a.bias_s_q : nullptr;
    const float mu = a.qmu[row], max_norm = __uint_as_float(*a.max_bits);
    for (int64_t w = warp; w * 32 < a.S; w += 4) {
      const uint32_t units = a.unit ? a.unit[row * a.W + w] : 0u;
      uint32_t on = a.match[row * a.W + w] | units;
      if (a.S - w * 32 < 32) on &= (1u << (a.S - w * 32)) - 1u;
      while (on) {  // the same for the whole warp; AHEAD keys' loads and sums are under way together
        int bit[AHEAD];
        bool has[AHEAD];
        uint2 kr[AHEAD], vr[AHEAD];
        float s[AHEAD], c[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          has[u] = on != 0u;
          bit[u] = has[u] ? __ffs(on) - 1 : bit[0];
          on &= on - 1u;
          const int64_t j = w * 32 + bit[u];
          kr[u] = *reinterpret_cast<const uint2*>(kb + j * a.ks_s + lane * 4);
          vr[u] = *reinterpret_cast<const uint2*>(vb + j * a.vs_s + lane * 4);
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          float k[4];
          four(kr[u], k);
          s[u] = q[0] * k[0] + q[1] * k[1] + q[2] * k[2] + q[3] * k[3];
          c[u] = qh[0] * k[0] + qh[1] * k[1] + qh[2] * k[2] + qh[3] * k[3];
        }
#pragma unroll
        for (int of = 16; of > 0; of >>= 1)
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            s[u] += __shfl_xor_sync(0xffffffffu, s[u], of);
            c[u] += __shfl_xor_sync(0xffffffffu, c[u], of);
          }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const int64_t j = w * 32 + bit[u];
          const float weight = (units >> bit[u]) & 1u ? 1.f
                               : atm_lsh_weight(c[u], mu, __frcp_rn(__fmul_rn(max_norm, a.dens[bk * a.dens_cap + j])), a.wtable);
          if (!has[u] || weight == 0.f) continue;
          float x = s[u] * a.scaling;
          if (brow) x += __bfloat162float(brow[j]);
          const float p = __expf(x - M) * weight;
          float v[4];
          four(vr[u], v);
#pragma unroll
          for (int i = 0; i < 4; ++i) num[i] += p * v[i];
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) part[warp][lane * 4 + i] = num[i];
    __syncthreads();
    o = part[0][d] + part[1][d] + part[2][d] + part[3][d];
  }
  float Mx = M, sink_term = 0.f;
  if (sinks != nullptr) {
    const float sk = sinks[h];
    Mx = fmaxf(M, sk);
    sink_term = expf(sk - Mx);
  }
  const float resc = (M == -INFINITY) ? 0.f : expf(M - Mx);
  out[((b * a.Sq + qi) * a.Hq + h) * D + d] = __float2bfloat16_rn(o * resc / (L * resc + sink_term));
}

// Rows of a block and CTAs per (KV head, block): one CTA per SM, at least four tiles each.
static int ast_rows(int rows) { return rows <= 32 ? 32 : 64; }
static int ast_splits(int64_t heads, int rows, int64_t S, int sm_count) {
  const int rp = ast_rows(rows);
  const int64_t lists = heads * sah_ceil_div((int64_t)rows, (int64_t)rp), tiles = sah_ceil_div(S, (int64_t)AST_TILE);
  int64_t n = sm_count / lists;
  if (n > tiles / 4) n = tiles / 4;
  return n < 1 ? 1 : (int)n;
}

// Where streaming every key beats gathering lists.  A key that has nothing to do with a query agrees
// with it in some table with probability f = 1 - (1 - 2^-K)^L, so the list of R rows holds about
// 1 - (1 - f)^R of the keys; a KV head has one list per q_block positions, and one pass over all keys
// per block of rows here.  Measured at 8 KV heads x 65500 keys, by lists times share of the keys:
// 11.1 (16 positions of 4 heads, 75 tables of 8 bits) 708 -> 144 us, 2.8 206 -> 116, 1.4 130 -> 112 and, 2
// heads, 112 -> 112, 1.2 (5 tables) 276 -> 144; 0.9 (2 positions, 40 tables) 107 -> 112, 0.5 93 -> 112.
// 8192 keys, 1.4: 40 -> 31 us.
static bool ast_default(int G, int Sq, int lsh_k, int lsh_l, int64_t blocks) {
  if (G > 4) return false;
  const int q_block = 4 / G < Sq ? 4 / G : Sq, lists = (Sq + q_block - 1) / q_block;
  const double miss = pow(1.0 - pow(0.5, lsh_k), lsh_l);
  return lists * (1.0 - pow(miss, G * q_block)) >= 1.2 * (double)blocks;
}
