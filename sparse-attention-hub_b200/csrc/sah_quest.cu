// Quest page top-k (research_attention/maskers/fixed/implementations/quest_top_k.py:108-196,
// utils/quest_utils.py): per-page minimum and maximum of every key channel, an upper bound of
// q.k per page from them, top pages, pages expanded to keys.
//
// The page bounds are kept per KV head (the reference repeats the keys over the query heads of
// a group first, which repeats the bounds), as [B][Hkv][D/8][page capacity][8]: the scoring
// kernel has one thread per page, and with eight channels of consecutive pages next to each
// other its 16-byte loads are coalesced.  The bound is a sum over the head dimension of
// dtype-rounded products; it is taken in the order of the reference's CPU row reduction so that
// page scores, and with them the chosen pages, are the reference's bit for bit: float32
// accumulation in vectors of 8 lanes (a bfloat16 load brings 16 elements and adds its two
// halves), four interleaved vector accumulators added in order, then the lanes in order.
#include "sah_common.cuh"

// ---- page bounds ---------------------------------------------------------------------------
template <typename T>
__global__ void quest_minmax_kernel(const T* __restrict__ k, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                                    int Hkv, int64_t S, int D, int page_size, int64_t page_begin,
                                    int64_t P_cap, T* __restrict__ pmin, T* __restrict__ pmax) {
  const int64_t page = page_begin + blockIdx.x;
  const int h = blockIdx.y;
  const int64_t b = blockIdx.z;
  const int64_t s0 = page * page_size;
  const int64_t s1 = s0 + page_size < S ? s0 + page_size : S;
  const T* base = k + b * ks_b + h * ks_h;
  for (int d = threadIdx.x; d < D; d += blockDim.x) {
    float lo = INFINITY, hi = -INFINITY;
#pragma unroll 4
    for (int64_t s = s0; s < s1; ++s) {
      const float x = sah_to_float<T>(base[s * ks_s + d]);
      lo = fminf(lo, x);
      hi = fmaxf(hi, x);
    }
    const int64_t o = ((((b * Hkv + h) * (D / 8) + d / 8) * P_cap + page) << 3) + (d & 7);
    pmin[o] = sah_from_float<T>(lo);
    pmax[o] = sah_from_float<T>(hi);
  }
}

extern "C" int sah_quest_page_minmax(const void* k, int dtype, int64_t ks_b, int64_t ks_h, int64_t ks_s,
                                     int B, int Hkv, int64_t S, int D, int page_size,
                                     int64_t page_begin, int64_t P_cap, void* pmin, void* pmax,
                                     void* stream) {
  SAH_REQUIRE(k && pmin && pmax, "quest_page_minmax: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && S > 0 && D > 0 && D % 8 == 0 && page_size > 0,
              "quest_page_minmax: bad extents (the head dimension must be a multiple of 8)");
  const int64_t P = sah_ceil_div(S, page_size);
  SAH_REQUIRE(page_begin >= 0 && page_begin <= P && P <= P_cap, "quest_page_minmax: bad page range");
  SAH_REQUIRE(Hkv <= 65535 && B <= 65535, "quest_page_minmax: too many heads or batches");
  if (page_begin == P) return SAH_OK;
  dim3 grid((unsigned)(P - page_begin), (unsigned)Hkv, (unsigned)B);
  const int threads = D >= 256 ? 256 : ((D + 31) / 32) * 32;
  SAH_DISPATCH_DTYPE(dtype, T, {
    quest_minmax_kernel<T><<<grid, threads, 0, (cudaStream_t)stream>>>(
        (const T*)k, ks_b, ks_h, ks_s, Hkv, S, D, page_size, page_begin, P_cap, (T*)pmin, (T*)pmax);
  });
  SAH_LAUNCH_CHECK("quest_page_minmax");
  return SAH_OK;
}

// ---- page scores ---------------------------------------------------------------------------
// The page bounds of a KV head are read once for up to four of its rows: a CTA of (pages, rows)
// threads copies its pages' bounds to shared memory, every 16-byte piece requested before the
// first is waited for.  Bound by that latency and by the rounded products, two per channel; in
// bfloat16 they are made in pairs (the product of two bfloat16 numbers rounds once either way).
// 256 rows x 512 pages x 128 channels: 14.2 us with every row reading the bounds for itself,
// 8.0 us now.  In float32, where a page's bounds are twice as long and there are no pairs, that gains
// where a launch is short of warps (32 rows x 512 pages 5.9 us row by row, 4.3 us staged; 512
// channels 16 and 9 us) and loses where it is not (256 x 512 11 and 15 us): from QS_DIRECT scores on
// and up to 256 channels a thread reads the bounds of its page for its own row.
#define QS_ROWS 4
#define QS_PAGES 128            // pages per CTA; halved until the bounds fit
#define QS_BOUND_BYTES(elt) ((elt) == 2 ? 96 * 1024 : 36 * 1024)
#define QS_DIRECT (48 * 1024)
#define QS_MAXD 512
#define QS_SMEM (160 * 1024)    // 139 KB at most: 32 pages of 512 float32 channels

template <typename T>
struct QuestVec {  // elements one vector load of the reference's reduction brings
  static constexpr int N = sizeof(T) == 2 ? 16 : 8;
};

// max(q lo, q hi) of eight channels, both products rounded to T
__device__ __forceinline__ void quest_max8(const __nv_bfloat16* q, const __nv_bfloat16* lo, const __nv_bfloat16* hi,
                                           float* out) {
  const uint4 qv = *reinterpret_cast<const uint4*>(q), a = *reinterpret_cast<const uint4*>(lo),
              c = *reinterpret_cast<const uint4*>(hi);
  const uint32_t qw[4] = {qv.x, qv.y, qv.z, qv.w}, aw[4] = {a.x, a.y, a.z, a.w}, cw[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162*>(&qw[i]);
    const __nv_bfloat162 m = __hmax2(__hmul2(x, *reinterpret_cast<const __nv_bfloat162*>(&aw[i])),
                                     __hmul2(x, *reinterpret_cast<const __nv_bfloat162*>(&cw[i])));
    const uint32_t u = *reinterpret_cast<const uint32_t*>(&m);
    out[2 * i] = __uint_as_float(u << 16);
    out[2 * i + 1] = __uint_as_float(u & 0xffff0000u);
  }
}
__device__ __forceinline__ void quest_max8(const float* q, const float* lo, const float* hi, float* out) {
  float qf[8], a[8], c[8];
  sah_load8<float>(q, qf);
  sah_load8<float>(lo, a);
  sah_load8<float>(hi, c);
#pragma unroll
  for (int l = 0; l < 8; ++l) out[l] = fmaxf(__fmul_rn(qf[l], a[l]), __fmul_rn(qf[l], c[l]));
}

// STAGED: bounds in shared memory, blockDim.y = QS_ROWS; else read where they lie, blockDim.y = 1
template <typename T, bool STAGED>
__global__ void __launch_bounds__(STAGED ? QS_PAGES * QS_ROWS : QS_PAGES)
quest_scores_kernel(const T* __restrict__ q, int64_t qs_b, int64_t qs_h, int64_t qs_q,
                    const T* __restrict__ pmin, const T* __restrict__ pmax, int64_t P_cap, int Hq,
                    int Hkv, int Sq, int64_t S, int D, int page_size, const T* __restrict__ bias,
                    int64_t bias_s_b, int64_t bias_s_q, T* __restrict__ scores) {
  sah_pdl_entry();
  extern __shared__ __align__(16) unsigned char qs_smem[];
  const int NP = blockDim.x, chunks = D / 8;
  T* lo_sm = reinterpret_cast<T*>(qs_smem);                 // [chunks][NP][8]
  T* hi_sm = lo_sm + (size_t)chunks * NP * 8;
  T* q_sm = STAGED ? hi_sm + (size_t)chunks * NP * 8 : lo_sm;  // [rows][D]
  const int G = Hq / Hkv, R = G * Sq;                       // rows that share a KV head
  const int64_t bk = blockIdx.z;                            // b * Hkv + kvh
  const int kvh = (int)(bk % Hkv);
  const int64_t b = bk / Hkv;
  const int r = blockIdx.y * blockDim.y + threadIdx.y;      // row r = g * Sq + qi of the KV head
  const int64_t P = (S + page_size - 1) / page_size;
  const int64_t page0 = (int64_t)blockIdx.x * NP;
  const int np = (int)(P - page0 < NP ? P - page0 : NP);
  const int tid = threadIdx.y * NP + threadIdx.x, nt = NP * QS_ROWS;
  // chunk c (channels 8c .. 8c+7) of page p: base + (c * P_cap + p) * 8
  constexpr int PIECES = 8 * (int)sizeof(T) / 16;           // 16-byte pieces of a chunk
  const T* lo_g = pmin + bk * (int64_t)D * P_cap + page0 * 8;
  const T* hi_g = pmax + bk * (int64_t)D * P_cap + page0 * 8;
  for (int i = tid; STAGED && i < chunks * NP * PIECES; i += nt) {
    const int c = i / (NP * PIECES), x = i - c * (NP * PIECES);  // piece x of the chunk's row of pages
    if (x < np * PIECES) {
      const int64_t src = c * P_cap * 8 + (int64_t)x * (8 / PIECES);
      const int dst = c * NP * 8 + x * (8 / PIECES);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(lo_sm + dst)),
                   "l"(lo_g + src) : "memory");
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(hi_sm + dst)),
                   "l"(hi_g + src) : "memory");
    }
  }
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  const int g = r / Sq, qi = r - g * Sq, h = kvh * G + g;
  if (r < R) {
    const T* qr = q + b * qs_b + h * qs_h + qi * qs_q;
    for (int d = threadIdx.x; d < D; d += NP) q_sm[threadIdx.y * D + d] = qr[d];
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
  const int64_t page = page0 + threadIdx.x;
  if (r >= R || page >= P) return;
  const int64_t row = (b * Hq + h) * Sq + qi;
  const T* lo = (STAGED ? lo_sm : lo_g) + threadIdx.x * 8;
  const T* hi = (STAGED ? hi_sm : hi_g) + threadIdx.x * 8;
  const T* qs = q_sm + threadIdx.y * D;
  const int64_t cstride = STAGED ? NP * 8 : P_cap * 8;

  constexpr int VEC = QuestVec<T>::N;
  const int nv = D / VEC;
  const int full = nv / 4;
  float acc[4][8];
#pragma unroll
  for (int kk = 0; kk < 4; ++kk)
#pragma unroll
    for (int l = 0; l < 8; ++l) acc[kk][l] = 0.f;

  // the 8 lane values one vector load contributes: max(q*lo, q*hi), products rounded to T
  auto load_vec = [&](int v, float* out) {
#pragma unroll
    for (int half = 0; half < VEC / 8; ++half) {
      const int c = v * (VEC / 8) + half;
      float m[8];
      quest_max8(qs + c * 8, lo + c * cstride, hi + c * cstride, m);
#pragma unroll
      for (int l = 0; l < 8; ++l) out[l] = half == 0 ? m[l] : __fadd_rn(out[l], m[l]);  // a bf16 load adds its two halves
    }
  };
  for (int i = 0; i < full; ++i) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float val[8];
      load_vec(i * 4 + kk, val);
#pragma unroll
      for (int l = 0; l < 8; ++l) acc[kk][l] = __fadd_rn(acc[kk][l], val[l]);
    }
  }
  for (int v = full * 4; v < nv; ++v) {
    float val[8];
    load_vec(v, val);
#pragma unroll
    for (int l = 0; l < 8; ++l) acc[0][l] = __fadd_rn(acc[0][l], val[l]);
  }
#pragma unroll
  for (int kk = 1; kk < 4; ++kk)
#pragma unroll
    for (int l = 0; l < 8; ++l) acc[0][l] = __fadd_rn(acc[0][l], acc[kk][l]);
  float fin = 0.f;
  for (int c = nv * (VEC / 8); c < chunks; ++c) {   // elements past the last whole vector come first
    float m[8];
    quest_max8(qs + c * 8, lo + c * cstride, hi + c * cstride, m);
#pragma unroll
    for (int l = 0; l < 8; ++l) fin = __fadd_rn(fin, m[l]);
  }
#pragma unroll
  for (int l = 0; l < 8; ++l) fin = __fadd_rn(fin, acc[0][l]);
  float sc = sah_round_to<T>(fin);

  if (bias != nullptr) {   // a page none of whose keys is allowed scores the lowest value
    const T* br = bias + b * bias_s_b + qi * bias_s_q;
    const int64_t s0 = page * page_size;
    const int64_t s1 = s0 + page_size < S ? s0 + page_size : S;
    bool any = false;
    for (int64_t s = s0; s < s1 && !any; ++s) any = sah_to_float<T>(br[s]) >= 0.f;
    if (!any) sc = sizeof(T) == 2 ? __uint_as_float(0xFF7F0000u) : -3.402823466e38f;
  }
  scores[row * P + page] = sah_from_float<T>(sc);
}

extern "C" int sah_quest_scores(const void* q, int dtype, int64_t qs_b, int64_t qs_h, int64_t qs_q,
                                const void* pmin, const void* pmax, int64_t P_cap, int B, int Hq,
                                int Hkv, int Sq, int64_t S, int D, int page_size, const void* bias,
                                int64_t bias_s_b, int64_t bias_s_h, int64_t bias_s_q, void* scores,
                                void* stream) {
  SAH_REQUIRE(q && pmin && pmax && scores, "quest_scores: null pointer");
  SAH_REQUIRE(B > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0 && Sq > 0 && S > 0 && page_size > 0,
              "quest_scores: bad extents");
  if (D % 8 != 0 || D > QS_MAXD)
    return sah_fail(SAH_ERR_UNSUPPORTED, "quest_scores: head dimension %d (multiples of 8 up to %d)", D,
                    QS_MAXD);
  if (bias != nullptr && bias_s_h != 0)
    return sah_fail(SAH_ERR_UNSUPPORTED, "quest_scores: the attention mask must be shared by the heads");
  const int64_t P = sah_ceil_div(S, page_size);
  SAH_REQUIRE(P <= P_cap, "quest_scores: page capacity below the page count");
  SAH_REQUIRE(((uintptr_t)pmin & 15) == 0 && ((uintptr_t)pmax & 15) == 0, "quest_scores: bounds must be 16-byte aligned");
  const int64_t rows = (int64_t)B * Hq * Sq;
  SAH_REQUIRE(rows <= 65535, "quest_scores: more than 65535 mask rows");
  const int64_t elt = dtype == SAH_BF16 ? 2 : 4;
  int pages = QS_PAGES;
  const bool direct = dtype != SAH_BF16 && rows * P >= QS_DIRECT && D <= 256;
  while (!direct && pages > 32 && (2 * pages * D * elt > QS_BOUND_BYTES(elt) || P <= pages / 2)) pages /= 2;
  const int qrows = direct ? 1 : QS_ROWS;
  const size_t smem = (size_t)((direct ? 0 : 2 * pages) + qrows) * D * elt;
  dim3 grid((unsigned)sah_ceil_div(P, pages), (unsigned)sah_ceil_div((int64_t)(Hq / Hkv) * Sq, qrows),
            (unsigned)((int64_t)B * Hkv));
  sah_prof_begin(SAH_PROF_QUEST, (cudaStream_t)stream);
  const dim3 block((unsigned)pages, (unsigned)qrows);
#define QS_LAUNCH(T, STAGED)                                                                                       \
  do {                                                                                                             \
    if (smem > 48 * 1024) {                                                                                        \
      const cudaError_t e = cudaFuncSetAttribute(                                                                  \
          quest_scores_kernel<T, STAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, QS_SMEM);                   \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "quest_scores attr: %s", cudaGetErrorString(e));         \
    }                                                                                                              \
    sah_launch_chain(quest_scores_kernel<T, STAGED>, grid, block, smem, (cudaStream_t)stream, (const T*)q, qs_b,   \
        qs_h, qs_q, (const T*)pmin, (const T*)pmax, P_cap, Hq, Hkv, Sq, S, D, page_size, (const T*)bias, bias_s_b, \
        bias_s_q, (T*)scores);                                                                                     \
  } while (0)
  if (dtype == SAH_BF16) QS_LAUNCH(__nv_bfloat16, true);
  else if (dtype != SAH_F32) return sah_fail(SAH_ERR_INVALID, "unknown dtype %d", dtype);
  else if (direct) QS_LAUNCH(float, false);
  else QS_LAUNCH(float, true);
#undef QS_LAUNCH
  SAH_LAUNCH_CHECK("quest_scores");
  sah_prof_end(SAH_PROF_QUEST, (cudaStream_t)stream);
  return SAH_OK;
}

// ---- chosen pages -> key bitmap --------------------------------------------------------------
template <typename T>
__global__ void quest_expand_kernel(const uint32_t* __restrict__ page_bits, int64_t Wp,
                                    const uint32_t* __restrict__ prev_bits, const T* __restrict__ bias,
                                    int64_t bias_s_b, int64_t bias_s_q, int Hq, int Sq, int64_t S,
                                    int64_t W, int page_size, uint32_t* __restrict__ out_bits) {
  sah_pdl_entry_early();
  const int64_t row = blockIdx.y;
  const int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= W) return;
  const uint32_t* pg = page_bits + row * Wp;
  uint32_t bits = 0u;
  const int64_t c0 = w * 32;
  if (page_size % 32 == 0) {   // the word lies inside one page
    const int64_t page = c0 / page_size;
    if (c0 < S && ((pg[page >> 5] >> (page & 31)) & 1u)) bits = 0xffffffffu;
  } else {
#pragma unroll 4
    for (int i = 0; i < 32; ++i) {
      const int64_t page = (c0 + i) / page_size;
      if (c0 + i < S && ((pg[page >> 5] >> (page & 31)) & 1u)) bits |= 1u << i;
    }
  }
  if (c0 + 32 > S) bits &= (c0 >= S) ? 0u : ((1u << (S - c0)) - 1u);
  if (prev_bits != nullptr) bits |= prev_bits[row * W + w];
  if (bias != nullptr && bits) {   // keys the attention mask forbids leave the mask (:188-191)
    const int qi = (int)(row % Sq);
    const int64_t b = row / Sq / Hq;
    const T* br = bias + b * bias_s_b + qi * bias_s_q;
    uint32_t allowed = 0u;
    for (int i = 0; i < 32; ++i)
      if (c0 + i < S && sah_to_float<T>(br[c0 + i]) >= 0.f) allowed |= 1u << i;
    bits &= allowed;
  }
  out_bits[row * W + w] = bits;
}

extern "C" int sah_quest_expand(const uint32_t* page_bits, int64_t Wp, const uint32_t* prev_bits,
                                const void* bias, int dtype, int64_t bias_s_b, int64_t bias_s_h,
                                int64_t bias_s_q, int B, int Hq, int Sq, int64_t S, int64_t W,
                                int page_size, uint32_t* out_bits, void* stream) {
  SAH_REQUIRE(page_bits && out_bits, "quest_expand: null pointer");
  SAH_REQUIRE(B > 0 && Hq > 0 && Sq > 0 && S > 0 && W * 32 >= S && page_size > 0, "quest_expand: bad extents");
  SAH_REQUIRE(Wp * 32 >= sah_ceil_div(S, page_size), "quest_expand: page bitmap too short");
  if (bias != nullptr && bias_s_h != 0)
    return sah_fail(SAH_ERR_UNSUPPORTED, "quest_expand: the attention mask must be shared by the heads");
  const int64_t rows = (int64_t)B * Hq * Sq;
  SAH_REQUIRE(rows <= 65535, "quest_expand: more than 65535 mask rows");
  dim3 grid((unsigned)sah_ceil_div(W, 256), (unsigned)rows);
  SAH_DISPATCH_DTYPE(dtype, T, {
    sah_launch_chain(quest_expand_kernel<T>, grid, 256, 0, (cudaStream_t)stream, page_bits, Wp, prev_bits,
        (const T*)bias, bias_s_b, bias_s_q, Hq, Sq, S, W, page_size, out_bits);
  });
  SAH_LAUNCH_CHECK("quest_expand");
  return SAH_OK;
}
