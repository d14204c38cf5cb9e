// PQCache kernels (maskers/fixed/implementations/pq_top_k.py and utils/pq_utils.py):
//   sah_pq_assign         nearest centroid of every key sub-vector (k-means assignment
//                         step, pq_utils.py:246-255 + :353; new-key quantisation,
//                         pq_top_k.py:388-404)
//   sah_pq_accumulate     per-cluster sums and counts of one Lloyd iteration
//   sah_pq_update         new centres, empty-cluster reseeding and centre shift
//                         (pq_utils.py:360-423)
//   sah_pq_scores         query-centroid lookup tables and the code stream
//                         (pq_top_k.py:406-490)
//
// A "group" is one (batch, KV head, sub-vector): groups = B * Hkv * n_sub,
// group id = (b * Hkv + kvh) * n_sub + sub.  Codes are bytes laid out
// [B][Hkv][capacity][n_sub], i.e. the n_sub codes of one key are contiguous, so the
// scoring stream reads one 16-byte word per key for n_sub = 16.
#include "sah_common.cuh"

#define PQ_MAX_SUBD 16
#define PQ_TILE 256

// Squared distance in the fixed order the CPU restatement follows: dimensions
// ascending, (x - c) * (x - c) rounded, then added.
__device__ __forceinline__ float pq_dist(const float* x, const float* c, int sub_d) {
  float d = 0.f;
  for (int j = 0; j < sub_d; ++j) {
    const float t = __fsub_rn(x[j], c[j]);
    d = __fadd_rn(d, __fmul_rn(t, t));
  }
  return d;
}

// The same distance with every operation rounded to the key dtype: what the
// reference's quantisation of appended keys computes, since there both the keys and
// the stored centroids are dtype tensors (pq_top_k.py:388-404).
template <typename T>
__device__ __forceinline__ float pq_dist_dtype(const float* x, const float* c, int sub_d) {
  float d = 0.f;
  for (int j = 0; j < sub_d; ++j) {
    const float t = sah_round_to<T>(__fsub_rn(x[j], c[j]));
    d = __fadd_rn(d, sah_round_to<T>(__fmul_rn(t, t)));
  }
  return sah_round_to<T>(d);
}

template <typename T, bool DTYPE_MATH>
__global__ void __launch_bounds__(PQ_TILE)
pq_assign_kernel(const T* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int Hkv,
                 int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub, int sub_d,
                 int n_cent, const float* __restrict__ centroids, uint8_t* __restrict__ codes,
                 int64_t cap, const int* __restrict__ done) {
  extern __shared__ float pq_cent_sm[];  // [n_cent][sub_d]
  if (done && *done) return;
  const int sub = blockIdx.y;
  const int64_t bk = blockIdx.z;
  const int kvh = (int)(bk % Hkv);
  const int64_t b = bk / Hkv;
  const int64_t grp = bk * n_sub + sub;
  for (int i = threadIdx.x; i < n_cent * sub_d; i += PQ_TILE)
    pq_cent_sm[i] = centroids[grp * n_cent * sub_d + i];
  __syncthreads();
  const int64_t j = key_begin + (int64_t)blockIdx.x * PQ_TILE + threadIdx.x;
  if (j >= key_end) return;
  const T* xr = x + b * xs_b + kvh * xs_h + j * xs_s + sub * sub_d;
  float xv[PQ_MAX_SUBD];
  for (int d = 0; d < sub_d; ++d) xv[d] = sah_to_float<T>(xr[d]);
  float best = INFINITY;
  int arg = 0;
  for (int c = 0; c < n_cent; ++c) {
    const float dist = DTYPE_MATH ? pq_dist_dtype<T>(xv, pq_cent_sm + c * sub_d, sub_d)
                                  : pq_dist(xv, pq_cent_sm + c * sub_d, sub_d);
    if (dist < best) { best = dist; arg = c; }  // first minimum wins, as argmin does
  }
  codes[(bk * cap + (j - init_offset)) * n_sub + sub] = (uint8_t)arg;
}

// The same for the keys that a decode step appends: a warp takes one sub-vector of one key and
// deals the centroids to its lanes, straight from global memory (8 heads x 16 sub-vectors x 1 key
// took 56 us with one thread walking all 256 centroids of a CTA's table, 7.8 us now, all latency).
#define PQ_FEW_KEYS 16
template <typename T, bool DTYPE_MATH>
__global__ void __launch_bounds__(256)
pq_assign_few_kernel(const T* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int Hkv,
                     int64_t key_begin, int n_keys, int64_t init_offset, int n_sub, int sub_d, int n_cent,
                     int64_t items, const float* __restrict__ centroids, uint8_t* __restrict__ codes,
                     int64_t cap, const int* __restrict__ done) {
  const int lane = threadIdx.x & 31;
  const int64_t item = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);  // (group, key)
  if (item >= items || (done && *done)) return;
  const int64_t grp = item / n_keys, j = key_begin + item % n_keys;
  const int sub = (int)(grp % n_sub);
  const int64_t bk = grp / n_sub;
  const T* xr = x + bk / Hkv * xs_b + bk % Hkv * xs_h + j * xs_s + sub * sub_d;
  float xv[PQ_MAX_SUBD];
#pragma unroll
  for (int d = 0; d < PQ_MAX_SUBD; ++d) xv[d] = d < sub_d ? sah_to_float<T>(xr[d]) : 0.f;
  float best = INFINITY;
  int arg = 256;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int c = i * 32 + lane;
    if (c < n_cent) {
      const float* cp = centroids + (grp * n_cent + c) * sub_d;
      float dist = 0.f;  // pq_dist / pq_dist_dtype with the sub-vector in registers
#pragma unroll
      for (int d = 0; d < PQ_MAX_SUBD; ++d)
        if (d < sub_d) {
          const float t = __fsub_rn(xv[d], cp[d]);
          if (DTYPE_MATH) {
            const float r = sah_round_to<T>(t);
            dist = __fadd_rn(dist, sah_round_to<T>(__fmul_rn(r, r)));
          } else {
            dist = __fadd_rn(dist, __fmul_rn(t, t));
          }
        }
      if (DTYPE_MATH) dist = sah_round_to<T>(dist);
      if (dist < best) { best = dist; arg = c; }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
    if (ob < best || (ob == best && oa < arg)) { best = ob; arg = oa; }  // first minimum wins
  }
  if (lane == 0) codes[(bk * cap + (j - init_offset)) * n_sub + sub] = (uint8_t)(arg < 256 ? arg : 0);
}

// `done`, where the calls of this file take it: a word on the device that is not 0 once the clustering
// has converged; the kernels of the iterations behind it return at once.
static int pq_assign_run(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s,
                         int B, int Hkv, int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub,
                         int sub_d, int n_cent, const float* centroids, uint8_t* codes, int64_t cap, int dtype_math,
                         const int* done, void* stream) {
  SAH_REQUIRE(x && centroids && codes, "pq_assign: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && n_sub > 0 && sub_d > 0 && n_cent > 0, "pq_assign: bad extents");
  SAH_REQUIRE(init_offset <= key_begin && key_begin <= key_end && key_end - init_offset <= cap,
              "pq_assign: bad key range");
  if (sub_d > PQ_MAX_SUBD || n_cent > 256)
    return sah_fail(SAH_ERR_UNSUPPORTED, "pq_assign: sub-vector dim %d (<= %d) / %d centroids (<= 256)",
                    sub_d, PQ_MAX_SUBD, n_cent);
  if (key_begin == key_end) return SAH_OK;
  if (key_end - key_begin <= PQ_FEW_KEYS) {
    const int n_keys = (int)(key_end - key_begin);
    const int64_t items = (int64_t)B * Hkv * n_sub * n_keys;
    const unsigned few = (unsigned)sah_ceil_div(items, (int64_t)8);
    SAH_DISPATCH_DTYPE(dtype, T, {
      if (dtype_math)
        pq_assign_few_kernel<T, true><<<few, 256, 0, (cudaStream_t)stream>>>(
            (const T*)x, xs_b, xs_h, xs_s, Hkv, key_begin, n_keys, init_offset, n_sub, sub_d, n_cent, items,
            centroids, codes, cap, done);
      else
        pq_assign_few_kernel<T, false><<<few, 256, 0, (cudaStream_t)stream>>>(
            (const T*)x, xs_b, xs_h, xs_s, Hkv, key_begin, n_keys, init_offset, n_sub, sub_d, n_cent, items,
            centroids, codes, cap, done);
    });
    SAH_LAUNCH_CHECK("pq_assign_few");
    return SAH_OK;
  }
  dim3 grid((unsigned)sah_ceil_div(key_end - key_begin, PQ_TILE), (unsigned)n_sub,
            (unsigned)((int64_t)B * Hkv));
  const size_t smem = (size_t)n_cent * sub_d * sizeof(float);
  SAH_DISPATCH_DTYPE(dtype, T, {
    if (dtype_math)
      pq_assign_kernel<T, true><<<grid, PQ_TILE, smem, (cudaStream_t)stream>>>(
          (const T*)x, xs_b, xs_h, xs_s, Hkv, key_begin, key_end, init_offset, n_sub, sub_d, n_cent,
          centroids, codes, cap, done);
    else
      pq_assign_kernel<T, false><<<grid, PQ_TILE, smem, (cudaStream_t)stream>>>(
          (const T*)x, xs_b, xs_h, xs_s, Hkv, key_begin, key_end, init_offset, n_sub, sub_d, n_cent,
          centroids, codes, cap, done);
  });
  SAH_LAUNCH_CHECK("pq_assign");
  return SAH_OK;
}

extern "C" int sah_pq_assign(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s,
                             int B, int Hkv, int64_t key_begin, int64_t key_end,
                             int64_t init_offset, int n_sub, int sub_d, int n_cent,
                             const float* centroids, uint8_t* codes, int64_t cap, int dtype_math,
                             void* stream) {
  return pq_assign_run(x, dtype, xs_b, xs_h, xs_s, B, Hkv, key_begin, key_end, init_offset, n_sub, sub_d, n_cent,
                       centroids, codes, cap, dtype_math, nullptr, stream);
}

#include "sah_pq_tc.cuh"

// The assignment step on the tensor cores; same codes as sah_pq_assign(dtype_math = 0).
static int pq_assign_tc_run(const void* x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int B, int Hkv,
                            int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub, int sub_d,
                            int n_cent, const float* centroids, uint8_t* codes, int64_t cap, int* errflag,
                            int sm_count, const int* done, void* stream) {
  SAH_REQUIRE(x && centroids && codes && errflag, "pq_assign_tc: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && n_sub > 0, "pq_assign_tc: bad extents");
  SAH_REQUIRE(init_offset <= key_begin && key_begin <= key_end && key_end - init_offset <= cap,
              "pq_assign_tc: bad key range");
  if (sub_d != 8 || n_cent < 16 || n_cent > 256 || n_cent % 16 != 0)
    return sah_fail(SAH_ERR_UNSUPPORTED, "pq_assign_tc: sub-vectors of 8 channels and 16..256 centroids in "
                    "multiples of 16 (got %d, %d)", sub_d, n_cent);
  SAH_REQUIRE((xs_s * 2) % 16 == 0 && (xs_h * 2) % 16 == 0 && (xs_b * 2) % 16 == 0 && ((uintptr_t)x % 16) == 0,
              "pq_assign_tc: key rows must be 16-byte aligned");
  if (key_begin == key_end) return SAH_OK;
  if (sm_count <= 0) sm_count = 148;
  // Four neighbouring sub-vectors per CTA (a key's 64 bytes, one 4-byte store of codes) when the
  // layout allows it, else one; also one while every (sub-vector, tile) has a group of warps to itself
  // (128 groups x 64 keys x 256 centroids 23.4 us by fours, 7.3 us one by one).  n_cent padded to a
  // power-of-two number of 32-column blocks.
  const int64_t tiles = sah_ceil_div(key_end - key_begin, (int64_t)PTC_TILE);
  auto ctas = [&](int64_t blocks) { return tiles == 1 ? blocks : (blocks * tiles + 1) / 2; };  // two tiles of a block each
  const int64_t groups = (int64_t)B * Hkv * n_sub;
  const int ns = n_sub % 4 == 0 && (reinterpret_cast<uintptr_t>(codes) & 3) == 0 && ctas(groups) > sm_count ? 4 : 1;
  const int64_t n_blocks = groups / ns;
  const unsigned grid = (unsigned)(ctas(n_blocks) < sm_count ? ctas(n_blocks) : sm_count);
  const cudaStream_t st = (cudaStream_t)stream;
#define PTC_LAUNCH(NS, NB)                                                                                       \
  do {                                                                                                           \
    static bool allowed[64] = {};                                                                                \
    const cudaError_t e = sah_allow_smem(pq_assign_tc_kernel<NS, NB>, PtcCfg<NS>::SMEM, allowed);                \
    if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "pq_assign_tc attr: %s", cudaGetErrorString(e));         \
    pq_assign_tc_kernel<NS, NB><<<grid, PTC_THREADS, PtcCfg<NS>::SMEM, st>>>(                                    \
        reinterpret_cast<const __nv_bfloat16*>(x), xs_b, xs_h, xs_s, Hkv, key_begin, key_end, init_offset,       \
        n_sub, n_cent, n_blocks, centroids, codes, cap, errflag, done);                                                \
  } while (0)
#define PTC_LAUNCH_NS(NS)                   \
  do {                                      \
    if (n_cent <= 32) PTC_LAUNCH(NS, 1);    \
    else if (n_cent <= 64) PTC_LAUNCH(NS, 2);  \
    else if (n_cent <= 128) PTC_LAUNCH(NS, 4); \
    else PTC_LAUNCH(NS, 8);                 \
  } while (0)
  if (ns == 4) PTC_LAUNCH_NS(4);
  else PTC_LAUNCH_NS(1);
#undef PTC_LAUNCH_NS
#undef PTC_LAUNCH
  SAH_LAUNCH_CHECK("pq_assign_tc");
  return SAH_OK;
}

extern "C" int sah_pq_assign_tc(const void* x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int B, int Hkv,
                                int64_t key_begin, int64_t key_end, int64_t init_offset, int n_sub,
                                int sub_d, int n_cent, const float* centroids, uint8_t* codes, int64_t cap,
                                int* errflag, int sm_count, void* stream) {
  return pq_assign_tc_run(x, xs_b, xs_h, xs_s, B, Hkv, key_begin, key_end, init_offset, n_sub, sub_d, n_cent,
                          centroids, codes, cap, errflag, sm_count, nullptr, stream);
}

// Cluster sums in fp64 (so that the summation order does not reach the fp32 result) and counts.
// A CTA takes strips of PQA_STRIP keys of one group: it sorts the strip's keys by code (a
// counting sort with integer atomics in shared memory), then two threads per centroid walk the
// centroid's keys, each adding half of the channels into fp64 registers that live across the
// strips; the registers go to global memory with one atomic per (centroid, channel) and CTA.
// Below 129 centroids several such pairs of lanes (`shares`) take every so many-th key of a centroid
// and add up in the warp (16 centroids, 128 groups x 65472 keys: 258 us in bfloat16 and 1374 us in
// float32 with a pair each, 76 us and 176 us this way).
// Bound: shared-memory integer atomics and L2 (every 32-byte sector of a key is fetched by the
// CTAs of two sub-vectors).  8 KV heads x 65472 keys x 16 sub-vectors: 96 us with eight keys of a
// centroid in flight, 122 us with four and three CTAs per SM; with one fp64 shared-memory atomic
// per key and channel -- a compare-and-swap loop -- it took 812 us.  Sub-vectors
// of more than 16 channels are cut into blocks of 16 (`cblocks`), a CTA each; the first block counts.
#define PQA_THREADS 512
#define PQA_STRIP 4096

template <typename T>
__global__ void __launch_bounds__(PQA_THREADS, 2)
pq_accumulate_kernel(const T* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s, int Hkv,
                     int64_t n_keys, int64_t init_offset, int n_sub, int sub_d, int n_cent, int cblocks, int shares, int vec8,
                     const uint8_t* __restrict__ codes, int64_t cap, double* __restrict__ sums,
                     int* __restrict__ counts, const int* __restrict__ done) {
  if (done && *done) return;
  __shared__ int pos_sm[256];              // histogram, then the next free slot of every centroid
  __shared__ int start_sm[257];
  __shared__ int scan_sm[33];
  __shared__ uint16_t order_sm[PQA_STRIP]; // key numbers of the strip, sorted by code
  constexpr int HALF = (PQ_MAX_SUBD + 1) / 2;
  constexpr int PER = PQA_STRIP / PQA_THREADS;
  const int tid = threadIdx.x;
  const int sub = blockIdx.y / cblocks, c_lo = (blockIdx.y - sub * cblocks) * PQ_MAX_SUBD;
  const int64_t bk = blockIdx.z;
  const int kvh = (int)(bk % Hkv);
  const int64_t b = bk / Hkv;
  const int64_t grp = bk * n_sub + sub;
  const int cent = (tid >> 1) / shares, share = (tid >> 1) - cent * shares;
  const int nch = sub_d - c_lo < PQ_MAX_SUBD ? sub_d - c_lo : PQ_MAX_SUBD;  // channels of this CTA
  const int half = (nch + 1) / 2;          // channels of the even threads
  const int d0 = c_lo + ((tid & 1) ? half : 0), nd = (tid & 1) ? nch - half : half;
  const T* xg = x + b * xs_b + kvh * xs_h + init_offset * xs_s + sub * sub_d + d0;
  const uint8_t* cg = codes + bk * cap * n_sub + sub;
  double acc[HALF];
  int count = 0;
#pragma unroll
  for (int i = 0; i < HALF; ++i) acc[i] = 0.0;
  for (int64_t j0 = (int64_t)blockIdx.x * PQA_STRIP; j0 < n_keys; j0 += (int64_t)gridDim.x * PQA_STRIP) {
    if (tid < 256) pos_sm[tid] = 0;
    int code[PER];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int64_t j = j0 + i * PQA_THREADS + tid;
      code[i] = j < n_keys ? cg[j * n_sub] : -1;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (code[i] >= 0) atomicAdd(&pos_sm[code[i]], 1);
    __syncthreads();
    int total;
    const int before = sah_block_excl_scan<int>(tid < 256 ? pos_sm[tid] : 0, scan_sm, &total);
    if (tid < 256) { start_sm[tid] = before; pos_sm[tid] = before; }
    if (tid == 0) start_sm[256] = total;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; ++i)
      if (code[i] >= 0) order_sm[atomicAdd(&pos_sm[code[i]], 1)] = (uint16_t)(i * PQA_THREADS + tid);
    __syncthreads();
    const int e1 = start_sm[cent + 1];
    int e = start_sm[cent];
    if (share == 0) count += e1 - e;
    e += share;
    const T* xs = xg + j0 * xs_s;
    if (sizeof(T) == 2 && vec8) {  // four channels in 8 aligned bytes; eight keys in flight
      for (; e + 7 * shares < e1; e += 8 * shares) {
        uint2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          v[u] = *reinterpret_cast<const uint2*>(xs + (int64_t)order_sm[e + u * shares] * xs_s);
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          acc[0] += (double)__uint_as_float(v[u].x << 16);
          acc[1] += (double)__uint_as_float(v[u].x & 0xffff0000u);
          acc[2] += (double)__uint_as_float(v[u].y << 16);
          acc[3] += (double)__uint_as_float(v[u].y & 0xffff0000u);
        }
      }
      {  // the last few, all in flight as well
        uint2 v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u)
          v[u] = e + u * shares < e1 ? *reinterpret_cast<const uint2*>(xs + (int64_t)order_sm[e + u * shares] * xs_s)
                                     : make_uint2(0u, 0u);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (e + u * shares < e1) {
            acc[0] += (double)__uint_as_float(v[u].x << 16);
            acc[1] += (double)__uint_as_float(v[u].x & 0xffff0000u);
            acc[2] += (double)__uint_as_float(v[u].y << 16);
            acc[3] += (double)__uint_as_float(v[u].y & 0xffff0000u);
          }
      }
    } else {
      for (; e < e1; e += shares) {
        const T* xr = xs + (int64_t)order_sm[e] * xs_s;
#pragma unroll
        for (int i = 0; i < HALF; ++i)
          if (i < nd) acc[i] += (double)sah_to_float<T>(xr[i]);
      }
    }
    __syncthreads();  // the sorted list and the starts are done with
  }
  bool any = count > 0;
  if (shares > 1) {  // up to 16 shares of a centroid lie in one warp
    const int width = shares < 16 ? shares : 16;
    for (int o = 1; o < width; o <<= 1)
#pragma unroll
      for (int i = 0; i < HALF; ++i) acc[i] += __shfl_xor_sync(0xffffffffu, acc[i], 2 * o);
    if (share % width != 0) return;
    any = shares > 16 || count > 0;
  }
  if (cent < n_cent && any) {
    double* out = sums + (grp * n_cent + cent) * sub_d + d0;
#pragma unroll
    for (int i = 0; i < HALF; ++i)
      if (i < nd) atomicAdd(out + i, acc[i]);
    if ((tid & 1) == 0 && c_lo == 0 && count > 0) atomicAdd(&counts[grp * n_cent + cent], count);
  }
}

static int pq_accumulate_run(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s, int B, int Hkv,
                             int64_t n_keys, int64_t init_offset, int n_sub, int sub_d, int n_cent,
                             const uint8_t* codes, int64_t cap, double* sums, int* counts, const int* done,
                             void* stream) {
  SAH_REQUIRE(x && codes && sums && counts, "pq_accumulate: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && n_sub > 0 && sub_d > 0 && n_cent > 0 && n_keys >= 0,
              "pq_accumulate: bad extents");
  if (n_keys == 0) return SAH_OK;
  // one wave of two CTAs per SM; the strips of a slice share the CTA's registers
  const int cblocks = (sub_d + PQ_MAX_SUBD - 1) / PQ_MAX_SUBD;
  const int64_t groups = (int64_t)B * Hkv * n_sub * cblocks;
  int64_t slices = (int64_t)2 * 148 / groups;
  if (slices < 1) slices = 1;
  const int64_t strips = sah_ceil_div(n_keys, (int64_t)PQA_STRIP);
  if (slices > strips) slices = strips;
  dim3 grid((unsigned)slices, (unsigned)(n_sub * cblocks), (unsigned)((int64_t)B * Hkv));
  // pairs of threads per centroid: what is left of 256 of them, a power of two
  int shares = 1;
  while (shares * 2 * n_cent <= PQA_THREADS / 2) shares *= 2;
  const int vec8 = sub_d == 8 && (reinterpret_cast<uintptr_t>(x) & 7) == 0 && xs_s % 4 == 0 && xs_h % 4 == 0 &&
                   xs_b % 4 == 0;
  SAH_DISPATCH_DTYPE(dtype, T, {
    pq_accumulate_kernel<T><<<grid, PQA_THREADS, 0, (cudaStream_t)stream>>>(
        (const T*)x, xs_b, xs_h, xs_s, Hkv, n_keys, init_offset, n_sub, sub_d, n_cent, cblocks, shares, vec8, codes, cap,
        sums, counts, done);
  });
  SAH_LAUNCH_CHECK("pq_accumulate");
  return SAH_OK;
}

extern "C" int sah_pq_accumulate(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s,
                                 int B, int Hkv, int64_t n_keys, int64_t init_offset, int n_sub,
                                 int sub_d, int n_cent, const uint8_t* codes, int64_t cap,
                                 double* sums, int* counts, void* stream) {
  return pq_accumulate_run(x, dtype, xs_b, xs_h, xs_s, B, Hkv, n_keys, init_offset, n_sub, sub_d, n_cent, codes, cap,
                           sums, counts, nullptr, stream);
}

// new centre = fp32(sum) / fp32(count); an empty cluster takes the key sub-vector at
// reseed[group][cluster] (pq_utils.py:384-396); shift2[group] = (sum over clusters of
// the centre's Euclidean move)^2, the quantity compared with the tolerance (:399-423).
// With `state` (the words that sah_pq_kmeans_step keeps) the sums and counts are cleared for the next
// iteration and the last block makes the comparison.
struct PqState {
  int done, iterations, err, open, ticket;
};
template <typename T>
__global__ void pq_update_kernel(const T* __restrict__ x, int64_t xs_b, int64_t xs_h, int64_t xs_s,
                                 int Hkv, int64_t init_offset, int n_sub, int sub_d, int n_cent,
                                 double* __restrict__ sums, int* __restrict__ counts,
                                 const int64_t* __restrict__ reseed, float* __restrict__ centroids,
                                 float* __restrict__ shift2, PqState* __restrict__ state, int* __restrict__ seen) {
  __shared__ float scratch[33];
  if (state && state->done) return;
  const int64_t grp = blockIdx.x;
  const int sub = (int)(grp % n_sub);
  const int64_t bk = grp / n_sub;
  const int kvh = (int)(bk % Hkv);
  const int64_t b = bk / Hkv;
  float move = 0.f;
  const int c = threadIdx.x;
  if (c < n_cent) {
    // everything that may be needed is requested before the first use, 16 channels at a time (a
    // channel at a time, each with its own loads, took 16 to 29 us for 128 groups of 256 centres of
    // 8 channels; 4.3 us this way)
    const int cnt = counts[grp * n_cent + c];
    const T* xr = nullptr;
    if (cnt <= 0) xr = x + b * xs_b + kvh * xs_h + (reseed[grp * n_cent + c] + init_offset) * xs_s + sub * sub_d;
    float d2 = 0.f;
    for (int c_lo = 0; c_lo < sub_d; c_lo += PQ_MAX_SUBD) {
      double* sp = sums + (grp * n_cent + c) * sub_d + c_lo;
      float* cp = centroids + (grp * n_cent + c) * sub_d + c_lo;
      const int nch = sub_d - c_lo;
      double sv[PQ_MAX_SUBD];
      float old[PQ_MAX_SUBD];
#pragma unroll
      for (int d = 0; d < PQ_MAX_SUBD; ++d) {
        sv[d] = d < nch ? sp[d] : 0.0;
        old[d] = d < nch ? cp[d] : 0.f;
      }
#pragma unroll
      for (int d = 0; d < PQ_MAX_SUBD; ++d)
        if (d < nch) {
          const float nv = cnt > 0 ? __fdiv_rn((float)sv[d], (float)cnt) : sah_to_float<T>(xr[c_lo + d]);
          const float t = __fsub_rn(nv, old[d]);
          d2 = __fadd_rn(d2, __fmul_rn(t, t));
          cp[d] = nv;
          if (state) sp[d] = 0.0;
        }
    }
    move = sqrtf(d2);
    if (state) counts[grp * n_cent + c] = 0;
  }
  float total;
  sah_block_excl_scan<float>(move, scratch, &total);
  if (threadIdx.x != 0) return;
  if (shift2) shift2[grp] = total * total;
  if (!state) return;
  if (!(total * total < 1e-4f)) atomicAdd(&state->open, 1);
  __threadfence();
  if (atomicAdd(&state->ticket, 1) == (int)gridDim.x - 1) {  // every block has read `done` by now
    state->iterations += 1;
    const int done = atomicExch(&state->open, 0) == 0;
    state->done = done;
    state->ticket = 0;
    if (seen) {
      seen[0] = done;
      seen[1] = state->iterations;
      seen[2] = state->err;
      __threadfence_system();
    }
  }
}

extern "C" int sah_pq_update(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s,
                             int B, int Hkv, int64_t init_offset, int n_sub, int sub_d, int n_cent,
                             const double* sums, const int* counts, const int64_t* reseed,
                             float* centroids, float* shift2, void* stream) {
  SAH_REQUIRE(x && sums && counts && reseed && centroids && shift2, "pq_update: null pointer");
  SAH_REQUIRE(n_cent > 0 && n_cent <= 256, "pq_update: 1..256 centroids");
  const int64_t groups = (int64_t)B * Hkv * n_sub;
  SAH_DISPATCH_DTYPE(dtype, T, {
    pq_update_kernel<T><<<(unsigned)groups, 256, 0, (cudaStream_t)stream>>>(
        (const T*)x, xs_b, xs_h, xs_s, Hkv, init_offset, n_sub, sub_d, n_cent, const_cast<double*>(sums),
        const_cast<int*>(counts), reseed, centroids, shift2, nullptr, nullptr);
  });
  SAH_LAUNCH_CHECK("pq_update");
  return SAH_OK;
}

extern "C" int sah_pq_kmeans_step(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s, int B, int Hkv,
                                  int64_t n_keys, int64_t init_offset, int n_sub, int sub_d, int n_cent, int what,
                                  const int64_t* reseed, float* centroids, uint8_t* codes, int64_t cap, double* sums,
                                  int* counts, int* state, int* seen, int use_tc, int sm_count, void* stream) {
  SAH_REQUIRE(x && centroids && codes && sums && counts && state && (reseed || !(what & SAH_KMEANS_UPDATE)),
              "pq_kmeans: null pointer");
  SAH_REQUIRE(B > 0 && Hkv > 0 && n_sub > 0 && sub_d > 0 && n_keys >= 0, "pq_kmeans: bad extents");
  SAH_REQUIRE(n_cent > 0 && n_cent <= 256, "pq_kmeans: 1..256 centroids");
  const int64_t groups = (int64_t)B * Hkv * n_sub;
  const cudaStream_t st = (cudaStream_t)stream;
  PqState* ps = reinterpret_cast<PqState*>(state);
  if (what & SAH_KMEANS_BEGIN) {
    cudaError_t e = cudaMemsetAsync(sums, 0, (size_t)(groups * n_cent * sub_d) * sizeof(double), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(counts, 0, (size_t)(groups * n_cent) * sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(state, 0, sizeof(PqState), st);
    if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "pq_kmeans: %s", cudaGetErrorString(e));
  }
  if (what & SAH_KMEANS_UPDATE) {
    SAH_DISPATCH_DTYPE(dtype, T, {
      pq_update_kernel<T><<<(unsigned)groups, 256, 0, st>>>((const T*)x, xs_b, xs_h, xs_s, Hkv, init_offset, n_sub,
                                                            sub_d, n_cent, sums, counts, reseed, centroids, nullptr, ps,
                                                            seen);
    });
    SAH_LAUNCH_CHECK("pq_update");
  }
  if (what & SAH_KMEANS_ASSIGN) {
    int rc = use_tc ? pq_assign_tc_run(x, xs_b, xs_h, xs_s, B, Hkv, init_offset, init_offset + n_keys, init_offset,
                                       n_sub, sub_d, n_cent, centroids, codes, cap, &ps->err, sm_count, &ps->done, stream)
                    : pq_assign_run(x, dtype, xs_b, xs_h, xs_s, B, Hkv, init_offset, init_offset + n_keys, init_offset,
                                    n_sub, sub_d, n_cent, centroids, codes, cap, 0, &ps->done, stream);
    if (rc == SAH_OK)
      rc = pq_accumulate_run(x, dtype, xs_b, xs_h, xs_s, B, Hkv, n_keys, init_offset, n_sub, sub_d, n_cent, codes, cap,
                             sums, counts, &ps->done, stream);
    if (rc != SAH_OK) return rc;
  }
  return SAH_OK;
}

extern "C" int sah_pq_kmeans(const void* x, int dtype, int64_t xs_b, int64_t xs_h, int64_t xs_s, int B, int Hkv,
                             int64_t n_keys, int64_t init_offset, int n_sub, int sub_d, int n_cent, int n_iter,
                             const int64_t* const* reseed, float* centroids, uint8_t* codes, int64_t cap,
                             double* sums, int* counts, int* state, int use_tc, int sm_count, void* stream) {
  SAH_REQUIRE(reseed && n_iter >= 0, "pq_kmeans: no re-seeding indices");
  for (int it = 0; it < n_iter; ++it) SAH_REQUIRE(reseed[it], "pq_kmeans: null pointer");
  int rc = SAH_OK;
  for (int it = 0; it <= n_iter && rc == SAH_OK; ++it)
    rc = sah_pq_kmeans_step(x, dtype, xs_b, xs_h, xs_s, B, Hkv, n_keys, init_offset, n_sub, sub_d, n_cent,
                            (it == 0 ? SAH_KMEANS_BEGIN : SAH_KMEANS_UPDATE) | (it < n_iter ? SAH_KMEANS_ASSIGN : 0),
                            it > 0 ? reseed[it - 1] : nullptr, centroids, codes, cap, sums, counts, state, nullptr, use_tc,
                            sm_count, stream);
  return rc;
}

// ---------------------------------------------------------------------------
// Scores.  Per CTA: the lookup tables of up to PQ_ROWS mask rows of one KV group
// (lut[r][sub][c] = q_sub . centroid, fma over ascending dims, rounded to the
// dtype), then one thread per key sums its n_sub table entries in ascending
// sub-vector order in fp32 and rounds once (the reference sums a dtype tensor
// with an fp32 accumulator, pq_top_k.py:481-488).
// ---------------------------------------------------------------------------
#define PQ_ROWS 4
#define PQ_SCORES_SMEM (200 * 1024)  // tables and queries of a CTA

// One CTA: builds the table of one (KV group, block of 4 rows) in shared memory --
// lut[sub][c][rr] = q_sub(row rblk*4 + rr) . centroid(sub, c), fma over ascending dims, rounded
// to the dtype; rows past R hold 0 -- then scores a contiguous range of the group's keys: a
// key's n_sub codes index one entry each (the four rows of a centroid side by side: four
// bfloat16 in 8 bytes, or four floats in 16).  The key range per CTA is sized so that the grid
// is about two CTAs per SM: the table is built a few hundred times per call.
// The query rows are staged in shared memory as floats; a centroid is read with 16-byte loads
// when its sub-vector allows it (VEC: sub_d * sizeof(T) is a multiple of 16).
template <typename T>
struct PqEntry;
template <>
struct PqEntry<float> {
  typedef float4 type;
  static __device__ __forceinline__ float4 pack(const float* v) { return make_float4(v[0], v[1], v[2], v[3]); }
  static __device__ __forceinline__ void add(float* s, const float4& e) {
    s[0] = __fadd_rn(s[0], e.x); s[1] = __fadd_rn(s[1], e.y);
    s[2] = __fadd_rn(s[2], e.z); s[3] = __fadd_rn(s[3], e.w);
  }
};
template <>
struct PqEntry<__nv_bfloat16> {
  typedef uint2 type;  // the table values are bfloat16 numbers: two per word
  static __device__ __forceinline__ uint2 pack(const float* v) {
    const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&lo), *reinterpret_cast<const uint32_t*>(&hi));
  }
  static __device__ __forceinline__ void add(float* s, const uint2& e) {
    s[0] = __fadd_rn(s[0], __uint_as_float(e.x << 16)); s[1] = __fadd_rn(s[1], __uint_as_float(e.x & 0xffff0000u));
    s[2] = __fadd_rn(s[2], __uint_as_float(e.y << 16)); s[3] = __fadd_rn(s[3], __uint_as_float(e.y & 0xffff0000u));
  }
};

// bytes of the table in front of the staged queries, which are read 16 bytes at a time
__host__ __device__ __forceinline__ size_t pq_table_bytes(size_t entry, int n_sub, int n_cent) {
  return (entry * (size_t)n_sub * (size_t)n_cent + 15) / 16 * 16;
}

template <typename T, bool VEC>
__global__ void __launch_bounds__(PQ_TILE)
pq_scores_kernel(const T* __restrict__ q, int64_t qs_b, int64_t qs_h, int64_t qs_q,
                 const T* __restrict__ centroids, const uint8_t* __restrict__ codes, int64_t cap, int Hq,
                 int Hkv, int Sq, int64_t n_keys, int64_t init_offset, int64_t S, int n_sub, int sub_d,
                 int n_cent, int64_t keys_per_cta, T* __restrict__ scores) {
  sah_pdl_entry();
  typedef typename PqEntry<T>::type Entry;
  extern __shared__ __align__(16) unsigned char pq_sm_raw[];
  const int G = Hq / Hkv;
  const int R = G * Sq;
  const int64_t bk = blockIdx.z;
  const int kvh = (int)(bk % Hkv);
  const int64_t b = bk / Hkv;
  const int rblk = blockIdx.y;
  const int entries = n_sub * n_cent;
  const int Dh = n_sub * sub_d;
  Entry* lut = reinterpret_cast<Entry*>(pq_sm_raw);                  // [n_sub][n_cent]
  float* q_sm = reinterpret_cast<float*>(pq_sm_raw + pq_table_bytes(sizeof(Entry), n_sub, n_cent));  // [Dh][PQ_ROWS]
  for (int idx = threadIdx.x; idx < PQ_ROWS * Dh; idx += PQ_TILE) {
    const int rr = idx / Dh, d = idx - rr * Dh;
    const int r = rblk * PQ_ROWS + rr;
    float v = 0.f;
    if (r < R) {
      const int g = r / Sq, qi = r - g * Sq;
      v = sah_to_float<T>(q[b * qs_b + (int64_t)(kvh * G + g) * qs_h + qi * qs_q + d]);
    }
    q_sm[d * PQ_ROWS + rr] = v;
  }
  __syncthreads();
  constexpr int PER16 = 16 / (int)sizeof(T);  // elements per 16-byte load
  // Four entries of a thread at a time, their centroids' first 16 bytes (all of them, for 8 bf16
  // channels) requested together; channels ascending.
  constexpr int AHEAD = 4;
  const int log_cent = (n_cent & (n_cent - 1)) == 0 ? 31 - __clz(n_cent) : -1;  // a division per entry otherwise
  for (int idx0 = threadIdx.x; idx0 < entries; idx0 += AHEAD * PQ_TILE) {
    uint4 first[AHEAD];
    if constexpr (VEC) {
#pragma unroll
      for (int n = 0; n < AHEAD; ++n)
        if (idx0 + n * PQ_TILE < entries)
          first[n] = *reinterpret_cast<const uint4*>(centroids + (bk * n_sub * (int64_t)n_cent + idx0 + n * PQ_TILE) * sub_d);
    }
#pragma unroll
    for (int n = 0; n < AHEAD; ++n) {
      const int idx = idx0 + n * PQ_TILE;
      if (idx >= entries) break;
      const int sub = log_cent >= 0 ? idx >> log_cent : idx / n_cent;
      const T* cp = centroids + (bk * n_sub * (int64_t)n_cent + idx) * sub_d;
      const float4* qv = reinterpret_cast<const float4*>(q_sm) + sub * sub_d;
      float acc[PQ_ROWS] = {0.f, 0.f, 0.f, 0.f};
      auto channel = [&](float c, const float4& x) {
        acc[0] = fmaf(x.x, c, acc[0]);
        acc[1] = fmaf(x.y, c, acc[1]);
        acc[2] = fmaf(x.z, c, acc[2]);
        acc[3] = fmaf(x.w, c, acc[3]);
      };
      if constexpr (VEC) {
        uint4 raw = first[n];
        for (int d0 = 0; d0 < sub_d; d0 += PER16) {
          if (d0 > 0) raw = *reinterpret_cast<const uint4*>(cp + d0);
          const T* cv = reinterpret_cast<const T*>(&raw);
#pragma unroll
          for (int e = 0; e < PER16; ++e) channel(sah_to_float<T>(cv[e]), qv[d0 + e]);
        }
      } else {
        for (int d = 0; d < sub_d; ++d) channel(sah_to_float<T>(cp[d]), qv[d]);
      }
      float out[PQ_ROWS];
#pragma unroll
      for (int rr = 0; rr < PQ_ROWS; ++rr) out[rr] = (rblk * PQ_ROWS + rr < R) ? sah_round_to<T>(acc[rr]) : 0.f;
      lut[idx] = PqEntry<T>::pack(out);
    }
  }
  __syncthreads();
  const bool vec = (n_sub == 16) && ((reinterpret_cast<uintptr_t>(codes) & 15) == 0);
  int64_t rowoff[PQ_ROWS];
#pragma unroll
  for (int rr = 0; rr < PQ_ROWS; ++rr) {
    const int r = rblk * PQ_ROWS + rr;
    const int g = r / Sq, qi = r - g * Sq;
    rowoff[rr] = r < R ? ((b * Hq + kvh * G + g) * Sq + qi) * S + init_offset : -1;
  }
  const int64_t j0 = (int64_t)blockIdx.x * keys_per_cta;
  const int64_t j1 = j0 + keys_per_cta < n_keys ? j0 + keys_per_cta : n_keys;
  // the codes of the next two keys of a thread are requested before the present one is scored
  uint4 ahead[2];
  auto fetch = [&](int64_t j) -> uint4 {
    return vec && j < j1 ? *reinterpret_cast<const uint4*>(codes + (bk * cap + j) * n_sub) : make_uint4(0u, 0u, 0u, 0u);
  };
  ahead[0] = fetch(j0 + threadIdx.x);
  ahead[1] = fetch(j0 + threadIdx.x + PQ_TILE);
  for (int64_t j = j0 + threadIdx.x; j < j1; j += PQ_TILE) {
    const uint8_t* cj = codes + (bk * cap + j) * n_sub;
    float s[PQ_ROWS] = {0.f, 0.f, 0.f, 0.f};
    if (vec) {
      const uint4 cv = ahead[0];
      ahead[0] = ahead[1];
      ahead[1] = fetch(j + 2 * PQ_TILE);
      const uint32_t w[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
      for (int sub = 0; sub < 16; ++sub) {
        const uint32_t c = (w[sub >> 2] >> ((sub & 3) * 8)) & 255u;
        PqEntry<T>::add(s, lut[sub * n_cent + c]);
      }
    } else {
      for (int sub = 0; sub < n_sub; ++sub) PqEntry<T>::add(s, lut[sub * n_cent + cj[sub]]);
    }
#pragma unroll
    for (int rr = 0; rr < PQ_ROWS; ++rr)
      if (rowoff[rr] >= 0) scores[rowoff[rr] + j] = sah_from_float<T>(s[rr]);
  }
}

extern "C" int64_t sah_pq_scores_ws_bytes(int B, int Hq, int Hkv, int Sq, int n_sub, int n_cent) {
  if (B <= 0 || Hq <= 0 || Hkv <= 0 || Sq <= 0 || n_sub <= 0 || n_cent <= 0) return 0;
  const int64_t R = (int64_t)(Hq / Hkv) * Sq;
  const int64_t rblocks = (R + PQ_ROWS - 1) / PQ_ROWS;
  return (int64_t)B * Hkv * rblocks * n_sub * n_cent * PQ_ROWS * (int64_t)sizeof(float);
}

extern "C" int sah_pq_scores(const void* q, int dtype, int64_t qs_b, int64_t qs_h, int64_t qs_q,
                             const void* centroids, const uint8_t* codes, int64_t cap, int B, int Hq,
                             int Hkv, int Sq, int64_t n_keys, int64_t init_offset, int64_t S,
                             int n_sub, int sub_d, int n_cent, void* scores, void* workspace,
                             int64_t workspace_bytes, void* stream) {
  SAH_REQUIRE(q && centroids && codes && scores, "pq_scores: null pointer");
  SAH_REQUIRE(B > 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0 && Sq > 0, "pq_scores: bad heads");
  SAH_REQUIRE(n_keys >= 0 && init_offset >= 0 && init_offset + n_keys <= S && n_keys <= cap,
              "pq_scores: bad key range");
  SAH_REQUIRE(n_cent <= 256, "pq_scores: codes are bytes, at most 256 centroids");
  (void)workspace_bytes;
  if (n_keys == 0) return SAH_OK;
  const int R = (Hq / Hkv) * Sq;
  const int rblocks = (R + PQ_ROWS - 1) / PQ_ROWS;
  const size_t esz = (dtype == SAH_BF16) ? 8 : 16;  // one table entry: the four rows of a centroid
  const size_t smem = pq_table_bytes(esz, n_sub, n_cent) + (size_t)PQ_ROWS * n_sub * sub_d * sizeof(float);
  if (smem > PQ_SCORES_SMEM)
    return sah_fail(SAH_ERR_UNSUPPORTED, "pq_scores: %d x %d lookup table does not fit", n_sub, n_cent);
  SAH_REQUIRE(rblocks <= 65535 && (int64_t)B * Hkv <= 65535, "pq_scores: too many rows per launch");
  cudaStream_t st = (cudaStream_t)stream;
  (void)workspace;  // the tables live in shared memory; the argument is kept for callers that pass one
  sah_prof_begin(SAH_PROF_PQ_SCORES, st);
  // about two CTAs per SM, each with a contiguous key range that is a multiple of the CTA width
  const int64_t groups = (int64_t)B * Hkv * rblocks;
  int64_t per_group = (2 * 148 + groups - 1) / groups;
  if (per_group < 1) per_group = 1;
  int64_t keys_per_cta = sah_ceil_div(sah_ceil_div(n_keys, per_group), PQ_TILE) * PQ_TILE;
  if (keys_per_cta < 2048) keys_per_cta = 2048;
  dim3 grid((unsigned)sah_ceil_div(n_keys, keys_per_cta), (unsigned)rblocks, (unsigned)((int64_t)B * Hkv));
  const int64_t tsz = (dtype == SAH_BF16) ? 2 : 4;
  const bool vecc = (sub_d * tsz) % 16 == 0 && (reinterpret_cast<uintptr_t>(centroids) & 15) == 0;
  static bool allowed[4][64] = {};
#define PQ_SCORES_LAUNCH(T, VEC, SLOT)                                                                    \
  do {                                                                                                    \
    if ((int)smem > 48 * 1024) {                                                                          \
      const cudaError_t e = sah_allow_smem(pq_scores_kernel<T, VEC>, PQ_SCORES_SMEM, allowed[SLOT]);      \
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "pq_scores attr: %s", cudaGetErrorString(e));   \
    }                                                                                                     \
    sah_launch_chain(pq_scores_kernel<T, VEC>, grid, PQ_TILE, smem, st, (const T*)q, qs_b, qs_h, qs_q, (const T*)centroids, \
                                                          codes, cap, Hq, Hkv, Sq, n_keys, init_offset, S, \
                                                          n_sub, sub_d, n_cent, keys_per_cta, (T*)scores); \
  } while (0)
  if (dtype == SAH_BF16) {
    if (vecc) PQ_SCORES_LAUNCH(__nv_bfloat16, true, 0);
    else PQ_SCORES_LAUNCH(__nv_bfloat16, false, 1);
  } else if (dtype == SAH_F32) {
    if (vecc) PQ_SCORES_LAUNCH(float, true, 2);
    else PQ_SCORES_LAUNCH(float, false, 3);
  } else {
    return sah_fail(SAH_ERR_INVALID, "pq_scores: unknown dtype %d", dtype);
  }
#undef PQ_SCORES_LAUNCH
  SAH_LAUNCH_CHECK("pq_scores");
  sah_prof_end(SAH_PROF_PQ_SCORES, st);
  return SAH_OK;
}
