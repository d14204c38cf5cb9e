// Exact per-row top-k by radix select over order-preserving integer keys, with ties going to the
// lowest column, in one launch: a row belongs to a cluster of up to eight CTAs, each with a
// contiguous range of its columns.  Only columns inside [col_begin, col_end) whose `prev` bit is
// clear compete; the row written is prev | winners.
//
// Two (16-bit keys: 11 + 5 bits) or three (32-bit keys: 11 + 11 + 10) histogram passes, most
// significant digit first, fix the k-th largest key T and how many keys equal to T are still
// needed; every CTA reads the other CTAs' histograms over distributed shared memory and finds the
// digit itself, one cluster barrier per digit.  Wide first digits because scores share their
// exponents: 8-bit digits put most keys of a warp into the same few counters.  One more pass
// emits; where the keys equal to T are more than are needed a counting pass in front of it orders
// them: a warp owns a contiguous run of columns, 32 lanes x 8 columns at a time, so reads are
// coalesced and a scan over the warps' counts is all the ordering that is left.
//
// The first pass leaves the keys, zero where a column does not compete, in shared memory (up to
// 81920 columns of 16 bits or 40960 of 32 per CTA), and the others test two 16-bit keys with one
// integer operation; a longer range is read and converted again in every pass.  Bound by
// instruction issue (the passes make about 20 instructions per 16-bit key) and, for short rows,
// by the barriers.  128 rows x 65536 bfloat16 scores: 35.2 us as three launches with a grid-wide
// histogram each, 45.6 us with the keys converted in every pass, 27.6 us now (32 rows x 8191: 23.5 us before, 10.7 us now).
// Rows of up to 2048 columns (page scores) take digits of 8 bits and CTAs of 64 to 256 threads: 32
// rows x 512 bfloat16 scores 7.0 us with the wide digits, 5.9 us this way.
#pragma once

#include "sah_common.cuh"
#include <cooperative_groups.h>

#define SAH_SELECT_THREADS 1024
#define SAH_SELECT_PER 4             // counters of a digit per thread: at least 512 threads of 2048 ...
#define SAH_SELECT_SHORT_BYTES 256   // ... and 64 of 256, for rows of up to 2048 columns
#define SAH_SELECT_MAX_CLUSTER 8
#define SAH_SELECT_KEY_BYTES (160 * 1024)  // keys of a CTA's columns in shared memory
#define SAH_SELECT_HALF_BYTES (90 * 1024)  // two such CTAs share an SM

// Keep the lowest n set bits of m.
__device__ __forceinline__ uint32_t sah_lowest_bits(uint32_t m, int n) {
  int c = __popc(m);
  if (n >= c) return m;
  if (n <= 0) return 0u;
  unsigned pos = __fns(m, 0, n + 1);  // position of the (n+1)-th set bit
  return m & ((1u << pos) - 1u);
}


// Eight keys from column c0 of a row, two 16-bit ones or one 32-bit one per word (anything past
// the end).  No key is 0: that would be a negative not-a-number, and -0 and not-a-numbers are
// made +0 and the positive one by an addition of +0.
template <typename T, int KEYBITS>
struct SahScoreKeys;
template <>
struct SahScoreKeys<__nv_bfloat16, 16> {
  const __nv_bfloat16* scores;
  int64_t S;
  const __nv_bfloat16* s;
  bool vec;
  __device__ __forceinline__ void open(int64_t row) {
    s = scores + row * S;
    vec = (reinterpret_cast<uintptr_t>(s) & 15) == 0;
  }
  static constexpr int AHEAD = 4;  // blocks requested together, as registers allow
  static constexpr bool BANDS = true;  // the previous mask may come as bands
  struct Raw { uint32_t w[4]; };
  __device__ __forceinline__ void load(int64_t c0, Raw& raw) const {
    uint32_t* w = raw.w;
    if (vec && c0 + 8 <= S) {
      const uint4 v = *reinterpret_cast<const uint4*>(s + c0);
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
      const uint16_t* u = reinterpret_cast<const uint16_t*>(s);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t lo = c0 + 2 * i < S ? u[c0 + 2 * i] : 0u, hi = c0 + 2 * i + 1 < S ? u[c0 + 2 * i + 1] : 0u;
        w[i] = lo | hi << 16;
      }
    }
  }
  __device__ __forceinline__ void make(const Raw& raw, uint32_t* w) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const __nv_bfloat162 z = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&raw.w[i]), __float2bfloat162_rn(0.f));
      const uint32_t u = *reinterpret_cast<const uint32_t*>(&z);
      w[i] = u ^ ((((u >> 15) & 0x00010001u) * 0xFFFFu) | 0x80008000u);
    }
  }
};
template <>
struct SahScoreKeys<float, 32> {
  const float* scores;
  int64_t S;
  const float* s;
  bool vec;
  __device__ __forceinline__ void open(int64_t row) {
    s = scores + row * S;
    vec = (reinterpret_cast<uintptr_t>(s) & 15) == 0;
  }
  static constexpr int AHEAD = 2;
  static constexpr bool BANDS = true;
  struct Raw { float f[8]; };
  __device__ __forceinline__ void load(int64_t c0, Raw& raw) const {
    float* f = raw.f;
    if (vec && c0 + 8 <= S) {
      sah_load8<float>(s + c0, f);
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = c0 + i < S ? s[c0 + i] : 0.f;
    }
  }
  __device__ __forceinline__ void make(const Raw& raw, uint32_t* w) const {
#pragma unroll
    for (int i = 0; i < 8; ++i) w[i] = sah_float_key(raw.f[i] + 0.0f);
  }
};

// SHORT: digits of 8 bits, whose 256 counters a small CTA clears and scans in no time
template <int KEYBITS, typename Keys, bool RESIDENT, bool SHORT>
__global__ void __launch_bounds__(SHORT ? SAH_SELECT_SHORT_BYTES : SAH_SELECT_THREADS)
sah_select_kernel(Keys keys, const uint32_t* __restrict__ prev_bits, const __grid_constant__ MaskBands bands, int Sq,
                  uint32_t* __restrict__ band_bits, uint32_t* __restrict__ out_bits, int64_t S, int64_t W, int64_t col_begin, int64_t col_end,
                  long long k) {
  sah_pdl_entry();
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  constexpr int NW = KEYBITS == 16 ? 4 : 8;  // words of eight keys
  constexpr int DIGIT = SHORT ? 8 : 11, DIGITS = (KEYBITS + DIGIT - 1) / DIGIT, BINS = 1 << DIGIT;
  extern __shared__ __align__(16) unsigned char sel_smem[];
  uint4* store = reinterpret_cast<uint4*>(sel_smem);  // [NW / 4][bytes of this CTA]
  __shared__ unsigned int hist[2][BINS];  // alternate digits: a CTA may count the next
                                                     // one while others still read this one
  __shared__ unsigned int scan[33];
  __shared__ unsigned int prefix_sm;
  __shared__ long long need_sm;
  __shared__ unsigned int ties_sm;  // keys equal to the prefix in the whole row
  __shared__ int mode_sm;           // 0: threshold, 1: all candidates, 2: none
  const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int64_t row = blockIdx.x / ranks;
  keys.open(row);
  // the previous mask: a bitmap, or (no bitmap) its bands, written out as a bitmap for whoever
  // reads that mask later if there is a place for it
  const unsigned char* pb = prev_bits == nullptr ? nullptr : reinterpret_cast<const unsigned char*>(prev_bits + row * W);
  unsigned char* bb = band_bits == nullptr ? nullptr : reinterpret_cast<unsigned char*>(band_bits + row * W);
  unsigned char* ob = reinterpret_cast<unsigned char*>(out_bits + row * W);
  if (col_begin < 0) col_begin = 0;
  if (col_end > S) col_end = S;

  // this CTA's words in bytes of eight columns; a warp's run in blocks of 32 bytes
  const int64_t y_lo = W * rank / ranks * 4, y_hi = W * (rank + 1) / ranks * 4;
  const int ny = (int)(y_hi - y_lo);
  const int blocks = (ny + 31) / 32;
  const int q_lo = (int)((int64_t)blocks * warp / nw), q_hi = (int)((int64_t)blocks * (warp + 1) / nw);
  if (pb != nullptr) pb += y_lo;
  if (bb != nullptr) bb += y_lo;
  ob += y_lo;
  // bytes [gap_lo, gap_hi) of this CTA lie between the bands that begin the row and the others:
  // nearly all of them, and empty
  const int64_t qpos = row % Sq;
  int gap_lo = 0, gap_hi = 0;
  if (Keys::BANDS && pb == nullptr) {
    int64_t a = 0, e = S;
#pragma unroll
    for (int i = 0; i < SAH_MAX_BANDS; ++i) {
      if (i >= bands.n) break;
      const int64_t lo = bands.lo_base[i] + qpos * bands.lo_qstep[i], hi = bands.hi_base[i] + qpos * bands.hi_qstep[i];
      if (lo <= 0) a = hi > a ? hi : a;
      else e = lo < e ? lo : e;
    }
    a = (a + 7) / 8 - y_lo;
    e = e / 8 - y_lo;
    gap_lo = (int)(a < 0 ? 0 : a > ny ? ny : a);
    gap_hi = (int)(e < 0 ? 0 : e > ny ? ny : e);
  }
  auto previous = [&](int y) -> unsigned int {
    if (!Keys::BANDS || pb != nullptr) return pb[y];
    return y >= gap_lo && y < gap_hi ? 0u : sah_band_bits(bands, qpos, (y_lo + y) * 8, 8, S, 0u);
  };
  // columns of byte y (of this CTA) that compete
  auto competing = [&](int y) -> unsigned int {
    const int64_t c0 = (y_lo + y) * 8;
    if (c0 >= col_end || c0 + 8 <= col_begin) return 0u;
    unsigned int m = ~previous(y) & 255u;
    if (c0 < col_begin) m &= 255u << (int)(col_begin - c0);
    if (c0 + 8 > col_end) m &= (1u << (int)(col_end - c0)) - 1u;
    return m;
  };
  // the byte's keys from memory, 0 where a column does not compete; false if none does
  auto finish = [&](const typename Keys::Raw& raw, unsigned int m, uint32_t* w) -> bool {
#pragma unroll
    for (int i = 0; i < NW; ++i) w[i] = 0u;
    if (m == 0u) return false;
    keys.make(raw, w);
    if (m != 255u) {
#pragma unroll
      for (int i = 0; i < NW; ++i) {
        if (NW == 4)
          w[i] &= ((m >> (2 * i)) & 1u ? 0xFFFFu : 0u) | ((m >> (2 * i + 1)) & 1u ? 0xFFFF0000u : 0u);
        else
          w[i] = (m >> i) & 1u ? w[i] : 0u;
      }
    }
    return true;
  };
  auto convert = [&](int y, uint32_t* w) -> bool {
    const unsigned int m = competing(y);
    typename Keys::Raw raw;
    if (m) keys.load((y_lo + y) * 8, raw);
    return finish(raw, m, w);
  };
  auto fetch = [&](int y, uint32_t* w) -> bool {
    if (!RESIDENT) return convert(y, w);
#pragma unroll
    for (int i = 0; i < NW / 4; ++i) {
      const uint4 v = store[i * ny + y];
      w[4 * i] = v.x; w[4 * i + 1] = v.y; w[4 * i + 2] = v.z; w[4 * i + 3] = v.w;
    }
    return true;
  };
  auto key_at = [](const uint32_t* w, int i) -> uint32_t {
    return NW == 8 ? w[i] : (i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu;
  };

  uint32_t prefix = 0u, pmask = 0u;
  long long need = k;
  int mode = k <= 0 ? 2 : 0;
  unsigned int ties = 0u;   // keys equal to the threshold in the whole row
  unsigned int lower = 0u;  // and in the CTAs in front of this one
#pragma unroll
  for (int d = 0; d < DIGITS; ++d) {
    const int bits = d == DIGITS - 1 ? KEYBITS - DIGIT * (DIGITS - 1) : DIGIT;
    const int shift = d == DIGITS - 1 ? 0 : KEYBITS - DIGIT * (d + 1);
    const int nbins = 1 << bits;
    unsigned int* h = hist[d & 1];
    if (mode == 0) {  // the same in the whole cluster
      for (int i = tid; i < nbins; i += nt) h[i] = 0u;
      if (tid == 0) mode_sm = 0;
      __syncthreads();
      if (d == 0) {
        // a few blocks' keys are requested before the first is converted
        constexpr int AHEAD = Keys::AHEAD;
        for (int q0 = q_lo; q0 < q_hi; q0 += AHEAD) {
          typename Keys::Raw raw[AHEAD];
          unsigned int m[AHEAD];
#pragma unroll
          for (int n = 0; n < AHEAD; ++n) {
            const int y = (q0 + n) * 32 + lane;
            m[n] = q0 + n < q_hi && y < ny ? competing(y) : 0u;
            if (m[n]) keys.load((y_lo + y) * 8, raw[n]);
          }
#pragma unroll
          for (int n = 0; n < AHEAD; ++n) {
            const int y = (q0 + n) * 32 + lane;
            if (q0 + n >= q_hi || y >= ny) break;
            uint32_t w[NW];
            const bool any = finish(raw[n], m[n], w);
            if (RESIDENT) {
#pragma unroll
              for (int i = 0; i < NW / 4; ++i)
                store[i * ny + y] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
            }
            if (any) {
#pragma unroll
              for (int i = 0; i < 8; ++i) {
                const uint32_t key = key_at(w, i);
                if (key) atomicAdd(&h[key >> shift], 1u);
              }
            }
          }
        }
      } else {
        for (int q = q_lo; q < q_hi; ++q) {
          const int y = q * 32 + lane;
          if (y >= ny) break;
          uint32_t w[NW];
          if (!fetch(y, w)) continue;
          bool any = true;
          if (NW == 4) {  // some half agrees with the prefix (nothing is left below the mask, so the test is exact)
            uint32_t z = 0u;
#pragma unroll
            for (int i = 0; i < NW; ++i) {
              const uint32_t x = (w[i] ^ (prefix * 0x00010001u)) & (pmask * 0x00010001u);
              z |= (x - 0x00010001u) & ~x;
            }
            any = (z & 0x80008000u) != 0u;
          }
          if (any) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint32_t key = key_at(w, i);
              if (((key ^ prefix) & pmask) == 0u && key) atomicAdd(&h[(key >> shift) & (nbins - 1)], 1u);
            }
          }
        }
      }
      if (ranks > 1) cluster.sync(); else __syncthreads();
      // thread t owns PER neighbouring bins, the highest first; all reads are on their way before
      // the first is added
      constexpr int PER = SAH_SELECT_PER;
      unsigned int cnt[PER], mine = 0u;
#pragma unroll
      for (int j = 0; j < PER; ++j) {
        const int bin = nbins - 1 - (tid * PER + j);
        cnt[j] = 0u;
        if (bin >= 0) {
          if (ranks == 1) {
            cnt[j] = h[bin];
          } else {
#pragma unroll
            for (int r = 0; r < SAH_SELECT_MAX_CLUSTER; ++r)
              if (r < ranks) cnt[j] += cluster.map_shared_rank(h, r)[bin];
          }
        }
        mine += cnt[j];
      }
      unsigned int total;
      unsigned int above = sah_block_excl_scan<unsigned int>(mine, scan, &total);
      if ((long long)total < need || (d == 0 && (long long)total <= need)) {
        if (tid == 0) mode_sm = 1;
      } else if ((long long)above < need && (long long)above + mine >= need) {
        bool found = false;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
          if (!found && (long long)above + cnt[j] >= need) {
            prefix_sm = prefix | ((uint32_t)(nbins - 1 - (tid * PER + j)) << shift);
            need_sm = need - above;
            ties_sm = cnt[j];
            found = true;
          }
          above += cnt[j];
        }
      }
      __syncthreads();
      mode = mode_sm;
      if (mode == 0) {
        prefix = prefix_sm;
        need = need_sm;
        ties = ties_sm;
        pmask |= (uint32_t)(nbins - 1) << shift;
        if (d == DIGITS - 1)
          for (int r = 0; r < rank; ++r) lower += cluster.map_shared_rank(h, r)[prefix & (nbins - 1)];
      }
      __syncthreads();  // before the shared state is written again
    }
  }

  // one bit per key of the byte: equal to the threshold
  auto equal = [&](const uint32_t* w) -> uint32_t {
    uint32_t eq = 0u;
    if (NW == 4) {
      uint32_t z[4], any = 0u;  // bits 15 and 31: the half is zero
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t x = w[i] ^ (prefix * 0x00010001u);
        z[i] = ~(((x & 0x7FFF7FFFu) + 0x7FFF7FFFu) | x) & 0x80008000u;
        any |= z[i];
      }
      if (any) {
#pragma unroll
        for (int i = 0; i < 4; ++i) eq |= ((z[i] >> 15) & 1u) << (2 * i) | (z[i] >> 31) << (2 * i + 1);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) eq |= (w[i % NW] == prefix ? 1u : 0u) << i;
    }
    return eq;
  };

  // keys equal to the threshold in the columns in front of this warp's
  long long quota = need;
  if (mode == 0 && (long long)ties > need) {
    unsigned int eq = 0u;
    for (int q = q_lo; q < q_hi; ++q) {
      const int y = q * 32 + lane;
      uint32_t w[NW];
      if (y < ny && fetch(y, w)) eq += __popc(equal(w));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) eq += __shfl_xor_sync(0xffffffffu, eq, o);
    unsigned int total;
    unsigned int before = sah_block_excl_scan<unsigned int>(lane == 0 ? eq : 0u, scan, &total);
    before = __shfl_sync(0xffffffffu, before, 0);
    quota = need - (long long)lower - (long long)before;
  }
  for (int q = q_lo; q < q_hi; ++q) {
    const int y = q * 32 + lane;
    const unsigned int prev = y < ny ? previous(y) : 0u;
    unsigned int gt = 0u, eq = 0u;
    if (mode == 1) {
      if (y < ny) gt = competing(y);
    } else if (mode == 0 && y < ny) {
      uint32_t w[NW];
      if (fetch(y, w)) {
        uint32_t below = 0u;  // the threshold is not 0, so a column that does not compete is below it
        if (NW == 4) {
#pragma unroll
          for (int i = 7; i >= 0; --i) below = __funnelshift_l(key_at(w, i) - prefix, below, 1);
        } else {
#pragma unroll
          for (int i = 0; i < 8; ++i) below |= (w[i % NW] < prefix ? 1u : 0u) << i;
        }
        eq = equal(w);
        gt = ~below & 255u & ~eq;
      }
    }
    if (mode == 0 && quota > 0 && __any_sync(0xffffffffu, eq != 0u)) {  // uniform but for the vote
      int incl = __popc(eq);
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      const long long left = quota - (incl - __popc(eq));
      gt |= sah_lowest_bits(eq, left > 8 ? 8 : left < 0 ? 0 : (int)left);
      quota -= __shfl_sync(0xffffffffu, incl, 31);
    }
    if (y < ny) ob[y] = (unsigned char)(prev | gt);
    if (Keys::BANDS && bb != nullptr && y < ny) bb[y] = (unsigned char)prev;
  }
  if (ranks > 1) cluster.sync();  // nobody leaves while its counters may be read
}

// CTAs per row: a power of two, as long as one wave holds all of them and each keeps 8192
// columns, one byte of the bitmap per thread and pass (with 2048 columns per CTA 32 rows x 8191
// bfloat16 scores took 20.4 us: the cluster barriers and the counters of the other CTAs cost more
// than the passes)
static inline int sah_select_ranks(int64_t rows, int64_t S) {
  int ranks = 1;
  while (ranks < SAH_SELECT_MAX_CLUSTER && rows * ranks * 2 <= sah_cluster_wave(ranks * 2) &&
         S >= (int64_t)ranks * 2 * 8192)
    ranks *= 2;
  return ranks;
}

// bytes of shared memory for the keys of a CTA's columns
static inline int64_t sah_select_key_bytes(int64_t rows, int64_t S, int64_t W, int keybits) {
  const int ranks = sah_select_ranks(rows, S);
  return (W + ranks - 1) / ranks * 4 * keybits;
}

template <int KEYBITS, typename Keys>
static inline int sah_select_launch(const Keys& keys, const uint32_t* prev_bits, uint32_t* out_bits, int64_t rows,
                                    int64_t S, int64_t W, int64_t col_begin, int64_t col_end, int64_t k,
                                    cudaStream_t st, const MaskBands& bands = MaskBands(), int Sq = 1,
                                    uint32_t* band_bits = nullptr) {
  const int ranks = sah_select_ranks(rows, S);
  const int64_t key_bytes = sah_select_key_bytes(rows, S, W, KEYBITS);
  const bool resident = key_bytes <= SAH_SELECT_KEY_BYTES;
  const int64_t row_bytes = W * 4 / ranks;  // a thread looks at one at a time
  const bool shrt = W * 4 <= SAH_SELECT_SHORT_BYTES;
  // half-size CTAs for shorter rows, and when rows queue for SMs that hold two of them (256 rows x
  // 65536 bfloat16 scores, of which an SM holds one: 59.0 us in half-size CTAs, 48.1 us in whole ones)
  const bool two = rows * ranks > 148 && key_bytes <= SAH_SELECT_HALF_BYTES;
  const int nt = shrt ? (row_bytes <= 64 ? 64 : row_bytes <= 128 ? 128 : 256)
                      : row_bytes <= SAH_SELECT_THREADS / 2 || two ? SAH_SELECT_THREADS / 2 : SAH_SELECT_THREADS;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * ranks));
  cfg.blockDim = dim3((unsigned)nt);
  cfg.dynamicSmemBytes = resident ? (size_t)key_bytes : 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = ranks > 1 ? 1 : 0;
  auto launch = [&](auto kernel) {
    (void)cudaLaunchKernelEx(&cfg, kernel, keys, prev_bits, bands, Sq, band_bits, out_bits, S, W, col_begin, col_end,
                             (long long)k);
  };
  if (shrt) {
    launch(sah_select_kernel<KEYBITS, Keys, true, true>);
  } else if (resident) {
    if (key_bytes > 24 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(sah_select_kernel<KEYBITS, Keys, true, false>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, SAH_SELECT_KEY_BYTES);
      if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "select attr: %s", cudaGetErrorString(e));
    }
    launch(sah_select_kernel<KEYBITS, Keys, true, false>);
  } else {
    launch(sah_select_kernel<KEYBITS, Keys, false, false>);
  }
  return SAH_OK;  // a launch error stays for SAH_LAUNCH_CHECK
}
