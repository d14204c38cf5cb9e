// Oracle top-p: the keys whose softmax weight reaches the row's threshold, the threshold being
// the sorted weight at which the cumulative mass passes top_p
// (research_attention/maskers/fixed/implementations/oracle_top_p.py:85-169).
//
// The reference sorts the exp weights of a row (bf16 values), takes a running sum in sorted
// order -- torch's CPU cumsum: one float32 accumulator, every prefix rounded to bf16 --
// normalises by the last prefix and searches for top_p.  The threshold is a value of the
// sorted list, so only sums at the ends of runs of equal values matter, and the weight is a
// function of d = logit - maximum, a non-positive bf16 number: exp rounds to 1 for |d| < 2^-10
// and to 0 from |d| = 128 on, which leaves 17 * 128 values of d.  A histogram over those replaces
// the sort (and a comparison of d replaces the second look-up of the weight), and the accumulator
// is replayed over the bins from the largest weight down.
//
// The replay runs in parallel, binade by binade of the accumulator.  Inside a binade of spacing u
// the accumulator is an integer A times u, and an add of v = (k + f) u moves it by k or k + 1
// whatever A is, unless f is exactly one half; then the sum goes to the even neighbour, so the
// move depends on A's parity and every later add of the same v moves by the even one of k, k + 1.
// A bin is therefore a function of A's parity (two moves), such functions compose, and a scan
// over the bins gives every prefix up to the first one that reaches the next binade; that bin is
// added run by run, and the scan starts again behind it.  One warp does this over the list of
// non-empty bins, 64 at a time, some two dozen scans for a row of 65536 keys (all threads over all
// bins, with four barriers per binade, took 28 us for it).
//
// A row is shared by a cluster of up to eight CTAs where there are few rows.  What bounds the
// kernel is the instruction issue of the three passes over the row (maximum, histogram, emit), so
// the logits of the first pass stay in shared memory (81920 columns per CTA; longer ranges are
// converted again in every pass), the second replaces them by their bins, and where it can a pass
// handles two 16-bit values per integer instruction; four blocks of a pass are requested at a time.
// 128 rows x 65536 keys: 186 us with scalar
// loads, two gathers of the weight per key from global memory and the accumulator replayed by one
// thread; 62 us with the logits converted in every pass; 47 us with the replay by all threads;
// 30 us now.
// ---------------------------------------------------------------------------
#include "sah_common.cuh"
#include <cooperative_groups.h>

#define TP_THREADS 1024
#define TP_D0 0xBA80                 // bf16 bits of -2^-10: smaller magnitudes have weight 1
#define TP_D1 0xC300                 // -128: weight 0 from here on
#define TP_BINS (TP_D1 - TP_D0 + 2)  // bin 0: weight 1; bins 1 .. : d = TP_D0 ..; last bin: weight 0
#define TP_PER 3                     // bins per thread
#define TP_MAX_CLUSTER 8
#define TP_ROW_BYTES (160 * 1024)    // logits of a CTA's columns in shared memory

struct ToppArgs {
  const void* scores;      // [rows][S] unscaled q.k in bf16
  float scaling;
  const void* bias;
  int64_t bias_s_b, bias_s_h, bias_s_q;
  const uint32_t* prev_bits;
  int Hq, Sq;
  int64_t S, W;
  float top_p;
  int or_prev;
  const uint16_t* exp_table;
  uint32_t* out_bits;
};

__device__ __forceinline__ float tp_block_max(float v, float* scratch32) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch32[threadIdx.x >> 5] = v;
  __syncthreads();
  float w = scratch32[threadIdx.x & 31];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) w = fmaxf(w, __shfl_xor_sync(0xffffffffu, w, o));
  __syncthreads();
  return w;
}

// Bins of two values d = logit - maximum (packed bf16): ascending bins have descending weights.
// As unsigned 16-bit numbers the d of bins 1 .. are TP_D0 .., the smaller magnitudes, +0 and the
// positive not-a-number (an infinite or NaN logit; counts as weight 1) are below.
__device__ __forceinline__ uint32_t tp_bins2(uint32_t d2) {
  constexpr uint32_t LO = (TP_D0 - 1) * 0x00010001u, HI = TP_D1 * 0x00010001u;
  return __vminu2(__vmaxu2(d2, LO), HI) - LO;  // neither half borrows
}
__device__ __forceinline__ uint32_t tp_pack2(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float tp_lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float tp_hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// 8 columns from column c0 of a row (zeros past the end); `vec`: rows are 16-byte aligned
__device__ __forceinline__ void tp_load8(const __nv_bfloat16* __restrict__ s, int64_t c0, int64_t S, bool vec,
                                         float* f) {
  if (vec && c0 + 8 <= S) {
    sah_unpack8(*reinterpret_cast<const uint4*>(s + c0), f);
  } else {
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = c0 + i < S ? __bfloat162float(s[c0 + i]) : 0.f;
  }
}

// moves of A for the bin's adds by A's parity at entry, clamped to TP_FAR (past any binade)
#define TP_FAR (1u << 25)
struct TpMove {
  unsigned int d0, d1;
};
__device__ __forceinline__ TpMove tp_then(const TpMove& f, const TpMove& g) {
  TpMove r;
  r.d0 = min(f.d0 + ((f.d0 & 1u) ? g.d1 : g.d0), TP_FAR);
  r.d1 = min(f.d1 + ((f.d1 & 1u) ? g.d0 : g.d1), TP_FAR);
  return r;
}
// One add of the positive bf16 value with bits `vb` to an accumulator whose binade has exponent
// field `ea` (spacing 2^(ea - 150)): A moves by `step` from an even A, by `first1` from an odd one
// (to an even A where the two differ).
__device__ __forceinline__ void tp_steps(unsigned int vb, int ea, unsigned int& step, unsigned int& first1) {
  int ev = (int)(vb >> 7);
  unsigned int m = vb & 127u;
  if (ev) m |= 128u; else ev = 1;   // v = m * 2^(ev - 134)
  const int sh = ea - 16 - ev;      // v / u = m * 2^-sh
  if (sh <= 0) {
    first1 = step = m << -sh;       // v is not above the accumulator, so at most 2^24
  } else if (sh > 8) {
    first1 = step = 0u;             // below half a spacing
  } else {
    const unsigned int k = m >> sh, rem = m & ((1u << sh) - 1u), half = 1u << (sh - 1);
    if (rem == half) {
      step = k + (k & 1u);
      first1 = k + 1u - (k & 1u);
    } else {
      first1 = step = k + (rem > half ? 1u : 0u);
    }
  }
}
// `count` such adds, as moves by A's parity at entry
__device__ __forceinline__ TpMove tp_move(unsigned int vb, unsigned int count, int ea) {
  unsigned int step, first1;
  tp_steps(vb, ea, step, first1);
  const unsigned long long rest = (unsigned long long)(count - 1u) * step;
  TpMove r;
  r.d0 = (unsigned int)min(rest + step, (unsigned long long)TP_FAR);
  r.d1 = (unsigned int)min(rest + first1, (unsigned long long)TP_FAR);
  return r;
}
// `count` adds of the bf16 value with bits `vb` to acc (not below the value; 0 before the first run,
// whose weight is 1: the maximum itself), binade by
// binade: all that stay below the next power of two at once, then one real add across it.
__device__ __forceinline__ float tp_add_run(float acc, unsigned int vb, unsigned int count) {
  const float v = __uint_as_float(vb << 16);
  if (acc == 0.f) {
    acc = v;
    --count;
  }
  while (count > 0u) {
    const unsigned int ea = __float_as_uint(acc) >> 23;
    unsigned int A = (__float_as_uint(acc) & 0x7FFFFFu) | 0x800000u, step, first1;
    tp_steps(vb, (int)ea, step, first1);
    const unsigned int first = (A & 1u) ? first1 : step, room = (1u << 24) - 1u - A;  // A may grow by `room`
    if (first <= room) {
      unsigned int more = step == 0u ? count - 1u : (room - first) / step;  // adds after the first
      if (more > count - 1u) more = count - 1u;
      A += first + more * step;
      count -= 1u + more;
      acc = __uint_as_float(ea << 23 | (A & 0x7FFFFFu));
      if (step == 0u) break;  // nothing moves any more
    }
    if (count > 0u) {
      acc = __fadd_rn(acc, v);
      --count;
    }
  }
  return acc;
}

template <bool RESIDENT>
__global__ void __launch_bounds__(TP_THREADS)
topp_select_kernel(ToppArgs a) {
  sah_pdl_entry();
  namespace cg = cooperative_groups;
  extern __shared__ __align__(16) uint4 tp_row[];     // logits, then bins, of this CTA's columns
  cg::cluster_group cluster = cg::this_cluster();
  __shared__ unsigned int hist[TP_PER * TP_THREADS];  // this CTA's counts; in rank 0 the row's
  __shared__ uint16_t weight[TP_PER * TP_THREADS];    // bf16 bits of exp(d) by bin
  __shared__ float scratch[32];
  __shared__ uint16_t list[TP_PER * TP_THREADS];      // non-empty bins of positive weight, ascending
  __shared__ float list_sum[TP_PER * TP_THREADS];     // the accumulator behind each of them
  __shared__ int scan_sm[33];
  __shared__ float max_sm;                            // this CTA's maximum
  __shared__ float acc_sm;
  __shared__ int cross_sm, pick_sm, thr_sm;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int64_t row = blockIdx.x / ranks;
  const int qi = (int)(row % a.Sq);
  const int64_t bh = row / a.Sq;
  const int h = (int)(bh % a.Hq);
  const int64_t b = bh / a.Hq;
  typedef __nv_bfloat16 T;
  const T* s = reinterpret_cast<const T*>(a.scores) + row * a.S;
  const T* bias = a.bias ? reinterpret_cast<const T*>(a.bias) + b * a.bias_s_b + h * a.bias_s_h +
                               qi * a.bias_s_q
                         : nullptr;
  const bool vec = (reinterpret_cast<uintptr_t>(s) & 15) == 0;
  const bool bias_vec = (reinterpret_cast<uintptr_t>(bias) & 15) == 0;
  const unsigned char* pb = reinterpret_cast<const unsigned char*>(a.prev_bits + row * a.W);

  // the row in bytes of the bitmap, 8 columns each, cut into one range per CTA of the cluster
  const int64_t nb = a.W * 4;
  const int64_t b_lo = nb * rank / ranks;
  const int ny = (int)(nb * (rank + 1) / ranks - b_lo);
  pb += b_lo;

  // scaled logits of a byte's columns, packed in pairs, previously active positions pushed to the
  // lowest value (:96-104) and columns past the end to -inf
  auto load = [&](int y) -> uint4 {
    const int64_t c0 = (b_lo + y) * 8;
    if (vec && c0 + 8 <= a.S) return *reinterpret_cast<const uint4*>(s + c0);
    const uint16_t* u = reinterpret_cast<const uint16_t*>(s);
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t lo = c0 + 2 * i < a.S ? u[c0 + 2 * i] : 0u, hi = c0 + 2 * i + 1 < a.S ? u[c0 + 2 * i + 1] : 0u;
      w[i] = lo | hi << 16;
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
  };
  auto scale = [&](int y, const uint4& raw, unsigned int act, uint32_t* w) {
    const int64_t c0 = (b_lo + y) * 8;
    w[0] = raw.x; w[1] = raw.y; w[2] = raw.z; w[3] = raw.w;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = tp_pack2(__fmul_rn(tp_lo(w[i]), a.scaling), __fmul_rn(tp_hi(w[i]), a.scaling));
    if (bias) {
      float bv[8];
      tp_load8(bias, c0, a.S, bias_vec, bv);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        w[i] = tp_pack2(__fadd_rn(tp_lo(w[i]), bv[2 * i]), __fadd_rn(tp_hi(w[i]), bv[2 * i + 1]));
    }
    if (act || c0 + 8 > a.S) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const uint32_t v = c0 + i >= a.S ? 0xFF80u : 0xFF7Fu;
        if (((act >> i) & 1u) || c0 + i >= a.S)
          w[i >> 1] = (i & 1) ? (w[i >> 1] & 0xFFFFu) | v << 16 : (w[i >> 1] & 0xFFFF0000u) | v;
      }
    }
  };
  auto convert = [&](int y, uint32_t* w) { scale(y, load(y), pb[y], w); };

  for (int i = tid; i < TP_PER * TP_THREADS; i += TP_THREADS) {
    hist[i] = 0u;
    // bin 0 has weight 1, the last bin 0 (and everything past it)
    const unsigned int e = i == 0 ? 0x3F80u : i >= TP_BINS - 1 ? 0u : a.exp_table[TP_D0 - 1 + i];
    weight[i] = (uint16_t)min(e, 0x3F80u);
  }

  float mx = -INFINITY;
  constexpr int AHEAD = 4;
  for (int y0 = tid; y0 < ny; y0 += AHEAD * TP_THREADS) {
    uint4 raw[AHEAD];
    unsigned int act[AHEAD];
#pragma unroll
    for (int n = 0; n < AHEAD; ++n) {
      const int y = y0 + n * TP_THREADS;
      raw[n] = make_uint4(0u, 0u, 0u, 0u);
      act[n] = 0u;
      if (y < ny) {
        raw[n] = load(y);
        act[n] = pb[y];
      }
    }
#pragma unroll
    for (int n = 0; n < AHEAD; ++n) {
      const int y = y0 + n * TP_THREADS;
      if (y >= ny) break;
      uint32_t w[4];
      scale(y, raw[n], act[n], w);
      if (RESIDENT) tp_row[y] = make_uint4(w[0], w[1], w[2], w[3]);
#pragma unroll
      for (int i = 0; i < 4; ++i) mx = fmaxf(fmaxf(mx, tp_lo(w[i])), tp_hi(w[i]));
    }
  }
  mx = tp_block_max(mx, scratch);
  if (ranks > 1) {
    if (tid == 0) max_sm = mx;
    cluster.sync();
    for (int r = 0; r < ranks; ++r) mx = fmaxf(mx, *cluster.map_shared_rank(&max_sm, r));
  }

  // histogram over d
  auto bins = [&](int y, uint32_t* w) {
    if (RESIDENT) {
      const uint4 v = tp_row[y];
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
      convert(y, w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      w[i] = tp_bins2(tp_pack2(__fsub_rn(tp_lo(w[i]), mx), __fsub_rn(tp_hi(w[i]), mx)));
  };
  for (int y = tid; y < ny; y += TP_THREADS) {
    uint32_t w[4];
    bins(y, w);
    if (RESIDENT) tp_row[y] = make_uint4(w[0], w[1], w[2], w[3]);
    const int64_t left = a.S - (b_lo + y) * 8;
    if (left >= 8) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        atomicAdd(&hist[w[i] & 0xFFFFu], 1u);
        atomicAdd(&hist[w[i] >> 16], 1u);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < left) atomicAdd(&hist[(i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu], 1u);
    }
  }
  __syncthreads();
  if (ranks > 1) {
    cluster.sync();
    if (rank != 0) {
      unsigned int* h0 = cluster.map_shared_rank(hist, 0);
      for (int i = tid; i < TP_BINS; i += TP_THREADS)
        if (hist[i] != 0u) atomicAdd(&h0[i], hist[i]);
    }
    cluster.sync();
  }

  if (rank == 0) {
    // the non-empty bins, thread t looks at bins 3 t .. 3 t + 2
    unsigned int val[TP_PER];
    bool full[TP_PER];
    int n_here = 0;
#pragma unroll
    for (int i = 0; i < TP_PER; ++i) {
      val[i] = weight[tid * TP_PER + i];
      full[i] = val[i] != 0u && hist[tid * TP_PER + i] != 0u;
      n_here += full[i] ? 1 : 0;
    }
    if (tid == 0) { pick_sm = -1; thr_sm = -1; cross_sm = TP_BINS; }
    int n_list;
    int at = sah_block_excl_scan<int>(n_here, scan_sm, &n_list);
#pragma unroll
    for (int i = 0; i < TP_PER; ++i)
      if (full[i]) list[at++] = (uint16_t)(tid * TP_PER + i);
    __syncthreads();
    // replay of the accumulator, largest weight first: lane l takes entries base + 2 l, + 1
    if (warp == 0) {
      float acc = 0.f;
      for (int base = 0; base < n_list;) {
        if (acc == 0.f) {
          const int bin = list[0];
          acc = tp_add_run(0.f, weight[bin], hist[bin]);
          if (lane == 0) list_sum[0] = acc;
          base = 1;
          continue;
        }
        const int ea = (int)(__float_as_uint(acc) >> 23);
        const unsigned int A0 = (__float_as_uint(acc) & 0x7FFFFFu) | 0x800000u;
        unsigned int v[2], c[2];
        TpMove mv[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int e = base + 2 * lane + i;
          v[i] = c[i] = 0u;
          mv[i].d0 = mv[i].d1 = 0u;
          if (e < n_list) {
            const int bin = list[e];
            v[i] = weight[bin];
            c[i] = hist[bin];
            mv[i] = tp_move(v[i], c[i], ea);
          }
        }
        TpMove all = tp_then(mv[0], mv[1]);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          TpMove left;
          left.d0 = __shfl_up_sync(0xffffffffu, all.d0, o);
          left.d1 = __shfl_up_sync(0xffffffffu, all.d1, o);
          if (lane >= o) all = tp_then(left, all);
        }
        TpMove ex;
        ex.d0 = __shfl_up_sync(0xffffffffu, all.d0, 1);
        ex.d1 = __shfl_up_sync(0xffffffffu, all.d1, 1);
        if (lane == 0) ex.d0 = ex.d1 = 0u;
        // A in front of this lane's entries and behind each of them; from the first that reaches
        // the next binade on the numbers mean nothing
        const unsigned int before = A0 + ((A0 & 1u) ? ex.d1 : ex.d0);
        const unsigned int mid = before + ((before & 1u) ? mv[0].d1 : mv[0].d0);
        const unsigned int end = mid + ((mid & 1u) ? mv[1].d1 : mv[1].d0);
        const unsigned int over = __ballot_sync(0xffffffffu, end >= (1u << 24));  // moves only add up
        const int first = over ? __ffs(over) - 1 : 32;
        auto value = [&](unsigned int A) { return __uint_as_float((uint32_t)ea << 23 | (A & 0x7FFFFFu)); };
        const int e0 = base + 2 * lane;
        if (lane < first) {
          if (e0 < n_list) list_sum[e0] = value(mid);
          if (e0 + 1 < n_list) list_sum[e0 + 1] = value(end);
        } else if (lane == first && mid < (1u << 24)) {
          list_sum[e0] = value(mid);
        }
        if (first == 32) {
          acc = value(__shfl_sync(0xffffffffu, end, 31));
          base += 64;
        } else {
          const bool second = __shfl_sync(0xffffffffu, mid, first) < (1u << 24);  // which of the lane's entries
          const unsigned int A = __shfl_sync(0xffffffffu, second ? mid : before, first);
          const unsigned int vb = __shfl_sync(0xffffffffu, second ? v[1] : v[0], first);
          const unsigned int n = __shfl_sync(0xffffffffu, second ? c[1] : c[0], first);
          acc = tp_add_run(value(A), vb, n);
          base += 2 * first + (second ? 1 : 0);
          if (lane == 0) list_sum[base] = acc;
          ++base;
        }
      }
      if (lane == 0) acc_sm = acc;
    }
    __syncthreads();

    // first run (largest value) whose normalised prefix exceeds top_p (:118-131)
    const float total = sah_round_to<T>(acc_sm);
    const float p = sah_round_to<T>(a.top_p);
    int best = TP_BINS;  // place in the list
    for (int e = tid; e < n_list; e += TP_THREADS)
      if (sah_round_to<T>(__fdiv_rn(sah_round_to<T>(list_sum[e]), total)) > p) {
        best = e;
        break;
      }
    if (best < TP_BINS) atomicMin(&cross_sm, best);
    // weight 0 among the keys: bins whose weight is 0
#pragma unroll
    for (int i = 0; i < TP_PER; ++i)
      if (val[i] == 0u && hist[tid * TP_PER + i] != 0u) pick_sm = 1;
    __syncthreads();
    // nothing exceeds top_p: the search position is clamped to the last sorted element (:127-130)
    unsigned int thr;
    if (cross_sm < TP_BINS) thr = weight[list[cross_sm]];
    else thr = (pick_sm > 0 || n_list == 0) ? 0u : weight[list[n_list - 1]];
    // the last bin that is selected (weight >= threshold, :158-160)
    int keep = -1;
#pragma unroll
    for (int i = 0; i < TP_PER; ++i)
      if (tid * TP_PER + i < TP_BINS && val[i] >= thr) keep = tid * TP_PER + i;
    if (keep >= 0) atomicMax(&thr_sm, keep);
    __syncthreads();
  }
  int last_bin;
  if (ranks > 1) {
    cluster.sync();
    last_bin = *cluster.map_shared_rank(&thr_sm, 0);
    cluster.sync();  // rank 0 may not leave while its threshold is being read
  } else {
    last_bin = thr_sm;
  }

  unsigned char* out = reinterpret_cast<unsigned char*>(a.out_bits + row * a.W) + b_lo;
  for (int y = tid; y < ny; y += TP_THREADS) {
    uint32_t w[4];
    if (RESIDENT) {
      const uint4 v = tp_row[y];
      w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
    } else {
      bins(y, w);
    }
    uint32_t bits = 0u;  // the sign of bin - (last_bin + 1)
#pragma unroll
    for (int i = 7; i >= 0; --i)
      bits = __funnelshift_l(((i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu) - (uint32_t)(last_bin + 1), bits, 1);
    const int64_t left = a.S - (b_lo + y) * 8;
    if (left < 8) bits &= left <= 0 ? 0u : (1u << (int)left) - 1u;
    out[y] = (unsigned char)(a.or_prev ? (bits | pb[y]) : bits);
  }
}

extern "C" int sah_topp_select(const void* scores, int dtype, float scaling, const void* bias,
                               int64_t bias_s_b, int64_t bias_s_h, int64_t bias_s_q, int B, int Hq,
                               int Sq, int64_t S, int64_t W, const uint32_t* prev_bits, float top_p,
                               const uint16_t* exp_table, int or_prev, uint32_t* out_bits,
                               void* stream) {
  SAH_REQUIRE(scores && prev_bits && exp_table && out_bits, "topp_select: null pointer");
  SAH_REQUIRE(B > 0 && Hq > 0 && Sq > 0 && S > 0 && W * 32 >= S, "topp_select: bad extents");
  SAH_REQUIRE(top_p >= 0.f && top_p <= 1.f, "topp_select: top_p must be in [0, 1]");
  if (dtype != SAH_BF16)
    return sah_fail(SAH_ERR_UNSUPPORTED,
                    "topp_select: bfloat16 only (a float32 row is accumulated in float64 by the "
                    "reference over values that do not fall into a small set)");
  ToppArgs a;
  a.scores = scores; a.scaling = scaling; a.bias = bias;
  a.bias_s_b = bias_s_b; a.bias_s_h = bias_s_h; a.bias_s_q = bias_s_q;
  a.prev_bits = prev_bits; a.Hq = Hq; a.Sq = Sq; a.S = S; a.W = W; a.top_p = top_p;
  a.or_prev = or_prev; a.exp_table = exp_table; a.out_bits = out_bits;
  const int64_t rows = (int64_t)B * Hq * Sq;
  SAH_REQUIRE(rows <= 2147483647, "topp_select: too many rows");
  // Few rows: several CTAs per row (a power of two, so that the bitmap bytes split evenly), as
  // long as one wave holds them all and each still has a pass of 8 columns per thread.
  int ranks = 1;
  while (ranks < TP_MAX_CLUSTER && rows * ranks * 2 <= sah_cluster_wave(ranks * 2) &&
         S >= (int64_t)ranks * 2 * 8 * TP_THREADS)
    ranks *= 2;
  sah_prof_begin(SAH_PROF_TOPP, (cudaStream_t)stream);
  const int64_t row_bytes = (W * 4 + ranks - 1) / ranks * 16;
  const bool resident = row_bytes <= TP_ROW_BYTES;
  if (resident) {
    const cudaError_t e = cudaFuncSetAttribute(topp_select_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               TP_ROW_BYTES);
    if (e != cudaSuccess) return sah_fail(SAH_ERR_CUDA, "topp_select attr: %s", cudaGetErrorString(e));
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(rows * ranks));
  cfg.blockDim = dim3(TP_THREADS);
  cfg.dynamicSmemBytes = resident ? (size_t)row_bytes : 0;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)ranks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // (a launch error stays for SAH_LAUNCH_CHECK)
  if (resident) (void)cudaLaunchKernelEx(&cfg, topp_select_kernel<true>, a);
  else (void)cudaLaunchKernelEx(&cfg, topp_select_kernel<false>, a);
  SAH_LAUNCH_CHECK("topp_select");
  sah_prof_end(SAH_PROF_TOPP, (cudaStream_t)stream);
  return SAH_OK;
}
