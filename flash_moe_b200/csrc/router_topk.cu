// Product-key router top-k for sm_100a.
//
// For every token the reference evaluates all nk*nk sums lp0[i] + lp1[j] and extracts the k
// largest by k rounds of arg-max (flash_moe/ops/triton/flash_router.py:8-194).  This kernel gets
// the same answer - same scores, same indices, same order, including the order among equal
// scores (ascending flat id i*nk + j) - from far less work:
//
//   1. sort each half descending (value, then lower index first);
//   2. a candidate at ranks (p, q) (0-based) has (p+1)*(q+1)-1 candidates that score at least
//      as high, so only the "staircase" (p+1)*(q+1) <= k can hold a score above the k-th
//      largest; its ~k ln k sums are formed in the input dtype like the reference does;
//   3. tau = k-th largest staircase score, found by a bitwise search on order-preserving keys;
//      every candidate scoring above tau is inside the staircase and is emitted;
//   4. the remaining slots go to candidates scoring exactly tau with the lowest flat ids.  These
//      may lie outside the staircase, so they are located exactly: per row i a binary search in
//      the sorted second half counts its ties, then rows are visited in index order.
//   5. the k winners are sorted by (score desc, flat id asc) and written out, optionally with
//      gates = exp(score) (and the row renormalisation of flash_moe/modules/flash_moe.py:80-85).
//
// One warp owns one token; all scratch lives in shared memory.
#include "common.cuh"
#include "warp_sort.cuh"

namespace fmoe {
namespace {

constexpr unsigned kFull = 0xFFFFFFFFu;

template <typename T> struct OrdLowBits;  // low bits of the order key that carry no information
template <> struct OrdLowBits<float> { static constexpr int value = 0; };
template <> struct OrdLowBits<__nv_bfloat16> { static constexpr int value = 16; };
template <> struct OrdLowBits<__half> { static constexpr int value = 13; };

__device__ __forceinline__ uint64_t make_key(uint32_t ord, uint32_t id) {
  return (static_cast<uint64_t>(ord) << 32) | static_cast<uint64_t>(0xFFFFFFFFu - id);
}
__device__ __forceinline__ uint32_t key_id(uint64_t key) { return 0xFFFFFFFFu - static_cast<uint32_t>(key); }
__device__ __forceinline__ float key_val(uint64_t key) { return ord_to_f32(static_cast<uint32_t>(key >> 32)); }

// Warp-cooperative bitonic sort (descending) of one or two arrays of n = 2^m keys in shared memory.
__device__ __forceinline__ void bitonic_desc(uint64_t* a, uint64_t* b, int n, int lane) {
  for (int size = 2; size <= n; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = lane; i < (n >> 1); i += 32) {
        const int lo = ((i & ~(stride - 1)) << 1) | (i & (stride - 1));
        const int hi = lo | stride;
        const bool desc = (lo & size) == 0;
        uint64_t x = a[lo], y = a[hi];
        if ((x < y) == desc) { a[lo] = y; a[hi] = x; }
        if (b != nullptr) {
          x = b[lo]; y = b[hi];
          if ((x < y) == desc) { b[lo] = y; b[hi] = x; }
        }
      }
      __syncwarp();
    }
  }
}

struct RouterSmemLayout {
  int cta_bytes;   // staircase table + row starts (shared by the CTA)
  int warp_bytes;  // per-warp scratch
  int off_keys, off_win, off_cs, off_cnt;
  int nkp, kp, kq, C, Cp;
};

template <typename T>
__global__ void router_topk_smem_kernel(const T* __restrict__ logp, int64_t ntok, int nk, int k, RouterSmemLayout L,
                                   T* __restrict__ scores, int64_t* __restrict__ indices, T* __restrict__ gates,
                                   int flags) {
  const int norm = flags & kTopkNorm;
  const bool token_rows = (flags & kTopkTokenRows) != 0;  // [T, 2, nk] instead of [2, T, nk]
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int kq = L.kq, C = L.C, nkp = L.nkp, kp = L.kp;

  // ---- staircase table, built once per CTA: entry c -> (p << 16) | q with (p+1)(q+1) <= k
  uint32_t* pq = reinterpret_cast<uint32_t*>(smem);
  int* rowstart = reinterpret_cast<int*>(smem) + L.Cp;
  if (warp == 0) {
    int running = 0;
    for (int base = 0; base < kq; base += 32) {
      const int p = base + lane;
      const int len = (p < kq) ? min(k / (p + 1), kq) : 0;
      int incl = len;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += up;
      }
      if (p < kq) rowstart[p] = running + incl - len;
      running += __shfl_sync(kFull, incl, 31);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {  // entry c lies in the last row whose start is <= c
    int lo = 0, hi = kq - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (rowstart[mid] <= c) lo = mid; else hi = mid - 1;
    }
    pq[c] = (static_cast<uint32_t>(lo) << 16) | static_cast<uint32_t>(c - rowstart[lo]);
  }
  __syncthreads();

  unsigned char* wbase = smem + L.cta_bytes + warp * L.warp_bytes;
  float* va = reinterpret_cast<float*>(wbase);
  float* vb = va + nk;
  uint64_t* ka = reinterpret_cast<uint64_t*>(wbase + L.off_keys);
  uint64_t* kb = ka + nkp;
  uint64_t* win = reinterpret_cast<uint64_t*>(wbase + L.off_win);
  uint32_t* cs = reinterpret_cast<uint32_t*>(wbase + L.off_cs);
  uint32_t* cnt = reinterpret_cast<uint32_t*>(wbase + L.off_cnt);
  constexpr int LOW = OrdLowBits<T>::value;

  for (int64_t t = static_cast<int64_t>(blockIdx.x) * nwarps + warp; t < ntok;
       t += static_cast<int64_t>(gridDim.x) * nwarps) {
    const T* a_row = token_rows ? logp + t * 2 * nk : logp + t * nk;
    const T* b_row = token_rows ? a_row + nk : logp + (ntok + t) * nk;
    // 1. load (canonicalising -0 to +0) and build sort keys
    for (int i = lane; i < nkp; i += 32) {
      if (i < nk) {
        const float a = to_f32<T>(a_row[i]) + 0.0f;
        const float b = to_f32<T>(b_row[i]) + 0.0f;
        va[i] = a;
        vb[i] = b;
        ka[i] = make_key(f32_to_ord(a), i);
        kb[i] = make_key(f32_to_ord(b), i);
      } else {
        ka[i] = 0;
        kb[i] = 0;
      }
    }
    __syncwarp();
    bitonic_desc(ka, kb, nkp, lane);

    // 2. staircase candidate scores, rounded to T like the reference's in-dtype add
    for (int c = lane; c < C; c += 32) {
      const uint32_t e = pq[c];
      const float s = round_to<T>(__fadd_rn(key_val(ka[e >> 16]), key_val(kb[e & 0xFFFFu])));
      cs[c] = f32_to_ord(s + 0.0f);
    }
    __syncwarp();

    // 3. tau = k-th largest candidate score (bitwise search over the order key)
    uint32_t tau = 0;
    for (int bit = 31; bit >= LOW; --bit) {
      const uint32_t trial = tau | (1u << bit);
      int n_ge = 0;
      for (int c = lane; c < C; c += 32) n_ge += (cs[c] >= trial) ? 1 : 0;
      n_ge = __reduce_add_sync(kFull, n_ge);
      if (n_ge >= k) tau = trial;
    }
    if (LOW > 0 && (tau >> 31) == 0) tau |= (1u << LOW) - 1u;  // negative values: dropped bits are all ones

    // emit everything strictly above tau
    int filled = 0;
    for (int base = 0; base < C; base += 32) {
      const int c = base + lane;
      const bool g = (c < C) && (cs[c] > tau);
      const unsigned bal = __ballot_sync(kFull, g);
      if (g) {
        const int pos = filled + __popc(bal & ((1u << lane) - 1u));
        const uint32_t e = pq[c];
        const uint32_t flat = key_id(ka[e >> 16]) * static_cast<uint32_t>(nk) + key_id(kb[e & 0xFFFFu]);
        if (pos < k) win[pos] = make_key(cs[c], flat);
      }
      filled += __popc(bal);
    }
    int need = k - filled;

    // 4. candidates equal to tau, lowest flat id first.  Row i ties with sorted-b positions [gt, ge).
    for (int i = lane; i < nk; i += 32) {
      const float a = va[i];
      int lo = 0, hi = nk;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (f32_to_ord(round_to<T>(__fadd_rn(a, key_val(kb[mid]))) + 0.0f) >= tau) lo = mid + 1; else hi = mid;
      }
      const int ge = lo;
      lo = 0; hi = ge;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (f32_to_ord(round_to<T>(__fadd_rn(a, key_val(kb[mid]))) + 0.0f) > tau) lo = mid + 1; else hi = mid;
      }
      cnt[i] = static_cast<uint32_t>(ge - lo);
    }
    __syncwarp();
    for (int base = 0; base < nk && need > 0; base += 32) {
      const int i = base + lane;
      unsigned has = __ballot_sync(kFull, (i < nk) && (cnt[i] > 0));
      while (has != 0 && need > 0) {
        const int row = base + __ffs(has) - 1;
        has &= has - 1;
        const float a = va[row];
        for (int jb = 0; jb < nk && need > 0; jb += 32) {
          const int j = jb + lane;
          const bool tie = (j < nk) && (f32_to_ord(round_to<T>(__fadd_rn(a, vb[j])) + 0.0f) == tau);
          const unsigned bal = __ballot_sync(kFull, tie);
          const int rank = __popc(bal & ((1u << lane) - 1u));
          if (tie && rank < need)
            win[filled + rank] = make_key(tau, static_cast<uint32_t>(row) * static_cast<uint32_t>(nk) + j);
          const int took = min(__popc(bal), need);
          filled += took;
          need -= took;
        }
      }
    }
    for (int r = filled + lane; r < kp; r += 32) win[r] = 0;
    __syncwarp();

    // 5. order the winners and write out
    bitonic_desc(win, nullptr, kp, lane);
    float gsum = 0.f;
    for (int r = lane; r < k; r += 32) {
      const uint64_t key = win[r];
      const float s = key_val(key);
      scores[t * k + r] = from_f32<T>(s);
      indices[t * k + r] = static_cast<int64_t>(key_id(key));
      if (gates != nullptr) {
        const T g = from_f32<T>(expf(s));
        gsum += to_f32<T>(g);
        if (!norm) gates[t * k + r] = g;
      }
    }
    if (gates != nullptr && norm) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) gsum += __shfl_xor_sync(kFull, gsum, d);
      const float denom = round_to<T>(gsum);
      for (int r = lane; r < k; r += 32) {
        const float g = round_to<T>(expf(key_val(win[r])));
        gates[t * k + r] = from_f32<T>(g / denom);
      }
    }
    __syncwarp();
  }
}


// ------------------------------------------------------------------------------------------
// Register-resident variant for num_keys <= 1024 (float32; 16-bit rows where it is the faster one, see launch_typed): each half is sorted by a shuffle-based bitonic
// network (E = padded num_keys / 32 keys per lane), sort keys are 32-bit for 16-bit dtypes
// (16-bit order key | inverted index) and 64-bit for float32.  Shared memory only holds the
// sorted halves (for the candidate gathers and binary searches), the index-order values, the
// candidate scores and the winners.
// ------------------------------------------------------------------------------------------
template <typename T> struct HalfKey;  // sort key of one router half
template <> struct HalfKey<float> {
  using type = uint64_t;
  static __device__ __forceinline__ uint64_t make(float v, uint32_t i) { return make_key(f32_to_ord(v), i); }
  static __device__ __forceinline__ float value(uint64_t k) { return key_val(k); }
  static __device__ __forceinline__ uint32_t id(uint64_t k) { return key_id(k); }
};
template <typename T16> struct HalfKey16 {
  using type = uint32_t;
  static __device__ __forceinline__ uint32_t make(float v, uint32_t i) {
    const T16 h = from_f32<T16>(v);  // exact: v came from a T16
    uint32_t b = *reinterpret_cast<const uint16_t*>(&h);
    b ^= (b >> 15) ? 0xFFFFu : 0x8000u;
    return (b << 16) | (0xFFFFu - i);
  }
  static __device__ __forceinline__ float value(uint32_t k) {
    uint32_t b = k >> 16;
    b ^= (b >> 15) ? 0x8000u : 0xFFFFu;
    const uint16_t raw = static_cast<uint16_t>(b);
    return to_f32<T16>(*reinterpret_cast<const T16*>(&raw));
  }
  static __device__ __forceinline__ uint32_t id(uint32_t k) { return 0xFFFFu - (k & 0xFFFFu); }
};
template <> struct HalfKey<__nv_bfloat16> {  // the upper half of the float is the value: no conversions
  using type = uint32_t;
  static __device__ __forceinline__ uint32_t make(float v, uint32_t i) {
    const uint32_t x = __float_as_uint(v);
    return ((x ^ (static_cast<uint32_t>(static_cast<int32_t>(x) >> 31) | 0x80000000u)) & 0xFFFF0000u) | (0xFFFFu - i);
  }
  static __device__ __forceinline__ float value(uint32_t k) {
    return __uint_as_float((k ^ (static_cast<int32_t>(k) < 0 ? 0x80000000u : 0xFFFFFFFFu)) & 0xFFFF0000u);
  }
  static __device__ __forceinline__ uint32_t id(uint32_t k) { return 0xFFFFu - (k & 0xFFFFu); }
};
template <> struct HalfKey<__half> : HalfKey16<__half> {};

// One lane's E consecutive elements of a row (element lane * E + r -> v[r]); entries past nk read as -inf.  Whole
// rows of 32 E elements at a 16-byte aligned address are fetched with one or a few vector loads.
// Rows are read past the L1 cache: with kTopkLateWait a CTA starts beside an unrelated kernel.
__device__ __forceinline__ float load_cg(const float* p) { return __ldcg(p); }
template <typename T>
__device__ __forceinline__ T load_cg(const T* p) {
  const unsigned short raw = __ldcg(reinterpret_cast<const unsigned short*>(p));
  return *reinterpret_cast<const T*>(&raw);
}

template <typename T, int E>
__device__ __forceinline__ void load_blocked(const T* row, int nk, int lane, float (&v)[E]) {
  constexpr int BYTES = E * static_cast<int>(sizeof(T));
  if (BYTES >= 4 && nk == 32 * E && (reinterpret_cast<uintptr_t>(row) & 15u) == 0) {
    __align__(16) T tmp[E];
    const T* src = row + lane * E;
    if constexpr (BYTES % 16 == 0) {
#pragma unroll
      for (int j = 0; j < BYTES / 16; ++j) reinterpret_cast<uint4*>(tmp)[j] = __ldcg(reinterpret_cast<const uint4*>(src) + j);
    } else if constexpr (BYTES == 8) {
      *reinterpret_cast<uint2*>(tmp) = __ldcg(reinterpret_cast<const uint2*>(src));
    } else if constexpr (BYTES == 4) {
      *reinterpret_cast<uint32_t*>(tmp) = __ldcg(reinterpret_cast<const unsigned int*>(src));
    }
#pragma unroll
    for (int r = 0; r < E; ++r) v[r] = to_f32<T>(tmp[r]);
  } else {
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int i = lane * E + r;
      v[r] = (i < nk) ? to_f32<T>(load_cg(row + i)) : -INFINITY;
    }
  }
}

// One lane's E consecutive entries of a per-warp shared-memory array (16-byte aligned base, 32 E entries)
template <int E>
__device__ __forceinline__ void store_blocked(float* base, int lane, const float (&v)[E]) {
  float* dst = base + lane * E;
  if constexpr (E % 4 == 0) {
#pragma unroll
    for (int j = 0; j < E / 4; ++j)
      reinterpret_cast<float4*>(dst)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
  } else if constexpr (E == 2) {
    *reinterpret_cast<float2*>(dst) = make_float2(v[0], v[1]);
  } else {
#pragma unroll
    for (int r = 0; r < E; ++r) dst[r] = v[r];
  }
}
template <int E>
__device__ __forceinline__ void store_blocked(uint16_t* base, int lane, const uint32_t (&v)[E]) {  // v[r] < 65536
  uint16_t* dst = base + lane * E;
  if constexpr (E % 8 == 0) {
#pragma unroll
    for (int j = 0; j < E / 8; ++j)
      reinterpret_cast<uint4*>(dst)[j] =
          make_uint4(v[8 * j] | (v[8 * j + 1] << 16), v[8 * j + 2] | (v[8 * j + 3] << 16),
                     v[8 * j + 4] | (v[8 * j + 5] << 16), v[8 * j + 6] | (v[8 * j + 7] << 16));
  } else if constexpr (E == 4) {
    *reinterpret_cast<uint2*>(dst) = make_uint2(v[0] | (v[1] << 16), v[2] | (v[3] << 16));
  } else if constexpr (E == 2) {
    *reinterpret_cast<uint32_t*>(dst) = v[0] | (v[1] << 16);
  } else {
#pragma unroll
    for (int r = 0; r < E; ++r) dst[r] = static_cast<uint16_t>(v[r]);
  }
}

constexpr int kTieCap = 256;  // entries of the per-warp list of candidates that tie with tau

struct RouterRegLayout {
  int cta_bytes, warp_bytes;
  int off_sorted, off_ids, off_win, off_cs, off_tl;
  int nkp, kp, kq, C, Cp;
};

// CPL > 0: the staircase candidates (at most 32 * CPL of them) stay in registers, CPL per lane, through the threshold
// search and the emit step, whose loops then have compile-time bounds and no shared-memory round trips between rounds.
template <typename T, int E, int CPL = 0>
__global__ void __launch_bounds__(256) router_topk_reg_kernel(const T* logp, int64_t ntok, int nk, int k,
                                                             RouterRegLayout L, T* __restrict__ scores,
                                                             int64_t* __restrict__ indices, T* __restrict__ gates,
                                                             int flags) {
  const int norm = flags & kTopkNorm;
  const bool from_logits = (flags & kTopkFromLogits) != 0;
  const bool token_rows = (flags & (kTopkFromLogits | kTopkTokenRows)) != 0;  // [T, 2, nk] instead of [2, T, nk]
  using HK = HalfKey<T>;
  using K = typename HK::type;
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int kq = L.kq, C = L.C, nkp = L.nkp, kp = L.kp;

  uint32_t* pq = reinterpret_cast<uint32_t*>(smem);
  int* rowstart = reinterpret_cast<int*>(smem) + L.Cp;
  if (warp == 0) {
    int running = 0;
    for (int base = 0; base < kq; base += 32) {
      const int p = base + lane;
      const int len = (p < kq) ? min(k / (p + 1), kq) : 0;
      int incl = len;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int up = __shfl_up_sync(kFull, incl, d);
        if (lane >= d) incl += up;
      }
      if (p < kq) rowstart[p] = running + incl - len;
      running += __shfl_sync(kFull, incl, 31);
    }
  }
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += blockDim.x) {  // entry c lies in the last row whose start is <= c
    int lo = 0, hi = kq - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (rowstart[mid] <= c) lo = mid; else hi = mid - 1;
    }
    pq[c] = (static_cast<uint32_t>(lo) << 16) | static_cast<uint32_t>(c - rowstart[lo]);
  }
  __syncthreads();
  // the staircase table above depends on k alone; the logits come from the previous kernel (kTopkLateWait: the one before)
  if (!(flags & kTopkLateWait)) pdl_wait();

  unsigned char* wbase = smem + L.cta_bytes + warp * L.warp_bytes;
  float* va = reinterpret_cast<float*>(wbase);  // index order
  float* vb = va + nkp;
  float* sa = reinterpret_cast<float*>(wbase + L.off_sorted);  // sorted, descending
  float* sb = sa + nkp;
  uint16_t* ia = reinterpret_cast<uint16_t*>(wbase + L.off_ids);
  uint16_t* ib = ia + nkp;
  uint64_t* win = reinterpret_cast<uint64_t*>(wbase + L.off_win);
  uint32_t* cs = reinterpret_cast<uint32_t*>(wbase + L.off_cs);
  uint32_t* tl = reinterpret_cast<uint32_t*>(wbase + L.off_tl);  // flat ids of candidates equal to tau
  int* tcnt = reinterpret_cast<int*>(tl + kTieCap);
  constexpr int LOW = OrdLowBits<T>::value;
  int nsteps = 0;  // binary-search steps covering [0, nk]
  while ((1 << nsteps) <= nk) ++nsteps;

  for (int64_t t = static_cast<int64_t>(blockIdx.x) * nwarps + warp; t < ntok;
       t += static_cast<int64_t>(gridDim.x) * nwarps) {
    if (t + static_cast<int64_t>(gridDim.x) * nwarps >= ntok) pdl_launch_dependents();  // last token of this warp
    // from_logits: the input is the raw router logits [T, 2*nk]; the per-half log-softmax
    // (flash_moe/modules/flash_moe.py:72) is applied here, rounded to T like torch does
    const T* a_row = token_rows ? logp + t * 2 * nk : logp + t * nk;
    const T* b_row = token_rows ? a_row + nk : logp + (ntok + t) * nk;
    // 1. per half: load (lane-blocked: element lane * E + r in register r), optional log-softmax, keep the
    //    index-order copy, sort in registers, store the rank-order values and ids.  The two halves run through ONE copy
    //    of this code (the loop is not unrolled): the unrolled sorting network is most of the kernel's instructions -
    //    at 16 keys per lane two copies alone exceed 70 KB - and only one half's keys are live at a time.
    //    Measured, 16384 tokens x 512 keys top-128 | 16384 x 1024 top-16 | 131072 x 256 top-32 | 4096 x 128 top-64 (us):
    //    this form 330 | 532 | 559 | 21.5; both halves unrolled side by side 348 | 663 | 539 | 22.5; keys dealt round-robin
    //    over the lanes (r * 32 + lane, 25-35 shuffle stages) unrolled side by side 304 | 584 | 803 | 25.6, in one copy
    //    476 | 962 - with 16 or 32 keys per lane few warps are resident and the two halves' independent chains hide
    //    each other's latency, which the single copy gives up and the smaller code buys back.
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      const T* row = h == 0 ? a_row : b_row;
      float* vh = h == 0 ? va : vb;
      float* sh = h == 0 ? sa : sb;
      uint16_t* ih = h == 0 ? ia : ib;
      K key[E];
      float lv[E];
      load_blocked<T, E>(row, nk, lane, lv);
      if (from_logits) {
        float m = -INFINITY;
#pragma unroll
        for (int r = 0; r < E; ++r) m = fmaxf(m, lv[r]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, d));
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < E; ++r)
          if (lane * E + r < nk) sum += expf(lv[r] - m);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
        const float lg = logf(sum);
#pragma unroll
        for (int r = 0; r < E; ++r) lv[r] = round_to<T>((lv[r] - m) - lg);
      }
#pragma unroll
      for (int r = 0; r < E; ++r) {
        const int i = lane * E + r;
        lv[r] += 0.0f;  // -0 -> +0
        key[r] = (i < nk) ? HK::make(lv[r], i) : K(0);
      }
      store_blocked<E>(vh, lane, lv);  // index order (entries past nk are never read)
      bitonic_desc_regs<E, K>(key, lane);
      uint32_t idr[E];
#pragma unroll
      for (int r = 0; r < E; ++r) {
        lv[r] = HK::value(key[r]);
        idr[r] = HK::id(key[r]) & 0xFFFFu;
      }
      store_blocked<E>(sh, lane, lv);  // rank order
      store_blocked<E>(ih, lane, idr);
    }
    __syncwarp();

    // 2. staircase candidate scores; track the smallest to narrow the threshold search
    uint32_t cmin = 0xFFFFFFFFu;
    uint32_t csr[CPL > 0 ? CPL : 1], pqr[CPL > 0 ? CPL : 1];
    auto pair_ord = [&](uint32_t e) { return f32_to_ord(round_to<T>(__fadd_rn(sa[e >> 16], sb[e & 0xFFFFu])) + 0.0f); };
    if constexpr (CPL > 0) {
#pragma unroll
      for (int j = 0; j < CPL; ++j) {
        const int c = 32 * j + lane;
        const bool in = c < C;
        pqr[j] = in ? pq[c] : 0u;
        const uint32_t o = pair_ord(pqr[j]);
        csr[j] = in ? o : 0u;  // 0 is below the key of every float, -inf included
        if (in) {
          cs[c] = o;  // the tie search below looks up single cells
          cmin = min(cmin, o);
        }
      }
    } else {
      for (int c = lane; c < C; c += 32) {
        cs[c] = pair_ord(pq[c]);
        cmin = min(cmin, cs[c]);
      }
    }
    cmin = __reduce_min_sync(kFull, cmin);
    __syncwarp();
    const uint32_t cmax = cs[0];  // ranks (0, 0): the largest sum

    // 3. tau = k-th largest candidate; all candidates agree on the bits above the top differing one
    uint32_t tau = cmax;
    if (cmax != cmin) {
      const int top = 31 - __clz(cmax ^ cmin);
      tau = cmax & ~((2u << top) - 1u);
      for (int bit = top; bit >= LOW; --bit) {
        const uint32_t trial = tau | (1u << bit);
        int n_ge = 0;
        if constexpr (CPL > 0) {
#pragma unroll
          for (int j = 0; j < CPL; ++j) n_ge += (csr[j] >= trial) ? 1 : 0;
        } else {
          for (int c = lane; c < C; c += 32) n_ge += (cs[c] >= trial) ? 1 : 0;
        }
        n_ge = __reduce_add_sync(kFull, n_ge);
        if (n_ge >= k) tau = trial;
      }
      if (LOW > 0 && (tau >> 31) == 0) tau |= (1u << LOW) - 1u;
    }

    // emit everything above tau; collect the staircase candidates equal to tau in the tie list
    int filled = 0, nties = 0;
    auto emit = [&](bool in, uint32_t v, auto cell) {
      const bool g = in && v > tau;
      const bool eq = in && v == tau;
      const unsigned bal = __ballot_sync(kFull, g);
      const unsigned beq = __ballot_sync(kFull, eq);
      if (g || eq) {
        const uint32_t e = cell();
        const uint32_t flat = static_cast<uint32_t>(ia[e >> 16]) * static_cast<uint32_t>(nk) + ib[e & 0xFFFFu];
        if (g) {
          const int pos = filled + __popc(bal & ((1u << lane) - 1u));
          if (pos < k) win[pos] = make_key(v, flat);
        } else {
          const int pos = nties + __popc(beq & ((1u << lane) - 1u));
          if (pos < kTieCap) tl[pos] = flat;
        }
      }
      filled += __popc(bal);
      nties += __popc(beq);
    };
    if constexpr (CPL > 0) {
#pragma unroll
      for (int j = 0; j < CPL; ++j)
        if (32 * j < C) emit(32 * j + lane < C, csr[j], [&] { return pqr[j]; });
    } else {
      for (int base = 0; base < C; base += 32) {
        const int c = base + lane;
        emit(c < C, (c < C) ? cs[c] : 0u, [&] { return pq[c]; });
      }
    }
    int need = k - filled;

    // 4. the remaining `need` slots go to the candidates equal to tau with the lowest flat ids.
    //    Outside the staircase every score is <= tau, and along a row (fixed rank p of the first
    //    half) the scores do not increase, so the ties outside the staircase are the runs that
    //    continue a row past its last staircase cell, plus runs from q = 0 in the rows below the
    //    staircase.  They are gathered in rank space into the tie list; if the list overflows, the
    //    exhaustive per-row search below takes over.
    if (lane == 0) *tcnt = nties;
    __syncwarp();
    for (int p = lane; p < kq; p += 32) {
      const int rs = rowstart[p];
      const int len = ((p + 1 < kq) ? rowstart[p + 1] : C) - rs;  // = min(k / (p + 1), kq) without the division
      if (len < nk && cs[rs + len - 1] >= tau) {
        const float a = sa[p];
        const uint32_t ida = static_cast<uint32_t>(ia[p]) * static_cast<uint32_t>(nk);
        for (int q = len; q < nk; ++q) {
          if (f32_to_ord(round_to<T>(__fadd_rn(a, sb[q])) + 0.0f) != tau) break;
          const int pos = atomicAdd(tcnt, 1);
          if (pos < kTieCap) tl[pos] = ida + ib[q];
        }
      }
    }
    {
      const float b0 = sb[0];
      for (int base = kq; base < nk; base += 32) {  // rows below the staircase: tie runs start at q = 0
        const int p = base + lane;
        const bool hit = (p < nk) && (f32_to_ord(round_to<T>(__fadd_rn(sa[p < nk ? p : 0], b0)) + 0.0f) == tau);
        if (hit) {
          const float a = sa[p];
          const uint32_t ida = static_cast<uint32_t>(ia[p]) * static_cast<uint32_t>(nk);
          for (int q = 0; q < nk; ++q) {
            if (f32_to_ord(round_to<T>(__fadd_rn(a, sb[q])) + 0.0f) != tau) break;
            const int pos = atomicAdd(tcnt, 1);
            if (pos < kTieCap) tl[pos] = ida + ib[q];
          }
        }
        if (__ballot_sync(kFull, hit) == 0u) break;  // the rows are sorted: no later row can tie
      }
    }
    __syncwarp();
    nties = *tcnt;
    __syncwarp();
    const bool tie_list_ok = nties <= kTieCap;
    if (tie_list_ok && need > 0 && nties <= 32) {
      // the usual case, a handful of ties: one id per lane, its rank among them by a round of shuffles
      const uint32_t id = lane < nties ? tl[lane] : 0xFFFFFFFFu;
      int rank = 0;
      for (int j = 0; j < nties; ++j) rank += (__shfl_sync(kFull, id, j) < id) ? 1 : 0;
      if (lane < nties && rank < need) win[filled + rank] = make_key(tau, id);
      filled += min(nties, need);
      need = k - filled;
    } else if (tie_list_ok && need > 0) {
      uint32_t phi = 0xFFFFFFFFu;  // ids <= phi are taken
      if (nties > need) {
        // phi = the need-th smallest id = the largest v with fewer than `need` ids below v
        uint32_t v = 0;
        const int topbit = 31 - __clz(static_cast<unsigned>(nk) * static_cast<unsigned>(nk));
        for (int bit = topbit; bit >= 0; --bit) {
          const uint32_t trial = v | (1u << bit);
          int below = 0;
          for (int i = lane; i < nties; i += 32) below += (tl[i] < trial) ? 1 : 0;
          below = __reduce_add_sync(kFull, below);
          if (below < need) v = trial;
        }
        phi = v;
      }
      for (int base = 0; base < nties; base += 32) {
        const int i = base + lane;
        const uint32_t id = (i < nties) ? tl[i] : 0xFFFFFFFFu;
        const bool take = (i < nties) && (id <= phi);
        const unsigned bal = __ballot_sync(kFull, take);
        if (take) win[filled + __popc(bal & ((1u << lane) - 1u))] = make_key(tau, id);
        filled += __popc(bal);
      }
      need = k - filled;
    }

    // 4b. overflow path (more than kTieCap ties, e.g. constant inputs): row i = r*32 + lane ties with
    //     sorted-b positions [gt, ge); rows are then visited in index order
    if (!tie_list_ok) {
    int lo_ge[E], hi_ge[E], lo_gt[E], hi_gt[E];
    float arow[E];
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int i = (r << 5) | lane;
      arow[r] = (i < nk) ? va[i] : 0.f;
      lo_ge[r] = 0; hi_ge[r] = (i < nk) ? nk : 0;
      lo_gt[r] = 0; hi_gt[r] = (i < nk) ? nk : 0;
    }
    for (int step = 0; step < nsteps; ++step) {
#pragma unroll
      for (int r = 0; r < E; ++r) {
        if (lo_ge[r] < hi_ge[r]) {
          const int mid = (lo_ge[r] + hi_ge[r]) >> 1;
          const uint32_t o = f32_to_ord(round_to<T>(__fadd_rn(arow[r], sb[mid])) + 0.0f);
          if (o >= tau) lo_ge[r] = mid + 1; else hi_ge[r] = mid;
        }
        if (lo_gt[r] < hi_gt[r]) {
          const int mid = (lo_gt[r] + hi_gt[r]) >> 1;
          const uint32_t o = f32_to_ord(round_to<T>(__fadd_rn(arow[r], sb[mid])) + 0.0f);
          if (o > tau) lo_gt[r] = mid + 1; else hi_gt[r] = mid;
        }
      }
    }
#pragma unroll
    for (int r = 0; r < E; ++r) {
      const int cnt = lo_ge[r] - lo_gt[r];
      unsigned has = __ballot_sync(kFull, cnt > 0);
      while (has != 0 && need > 0) {
        const int row = (r << 5) + __ffs(has) - 1;
        has &= has - 1;
        const float a = va[row];
        for (int jb = 0; jb < nk && need > 0; jb += 32) {
          const int j = jb + lane;
          const bool tie = (j < nk) && (f32_to_ord(round_to<T>(__fadd_rn(a, vb[j])) + 0.0f) == tau);
          const unsigned bal = __ballot_sync(kFull, tie);
          const int rank = __popc(bal & ((1u << lane) - 1u));
          if (tie && rank < need)
            win[filled + rank] = make_key(tau, static_cast<uint32_t>(row) * static_cast<uint32_t>(nk) + j);
          const int took = min(__popc(bal), need);
          filled += took;
          need -= took;
        }
      }
    }
    }  // overflow path
    for (int r = filled + lane; r < kp; r += 32) win[r] = 0;
    __syncwarp();

    // 5. order the winners (registers when they fit, shared memory otherwise) and write out
    if (sizeof(T) == 2 && kp == 64 && nk <= 256) {
      // 16-bit scores and 16-bit flat ids: sort 32-bit keys
      uint32_t w[2];
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint64_t key = win[lane * 2 + r];
        w[r] = key == 0 ? 0u : static_cast<uint32_t>(HalfKey<T>::make(key_val(key), key_id(key)));
      }
      bitonic_desc_regs<2, uint32_t>(w, lane);
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        const uint32_t key32 = w[r];
        const float sc = static_cast<float>(HalfKey<T>::value(static_cast<typename HalfKey<T>::type>(key32)));
        win[lane * 2 + r] = make_key(f32_to_ord(sc + 0.0f), HalfKey<T>::id(static_cast<typename HalfKey<T>::type>(key32)));
      }
    } else if (kp <= 32) {
      uint64_t w[1] = {lane < kp ? win[lane] : 0};
      bitonic_desc_regs<1, uint64_t>(w, lane);
      if (lane < kp) win[lane] = w[0];
    } else if (kp == 64) {
      uint64_t w[2] = {win[2 * lane], win[2 * lane + 1]};
      bitonic_desc_regs<2, uint64_t>(w, lane);
      win[2 * lane] = w[0]; win[2 * lane + 1] = w[1];
    } else if (kp == 128) {
      uint64_t w[4] = {win[4 * lane], win[4 * lane + 1], win[4 * lane + 2], win[4 * lane + 3]};
      bitonic_desc_regs<4, uint64_t>(w, lane);
      win[4 * lane] = w[0]; win[4 * lane + 1] = w[1]; win[4 * lane + 2] = w[2]; win[4 * lane + 3] = w[3];
    } else {
      bitonic_desc(win, nullptr, kp, lane);
    }
    __syncwarp();
    float gsum = 0.f;
    for (int r = lane; r < k; r += 32) {
      const uint64_t key = win[r];
      const float s = key_val(key);
      scores[t * k + r] = from_f32<T>(s);
      indices[t * k + r] = static_cast<int64_t>(key_id(key));
      if (gates != nullptr) {
        const T g = from_f32<T>(expf(s));
        gsum += to_f32<T>(g);
        if (!norm) gates[t * k + r] = g;
      }
    }
    if (gates != nullptr && norm) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) gsum += __shfl_xor_sync(kFull, gsum, d);
      const float denom = round_to<T>(gsum);
      for (int r = lane; r < k; r += 32) {
        const float g = round_to<T>(expf(key_val(win[r])));
        gates[t * k + r] = from_f32<T>(g / denom);
      }
    }
    __syncwarp();
  }
  // one waiting CTA keeps the grid from ending; more would keep later CTAs from starting
  if ((flags & kTopkLateWait) && blockIdx.x == gridDim.x - 1) pdl_wait();
}

RouterRegLayout make_reg_layout(int nk, int k) {
  RouterRegLayout L{};
  L.nkp = next_pow2(nk) < 32 ? 32 : next_pow2(nk);
  L.kp = next_pow2(k);
  L.kq = k < nk ? k : nk;
  int C = 0;
  for (int p = 0; p < L.kq; ++p) C += (k / (p + 1) < L.kq) ? k / (p + 1) : L.kq;
  L.C = C;
  L.Cp = (C + 3) / 4 * 4;
  L.cta_bytes = static_cast<int>(align_up(static_cast<size_t>(L.Cp) * 4 + static_cast<size_t>(L.kq) * 4, 16));
  int off = 2 * L.nkp * 4;
  L.off_sorted = off;
  off += 2 * L.nkp * 4;
  L.off_ids = off;
  off += 2 * L.nkp * 2;
  off = static_cast<int>(align_up(off, 16));
  L.off_win = off;
  off += (L.kp < 32 ? 32 : L.kp) * 8;
  L.off_cs = off;
  off += L.Cp * 4;
  L.off_tl = off;
  off += (kTieCap + 4) * 4;
  L.warp_bytes = static_cast<int>(align_up(off, 16));
  return L;
}

// ------------------------------------------------------------------------------------------
// 16-bit inputs, num_keys <= 1024, top_k <= 128: only the sums that can be among the k largest are ever formed.
//
//   1. The 32 lane maxima of each half, sorted (both halves in one packed 16-bit network), give a lower bound on the k-th
//      largest sum: first the best rectangle (p maxima of one half and ceil(k / p) of the other make at least k sums of at
//      least A_p + B_ceil(k/p)), then, by bisection, the largest value that k of the 32 x 32 sums reach.
//   2. A key whose sum with the other half's maximum stays below the bound is dropped (a superset is kept where rounding
//      or a non-finite value blurs the test).  What is left - 25 of 128 keys at top-64, 56 of 512 at top-128 for normal
//      logits; 41 and 105 with the rectangle alone - is compacted and sorted.
//      Where that still keeps most keys, raise_level bounds the sums again.
//   3. Each row of the first half counts its sums at or above the bound by a binary search (they do not increase along a
//      row).  Where there are at most 2 k in all - raising the bound by bisection if there are more - they are the only
//      candidates: numbered through a running maximum over marks at the rows' first numbers, formed, and sorted as 32-bit keys
//      (level of the score above the bound | inverted flat id), which puts ties in the order of their ids as well.
//      Levels too far apart for that are sorted as 64-bit keys.
//   4. Otherwise (long runs of equal sums, non-finite values) the level of the k-th sum is found exactly, the sums above it are
//      taken, and the ties with the lowest flat ids fill the rest.
//
// Bound by one token's chain of dependent instructions and by instruction issue (with all keys kept, a threshold search over the
// staircase (p + 1)(q + 1) <= k and a separate treatment of ties a token of 512 keys, top-128 took 7100 instructions).  us, that
// form -> this one: 16384 x 512 keys top-128 217 -> 104, 131072 x 256 top-32 359 -> 262, 16384 x 128 top-64 53.5 -> 39.2,
// 4096 x 128 top-64 18.7 -> 12.6, 8192 x 1024 top-64 102 -> 78, one token 7.5 -> 6.0; logits 100 times smaller, whose sums tie in
// long runs, 2000 x 512 top-128 606 -> 60.  Measured and not kept: both halves sorted (16384 x 512 top-128 152, 122 with the second
// alone), four CTAs per SM for 512 keys instead of six (122, 107), rows counted 32 at a time (108, 104 with 64).
// ------------------------------------------------------------------------------------------
struct RouterPrunedLayout {
  int warp_bytes;
  int off_ids, off_win, off_runs;
  int nkp;
};

constexpr int kPrunedMaxK = 128;  // at most 256 candidates, eight per lane

// Sorts the n <= 32 R keys of `list` (shared memory) into values and ids in rank order (the values may lie over the list).
template <typename T, int R, bool UNROLLED>
__device__ __noinline__ void sort_list(const uint32_t* list, int n, float* sv, uint16_t* si, int lane) {
  using HK = HalfKey<T>;
  uint32_t a[R];
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = lane * R + r < n ? list[lane * R + r] : 0u;
  sort_desc<R, UNROLLED>(a, lane);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane * R + r;
    if (i < n) {
      sv[i] = HK::value(a[r]);
      si[i] = static_cast<uint16_t>(HK::id(a[r]));
    }
  }
  __syncwarp();
}

// Sort of the 32 lanes, descending, of both 16-bit halves of v at once
__device__ __forceinline__ uint32_t sort_lanes_packed(uint32_t v, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int step = size >> 1; step > 0; step >>= 1) {
      const uint32_t other = __shfl_xor_sync(kFull, v, step);
      const bool desc = size == 32 || (lane & size) == 0;
      v = (((lane & step) == 0) == desc) ? __vmaxu2(v, other) : __vminu2(v, other);
    }
  return v;
}

// Order level of a sum in the type of the input: larger sum <=> larger level, -0 as +0
template <typename T>
__device__ __forceinline__ uint32_t sum_level(float s) {
  return HalfKey<T>::make(round_to<T>(s) + 0.0f, 0) >> 16;
}

// The lowest key of each half that can be in a sum of order level `level` or above (ta, tb: the halves' largest values); left as
// it is where there is no such bound.
template <typename T>
__device__ __forceinline__ void lowest_keys(uint32_t level, float ta, float tb, uint32_t& thr0, uint32_t& thr1) {
  using HK = HalfKey<T>;
  const float bound = HK::value(level << 16);
  // round(a + b) >= bound needs a + b >= bound less one step of T there; the threshold's key is rounded to T too
  constexpr float kStep = OrdLowBits<T>::value == 16 ? 0.0078125f : 0.0009765625f;
  const float low = bound - (fabsf(bound) * kStep + 1e-7f);
  const float xa = low - tb, xb = low - ta, blur = (fabsf(bound) + fabsf(ta) + fabsf(tb)) * 1e-6f + 1e-7f;
  const float ya = xa - (fabsf(xa) * kStep + blur), yb = xb - (fabsf(xb) * kStep + blur);
  if (ya > -INFINITY && yb > -INFINITY) {
    thr0 = max(HK::make(round_to<T>(ya), 0) & 0xFFFF0000u, 1u);
    thr1 = max(HK::make(round_to<T>(yb), 0) & 0xFFFF0000u, 1u);
  }
}

// Keeps the keys of `list` from `th` on, in their order; returns how many they are.
__device__ __forceinline__ int keep_from(uint32_t* list, int n, uint32_t th, int lane) {
  int kept = 0;
#pragma unroll 2
  for (int base = 0; base < n; base += 32) {  // in place: a key never moves up
    const uint32_t kv = base + lane < n ? list[base + lane] : 0u;
    const unsigned bal = __ballot_sync(kFull, kv >= th);
    if (kv >= th) list[kept + __popc(bal & ((1u << lane) - 1u))] = kv;
    kept += __popc(bal);
    __syncwarp();
  }
  return kept;
}

// Where a key holds nearly all of the probability of its half, the k largest sums are those of its row and of the column of the
// other half's largest key.  The lane maxima show 32 sums of each, and their bound then keeps most keys of both halves.  Here
// row and column are counted whole: the level goes up (by bisection) to one that k of their sums reach, the keys below it go.
// Returns the level and the number of keys kept of each half (16 bits each).
// us, the kernel of before, which dropped fewer keys -> this one without this step -> with it, tokens with 0.99 of the probability
// in one key of each half: 2000 x 512 keys top-128 43 -> 61 -> 29, 2000 x 1024 top-64 60 -> 119 -> 37, 65536 x 256 top-64 393 ->
// 463 -> 277; ordinary tokens as before (16384 x 512 top-128 106.5) or up to 2 % slower alone (65536 x 256 top-64 182, 186).
template <typename T>
__device__ __noinline__ uint2 raise_level(uint32_t* rows, uint32_t* cols, int na, int nb, int k, uint32_t level, int lane) {
  using HK = HalfKey<T>;
  float top[2], second[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t* list = h == 0 ? rows : cols;
    uint32_t first = 0, next = 0;
    for (int i = lane; i < (h == 0 ? na : nb); i += 32) {
      const uint32_t kv = list[i];
      next = max(next, min(first, kv));
      first = max(first, kv);
    }
    const uint32_t best = __reduce_max_sync(kFull, first);
    next = __reduce_max_sync(kFull, first == best ? next : first);
    top[h] = HK::value(best);
    second[h] = next != 0 ? HK::value(next) : top[h];
  }
  const float from = HK::value(level << 16);
  float lo = from, hi = fmaxf(__fadd_rn(top[0], second[1]), __fadd_rn(second[0], top[1]));
#pragma unroll 1
  for (int step = 0; step < 6; ++step) {
    const float mid = 0.5f * lo + 0.5f * hi;
    if (!(mid > from && mid < hi)) break;
    int n = 0;  // the sum of the two largest keys is counted in the row and in the column
#pragma unroll 4
    for (int i = lane; i < na; i += 32) n += __fadd_rn(HK::value(rows[i]), top[1]) >= mid ? 1 : 0;
#pragma unroll 4
    for (int i = lane; i < nb; i += 32) n += __fadd_rn(top[0], HK::value(cols[i])) >= mid ? 1 : 0;
    if (static_cast<int>(__reduce_add_sync(kFull, n)) > k) lo = mid;
    else hi = mid;
  }
  if (lo > from) {
    level = sum_level<T>(lo);
    uint32_t thr0 = 1, thr1 = 1;
    lowest_keys<T>(level, top[0], top[1], thr0, thr1);
    na = keep_from(rows, na, thr0, lane);
    nb = keep_from(cols, nb, thr1, lane);
  }
  return make_uint2(level, na | nb << 16);
}

// Step 4 of the kernel below, for the rare rows: exactly k winners as 64-bit keys (level, inverted flat id), in order.  At least k
// sums reach level lo, fewer level hi.  rows: the keys kept of the first half (na, in the order of their ids); sb, ib: the second
// half sorted (nb); runs: scratch, na entries.
template <typename T>
__device__ __noinline__ void select_exactly(uint32_t* rows, const float* sb, const uint16_t* ib, int na, int nb, int nk, int k,
                                            uint32_t lo, uint32_t hi, uint16_t* runs, uint64_t* win, int lane) {
  using HK = HalfKey<T>;
  auto level = [&](int p, int q) { return sum_level<T>(__fadd_rn(HK::value(rows[p]), sb[q])); };
  const int first = 1 << (31 - __clz(nb));
  auto reach = [&](int p, uint32_t x) {  // sums of row p at or above level x
    int n = 0;
    for (int w = first; w > 0; w >>= 1)
      if (n + w <= nb && level(p, n + w - 1) >= x) n += w;
    return n;
  };
  int kept = 0;  // rows that reach lo at all (a row never moves up)
  for (int base = 0; base < na; base += 32) {
    const int p = base + lane;
    const uint32_t row = p < na ? rows[p] : 0u;
    const bool keep = p < na && (lo == 0 || level(p, 0) >= lo);
    const unsigned bal = __ballot_sync(kFull, keep);
    if (keep) rows[kept + __popc(bal & ((1u << lane) - 1u))] = row;
    kept += __popc(bal);
    __syncwarp();
  }
  na = kept;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    int n = 0;
    for (int p = lane; p < na; p += 32) n += reach(p, mid);
    if (static_cast<int>(__reduce_add_sync(kFull, n)) >= k) lo = mid;
    else hi = mid;
  }
  // everything above (fewer than k <= 128); the runs of ties: (first column rank << 8) | columns, counted up to 255: a row that is
  // taken whole has fewer than k
  auto row_id = [&](int p) { return HK::id(rows[p]); };
  auto flat_id = [&](int p, int q) { return row_id(p) * static_cast<uint32_t>(nk) + ib[q]; };
  int filled = 0;
  for (int base = 0; base < na; base += 32) {
    const int p = base + lane;
    int n = 0;
    if (p < na) {
      n = reach(p, hi);
      runs[p] = static_cast<uint16_t>(n << 8 | min(max(reach(p, lo) - n, 0), 255));
    }
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += up;
    }
    for (int q = 0; q < n && filled + incl - n + q < k; ++q) win[filled + incl - n + q] = make_key(level(p, q), flat_id(p, q));
    filled += __shfl_sync(kFull, incl, 31);
  }
  __syncwarp();
  // ties with the lowest flat ids: the rows whose id is below `row` whole (the largest id for which they do not suffice), then
  // the lowest column ids of that row
  const int need = k - filled;
  uint32_t row = 0;
  int whole = 0;  // ties in the rows below `row`
  for (int bit = 31 - __clz(nk); bit >= 0; --bit) {
    const uint32_t trial = row | (1u << bit);
    int n = 0;
    for (int p = lane; p < na; p += 32) n += row_id(p) < trial ? static_cast<int>(runs[p] & 0xFFu) : 0;
    n = __reduce_add_sync(kFull, n);
    if (n < need) {
      row = trial;
      whole = n;
    }
  }
  int at = filled;
  for (int base = 0; base < na; base += 32) {
    const int p = base + lane;
    const bool take = p < na && row_id(p) < row;
    const uint32_t run = take ? runs[p] : 0u;
    const int n = run & 0xFFu;
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int up = __shfl_up_sync(kFull, incl, d);
      if (lane >= d) incl += up;
    }
    for (int q = 0; q < n && at + incl - n + q < k; ++q) win[at + incl - n + q] = make_key(lo, flat_id(p, (run >> 8) + q));
    at += __shfl_sync(kFull, incl, 31);
    const unsigned here = __ballot_sync(kFull, p < na && row_id(p) == row);
    if (here != 0) {
      const int split = base + __ffs(here) - 1, from = runs[split] >> 8, cols = max(reach(split, lo) - from, 0);
      const int rest = need - whole;
      uint32_t phi = 0;  // the largest id with fewer than `rest` column ids of the run below it: those and phi are taken
      for (int bit = 31 - __clz(nk); bit >= 0; --bit) {
        const uint32_t trial = phi | (1u << bit);
        int under = 0;
        for (int q = lane; q < cols; q += 32) under += ib[from + q] < trial ? 1 : 0;
        if (static_cast<int>(__reduce_add_sync(kFull, under)) < rest) phi = trial;
      }
      int done = filled + whole;
      for (int c = 0; c < cols; c += 32) {
        const bool in = c + lane < cols && ib[from + min(c + lane, cols - 1)] <= phi;
        const unsigned bal = __ballot_sync(kFull, in);
        const int pos = done + __popc(bal & ((1u << lane) - 1u));
        if (in && pos < k) win[pos] = make_key(lo, flat_id(split, from + c + lane));
        done += __popc(bal);
      }
    }
  }
  filled = min(k, filled + whole + max(need - whole, 0));
  int kp = 1;
  while (kp < k) kp <<= 1;
  __syncwarp();
  for (int r = filled + lane; r < kp; r += 32) win[r] = 0;
  __syncwarp();
  bitonic_desc(win, nullptr, kp, lane);
}

// The numbered candidates as 64-bit keys (level, inverted flat id), sorted over the rows and values that they come from
// (32 R keys are at most the 2 nkp entries of those); the first k to `win`.  For levels too far apart for 32-bit keys.
template <typename T, int R>
__device__ __noinline__ void sort_wide(const uint32_t* rows, const float* sb, const uint16_t* ib, const uint32_t* marks, int found,
                                       int nk, int k, uint64_t* keys, uint64_t* win, int lane) {
  using HK = HalfKey<T>;
  uint64_t cand[R];
  uint32_t carry = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = 32 * r + lane;
    uint32_t m = marks[i];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) m = max(m, __shfl_up_sync(kFull, m, d));
    m = max(m, carry);
    carry = __shfl_sync(kFull, m, 31);
    cand[r] = 0;
    if (i < found) {
      const int p = m >> 16, q = i - static_cast<int>(m & 0xFFFFu);
      cand[r] = make_key(sum_level<T>(__fadd_rn(HK::value(rows[p]), sb[q])), HK::id(rows[p]) * static_cast<uint32_t>(nk) + ib[q]);
    }
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) keys[32 * r + lane] = cand[r];
  __syncwarp();
  bitonic_desc(keys, nullptr, 32 * R, lane);
  for (int r = lane; r < k; r += 32) win[r] = keys[r];
  __syncwarp();
}

// E: keys per lane and half; R: candidates per lane, 32 R >= 2 k
template <typename T, int E, int R>
__global__ void __launch_bounds__(128, E <= 8 ? 7 : E <= 16 ? 6 : 4)
router_topk_pruned_kernel(const T* logp, int64_t ntok, int nk, int k, RouterPrunedLayout L,
                          T* __restrict__ scores, int64_t* __restrict__ indices, T* __restrict__ gates, int flags) {
  using HK = HalfKey<T>;
  constexpr bool kKeysInRegs = E <= 16;  // both halves' keys stay in registers up to the compaction
  constexpr int kCap = 32 * R;
  const int norm = flags & kTopkNorm;
  const bool from_logits = (flags & kTopkFromLogits) != 0;
  const bool token_rows = (flags & (kTopkFromLogits | kTopkTokenRows)) != 0;  // [T, 2, nk] instead of [2, T, nk]
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int nwarps = blockDim.x >> 5;
  const int nkp = L.nkp;
  if (!(flags & kTopkLateWait)) pdl_wait();  // the logits come from the previous kernel (kTopkLateWait: the one before)

  unsigned char* wbase = smem + warp * L.warp_bytes;
  uint32_t* rows = reinterpret_cast<uint32_t*>(wbase);  // keys kept of the first half, in the order of their ids
  uint32_t* cols = rows + nkp;                           // of the second half ...
  float* sb = reinterpret_cast<float*>(cols);            // ... then its values in rank order
  uint16_t* ib = reinterpret_cast<uint16_t*>(wbase + L.off_ids);
  uint32_t* win32 = reinterpret_cast<uint32_t*>(wbase + L.off_win);  // marks, then the winners' 32-bit keys ...
  uint64_t* win = reinterpret_cast<uint64_t*>(wbase + L.off_win);    // ... or their 64-bit keys (rare)
  const int qrank = (k + lane) / (lane + 1);  // ceil(k / (lane + 1)): the rank that pairs with rank lane + 1 of half 0
  int idbits = 1;
  while (idbits < 31 && (1 << idbits) < nk * nk) ++idbits;
  const uint32_t idmask = (1u << idbits) - 1u;

  for (int64_t t = static_cast<int64_t>(blockIdx.x) * nwarps + warp; t < ntok;
       t += static_cast<int64_t>(gridDim.x) * nwarps) {
    if (t + static_cast<int64_t>(gridDim.x) * nwarps >= ntok) pdl_launch_dependents();  // last token of this warp
    // 1. load both halves (lane-blocked: element lane * E + r in register r), from_logits: the per-half log-softmax
    //    (flash_moe/modules/flash_moe.py:72) rounded to T like torch does; lane maxima
    const T* a_row = token_rows ? logp + t * 2 * nk : logp + t * nk;
    const T* b_row = token_rows ? a_row + nk : logp + (ntok + t) * nk;
    uint32_t key[kKeysInRegs ? 2 : 1][E];
    uint32_t v = 0;      // this lane's maximum of both halves (16-bit order keys)
    float poison = 0.f;  // NaN once a value is not finite
    auto load_half = [&](int h, uint32_t (&kk)[E]) {
      float lv[E];
      load_blocked<T, E>(h == 0 ? a_row : b_row, nk, lane, lv);
      if (from_logits) {
        float m = -INFINITY;
#pragma unroll
        for (int r = 0; r < E; ++r) m = fmaxf(m, lv[r]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, d));
        float sum = 0.f;
#pragma unroll
        for (int r = 0; r < E; ++r)
          if (lane * E + r < nk) sum += expf(lv[r] - m);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
        const float lg = logf(sum);
#pragma unroll
        for (int r = 0; r < E; ++r) lv[r] = round_to<T>((lv[r] - m) - lg);
      }
      uint32_t best = 0;
#pragma unroll
      for (int r = 0; r < E; ++r) {
        const bool in = lane * E + r < nk;
        kk[r] = in ? HK::make(lv[r] + 0.0f, lane * E + r) : 0u;  // -0 -> +0
        best = max(best, kk[r]);
        if (in) poison = fmaf(lv[r], 0.f, poison);
      }
      v |= h == 0 ? best >> 16 : best & 0xFFFF0000u;
    };
    if constexpr (kKeysInRegs) {
      load_half(0, key[0]);
      load_half(1, key[1]);
    } else {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        load_half(h, key[0]);
        store_blocked<E>(reinterpret_cast<float*>(h == 0 ? rows : cols), lane, reinterpret_cast<const float (&)[E]>(key[0]));
      }
    }
    // 2. lower bound on the k-th largest sum from the sorted lane maxima (0: absent), and the keys it leaves
    uint32_t level = 0;          // order level of the bound: at least k sums reach it
    uint32_t cmax = 0;           // level of the largest sum
    uint32_t thr0 = 1, thr1 = 1;  // keys from here on are kept (0 pads the rows)
    bool ordinary = __all_sync(kFull, poison == 0.f);  // no NaN, no +inf (-inf is but the lowest value)
    if (!ordinary) {
      constexpr uint32_t kMinusInf = OrdLowBits<T>::value == 16 ? 0x007Fu : 0x03FFu;
      bool ok = true;
#pragma unroll(kKeysInRegs ? E : 1)
      for (int r = 0; r < E; ++r) {
        const uint32_t a = kKeysInRegs ? key[0][r] : rows[lane * E + r];
        const uint32_t b = kKeysInRegs ? key[kKeysInRegs ? 1 : 0][r] : cols[lane * E + r];
        ok = ok && (a == 0 || (a >> 16) - kMinusInf < 0xFFFFu - 2 * kMinusInf);  // the level of +inf is 0xFFFF - kMinusInf
        ok = ok && (b == 0 || (b >> 16) - kMinusInf < 0xFFFFu - 2 * kMinusInf);
      }
      ordinary = __all_sync(kFull, ok);
    }
    if (ordinary) {
      v = sort_lanes_packed(v, lane);
      const uint32_t other = __shfl_sync(kFull, v, qrank <= 32 ? qrank - 1 : 0);
      const uint32_t ka = v << 16, kb = other & 0xFFFF0000u;
      uint32_t rect = 0;
      if (qrank <= 32 && ka != 0 && kb != 0) rect = f32_to_ord(__fadd_rn(HK::value(ka), HK::value(kb)));
      rect = __reduce_max_sync(kFull, rect);
      const uint32_t top = __shfl_sync(kFull, v, 0);
      const float ta = HK::value(top << 16), tb = HK::value(top);
      cmax = sum_level<T>(__fadd_rn(ta, tb));
      if (rect != 0) {
        const float a = ka != 0 ? HK::value(ka) : -INFINITY;
        const float b = (v & 0xFFFF0000u) != 0 ? HK::value(v & 0xFFFF0000u) : -INFINITY;
        float lo = ord_to_f32(rect), hi = __fadd_rn(ta, tb);
#pragma unroll 1
        for (int step = 0; step < 5; ++step) {
          const float mid = 0.5f * lo + 0.5f * hi;
          int n = 0;  // sums of this lane's maximum of the first half that reach mid (at most 31 are counted)
#pragma unroll
          for (int w = 16; w > 0; w >>= 1)
            if (__fadd_rn(a, __shfl_sync(kFull, b, n + w - 1)) >= mid) n += w;
          if (static_cast<int>(__reduce_add_sync(kFull, n)) >= k) lo = mid;
          else hi = mid;
        }
        level = sum_level<T>(lo);
        lowest_keys<T>(level, ta, tb, thr0, thr1);
      }
    }
    int na = 0, nb = 0;
    if constexpr (kKeysInRegs) {
      uint32_t cnt = 0;
#pragma unroll
      for (int r = 0; r < E; ++r) cnt += (key[0][r] >= thr0 ? 1u : 0u) + (key[1][r] >= thr1 ? 0x10000u : 0u);
      const uint32_t mine = cnt;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t up = __shfl_up_sync(kFull, cnt, d);
        if (lane >= d) cnt += up;
      }
      const uint32_t total = __shfl_sync(kFull, cnt, 31);
      na = total & 0xFFFFu;
      nb = total >> 16;
      cnt -= mine;
      uint32_t* da = rows + (cnt & 0xFFFFu);
      uint32_t* db = cols + (cnt >> 16);
#pragma unroll
      for (int r = 0; r < E; ++r) {
        if (key[0][r] >= thr0) *da++ = key[0][r];
        if (key[1][r] >= thr1) *db++ = key[1][r];
      }
      __syncwarp();
    } else {
      __syncwarp();
      na = keep_from(rows, nkp, thr0, lane);
      nb = keep_from(cols, nkp, thr1, lane);
    }
    // Far more keys than the k sums can need, and not because of ties.  An ordinary row keeps 0.8 k, one in a hundred 3 k; from
    // 3 k on ordinary tokens took 3 % longer (65536 x 256 top-64: 185 and 190 us).  Up to top-32 the bound above is close enough.
    if ((R >= 4 || E >= 16) && na + nb > max(min(6 * k, nk + nk / 2), 64) && level != 0 && cmax - level > 8) {
      const uint2 raised = raise_level<T>(rows, cols, na, nb, k, level, lane);
      level = raised.x;
      na = raised.y & 0xFFFFu;
      nb = raised.y >> 16;
    }
    if (nb <= 32) sort_list<T, 1, true>(cols, nb, sb, ib, lane);
    else if (E <= 2 || nb <= 64) sort_list<T, 2, true>(cols, nb, sb, ib, lane);
    else if (E <= 4 || nb <= 128) sort_list<T, 4, false>(cols, nb, sb, ib, lane);
    else if (E <= 8 || nb <= 256) sort_list<T, 8, false>(cols, nb, sb, ib, lane);
    else if (E <= 16 || nb <= 512) sort_list<T, 16, false>(cols, nb, sb, ib, lane);
    else sort_list<T, E >= 32 ? 32 : 16, false>(cols, nb, sb, ib, lane);

    // 3. the sums that reach the bound, or a higher level if those are too many: row counts, then marks at the rows' first
    //    numbers; lo: at least k sums reach it, hi: fewer do
    uint32_t lo = level, hi = cmax + 1, step = OrdLowBits<T>::value == 16 ? 1 : 8;
    int found = 0;
    bool listed = false;  // the candidates are found and marked
#pragma unroll 1
    for (level = level != 0 ? level : (lo + hi) >> 1; ordinary; level = max(lo + 1, min(lo + step, (lo + hi) >> 1))) {
      // a sum rounds to the level or above from `edge` on: half way from the level below, or the next float if that rounds down
      const float value = HK::value(level << 16), under = HK::value((level == 0x8000u ? 0x7FFEu : level - 1) << 16);  // 0x7FFF: -0
      if (!(fabsf(value) < INFINITY && fabsf(under) < INFINITY)) break;
      float edge = 0.5f * value + 0.5f * under;
      if (sum_level<T>(edge) < level) edge = ord_to_f32(f32_to_ord(edge) + 1u);
#pragma unroll
      for (int r = 0; r < R; ++r) win32[32 * r + lane] = 0;
      __syncwarp();
      found = 0;
      const int first = 1 << (31 - __clz(nb));
      auto mark = [&](int p, int n, int start) {
        if (n > 0 && start < kCap) win32[start] = (static_cast<uint32_t>(p) << 16) | static_cast<uint32_t>(start);
      };
      auto up_to = [&](uint32_t v_) {  // inclusive sum over the lanes
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t up = __shfl_up_sync(kFull, v_, d);
          if (lane >= d) v_ += up;
        }
        return v_;
      };
      if (E <= 16 && na <= 32) {
        const float a = lane < na ? HK::value(rows[lane]) : -INFINITY;
        int n = 0;  // sums of the row that reach the edge
        for (int w = first; w > 0; w >>= 1)
          if (n + w <= nb && __fadd_rn(a, sb[n + w - 1]) >= edge) n += w;
        const int incl = up_to(n);
        found = __shfl_sync(kFull, incl, 31);
        mark(lane, n, incl - n);
      } else {
#pragma unroll 1
        for (int base = 0; base < na && found <= kCap; base += 64) {  // two rows per lane, both searches at once
          const int p = base + lane;
          const float a0 = p < na ? HK::value(rows[p]) : -INFINITY, a1 = p + 32 < na ? HK::value(rows[p + 32]) : -INFINITY;
          int n0 = 0, n1 = 0;
          for (int w = first; w > 0; w >>= 1) {
            if (n0 + w <= nb && __fadd_rn(a0, sb[n0 + w - 1]) >= edge) n0 += w;
            if (n1 + w <= nb && __fadd_rn(a1, sb[n1 + w - 1]) >= edge) n1 += w;
          }
          const uint32_t both = static_cast<uint32_t>(n0) | static_cast<uint32_t>(n1) << 16, incl = up_to(both);
          const uint32_t total = __shfl_sync(kFull, incl, 31);
          const int all0 = total & 0xFFFFu, before0 = (incl - both) & 0xFFFFu, before1 = (incl - both) >> 16;
          mark(p, n0, found + before0);
          mark(p + 32, n1, found + all0 + before1);
          found += all0 + static_cast<int>(total >> 16);
        }
      }
      __syncwarp();
      if (found >= k && found <= kCap) {
        listed = true;
        break;
      }
      if (found < k) {
        hi = level;
      } else {
        lo = level;
        step *= 2;
      }
      if (hi - lo <= 1) break;
    }
    const bool few = listed && cmax - level < (1u << (32 - idbits)) - 1u;  // they fit 32-bit keys
    if (few) {
      uint32_t cand[R];
      uint32_t carry = 0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int i = 32 * r + lane;
        uint32_t m = win32[i];  // (row << 16) | number of the row's first candidate
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) m = max(m, __shfl_up_sync(kFull, m, d));
        m = max(m, carry);
        carry = __shfl_sync(kFull, m, 31);
        cand[r] = 0;
        if (i < found) {
          const int p = m >> 16, q = i - static_cast<int>(m & 0xFFFFu);
          const uint32_t row = rows[p], flat = HK::id(row) * static_cast<uint32_t>(nk) + ib[q];
          cand[r] = ((sum_level<T>(__fadd_rn(HK::value(row), sb[q])) - level + 1u) << idbits) | (idmask - flat);
        }
      }
      sort_desc<R, (R <= 4)>(cand, lane);
      __syncwarp();  // the marks have been read
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (lane * R + r < k) win32[lane * R + r] = cand[r];
      __syncwarp();
    } else if (listed) {
      sort_wide<T, R>(rows, sb, ib, win32, found, nk, k, reinterpret_cast<uint64_t*>(wbase), win, lane);
    } else {
      select_exactly<T>(rows, sb, ib, na, nb, nk, k, lo, ordinary ? hi : 0x10000u, reinterpret_cast<uint16_t*>(wbase + L.off_runs),
                        win, lane);
    }

    // 4. write out
    float gsum = 0.f;
    for (int r = lane; r < k; r += 32) {
      uint32_t lv, id;
      if (few) {
        const uint32_t w = win32[r];
        lv = (w >> idbits) - 1u + level;
        id = idmask - (w & idmask);
      } else {
        const uint64_t ky = win[r];
        lv = static_cast<uint32_t>(ky >> 32);
        id = key_id(ky);
      }
      const float s = HK::value(lv << 16);
      scores[t * k + r] = from_f32<T>(s);
      indices[t * k + r] = static_cast<int64_t>(id);
      if (gates != nullptr) {
        const T g = from_f32<T>(expf(s));
        gsum += to_f32<T>(g);
        if (!norm) gates[t * k + r] = g;
      }
    }
    if (gates != nullptr && norm) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) gsum += __shfl_xor_sync(kFull, gsum, d);
      const float denom = round_to<T>(gsum);
      for (int r = lane; r < k; r += 32) {  // this lane's own scores, written above
        const float g = round_to<T>(expf(to_f32<T>(scores[t * k + r])));
        gates[t * k + r] = from_f32<T>(g / denom);
      }
    }
    __syncwarp();
  }
  // one waiting CTA keeps the grid from ending; more would keep later CTAs from starting
  if ((flags & kTopkLateWait) && blockIdx.x == gridDim.x - 1) pdl_wait();
}

template <typename T, int E, int R>
int launch_pruned_candidates(const void* logp, int64_t T_, int nk, int k, void* scores, int64_t* indices, void* gates, int norm,
                             cudaStream_t stream) {
  RouterPrunedLayout L{};
  L.nkp = next_pow2(nk) < 32 ? 32 : next_pow2(nk);
  if (32 * R > L.nkp) return FMOE_ERR_UNSUPPORTED;  // sort_wide lays 32 R 64-bit keys over the two lists (launch_typed)
  L.off_ids = 2 * L.nkp * 4;
  L.off_win = L.off_ids + L.nkp * 2;
  L.off_runs = L.off_win + 32 * R * 4;
  L.warp_bytes = L.off_runs + L.nkp * 2;  // 1024 keys: four CTAs per SM as the registers allow, top-16 of 2000 tokens 35 -> 27 us
  static_assert(E < 32 || 4 * (E * 32 * (4 + 4 + 2 + 2) + 32 * R * 4) + 1024 <= 228 * 1024 / 4, "four CTAs per SM");
  const int warps = 4;
  const int smem = warps * L.warp_bytes;
  auto kern = router_topk_pruned_kernel<T, E, R>;
  FMOE_CUDA_TRY(allow_smem(kern, smem));
  if (norm & kTopkLateWait) FMOE_CUDA_TRY(prefer_smem(kern));
  int per_sm = 1;
  FMOE_CUDA_TRY(resident_ctas(kern, warps * 32, smem, &per_sm));
  if (per_sm < 1) per_sm = 1;
  const int64_t want = (T_ + warps - 1) / warps;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * per_sm;
  const int grid = static_cast<int>(want < cap ? want : cap);
  FMOE_CUDA_TRY(launch_pdl(2, kern, dim3(grid), dim3(warps * 32), smem, stream, 1, static_cast<const T*>(logp), T_, nk, k, L,
                           static_cast<T*>(scores), indices, static_cast<T*>(gates), norm));
  return FMOE_OK;
}

template <typename T, int E>
int launch_pruned(const void* logp, int64_t T_, int nk, int k, void* scores, int64_t* indices, void* gates, int norm,
                  cudaStream_t stream) {
  if (k <= 16) return launch_pruned_candidates<T, E, 1>(logp, T_, nk, k, scores, indices, gates, norm, stream);
  if (k <= 32) return launch_pruned_candidates<T, E, 2>(logp, T_, nk, k, scores, indices, gates, norm, stream);
  if (k <= 64) return launch_pruned_candidates<T, E, 4>(logp, T_, nk, k, scores, indices, gates, norm, stream);
  return launch_pruned_candidates<T, E, 8>(logp, T_, nk, k, scores, indices, gates, norm, stream);
}

template <typename T, int E, int CPL = 0>
int launch_reg(const void* logp, int64_t T_, int nk, int k, const RouterRegLayout& L, int warps, void* scores,
               int64_t* indices, void* gates, int norm, cudaStream_t stream) {
  const int smem = L.cta_bytes + warps * L.warp_bytes;
  auto kern = router_topk_reg_kernel<T, E, CPL>;
  FMOE_CUDA_TRY(allow_smem(kern, smem));
  if (norm & kTopkLateWait) FMOE_CUDA_TRY(prefer_smem(kern));
  int per_sm = 1;
  FMOE_CUDA_TRY(resident_ctas(kern, warps * 32, smem, &per_sm));
  if (per_sm < 1) per_sm = 1;
  const int64_t want = (T_ + warps - 1) / warps;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * per_sm;
  const int grid = static_cast<int>(want < cap ? want : cap);
  FMOE_CUDA_TRY(launch_pdl(2, kern, dim3(grid), dim3(warps * 32), smem, stream, 1, static_cast<const T*>(logp), T_, nk, k, L,
                           static_cast<T*>(scores), indices, static_cast<T*>(gates), norm));
  return FMOE_OK;
}

// register kernel when the halves fit 32 keys per lane and the per-warp scratch stays small
template <typename T>
int launch_typed(const void* logp, int64_t T_, int nk, int k, void* scores, int64_t* indices, void* gates, int norm,
                 cudaStream_t stream);

RouterSmemLayout make_layout(int nk, int k) {
  RouterSmemLayout L{};
  L.nkp = next_pow2(nk);
  L.kp = next_pow2(k);
  L.kq = k < nk ? k : nk;
  int C = 0;
  for (int p = 0; p < L.kq; ++p) C += (k / (p + 1) < L.kq) ? k / (p + 1) : L.kq;
  L.C = C;
  L.Cp = (C + 3) / 4 * 4;
  L.cta_bytes = static_cast<int>(align_up(static_cast<size_t>(L.Cp) * 4 + static_cast<size_t>(L.kq) * 4, 16));
  int off = 2 * nk * 4;
  off = static_cast<int>(align_up(off, 16));
  L.off_keys = off;
  off += 2 * L.nkp * 8;
  L.off_win = off;
  off += L.kp * 8;
  L.off_cs = off;
  off += L.Cp * 4;
  L.off_cnt = off;
  off += nk * 4;
  L.warp_bytes = static_cast<int>(align_up(off, 16));
  return L;
}

template <typename T>
int launch_smem(const void* logp, int64_t T_, int nk, int k, void* scores, int64_t* indices, void* gates, int norm,
                 cudaStream_t stream) {
  const RouterSmemLayout L = make_layout(nk, k);
  constexpr int kMaxSmem = 227 * 1024;
  int warps = 8;
  while (warps > 1 && L.cta_bytes + warps * L.warp_bytes > kMaxSmem / 2) warps >>= 1;  // keep >= 2 CTAs/SM if possible
  if (L.cta_bytes + warps * L.warp_bytes > kMaxSmem) return FMOE_ERR_UNSUPPORTED;
  const int smem = L.cta_bytes + warps * L.warp_bytes;
  auto kern = router_topk_smem_kernel<T>;
  FMOE_CUDA_TRY(allow_smem(kern, smem));
  int per_sm = 1;
  FMOE_CUDA_TRY(resident_ctas(kern, warps * 32, smem, &per_sm));
  if (per_sm < 1) per_sm = 1;
  const int64_t want = (T_ + warps - 1) / warps;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * per_sm;
  const int grid = static_cast<int>(want < cap ? want : cap);
  kern<<<grid, warps * 32, smem, stream>>>(static_cast<const T*>(logp), T_, nk, k, L, static_cast<T*>(scores), indices,
                                           static_cast<T*>(gates), norm);
  FMOE_LAUNCH_CHECK();
  return FMOE_OK;
}


template <typename T>
int launch_typed(const void* logp, int64_t T_, int nk, int k, void* scores, int64_t* indices, void* gates, int norm,
                 cudaStream_t stream) {
  if constexpr (sizeof(T) == 2) {
    // Not for one key per lane, nor where more than half of a short row is wanted: there the two halves' lists do not hold the
    // 64-bit keys of all candidates (sort_wide).  With lists of 32 R entries the pruned kernel is the faster one there too (us,
    // whole rows and pruned: 20000 x 32 top-4 33 and 33, top-16 37 and 33, 16384 x 64 top-48 51 and 39, 16384 x 100 top-70 74
    // and 61, 4096 x 128 top-128 33 and 25), which no call takes yet.
    const bool prune = nk > 32 && (nk > 128 || 2 * k <= nk);
    if (nk <= 1024 && k <= kPrunedMaxK && prune) {
      switch ((next_pow2(nk) < 32 ? 32 : next_pow2(nk)) / 32) {
        case 2: return launch_pruned<T, 2>(logp, T_, nk, k, scores, indices, gates, norm, stream);
        case 4: return launch_pruned<T, 4>(logp, T_, nk, k, scores, indices, gates, norm, stream);
        case 8: return launch_pruned<T, 8>(logp, T_, nk, k, scores, indices, gates, norm, stream);
        case 16: return launch_pruned<T, 16>(logp, T_, nk, k, scores, indices, gates, norm, stream);
        default: return launch_pruned<T, 32>(logp, T_, nk, k, scores, indices, gates, norm, stream);
      }
    }
  }
  // float32, and the 16-bit shapes the pruned kernel leaves
  if (nk <= 1024) {
    const RouterRegLayout L = make_reg_layout(nk, k);
    // few tokens per SM: small CTAs spread them over more SMs
    int warps = 4;
    while (warps > 1 && L.cta_bytes + warps * L.warp_bytes > 96 * 1024) warps >>= 1;
    if (L.cta_bytes + warps * L.warp_bytes <= 200 * 1024) {
      switch (L.nkp / 32) {
        case 1: return launch_reg<T, 1>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        case 2: return launch_reg<T, 2>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        case 4:
          if constexpr (sizeof(T) == 2)  // 16384 x 100 keys top-70: 72.6 us with the candidates in shared memory, 68.8 in registers
            if (L.C > 128 && L.C <= 320)
              return launch_reg<T, 4, 10>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
          return launch_reg<T, 4>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        case 8: return launch_reg<T, 8>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        case 16: return launch_reg<T, 16>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        case 32: return launch_reg<T, 32>(logp, T_, nk, k, L, warps, scores, indices, gates, norm, stream);
        default: break;
      }
    }
  }
  if (norm & kTopkFromLogits) return FMOE_ERR_UNSUPPORTED;  // raw logits are only accepted by the register kernel
  return launch_smem<T>(logp, T_, nk, k, scores, indices, gates, norm, stream);
}

}  // namespace

int launch_router_topk(const void* log_probs, int dtype, int64_t T, int nk, int k, void* scores, int64_t* indices,
                       void* gates, int norm, cudaStream_t stream) {
  if (T < 0 || nk <= 0 || k < 0 || k > nk) return FMOE_ERR_BAD_ARG;
  if (nk > 32768) return FMOE_ERR_UNSUPPORTED;  // flat ids and the (p, q) table are 32/16-bit
  if (T == 0 || k == 0) return FMOE_OK;
  if (log_probs == nullptr || scores == nullptr || indices == nullptr) return FMOE_ERR_BAD_ARG;
  switch (dtype) {
    case FMOE_DTYPE_F32: return launch_typed<float>(log_probs, T, nk, k, scores, indices, gates, norm, stream);
    case FMOE_DTYPE_BF16: return launch_typed<__nv_bfloat16>(log_probs, T, nk, k, scores, indices, gates, norm, stream);
    case FMOE_DTYPE_F16: return launch_typed<__half>(log_probs, T, nk, k, scores, indices, gates, norm, stream);
    default: return FMOE_ERR_BAD_ARG;
  }
}

}  // namespace fmoe
