// Sorting networks of one warp, keys in registers.
#pragma once
#include <cstdint>

namespace fmoe {

__device__ __forceinline__ uint32_t shfl_xor_key(uint32_t v, int m) { return __shfl_xor_sync(0xFFFFFFFFu, v, m); }
__device__ __forceinline__ uint64_t shfl_xor_key(uint64_t v, int m) {
  return static_cast<uint64_t>(__shfl_xor_sync(0xFFFFFFFFu, static_cast<unsigned long long>(v), m));
}

// Descending bitonic sort of 32*E keys in the lane-blocked layout: element i = lane * E + r sits in a[r].  Strides
// below E exchange two registers of one lane (no shuffle: 15 shuffle stages for any E >= 1 instead of up to 35 with
// the keys dealt round-robin over the lanes); the direction of a block folds into the comparison predicate, so an
// exchange costs one compare and two selects per pair and a shuffle stage one shuffle, one compare and one select per key.
template <int E, typename K>
__device__ __forceinline__ void bitonic_desc_regs(K (&a)[E], int lane) {
  constexpr int n = 32 * E;
#pragma unroll
  for (int size = 2; size <= n; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      if (stride >= E) {
        const int ls = stride / E;
        const bool desc = (size == n) || (((lane * E) & size) == 0);  // size >= 2 E here: decided by the lane
        const bool keep_max = ((lane & ls) == 0) == desc;
#pragma unroll
        for (int r = 0; r < E; ++r) {
          const K other = shfl_xor_key(a[r], ls);
          a[r] = ((other > a[r]) == keep_max) ? other : a[r];
        }
      } else {
#pragma unroll
        for (int r = 0; r < E; ++r) {
          if ((r & stride) == 0) {
            const bool desc = (size == n) || (size < E ? ((r & size) == 0) : (((lane * E) & size) == 0));
            const K x = a[r], y = a[r | stride];
            const bool sw = (x < y) == desc;
            a[r] = sw ? y : x;
            a[r | stride] = sw ? x : y;
          }
        }
      }
    }
  }
}

// Descending bitonic sort of 32 R keys in the lane-blocked layout (element lane * R + r in a[r]).  UNROLLED = false: as
// loops, with only the stages inside a lane unrolled - kernels whose straight-line code exceeds the instruction cache spend
// two thirds of their time fetching it (512 keys, top-128: 352 us with everything unrolled, 201 us with loops).
template <int R, bool UNROLLED>
__device__ __forceinline__ void sort_desc(uint32_t (&a)[R], int lane) {
  if constexpr (UNROLLED) {
    bitonic_desc_regs<R, uint32_t>(a, lane);
  } else {
    auto inside = [&](int from, bool desc_lane, bool by_reg, int size) {
#pragma unroll
      for (int step = R >> 1; step > 0; step >>= 1) {
        if (step > from) continue;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if ((r & step) == 0) {
            const bool desc = by_reg ? (r & size) == 0 : desc_lane;
            const uint32_t lo = min(a[r], a[r | step]), hi = max(a[r], a[r | step]);
            a[r] = desc ? hi : lo;
            a[r | step] = desc ? lo : hi;
          }
        }
      }
    };
#pragma unroll
    for (int size = 2; size < R; size <<= 1) inside(size >> 1, true, true, size);
    if (R > 1) inside(R >> 1, (lane & 1) == 0, false, 0);
#pragma unroll 1
    for (int ls2 = 2; ls2 <= 32; ls2 <<= 1) {  // blocks of ls2 lanes
      const bool desc = ls2 == 32 || (lane & ls2) == 0;
#pragma unroll 1
      for (int ls = ls2 >> 1; ls > 0; ls >>= 1) {
        const bool keep_max = ((lane & ls) == 0) == desc;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t other = __shfl_xor_sync(0xFFFFFFFFu, a[r], ls);
          a[r] = keep_max ? max(a[r], other) : min(a[r], other);
        }
      }
      if (R > 1) inside(R >> 1, desc, false, 0);
    }
  }
}

}  // namespace fmoe
