// Which mbarrier phases a group of normalising warps of router_gemm_bn_kernel waits for before it touches the x tile of a
// k-block.  Plain C++ as well as CUDA, so that the rule can be run on a host.
//
// k-block kb sits in stage kb % kStages and is normalised by group kb % kGroups.  A parity wait only tells a phase from the one
// after it: on a barrier that is still two phases behind it returns at once.  Where kStages is a multiple of kGroups a stage
// always belongs to one group, which has seen every earlier phase of its `full` barrier itself.  Otherwise the phase before is
// another group's k-block, kb - kStages, and copies may land out of order: the tile of kb - kGroups, then that of kb - kStages.
// The group therefore first waits for the stage's `empty` phase, that the MMAs of kb - kStages have ended; the copy of
// k-block kb, which `full` stands for, is only requested behind that phase, so nothing is waited for twice.  That wait is never
// two phases early: the producer saw the phase before it when it requested kb - kStages, ahead of the k-block kb - kGroups
// whose tile this group has had.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define FMOE_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define FMOE_HOST_DEVICE inline
#endif

namespace fmoe {

template <int kStages, int kGroups>
struct NormaliseWaits {
  static_assert(kStages >= kGroups, "a group's k-block before this one is requested behind the stage's last use");
  static constexpr bool kOwnStages = kStages % kGroups == 0;
  // whether k-block kb is behind a phase of `empty`, and that phase's parity
  static FMOE_HOST_DEVICE bool behind_empty(int kb) { return !kOwnStages && kb >= kStages; }
  static FMOE_HOST_DEVICE uint32_t empty_parity(int kb) { return static_cast<uint32_t>(kb / kStages - 1) & 1u; }
  static FMOE_HOST_DEVICE uint32_t full_parity(int kb) { return static_cast<uint32_t>(kb / kStages) & 1u; }
};

}  // namespace fmoe
