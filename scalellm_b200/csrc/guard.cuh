// guard.cuh — mbarrier waits that end.  A wait that runs out marks the CTA (a word of its shared memory); every later
// wait of the CTA then returns at once, so all roles leave their loops, the CTA lets its copies in flight land
// (guard_drain), frees its tensor memory and returns.  A marked CTA writes NaN instead of results: the caller sees it.
#pragma once

#include "common.cuh"

namespace b200 {

constexpr uint32_t GUARD_TRIES = 1u << 22;   // of mbarrier.try_wait, which itself waits: seconds, where a wait takes us

__device__ __forceinline__ void guard_wait(uint64_t* bar, uint32_t parity, volatile uint32_t* dead) {
  if (mbar_try_wait(bar, parity)) return;
  for (uint32_t i = 0; i < GUARD_TRIES; ++i) {
    if (mbar_try_wait(bar, parity)) return;
    if ((i & 255u) == 255u && *dead) return;
  }
  *dead = 1u;
}
// Called by one thread at the end of a marked CTA: time for bulk copies that nobody waited for to land.
__device__ __forceinline__ void guard_drain() {
  for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

}  // namespace b200
