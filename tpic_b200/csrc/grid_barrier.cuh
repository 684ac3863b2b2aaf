// A barrier over all CTAs of a cooperative launch, with bounded waits.
//
// Two words, zero between launches: arrivals and departures; the last CTA to
// leave zeroes both. A CTA whose poll runs out reports false to its threads,
// which leave the kernel; the other CTAs then run out at their next barrier.
#pragma once

#include "common.cuh"

namespace tpicb200 {

constexpr uint32_t kGridBarrierPolls = 1u << 22;

__device__ __forceinline__ uint32_t load_acquire(const unsigned* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

struct GridBarrier {
  unsigned* words;
  uint32_t arrivals = 0;
  bool failed = false;
  __device__ explicit GridBarrier(unsigned* w) : words(w) {}

  // Every thread of every CTA; false when it gave up (for the whole CTA).
  __device__ __forceinline__ bool wait() {
    __syncthreads();
    if (threadIdx.x == 0) {
      arrivals += gridDim.x;
      // The CTA's writes are ordered before the arrival (the barrier above and
      // the release), the others' before what follows the acquire.
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(words) : "memory");
      uint32_t poll = 0;
      while (load_acquire(words) < arrivals && poll < kGridBarrierPolls) ++poll;
      failed = poll == kGridBarrierPolls;
    }
    return !__syncthreads_or(failed);
  }
  __device__ __forceinline__ void leave() {
    if (threadIdx.x == 0 && !failed && atomicAdd(words + 1, 1u) == gridDim.x - 1) {
      words[0] = 0;
      words[1] = 0;
    }
  }
};

}  // namespace tpicb200
