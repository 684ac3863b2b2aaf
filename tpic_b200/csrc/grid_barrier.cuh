// A barrier over all CTAs of a cooperative launch, with bounded waits.
//
// Two words, zero between launches: arrivals, and departures with those of
// CTAs that gave up counted in the upper half. A CTA whose polls run out reports
// false to its threads, which do no more work; the others then run out at their
// next wait. Where every CTA departs on every way out, the last one to do so zeroes
// the words, so a launch that failed spoils none after it; that CTA also learns of
// the failure and, by leave(), can put the outputs in order, all the other CTAs'
// writes being done. A kernel whose host reads of the failure may end without
// departing: the host then clears the words.
#pragma once

#include "common.cuh"

namespace tpicb200 {

constexpr uint32_t kGridBarrierPolls = 1u << 22;
constexpr int kGridBarrierWords = 2;

// The bound of a barrier's waits, and for tests the wait (from 1) at which CTA
// 0 expects more arrivals than there ever are (0: none).
struct GridWaits {
  uint32_t polls, stall;
};

__device__ __forceinline__ uint32_t load_acquire(const unsigned* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// kStall: the waits look at the stall.
template <bool kStall>
struct GridBarrier {
  static constexpr uint32_t kFailed = 1u << 16;  // above any number of CTAs resident at once
  unsigned* words;
  GridWaits waits;
  uint32_t arrivals = 0, number = 0;
  bool failed = false;
  __device__ GridBarrier(unsigned* w, GridWaits limits) : words(w), waits(limits) {}

  // Every thread of every CTA; false when it gave up (for the whole CTA).
  __device__ __forceinline__ bool wait() {
    __syncthreads();
    if (threadIdx.x == 0) {
      arrivals += gridDim.x;
      uint32_t expected = arrivals;
      if (kStall && ++number == waits.stall && blockIdx.x == 0) expected = 0xffffffffu;
      // The CTA's writes are ordered before the arrival (the barrier above and
      // the release), the others' before what follows the acquire.
      asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(words) : "memory");
      uint32_t poll = 0;
      while (load_acquire(words) < expected && poll < waits.polls) ++poll;
      failed = poll == waits.polls;
    }
    return !__syncthreads_or(failed);
  }

  enum Exit { kOther, kLast, kLastOfFailed };
  // One thread of every CTA, once, on every way out of the kernel.
  __device__ __forceinline__ Exit depart() {
    const uint32_t before = atomicAdd(words + 1, failed ? kFailed + 1 : 1u);
    if (before % kFailed != gridDim.x - 1) return kOther;
    words[0] = words[1] = 0;
    return failed || before >= kFailed ? kLastOfFailed : kLast;
  }
  // The same by every thread, all of which get the answer; what the CTAs have
  // written is then done where the last one goes on.
  __device__ __forceinline__ Exit leave() {
    __syncthreads();
    Exit exit = kOther;
    if (threadIdx.x == 0) {
      __threadfence();
      exit = depart();
      __threadfence();
    }
    const bool last = __syncthreads_or(exit != kOther), any_failed = __syncthreads_or(exit == kLastOfFailed);
    return any_failed ? kLastOfFailed : last ? kLast : kOther;
  }
};

}  // namespace tpicb200
