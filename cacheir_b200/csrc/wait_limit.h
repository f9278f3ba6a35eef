// How long a bounded wait goes on. Plain C++: the kernels and a host program that moves the clock by hand share it.
//
// A wait looks at its barrier again and again. For kWaitNs it goes by the clock. But that runs also while the program does not (another process has
// the GPU, the machine is suspended), so that a wait that the clock has ended goes on by its looks: the time between two of them counts only up to what a look can
// take, and after a pause there is still time to see what has arrived meanwhile.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define CB200_BOTH __host__ __device__
#else
#define CB200_BOTH
#endif

namespace cb200 {

constexpr uint32_t kWaitNs = 500u * 1000u * 1000u;         // by the clock, and as long again by looks: then a wait gives up and says so
constexpr uint32_t kSuspendNs = 20u * 1000u;               // for how long a look may suspend its thread
constexpr uint32_t kLookNs = 5 * kSuspendNs;

// look(): has the phase ended? clock(): nanoseconds, of which 32 bits are enough
template <typename Look, typename Clock>
CB200_BOTH inline bool wait_by_looks(Look look, Clock clock) {
  uint32_t seen = clock(), waited = 0;
  while (!look()) {
    const uint32_t now = clock(), gap = now - seen;
    waited += (gap < kLookNs ? gap : kLookNs) + 1;         // (at least 1: the wait ends on any clock)
    seen = now;
    if (waited > kWaitNs) return false;
  }
  return true;
}

}  // namespace cb200
