// barrier.h -- the arithmetic of the grid barrier's arrival count (roundloop.cu),
// in a header of its own that a host compiler takes too.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define PCC_HOST_DEVICE __host__ __device__
#else
#define PCC_HOST_DEVICE
#endif

namespace pcc {

// Arrivals are counted in 32 bits and never reset, 2 to 7 barriers a round of up
// to 304 CTAs each, so a run of millions of rounds passes 2^32.  The count
// starts a little below it: every run of some barriers passes it.
constexpr uint32_t kBarrierStart = 0u - 512u;

// Whether `count` arrivals include the `target`-th, modulo 2^32.  The two are
// never further apart than the CTAs of the grid: a CTA arrives once at each
// barrier, and at the next one only after all others have arrived.
PCC_HOST_DEVICE inline bool BarrierReached(uint32_t count, uint32_t target) {
  return static_cast<int32_t>(count - target) >= 0;
}

}  // namespace pcc
