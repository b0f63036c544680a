// Counting arrivals modulo 2^32 (plain C++: also compiled by the host compiler for its test).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define PM_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define PM_HOST_DEVICE inline
#endif

namespace pacmap {

// The counter of a launch starts here, one arrival before it wraps, so that every launch takes it over the end.
constexpr uint32_t ARRIVALS_START = 0xFFFFFFFFu;

// What the counter must reach for `blocks` blocks to have arrived `round` times each.
PM_HOST_DEVICE uint32_t arrivals_wanted(uint32_t round, uint32_t blocks) { return ARRIVALS_START + round * blocks; }

// Whether the counter has reached `wanted`. It is never more than 2 * blocks away (a block arrives for the next round
// only after the wait of this one), so the sign of the difference decides, also where either has wrapped: 592 blocks
// count to 2^32 in 7.3 million rounds.
PM_HOST_DEVICE bool arrivals_reached(uint32_t seen, uint32_t wanted) { return static_cast<int32_t>(seen - wanted) >= 0; }

}  // namespace pacmap
