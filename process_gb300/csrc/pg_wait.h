// Counting arrivals at a wait.
#pragma once
#include <cstdint>
#if !defined(__CUDACC__) && !defined(__host__)
#define __host__
#define __device__
#endif

namespace pg {

// Whether a count that goes up by one per arrival has reached target.  Both
// wrap at 2^32 (a loop of many steps counts on), so they are compared by their
// difference, which stays far below 2^31.
__host__ __device__ inline bool arrived(uint32_t count, uint32_t target) { return int32_t(count - target) >= 0; }

}  // namespace pg
