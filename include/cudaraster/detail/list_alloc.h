// list_alloc.h -- arithmetic of the tile lists' allocation: host and device,
// plain C++, so that it can be checked without a GPU. Totals are 64-bit: a
// viewport's 1,024 tiles with 2^21 entries each already pass 2^31, while list
// indices are 32-bit, so lists that end beyond 2^31 - 1 never fit, whatever the
// capacity.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define CR_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CR_HOST_DEVICE inline
#endif

namespace cr {

constexpr int64_t kMaxListEntries = 0x7FFFFFFF;

// Entries of four neighbouring tiles (a tile has at most one per subtriangle).
CR_HOST_DEVICE uint64_t entriesOf4(const int32_t* counts) {
    return (uint64_t)(uint32_t)counts[0] + (uint32_t)counts[1] + (uint32_t)counts[2] + (uint32_t)counts[3];
}

// Whether lists that end at entry `end` fit into memory for `capacity` entries.
CR_HOST_DEVICE bool listsFit(uint64_t end, int64_t capacity) {
    return end <= (uint64_t)(capacity < kMaxListEntries ? capacity : kMaxListEntries);
}

// A total as the 32-bit counters report it: saturated.
CR_HOST_DEVICE int32_t reportedEntries(uint64_t total) {
    return (int32_t)(total < (uint64_t)kMaxListEntries ? total : (uint64_t)kMaxListEntries);
}

// Whether the list memory has an entry `index`.
CR_HOST_DEVICE bool listHolds(int32_t index, int64_t capacity) { return (uint64_t)(uint32_t)index < (uint64_t)capacity && index >= 0; }

}  // namespace cr
