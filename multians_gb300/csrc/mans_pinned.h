// Whether a buffer lies inside one range of memory.
#pragma once

#include <cstdint>

namespace mans {

// [p, p + bytes) inside [start, start + size); a range of no size holds
// nothing, and neither sum wraps.
inline bool range_covers(uint64_t start, uint64_t size, uint64_t p, uint64_t bytes) {
    return size != 0 && p >= start && bytes <= size && p - start <= size - bytes;
}

}  // namespace mans
