// Host-only rules of the engine, without CUDA.
#pragma once

#include <cstdint>

namespace tbr {

// Whether the bytes [p, p + bytes) all lie within [start, start + size).
inline bool range_holds(uint64_t start, uint64_t size, uint64_t p, uint64_t bytes) {
    return p >= start && bytes <= size && p - start <= size - bytes;
}

}  // namespace tbr
