// Host planes going up: those that follow one another in one piece of host memory go as one
// copy (a call per plane took a third of the encode of 12 small frames).
#pragma once

#include <stddef.h>
#include <stdint.h>

namespace mmr {

// Where a host address lies: a pinned or registered range, or (lo == nullptr) ordinary memory.
struct HostRange {
    const uint8_t *lo = nullptr, *hi = nullptr;
};

// The pending copy. One copy never spans two pinned ranges, nor pinned and ordinary memory:
// buffers that were pinned separately can be neighbours, and the runtime takes a copy for
// that of the range that it starts in. range_of(p) is asked once per copy for pinned memory
// (planes in a range known already need no question) and once per plane for ordinary memory.
struct PlaneUploads {
    const uint8_t *src = nullptr;
    uint8_t *dst = nullptr;
    size_t bytes = 0;
    HostRange range;

    template <class RangeOf>
    void start(const uint8_t *p, uint8_t *to, size_t n, RangeOf range_of) {
        src = p;
        dst = to;
        bytes = n;
        if (!range.lo || p < range.lo || p >= range.hi) range = range_of(p);
    }

    // Whether `more` bytes at p continue the pending copy.
    template <class RangeOf>
    bool append(const uint8_t *p, size_t more, RangeOf range_of) {
        if (!bytes || p != src + bytes) return false;
        if (range.lo ? p + more > range.hi : range_of(p).lo != nullptr) return false;
        bytes += more;
        return true;
    }
};

}  // namespace mmr
