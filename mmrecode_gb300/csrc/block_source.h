// Where the samples of an encoder's block come from (read_block, encoder.rs:392-402).
#pragma once

#include <stddef.h>
#include <stdint.h>

#include "common.h"

namespace mmr {

struct BlockSource {
    const uint8_t *plane;
    size_t stride;
    uint32_t x0, y0, pw, ph, tq;
};

// Row r of the block's samples as the bytes of a Pair {x, y} of words, sample 0 lowest: rows
// and columns past the plane repeat its last. load8 reads a Pair at an aligned address, load1
// a byte. Nothing outside the plane's storage is read, `stride` bytes a row, although
// unaligned samples come from the two aligned words that hold them: of those only a row's
// first and last may reach past the storage, and they are read by byte.
template <class Pair, class Load8, class Load1>
MMR_HD Pair plane_row(const BlockSource &B, uint32_t r, Load8 load8, Load1 load1) {
    const uint32_t y = B.y0 + r < B.ph - 1 ? B.y0 + r : B.ph - 1;
    const uint8_t *row = B.plane + (size_t)y * B.stride;
    const uintptr_t a = reinterpret_cast<uintptr_t>(row + B.x0);
    const uint32_t sh = (uint32_t)(a & 7) * 8;
    // (x0 - 1 < stride - 16: neither the row's first eight bytes nor among its last fifteen. Testing
    // the addresses against the storage cost 1.5 to 5 % of an encode)
    if (B.x0 + 8 <= B.pw && (sh == 0 || B.x0 - 1 < (uint32_t)B.stride - 16)) {
        const Pair *q = reinterpret_cast<const Pair *>(a & ~(uintptr_t)7);
        const Pair v = load8(q);
        if (sh == 0) return v;
        const Pair n = load8(q + 1);
        const unsigned long long s = ((unsigned long long)v.y << 32 | v.x) >> sh | ((unsigned long long)n.y << 32 | n.x) << (64 - sh);
        return Pair{(uint32_t)s, (uint32_t)(s >> 32)};
    }
    Pair w{0, 0};
#if defined(__CUDA_ARCH__)
#pragma unroll
#endif
    for (uint32_t x = 0; x < 4; x++) {
        const uint32_t lo = B.x0 + x, hi = lo + 4, last = B.pw - 1;
        w.x |= (uint32_t)load1(row + (lo < last ? lo : last)) << (8 * x);
        w.y |= (uint32_t)load1(row + (hi < last ? hi : last)) << (8 * x);
    }
    return w;
}

}  // namespace mmr
