// Host-only harness: the reads an encoder's block makes of its plane
// (mmrecode_gb300/csrc/block_source.h).
#include <stddef.h>
#include <stdint.h>

#include "block_source.h"

// Row r of the block at (x0, y0) of a plane; *outside: bytes read outside its storage.
extern "C" uint64_t mmr_test_source_row(const uint8_t *plane, size_t stride, uint32_t pw, uint32_t ph, uint32_t x0,
                                        uint32_t y0, uint32_t r, uint32_t *outside) {
    const uint8_t *end = plane + stride * ph;
    uint32_t bad = 0;
    auto byte = [&](const uint8_t *p) -> uint8_t {
        if (p < plane || p >= end) {
            bad++;
            return 0x5a;
        }
        return *p;
    };
    struct Pair {
        uint32_t x, y;
    };
    auto word = [&](const Pair *p) {
        const uint8_t *b = reinterpret_cast<const uint8_t *>(p);
        Pair v{0, 0};
        for (int i = 0; i < 4; i++) {
            v.x |= (uint32_t)byte(b + i) << (8 * i);
            v.y |= (uint32_t)byte(b + 4 + i) << (8 * i);
        }
        return v;
    };
    const mmr::BlockSource B{plane, stride, x0, y0, pw, ph, 0};
    const Pair v = mmr::plane_row<Pair>(B, r, word, byte);
    *outside = bad;
    return (uint64_t)v.y << 32 | v.x;
}
