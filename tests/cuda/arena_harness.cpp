// Host-only harness for the device-memory rules (mmrecode_gb300/csrc/arena.h).
#include <stddef.h>
#include <stdint.h>

#include "arena.h"

struct TestFrame {
    uint64_t len, planar, blocks, intervals, planes, host_out;
};

static mmr::FrameNeed need_of(const TestFrame &t) {
    mmr::FrameNeed f;
    f.len = t.len;
    f.planar = t.planar;
    f.blocks = t.blocks;
    f.intervals = t.intervals;
    f.sliced = f.host_in = true;
    f.planes = t.planes != 0;
    f.host_out = t.host_out;
    return f;
}

// A batch of requests held to what is reserved for them (limited) or not: bytes reserved,
// bytes of the plan taken, of the plan of an unlimited batch; its paths.
extern "C" void mmr_test_arena(const TestFrame *frames, size_t n, int limited, uint64_t *out) {
    uint64_t reserved = 0, bits = 0;
    for (size_t i = 0; i < n; i++) {
        reserved += mmr::reserved_bytes(need_of(frames[i]));
        bits += 8 * frames[i].len;
    }
    auto need = [&](const mmr::SlicePlan &s) {
        uint64_t b = 0;
        for (size_t i = 0; i < n; i++) b += mmr::frame_bytes(need_of(frames[i]), s.bits, s.paths);
        return b;
    };
    const mmr::SlicePlan p = mmr::batch_slices(bits, limited ? reserved : 0, need);
    out[0] = reserved;
    out[1] = need(p);
    out[2] = need(mmr::auto_slices(bits));
    out[3] = p.paths;
}
