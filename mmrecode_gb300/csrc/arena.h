// Device memory of a batch's MJPEG frames, from their headers: what the engine's arenas
// take, what the server reserves for a request, and the slices that fit between the two.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <algorithm>

#include "plan.h"

namespace mmr {

// Slice size, and lead and number of the speculative decodes per slice of a batch.
struct SlicePlan {
    uint32_t bits, lead, paths;
};

// Small batches leave the GPU idle, so their time is that of one thread's slice: short
// slices, and every block of the MCU guessed, which finds the true state after 250 to
// 500 bits (99 % of starts) where one guess takes 1,000 to 5,000. Large batches are
// bound by the instructions of all threads: long slices and one guess. Measured, us,
// by slice bits / lead / paths:
//   one 320x240 4:2:0 frame (0.13 Mbit)   256/384/6 307   512/384/6 317   1024/384/6 352
//   one 1080p 4:2:2 frame (9 Mbit)        256/384/6 350   512/384/6 327   1024/384/6 359
//   30 VGA 4:2:0 frames (14 Mbit)         512/384/6 471   1024/384/6 421  1024/1024/1 492   2048/768/1 544
//   64 mixed frames (four of 106 Mbit)    1024/1024/1 3271   2048/768/1 3079   4096/768/1 3128
//   300 1080p frames (eight of 341 Mbit)  2048/768/1 7930   4096/768/1 7469   2048/384/4 11003
// and with the present kernels, near the lines between them (VGA 4:2:0 frames of 0.48 Mbit
// to planes, 1080p 4:2:2 ones of 9 Mbit to RGB; the plan taken is the first):
//   20 VGA (10 Mbit)     512/384/6 290    1024/384/6 292
//   28 VGA (13 Mbit)     1024/384/6 318   512/384/6 330    1024/1024/1 384
//   3 1080p (27 Mbit)    1024/384/6 290   2048/768/1 326   1024/1024/1 305
//   4 1080p (36 Mbit)    2048/768/1 339   1024/384/6 353   2048/384/6 352
//   5 1080p (45 Mbit)    2048/768/1 390   1024/384/6 372   2048/384/6 382
//   16 1080p (144 Mbit)  2048/768/1 562   4096/768/1 705   2048/384/6 719
//   20 1080p (180 Mbit)  4096/768/1 723   2048/768/1 599
//   28 1080p (252 Mbit)  4096/768/1 815   2048/768/1 871
// (so the last line could lie nearer 200 Mbit).
inline SlicePlan auto_slices(uint64_t total_bits) {
    if (total_bits <= 2u << 20) return SlicePlan{256, 384, 6};
    if (total_bits <= 12u << 20) return SlicePlan{512, 384, 6};
    if (total_bits <= 32u << 20) return SlicePlan{1024, 384, 6};
    if (total_bits <= 160u << 20) return SlicePlan{2048, 768, 1};
    return SlicePlan{4096, 768, 1};
}

// The plan of larger batches, where the records of several guesses (1.7 KB a slice) have
// no room: a tenth of the memory.
inline SlicePlan lean_slices(uint64_t total_bits) {
    const SlicePlan p = auto_slices(total_bits);
    return p.paths > 1 ? SlicePlan{2048, 768, 1} : p;
}

// Slots of a frame (jpeg_slices.cu: an interval's begin at its bits / slice_bits plus its
// number), in whole CTAs.
inline uint64_t slice_slots(uint64_t len, uint64_t intervals, uint32_t slice_bits) {
    const uint64_t n = (8 * len + slice_bits - 1) / slice_bits + intervals;
    return (n + kSliceThreads - 1) / kSliceThreads * kSliceThreads;
}

// A frame as its headers describe it.
struct FrameNeed {
    uint64_t len = 0;        // packet
    uint64_t planar = 0;     // samples
    uint64_t blocks = 0;     // coefficient blocks, those of padding included
    uint64_t intervals = 0;  // restart intervals
    bool sliced = false;     // decoded in slices (at most four components)
    bool host_in = false;    // the packet goes up
    bool planes = false;     // planes of its own besides the output (RGB)
    uint64_t host_out = 0;   // output bytes that go down
};

// Device bytes of a frame in a batch decoded with such slices (records of `paths` guesses).
inline uint64_t frame_bytes(const FrameNeed &f, uint32_t slice_bits, uint32_t paths) {
    auto pad = [](uint64_t v) { return (v + 255) / 256 * 256; };
    uint64_t b = pad(f.len) * (f.host_in ? 2 : 1) + 512;            // tokens, packet
    b += f.len / 512 + 64;                                          // marker scan: tile counts and their groups
    b += f.blocks * (128 + 4 + 16);                                 // levels, DC, exact queue
    b += (f.planes ? pad(f.planar) : 0) + pad(f.host_out);
    b += f.intervals * (sizeof(RstEntry) + sizeof(Diag) + 8 + sizeof(IvInfo) + 8 + 4);
    if (f.sliced)
        b += slice_slots(f.len, f.intervals, slice_bits) *
             (4 + sizeof(SliceSync) + sizeof(SlicePrefix) + sizeof(SliceEvent) + paths * sizeof(SliceSpec));
    return b;
}

// What the server reserves for a frame: 8 bytes per compressed byte and 5.5 per sample,
// which the lean plan's arenas stay below but for frames of one or two blocks per restart
// interval, and of much padding. In a batch of such requests the engine takes more guesses
// only where they fit the sum (batch_slices).
inline uint64_t reserved_bytes(const FrameNeed &f) {
    const uint64_t usual = 8 * f.len + f.planar * 9 / 2 + f.planar + 65536 + f.host_out;
    return std::max(usual, frame_bytes(f, lean_slices(0).bits, 1) + 16384);  // (+ tables and frame records)
}

// The slices of a batch of `total_bits` compressed bits, held to `limit` device bytes (0: not
// held). need(plan): its bytes.
template <class Need>
inline SlicePlan batch_slices(uint64_t total_bits, uint64_t limit, Need need) {
    const SlicePlan p = auto_slices(total_bits);
    return limit == 0 || p.paths == 1 || need(p) <= limit ? p : lean_slices(total_bits);
}

}  // namespace mmr
