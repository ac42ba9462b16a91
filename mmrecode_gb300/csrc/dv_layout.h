// Where each block of a DV25 frame lands in its planes (dv/src/decoder.rs:395-505), as a
// table per system built on the host: a thread of the transform would spend more
// instructions on the macroblock coordinates than on its share of the transform.
#pragma once

#include <stdint.h>

#include "tables.h"

namespace mmr {

constexpr uint32_t kDvBlocks525 = 10 * 27 * 30, kDvBlocks625 = 12 * 27 * 30;
constexpr uint32_t kDvPlaceEntries = kDvBlocks525 + kDvBlocks625;  // 525/60, then 625/50

// Entry: byte offset of the block's first sample in the planar frame, and:
constexpr uint32_t kDvPlaceChroma = 1u << 31;  // rows are the chroma width apart (else the luma width)
constexpr uint32_t kDvPlaceSplit = 1u << 30;   // put_split_chroma: columns 4..7 go eight rows further down
constexpr uint32_t kDvPlaceOffset = kDvPlaceSplit - 1;

// macroblock_coordinates (decoder.rs:395-422), in 8-sample units
inline void dv_mb_coords(bool pal, uint32_t seqs, uint32_t sequence, uint32_t slot, uint32_t m, uint32_t *mbx,
                         uint32_t *mby) {
    static const uint32_t off[5] = {2, 6, 8, 0, 4}, shuf3[5] = {18, 9, 27, 0, 36}, lstart[5] = {9, 4, 13, 0, 18};
    if (pal) {
        // SERPENT1[slot] = 0,1,2,2,1,0 repeating
        const uint32_t s6 = slot % 6, serp1 = s6 < 3 ? s6 : 5 - s6;
        *mbx = (shuf3[m] + slot / 3) * 2;
        *mby = (serp1 + ((sequence + off[m]) % seqs) * 3) * 2;
    } else {
        const uint32_t row = (sequence + off[m]) % seqs, k = slot + ((m == 1 || m == 2) ? 3 : 0);
        const uint32_t x = lstart[m] + k / 6;
        // SERPENT2[k] = 0..5,5..0 repeating
        const uint32_t k12 = k % 12, serp2 = k12 < 6 ? k12 : 11 - k12;
        uint32_t y = serp2 + row * 6;
        if (x > 21) y = y * 2 - row * 6;
        *mbx = x * 4;
        *mby = y;
    }
}

inline void fill_dv_place(uint32_t *table) {
    for (int pal = 0; pal < 2; pal++) {
        const uint32_t seqs = pal ? 12 : 10, W = 720, H = pal ? 576 : 480, cw = pal ? 360 : 180, ch = pal ? 288 : 480;
        for (uint32_t b = 0; b < seqs * 27 * 30; b++) {
            const uint32_t seg = b / 30, j = b % 30, m = j / 6, bi = j % 6;
            uint32_t mbx, mby;
            dv_mb_coords(pal != 0, seqs, seg / 27, seg % 27, m, &mbx, &mby);
            const uint32_t X = mbx * 8, Y = mby * 8;
            const bool square = pal || mbx >= 88;  // luma 2x2 (else 4x1)
            uint32_t e;
            if (bi < 4) {
                e = square ? (Y + (bi >> 1) * 8) * W + X + (bi & 1) * 8 : Y * W + X + bi * 8;
            } else {
                const uint32_t plane = W * H + (bi == 4 ? cw * ch : 0);  // block 4 is Cr, the last plane
                e = plane + (pal ? Y / 2 * cw + X / 2 : Y * cw + X / 4);
                e |= kDvPlaceChroma | (!pal && square ? kDvPlaceSplit : 0);
            }
            *table++ = e;
        }
    }
}

}  // namespace mmr
