// Device-visible plan records for one decode batch (host builds, kernels read).
#pragma once

#include "common.h"

namespace mmr {

// ---------------------------------------------------------------- MJPEG ----

// Canonical-Huffman lookup for one DHT table (crates/codecs/mjpeg/src/entropy.rs:18-70).
// fast[] resolves every code of length <= 9 from the next 9 bits; longer codes use
// maxcode/valptr (JPEG Annex F.2.2.3), which for canonical codes finds the same
// code as the reference's length-by-length search.
constexpr int kHuffFastBits = 11;
constexpr uint32_t kFastEob = 1u << 12;
constexpr uint32_t kFastCode = 1u << 13;
constexpr uint32_t kFastPair = kFastEob | kFastCode;  // (no single entry has both)

struct HuffLut {
    uint16_t fast[512];    // (length << 8) | symbol; 0 when the code is longer than 9 bits or absent
    // Whole symbols within the next 11 bits: value << 16 | eob << 12 | advance << 5 |
    // total bits (code + magnitude). advance moves the coefficient index k: 1 for a
    // DC difference (size 0..11), run + 1 for an AC level (size 1..10), 16 for ZRL;
    // EOB sets k to 64. Codes of at most 11 bits whose magnitude bits reach past
    // them: size << 16 | kFastCode | advance << 5 | code length (the magnitude is
    // read from the bits after the code). 0: slow path (codes longer than 11 bits,
    // and every symbol the reference rejects).
    uint32_t fastv[1 << kHuffFastBits];
    // fastv with two AC symbols in one entry where both lie whole within the next
    // 11 bits, the first not EOB, with levels in -64..63 and -32..31:
    //   level2 << 26 | level1 << 19 | advance2 << 14 | kFastPair | advance1 << 5 | total bits
    // (advance2 0: the second is EOB). The same as fastv for DC tables. No kernel reads
    // them any more (skip, below); the table tests check them with the rest of the record.
    uint32_t fastp[1 << kHuffFastBits];
    int32_t maxcode[18];   // largest code of each length 1..16, -1 if none
    int32_t valptr[18];    // symbol index of a length's first code, minus that code
    uint32_t sym_off;      // first symbol in the symbol pool
    uint32_t nsym;
    uint32_t pad[2];       // size multiple of 16
};

// The canonical code by itself (HuffLut's fields of the same names), for decodes that go
// symbol by symbol with the reference's checks.
struct HuffCanon {
    uint16_t fast[512];
    int32_t maxcode[18];
    int32_t valptr[18];
    uint32_t sym_off;
    uint32_t pad[3];
};

// Lookups of the chunked decoder (jpeg_slices.cu), per table. Canonical codes of more
// than 11 bits are the last of the code space, from the 32-bit left-aligned code
// `first_long` on, so one table serves both: the entry of a window w (the next 32 bits)
// is lut_entry_index(w): its 11-bit prefix, plus one entry per 16-bit pattern from
// first_long on (192 of them for Annex K's AC tables), without a second lookup.
//   sym   code bits | size << 5 | advance << 9 (size: magnitude bits after the code;
//         advance of the coefficient index: 1 for a DC difference, run + 1 for an AC
//         level, 16 for ZRL, kSymEob for EOB, so that a block ends with an index of 64
//         or from 97 to 159 and an overrun lies between); 0 for bits no code matches
//         and for symbols the reference rejects.
//   skip  for decodes that only follow positions, made on the device (skip_entry_of).
//         Byte 3: advance of the first symbol, byte 2: its bits, magnitude included;
//         bytes 1 and 0: the same
//         of the first two where the second's code lies within the 11 bits too (else of
//         the first); 0 where sym is 0.
constexpr uint32_t kSymEob = 96;

struct LutMeta {
    uint32_t off;         // first entry in sym and skip (a multiple of 8)
    uint32_t len;         // entries
    uint32_t first_long;  // 0xffffffff: no codes of more than 11 bits
    uint32_t last;        // windows are clamped to it (the first pattern past the last code, an
                          // invalid one); 0xffffffff where the table covers every pattern
};

// Long-code patterns a table may have to be kept in shared memory (such tables cover
// every pattern and need no clamp).
constexpr uint32_t kSharedLong = 512;
constexpr uint32_t kSharedTab = (1u << kHuffFastBits) + kSharedLong;
constexpr uint32_t kSharedTabs = 2;  // DC and AC tables a CTA keeps in shared memory, of each

// Whether a table can be read from shared memory, where windows are not clamped.
MMR_HD bool lut_fits_shared(const LutMeta &m) { return m.last == 0xffffffffu && m.len <= kSharedTab; }

MMR_HD uint32_t lut_entry_index(uint32_t w, uint32_t first_long) {
    return (w >> (32 - kHuffFastBits)) + (((w > first_long ? w : first_long) - first_long) >> 16);
}

// The skip entry x of a table, from its sym entries.
MMR_HD uint32_t skip_entry_of(const uint16_t *sym, uint32_t first_long, uint32_t x) {
    constexpr uint32_t FB = kHuffFastBits;
    const uint32_t e = sym[x];
    if (!e) return 0;
    const uint32_t cl = e & 31, len = cl + ((e >> 5) & 15), adv = e >> 9;
    uint32_t len2 = len, adv2 = adv;
    // (windows below first_long have no long entries before theirs: x is the prefix)
    if (cl <= FB && adv < kSymEob && len < FB) {
        const uint32_t y = (x << len) & ((1u << FB) - 1);  // what is left of the 11 bits, then zeros
        const uint32_t e2 = y << (32 - FB) < first_long ? sym[y] : 0;
        if (e2 && (e2 & 31) <= FB - len) {
            len2 += (e2 & 31) + ((e2 >> 5) & 15);
            adv2 += e2 >> 9;
        }
    }
    return adv << 24 | len << 16 | adv2 << 8 | len2;
}

// One frame component (SOF0 order).
struct JComp {
    uint32_t plane_w, plane_h;  // visible samples (decoder.rs:440-445)
    uint32_t bw, bh;            // block grid covered by the MCUs
    uint32_t blk_base;          // frame-relative index of block (0,0)
    uint32_t out_off;           // offset of this plane in the frame's planar buffer
    uint8_t h, v, q, pad;       // sampling factors and quantisation slot
    uint32_t pad2;
};

// One block of an MCU, in the scan's component order (decoder.rs:374-400).
struct JSched {
    uint16_t comp;   // frame component index
    uint8_t bx, by;  // block position inside the MCU
    uint8_t dc, ac;  // Huffman table slots
    uint8_t pad[2];
};

// Everything the entropy decoders need for one MCU block position, in one
// 32-byte record (parallel to the schedule): lookups, DC quantiser, and the
// block index of MCU (mx, my) as base_off + mx * mul_x + my * mul_y.
struct JBlockRec {
    uint32_t dc_lut, ac_lut;
    uint32_t base_off;  // frame-relative block of MCU (0, 0)
    uint32_t mul_y;
    uint32_t mul_x;
    uint32_t comp;      // frame component (scan components = frame components)
    int32_t q0;         // DC quantiser
    uint32_t local;     // comp | DC table << 8 | AC table << 16, numbered within the frame
};
constexpr uint32_t kMostPaths = 6;
constexpr uint32_t kMaxSched = 64;  // blocks per MCU of a frame with at most four components

struct JFrame {
    const uint8_t *in;      // packet (device)
    uint8_t *tok;           // unstuffed entropy-coded bytes (device), capacity in_len
    uint8_t *planes;        // planar samples (device): the output itself, or scratch for RGB output
    uint32_t in_len;
    uint32_t data_start;    // first entropy-coded byte
    uint32_t width, height;
    uint32_t ncomp, interleaved;
    uint32_t mcu_cols, mcu_rows, total_mcus;
    uint32_t ri;            // MCUs per restart interval (total_mcus when there is no DRI)
    uint32_t n_intervals;
    uint32_t item_base;     // first (frame, interval) work item
    uint32_t sched_off, sched_len;
    uint32_t comp_off;
    uint32_t lut[8];        // HuffLut index of DC 0..3 then AC 0..3; UINT32_MAX when undefined
    uint32_t quant_off;     // 4 tables x 64 entries, natural order
    uint32_t rst_off;       // restart table (capacity n_intervals)
    uint32_t tile_first;    // first marker-scan tile
    uint32_t decode;        // 0: the header already failed; only the marker scan runs
    uint64_t blk_off;       // first block in the coefficient arena
    uint32_t n_blocks;
    uint32_t item;          // caller's batch item
    uint32_t slot_first;    // first slice slot of the chunked entropy decoder
    uint32_t slot_count;    // slots reserved: ceil(8 * in_len / slice_bits) + n_intervals, in whole CTAs
    uint32_t slice_bits;    // bits per slice (multiple of 32, >= 128)
    uint32_t n_dc, n_ac;    // distinct DC and AC tables of the scan, and the first four of each
    uint32_t dc_id[4], ac_id[4];
    uint32_t lead, paths;   // of the speculative decodes: bits before a slice, and how many (1..kMostPaths)
    uint32_t shared_tabs;   // 1: they fit a CTA's shared memory (kSharedTabs of each, kSharedLong)
};

// --------------------------------------------- chunked entropy decoding ----
//
// Decoder states are block boundaries, packed as (bit position << 8) | block of the
// MCU that starts there, the position counted from the interval's first entropy-coded
// token.

constexpr int kSliceThreads = 128;  // slots per CTA; frames reserve whole CTAs

// One restart interval (the whole scan without DRI) of a frame with <= 4 components.
struct IvInfo {
    uint32_t start;       // first token
    uint32_t barrier;     // tokens before the RST marker (or the end of the scan) that ends it
    uint32_t slot_first;  // first slice slot
    uint32_t n_slices;    // 0: not decoded (header failure, or no RST precedes it)
    uint32_t blocks;      // coefficient blocks in the interval
    uint32_t flags;       // bit 0: the barrier is an RST marker
    uint32_t frame;
    uint32_t pad;
};

// Where the true decode of a slice met its speculative decode.
constexpr uint32_t kMatchNone = 0xffffffffu;
constexpr uint32_t kMatchStart = 0xfffffffeu;  // a first slice: the speculative decode is the true one

// Per slice: the state its decode starts from and what that decode produced.
struct SliceSync {
    unsigned long long start;  // start state (guess marker until it is settled)
    unsigned long long exit;   // first block boundary at or past the slice end
    uint32_t blocks;           // blocks that start in [start, exit)
    int32_t dc[4];             // sum of their DC differences, per scan component
    uint32_t q;                // checkpoint where it met the speculative decode (kMatch*)
};

// A block boundary of the speculative decode and the counts accumulated before it.
struct SlicePoint {
    unsigned long long state;
    uint32_t blocks;
    int32_t dc[4];
    uint32_t pad;  // SliceSpec::exit: bit q set when cp[q] is on the way to it
};

// Checkpoints: the first block boundary 0, 64, 128, 256, 512, 768, 1024 and 1536 bits
// into a slice (those inside it).
constexpr int kSliceCheckpoints = 8;

struct SliceSpec {
    SlicePoint exit;                      // end of the speculative decode
    SlicePoint cp[kSliceCheckpoints];
};

// Blocks that a slice decodes: of the n that start in it, those up to the interval's last
// of `blocks`; the first is block `base` of the interval, block si of the MCU. After an
// error in the scan, slices start where guesses met and base sums what those counted: one
// whose si is not base's place in the MCU would go past the interval's last MCU (into
// another component's blocks, another frame's, or past the arena) and decodes nothing. (For
// true states the two agree, and what an error leaves behind is never shown.)
MMR_HD uint32_t slice_share(uint32_t n, uint32_t base, uint32_t blocks, uint32_t si, uint32_t sched_len) {
    if (base >= blocks || base % sched_len != si) return 0;
    return n < blocks - base ? n : blocks - base;
}

// Block index and DC predictors at a slice's start (interval-relative).
struct SlicePrefix {
    uint32_t base;
    uint32_t pad;
    long long dc[4];
};

// The first event of a slice's final decode: an error, or the interval's last block done.
struct SliceEvent {
    Diag diag;          // error; for completion, offset = tokens consumed by the interval
    uint32_t complete;
};

// Written by the kernels, copied back to the host.
struct JState {
    unsigned long long term;  // (offset << 9) | (truncated << 8) | code of the first terminator; ~0 if none
    uint32_t n_tokens;
    uint32_t n_rst;
    uint32_t bad_interval;    // first interval that failed (UINT32_MAX if none)
    uint32_t pad;
    Diag diag;                // that interval's diagnostic (offset = tokens consumed)
};

struct RstEntry {
    uint32_t tok;     // tokens before the marker
    uint32_t number;  // n of RSTn
};

// One (frame, component) run of coefficient blocks, for the transform kernel.
struct JBlockRange {
    uint64_t first;  // first global block
    uint32_t frame;
    uint32_t comp;   // frame component index
};

// ---------------------------------------------------------------- DV25 -----

struct DvFrame {
    const uint8_t *in;   // 120000 / 144000 bytes (device)
    uint8_t *planes;     // planar samples (device): the output itself, or scratch for RGB output
    uint32_t pal;        // 0: 525/60, 1: 625/50
    uint32_t sequences;  // 10 or 12
    uint32_t width, height, cw, ch;
    uint32_t conceal;
    uint32_t item;
    uint64_t blk_off;    // first block in the DV coefficient arena (sequences*27*30 blocks)
    uint32_t seg_first;  // first segment in the segment arrays
};

struct DvState {
    uint32_t bad_segment;  // first failing segment (sequence*27+slot), UINT32_MAX if none
    uint32_t failed;       // number of failing segments
    Diag diag;
};

// ---------------------------------------------------------------- colour ---

// One frame to convert to interleaved RGB24 (crates/cli/src/terminal_preview.rs:7159-7236, 1:1).
struct RgbJob {
    const uint8_t *planes;
    uint8_t *out;
    uint32_t w, h;
    uint32_t lw, lh, cbw, cbh, crw, crh;
    uint32_t cb_off, cr_off;  // offsets of Cb / Cr in planes (Y at 0)
    uint32_t limited;         // ColorRange::Limited
    uint32_t gray;
    uint32_t item;
    uint32_t pad;
};

}  // namespace mmr
