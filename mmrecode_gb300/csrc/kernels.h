// Kernel launchers (host-callable) for the MJPEG and DV25 decode stages.
#pragma once

#include <cuda_runtime.h>

#include "plan.h"

namespace mmr {

constexpr int kScanTile = 4096;  // bytes of entropy-coded data per marker-scan warp

// Packet-relative first byte of a frame's first tile: its address is the 16-byte line that
// data_start lies in, so that it may lie before the packet. (The host sizes by it too.)
MMR_HD long long scan_base(const uint8_t *in, uint32_t data_start) {
    return (long long)data_start - (long long)((reinterpret_cast<uintptr_t>(in) + data_start) & 15);
}

struct JpegLaunch {
    const JFrame *frames;        // device
    JState *states;              // device
    uint32_t n_frames;
    bool early;                  // begin_kernel's (a small batch)
    const uint32_t *tile_first;  // n_frames + 1 prefix of marker-scan tiles
    uint32_t n_tiles;
    unsigned long long *tile_cnt;    // per tile: tokens, and restart markers << 32
    unsigned long long *tile_group;  // their sums over a frame's groups of 64 tiles (zeroed per batch)
    RstEntry *rsts;
    const JSched *sched;
    const JBlockRec *brec;       // parallel to sched
    const JComp *comps;
    const HuffLut *luts;         // only when a frame has more than four components
    uint32_t n_luts;
    const uint8_t *symbols;
    const uint16_t *quant;       // natural order
    const uint2 *items;          // (frame, interval); frames with <= 4 components first
    uint32_t n_items_small;
    uint32_t n_items;
    Diag *results;               // per item
    int16_t *coef;               // 64 levels per block
    int32_t *dc;                 // dequantised DC per block
    const JBlockRange *ranges;
    uint32_t n_ranges;
    const uint32_t *idct_cta_first;  // n_ranges + 1 prefix of transform CTAs (idct_ctas per range)
    uint32_t n_idct_ctas;
    uint32_t idct_tiles;         // tiles of 64 blocks per transform CTA
    uint64_t n_blocks;
    uint32_t *item_ok;           // per batch item: 1 while decoding has not failed
    ulonglong2 *fix;             // blocks the fp32 IDCT could not fully decide: (block, sample mask)
    uint32_t *fix_count;         // entries, samples, slices decoded again by the sync passes, slices, unused,
                                 // those decoded again whole (8 counters, zeroed per batch)
    uint32_t fixup_grid;         // CTAs of the grid-stride fixup pass
    // chunked entropy decoder (frames with <= 4 components; items [0, n_items_small))
    uint32_t n_slots;
    uint32_t *slot_item;         // per slot: item, UINT32_MAX when unused
    IvInfo *ivs;                 // per item
    SliceSync *sync;             // per slot
    SliceSpec *spec;             // paths x n_slots
    uint32_t paths;              // most speculative decodes per slice of any frame
    SlicePrefix *prefix;         // per slot
    SliceEvent *events;          // per slot
    unsigned long long *iv_key;  // per item: first slice that reports an event
    uint32_t *iv_pend;           // per item: first slice still to settle after the sync passes
    uint32_t *sync_left;         // intervals the sync passes left unsettled (zeroed per batch)
    const LutMeta *lut_meta;     // per LUT, its entries in:
    const uint16_t *sym;
    uint32_t *skip;              // written by slice_plan_kernel
    const HuffCanon *canon;
    const long long *fixw;       // fixed-point IDCT weights (exact_fixed.h)
};

// Sync passes before the serial fix-up walk: the first settles the slices inside each
// CTA, the others what changed across CTA boundaries.
constexpr int kSyncPasses = 2;

void launch_jpeg_scan(const JpegLaunch &L, cudaStream_t s);
void launch_jpeg_entropy(const JpegLaunch &L, cudaStream_t s);   // frames with > 4 components
// frames with <= 4 components; marks (optional, 3 events) are recorded after the
// speculative pass, after the sync passes + prefix, and after the final decode
// (as external event nodes when the stream is being captured into a graph)
void launch_jpeg_slices(const JpegLaunch &L, cudaStream_t s, cudaEvent_t *marks = nullptr, bool capturing = false);
int jpeg_slice_launches(const JpegLaunch &L);
void launch_jpeg_idct(const JpegLaunch &L, cudaStream_t s);
uint32_t idct_ctas(uint32_t blocks, uint32_t tiles);

// MJPEG frames decoded straight to RGB24 (three components, chroma 1x1, luma
// 1x1, 2x1 or 2x2): one launch per layout, a CTA per strip of MCUs.
struct FusedJob {
    uint32_t frame;     // JFrame index
    uint32_t groups_x;  // CTAs per MCU row
    uint32_t strips;    // strips per CTA
    uint32_t width, height;
    uint8_t *out;       // width * height * 3 bytes
};

struct FusedLaunch {
    const FusedJob *jobs;
    const uint32_t *cta_first;  // n_jobs + 1 prefix of CTAs (groups_x * mcu_rows per job)
    uint32_t n_jobs;
    uint32_t n_ctas;
};

int fused_variant(uint32_t hmax, uint32_t vmax);  // 0: 1x1, 1: 2x1, 2: 2x2, -1: not fused
// launch slot of a layout variant with a narrow or wide strip (MCUs per CTA:
// 8 or 16 at 1x1, 4 or 8 otherwise); kFusedSlots launches, one per slot
constexpr int kFusedSlots = 6;
int fused_slot(int variant, bool wide);
uint32_t fused_slot_mcus(int slot);
uint32_t fused_groups_x(int slot, uint32_t mcu_cols, uint32_t strips);
void launch_jpeg_idct_rgb(const JpegLaunch &L, const FusedLaunch *FL, cudaStream_t s);  // FL[kFusedSlots]
int fused_launches(const FusedLaunch &FL);

struct DvLaunch {
    const DvFrame *frames;
    DvState *states;
    uint32_t n_frames;
    const uint32_t *seg_first;   // n_frames + 1 prefix of segments
    uint32_t n_segments;
    uint8_t *seg_err;            // per segment: DiagKind (0 = ok)
    int16_t *coef;               // 64 per block, natural order
    uint8_t *modes;              // per block: 1 = 2-4-8
    const uint32_t *vlc;         // two-level VLC table
    const long long *fixw;       // fixed-point transform weights: 8-8 then 2-4-8 (exact_fixed.h)
    const uint32_t *place;       // where blocks land (dv_layout.h)
    bool early;                  // begin_kernel's (a small batch)
    uint64_t n_blocks;           // less than 2^32
    uint32_t frame_blocks;       // of every frame, 0 when they differ
    uint32_t *item_ok;
};

void launch_dv_decode(const DvLaunch &L, cudaStream_t s);
void launch_dv_idct(const DvLaunch &L, cudaStream_t s);

struct RgbLaunch {
    const RgbJob *jobs;
    const uint32_t *cta_first;  // n_jobs + 1 prefix of CTAs (rgb_ctas per job)
    uint32_t n_jobs;
    uint32_t n_ctas;
    const uint32_t *item_ok;
};

uint32_t rgb_ctas(uint32_t w, uint32_t h);
void launch_rgb(const RgbLaunch &L, cudaStream_t s);

// DV VLC lookup: level-1 indexed by the next 10 bits; long codes index a
// 64-entry level-2 block with the following 6 bits. Entry layout:
//   bit 31 set: level-2 block at bits 0..15 (entry index)
//   otherwise: len (bits 0..4), run (bits 5..11), level + 256 (bits 12..20); len 0 = no code
constexpr int kDvVlcL1Bits = 10;
// The DV code's table: 32 level-1 entries, those of the 16-bit windows from kDvVlcLong
// on, have level-2 blocks, in window order.
constexpr uint32_t kDvVlcLong = 0xf800;
constexpr size_t kDvVlcEntries = (1u << kDvVlcL1Bits) + (0x10000u - kDvVlcLong);

}  // namespace mmr
