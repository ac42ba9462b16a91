// DV25 decode kernels for sm_103a.
//
//   segment    a warp per video segment (5 macroblocks, 30 blocks), persistent CTAs: DIF
//              identifiers vs the canonical layout (crates/codecs/dv/src/dif.rs:181-253),
//              DC/mode/class fields, VLC decode and the three-level spill of
//              unused bits -- block region (a lane per block), macroblock pool
//              (a lane per macroblock), segment pool (one lane)
//              (dv/src/decoder.rs:152-317); writes every dequantised coefficient.
//   resolve    first failing segment per frame (sequential semantics).
//   idct       eight threads per block (one per output row), 8 blocks per CTA:
//              fp32 separable 8-8 / 2-4-8 transform with a proven error bound;
//              samples within it of a rounding boundary are settled by the warp in
//              exact fixed point, or in the reference's binary64 order for genuine
//              near-ties (decoder.rs:520-602, dv_idct_core.h); then placement
//              (decoder.rs:395-505).
#include <cuda_runtime.h>

#include <algorithm>

#include "dv_idct_core.h"
#include "dv_layout.h"
#include "kernels.h"
#include "launch.h"
#include "rounding.h"
#include "tables.h"

namespace mmr {

__constant__ int c_dv_zz88[64] = MMR_ZIGZAG_INIT;
__constant__ int c_dv_zz248[64] = MMR_DV_ZIGZAG_248_INIT;
__constant__ uint8_t c_dv_shifts[88] = MMR_DV_QUANT_SHIFTS_INIT;
__constant__ int c_dv_qoff[4] = MMR_DV_QUANT_OFFSET_INIT;
__constant__ int32_t c_dv_w88[64] = MMR_DV_IWEIGHT_88_INIT;
__constant__ int32_t c_dv_w248[64] = MMR_DV_IWEIGHT_248_INIT;

namespace {

// dif.rs:235-253 expected_id
__device__ __forceinline__ void expected_id(uint32_t pos, uint32_t *section, uint32_t *number) {
    if (pos == 0) {
        *section = 0;
        *number = 0;
    } else if (pos <= 2) {
        *section = 1;
        *number = pos - 1;
    } else if (pos <= 5) {
        *section = 2;
        *number = pos - 3;
    } else {
        uint32_t av = pos - 6;
        if (av % 16 == 0) {
            *section = 3;
            *number = av / 16;
        } else {
            *section = 4;
            *number = (av - av / 16 - 1) & 0xff;
        }
    }
}

// ---- bit buffers (MSB-first, 32-bit words) ----

__device__ __forceinline__ uint32_t get32(const uint32_t *w, uint32_t bit) {
    uint32_t i = bit >> 5, r = bit & 31;
    uint32_t hi = w[i] << r;
    return r ? hi | (w[i + 1] >> (32 - r)) : hi;
}

// Appends bits [start, start+n) of src to dst (which holds dn bits, zero beyond).
__device__ __forceinline__ void append_bits(uint32_t *dst, uint32_t &dn, const uint32_t *src, uint32_t start,
                                            uint32_t n) {
    while (n) {
        uint32_t k = n < 32 ? n : 32;
        uint32_t v = get32(src, start) >> (32 - k);  // k bits, right-aligned
        uint32_t i = dn >> 5, r = dn & 31;
        // place v's k bits at bit offset r of word i
        uint64_t sh = (uint64_t)v << (64 - r - k);
        dst[i] |= (uint32_t)(sh >> 32);
        if (r + k > 32) dst[i + 1] |= (uint32_t)sh;
        dn += k;
        start += k;
        n -= k;
    }
}

struct DvBlock {
    uint8_t position;
    uint8_t mode;     // 1 = 2-4-8
    uint8_t cls;
    uint8_t plen;
    uint16_t pval;    // partial bits (< 16), right-aligned
};

// A warp takes a video segment at a time (dv/src/decoder.rs:152-317), in the
// reference's three levels:
//   1. a lane per block (30): DC/mode/class and the AC codes inside the
//      block's own region of its macroblock's payload, the region's bits in registers;
//   2. a lane per macroblock (5): the leftover bits of its complete blocks, in
//      block order, make the macroblock pool, which its incomplete blocks
//      consume in order (decode_macroblock, decoder.rs:193-243);
//   3. one lane: the macroblock pools' leftovers, in macroblock order, make the segment
//      pool, which the segment's incomplete blocks consume in order
//      (consume_pool_for_macroblocks, decoder.rs:225-233).
// Payload, pools and dequantised coefficients stay in shared memory; every
// block's 64 coefficients (zeros included) then leave as 16-byte stores. CTAs are
// persistent: the VLC table and the dequantisation tables, which the lanes index
// freely, are copied to shared memory once (constant memory and L1 served such
// lookups a lane at a time).
//
// Each level is a chain of lookups, so warps go their own ways: with four segments to a
// CTA and a thread per block, then per macroblock, then per segment, half of all warp time
// was spent at the barriers between them (a call of 1000 NTSC frames, 270,000 segments,
// transform included: 2325 us, then 1955; 1775 with the transform's later steps). More CTAs
// per SM gain nothing.
constexpr int kSegThreads = 128;
constexpr int kSegWarps = kSegThreads / 32;
constexpr int kSegCtasPerSm = 6;

struct SegWarp {
    __align__(16) int16_t coef[30][64];
    uint32_t pay[5 * 19 + 5];  // payload words of the five macroblocks (+5: reads past the end)
    uint32_t mbpool[5][20];
    uint32_t segpool[5 * 19 + 2];
    DvBlock blk[30];
    uint16_t left_start[30], left_len[30];  // unused bits of a complete block's region
    uint16_t mb_pos[5], mb_len[5];
    uint8_t qno[5];
};

struct SegSmem {
    __align__(16) uint32_t vlc[kDvVlcEntries];
    uint32_t dequant[2][64];            // per mode and zigzag index: weight | natural index << 16 | 8 * area << 24
    uint32_t shifts[22];                // per quantiser row: the four areas' shifts, a byte each
    SegWarp warp[kSegWarps];
};

// Entry of the next 16 bits. The codes of more than kDvVlcL1Bits bits are the last of
// the code space, so the level-2 blocks follow one another in code order and one index
// reaches both levels (dv_vlc_one_index checks the table).
__device__ __forceinline__ uint32_t vlc_entry(const SegSmem &S, uint32_t w16) {
    return S.vlc[w16 < kDvVlcLong ? w16 >> (16 - kDvVlcL1Bits) : (1u << kDvVlcL1Bits) + w16 - kDvVlcLong];
}

// A block's dequantisation: its table, and its quantiser row's shifts
// (inverse_factor_for_encoding, decoder.rs:290-310).
struct Dequant {
    const uint32_t *table;
    uint32_t shifts;
    int16_t *coef;
};

__device__ __forceinline__ Dequant dequant_of(const SegSmem &S, SegWarp &W, const DvBlock &b, uint32_t block, uint32_t qno) {
    Dequant d;
    d.table = S.dequant[b.mode];
    d.shifts = S.shifts[qno + (uint32_t)c_dv_qoff[b.cls]] + (b.cls == 3 ? 0x02020202u : 0x01010101u);
    d.coef = W.coef[block];
    return d;
}

// Moves the position past the entry's run; true when that completes the block, else its
// level is stored (a zero level changes nothing).
__device__ __forceinline__ bool take_level(const Dequant &d, uint32_t e, uint32_t &p) {
    p += ((e >> 5) & 127) + 1;
    if (p >= 64) return true;
    const uint32_t t = d.table[p];
    const int32_t level = (int32_t)((e >> 12) & 511) - 256;
    const int32_t factor = (int32_t)((t & 0xffff) << ((d.shifts >> (t >> 24)) & 0xff));
    d.coef[(t >> 16) & 63] = (int16_t)((level * factor + 8192) >> 14);
    return false;
}

// consume_ac (decoder.rs:245-284) on a pool, the virtual stream (partial bits ++
// buf[pos, end)). On completion pos is left after the EOB; otherwise the remaining
// bits become the block's partial and pos == end.
// Returns whether the block is complete.
__device__ bool consume_pool(const SegSmem &S, SegWarp &W, uint32_t block, uint32_t qno, const uint32_t *buf,
                             uint32_t &pos, uint32_t end, bool &bad_vlc) {
    DvBlock &b = W.blk[block];
    const Dequant d = dequant_of(S, W, b, block, qno);
    bool complete = false;
    uint32_t p = b.position, plen = b.plen, avail = plen + (end - pos);
    uint32_t w16 = get32(buf, pos) >> 16;
    if (plen) w16 = (((uint32_t)b.pval << (16 - plen)) | (w16 >> plen)) & 0xffffu;
    b.plen = 0;
    b.pval = 0;
    for (;;) {
        const uint32_t e = vlc_entry(S, w16), len = e & 31;
        if (len == 0) {  // unreachable: the DV VLC code is complete (Kraft sum 1)
            bad_vlc = true;
            pos = end;
            break;
        }
        if (len > avail) {  // fewer than 16 bits: the next partial
            b.pval = (uint16_t)(w16 >> (16 - avail));
            b.plen = (uint8_t)avail;
            pos = end;
            break;
        }
        avail -= len;
        pos += len - plen;  // (a partial never holds a whole code)
        plen = 0;
        if (take_level(d, e, p)) {
            complete = true;
            break;
        }
        w16 = get32(buf, pos) >> 16;
    }
    b.position = (uint8_t)p;
    return complete;
}

// The frame of segment g: 32 probes a step.
__device__ __forceinline__ uint32_t frame_of(const DvLaunch &L, uint32_t g) {
    uint32_t lo = 0, hi = L.n_frames;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, at = lo + (threadIdx.x & 31) * step;
        const uint32_t below = __ballot_sync(0xffffffffu, at < hi && L.seg_first[at] <= g);
        lo += (uint32_t)(31 - __clz(below)) * step;  // (lane 0's probe always holds)
        hi = min(lo + step, hi);
    }
    return lo;
}

__global__ void __launch_bounds__(kSegThreads, kSegCtasPerSm) segment_kernel(DvLaunch L) {
    begin_kernel(L.early);
    __shared__ SegSmem S;
    for (uint32_t i = threadIdx.x; i < (uint32_t)kDvVlcEntries; i += kSegThreads) S.vlc[i] = __ldg(L.vlc + i);
    for (uint32_t i = threadIdx.x; i < 128; i += kSegThreads) {
        const uint32_t p = i & 63, m = i >> 6;
        const uint32_t area = p <= 5 ? 0 : p <= 20 ? 1 : p <= 42 ? 2 : 3;
        S.dequant[m][p] = (uint32_t)(m ? c_dv_w248[p] : c_dv_w88[p]) |
                          (uint32_t)(m ? c_dv_zz248[p] : c_dv_zz88[p]) << 16 | area << 27;
    }
    if (threadIdx.x < 22) {
        const uint32_t t = threadIdx.x;
        S.shifts[t] = c_dv_shifts[t * 4] | c_dv_shifts[t * 4 + 1] << 8 | c_dv_shifts[t * 4 + 2] << 16 |
                      (uint32_t)c_dv_shifts[t * 4 + 3] << 24;
    }
    __syncthreads();
    const uint32_t t = threadIdx.x & 31;
    SegWarp &W = S.warp[threadIdx.x >> 5];
    for (uint32_t g = blockIdx.x * kSegWarps + (threadIdx.x >> 5); g < L.n_segments; g += gridDim.x * kSegWarps) {
        const uint32_t f = frame_of(L, g);
        const uint32_t local = g - L.seg_first[f], sequence = local / 27, slot = local % 27;
        const uint8_t *in = L.frames[f].in;
        // macroblock records: DIF block, its identifier against the canonical layout
        // (dif.rs:181-253), quantiser
        uint32_t off = 0;  // byte offset of the lane's macroblock's DIF block in the frame
        bool damaged = false;
        if (t < 5) {
            const uint32_t vn = slot * 5 + t, pos = 7 + (vn / 15) * 16 + vn % 15;  // DIF block of the sequence
            off = (sequence * 150 + pos) * 80;
            const uint8_t *b = in + off;
            uint32_t es, en;
            expected_id(pos, &es, &en);
            damaged = (uint32_t)(b[0] >> 5) != es || (uint32_t)(b[1] >> 4) != sequence || (uint32_t)b[2] != en;
            W.qno[t] = b[3] & 0x0f;
        }
        damaged = __any_sync(0xffffffffu, damaged);
        // payload words (bytes 4..80 of each DIF block), big-endian
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            const uint32_t wi = k * 32 + t, m = min(wi / 19, 4u);
            const uint8_t *src = in + __shfl_sync(0xffffffffu, off, m) + 4 + (wi - m * 19) * 4;
            uint32_t v = 0;
            if (wi < 95) {
                if ((reinterpret_cast<uintptr_t>(src) & 3) == 0)
                    v = __byte_perm(__ldg(reinterpret_cast<const uint32_t *>(src)), 0, 0x0123);
                else
                    v = ((uint32_t)src[0] << 24) | ((uint32_t)src[1] << 16) | ((uint32_t)src[2] << 8) | (uint32_t)src[3];
            }
            if (wi < 100) W.pay[wi] = v;
        }
        for (uint32_t i = t; i < 240; i += 32) reinterpret_cast<int4 *>(&W.coef[0][0])[i] = make_int4(0, 0, 0, 0);
        for (uint32_t i = t; i < 100; i += 32) (&W.mbpool[0][0])[i] = 0;
        for (uint32_t i = t; i < 97; i += 32) W.segpool[i] = 0;
        __syncwarp();
        uint16_t kind = kDvDamagedId;
        uint32_t mode = 0;
        if (!damaged) {  // (uniform)
            // 1. a lane per block: its own region
            bool complete = true, bad = false;
            if (t < 30) {
                const uint32_t m = t / 6, bi = t % 6;
                DvBlock B{};
                uint16_t ls = 0, ll = 0;
                const uint32_t *w = W.pay + m * 19;
                const uint32_t r0 = bi < 4 ? bi * 112 : 448 + (bi - 4) * 80, bits = bi < 4 ? 112 : 80;
                const uint32_t head = get32(w, r0) >> 20;  // 12 bits: dc(9) mode(1) class(2)
                int32_t dc = (int32_t)(head >> 3);
                if (dc & 0x100) dc -= 512;
                B.mode = (head >> 2) & 1;
                B.cls = head & 3;
                mode = B.mode;
                const Dequant d = dequant_of(S, W, B, t, W.qno[m]);
                d.coef[0] = (int16_t)(dc * 4 + 1024);
                // the region's bits after the header (at most 100), left-aligned
                const uint32_t at = r0 + 12, i = at >> 5, o = at & 31;
                uint32_t a0 = __funnelshift_l(w[i + 1], w[i], o), a1 = __funnelshift_l(w[i + 2], w[i + 1], o);
                uint32_t a2 = __funnelshift_l(w[i + 3], w[i + 2], o), a3 = __funnelshift_l(w[i + 4], w[i + 3], o);
                uint32_t left = bits - 12, p = 0;
                for (;;) {
                    const uint32_t e = vlc_entry(S, a0 >> 16), len = e & 31;
                    if (len == 0) bad = true;  // unreachable: the code is complete
                    if (len == 0 || len > left) {
                        B.pval = (uint16_t)(left < 16 ? a0 >> 16 >> (16 - left) : 0);  // the partial
                        B.plen = (uint8_t)(left < 16 ? left : 0);
                        complete = false;
                        break;
                    }
                    a0 = __funnelshift_l(a1, a0, len);
                    a1 = __funnelshift_l(a2, a1, len);
                    a2 = __funnelshift_l(a3, a2, len);
                    a3 <<= len;
                    left -= len;
                    if (take_level(d, e, p)) {
                        ls = (uint16_t)(r0 + bits - left);
                        ll = (uint16_t)left;
                        break;
                    }
                }
                B.position = (uint8_t)p;
                W.blk[t] = B;
                W.left_start[t] = ls;
                W.left_len[t] = ll;
            }
            uint32_t open = __ballot_sync(0xffffffffu, !complete);  // incomplete blocks
            __syncwarp();
            // 2. a lane per macroblock: its pool
            uint32_t mine = 0;
            if (t < 5) {
                const uint32_t *w = W.pay + t * 19;
                const uint32_t j0 = t * 6;
                mine = (open >> j0) & 63;
                uint32_t pos = 0, mbn = 0;
                for (uint32_t done = ~mine & 63; done; done &= done - 1) {
                    const uint32_t j = j0 + __ffs(done) - 1;
                    append_bits(W.mbpool[t], mbn, w, W.left_start[j], W.left_len[j]);
                }
                for (uint32_t left = mine; left && pos < mbn; left &= left - 1) {
                    const uint32_t k = __ffs(left) - 1;
                    if (consume_pool(S, W, j0 + k, W.qno[t], W.mbpool[t], pos, mbn, bad)) mine ^= 1u << k;
                }
                W.mb_pos[t] = (uint16_t)pos;
                W.mb_len[t] = (uint16_t)mbn;
                mine <<= j0;
            }
            open = __reduce_or_sync(0xffffffffu, mine);
            __syncwarp();
            // 3. one lane: the segment's pool
            if (t == 0 && open) {
                uint32_t pos = 0, segn = 0;
                for (uint32_t m = 0; m < 5; m++)
                    if (W.mb_pos[m] < W.mb_len[m])
                        append_bits(W.segpool, segn, W.mbpool[m], W.mb_pos[m], W.mb_len[m] - W.mb_pos[m]);
                for (uint32_t left = open; left && pos < segn; left &= left - 1) {
                    const uint32_t j = __ffs(left) - 1;
                    if (consume_pool(S, W, j, W.qno[j / 6], W.segpool, pos, segn, bad)) open ^= 1u << j;
                }
            }
            open = __shfl_sync(0xffffffffu, open, 0);
            kind = __any_sync(0xffffffffu, bad) ? kDvBadVlc : open ? kDvIncomplete : kDiagNone;
            __syncwarp();
        }
        // coefficients out, modes, result
        int4 *dst = reinterpret_cast<int4 *>(L.coef + (uint64_t)g * 30 * 64);
        const int4 *src = reinterpret_cast<const int4 *>(&W.coef[0][0]);
        for (uint32_t i = t; i < 240; i += 32) dst[i] = src[i];
        if (t < 30) L.modes[(uint64_t)g * 30 + t] = (uint8_t)mode;
        if (t == 0) {
            L.seg_err[g] = (uint8_t)kind;
            if (kind != kDiagNone) {
                atomicMin(&L.states[f].bad_segment, local);
                atomicAdd(&L.states[f].failed, 1u);
            }
        }
        __syncwarp();  // the coefficients are read
    }
}

__global__ void dv_resolve_kernel(DvLaunch L) {
    begin_kernel(L.early);
    uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= L.n_frames) return;
    DvState *st = &L.states[f];
    uint32_t bad = st->bad_segment;
    if (bad != 0xffffffffu) {
        uint16_t kind = L.seg_err[L.frames[f].seg_first + bad];
        st->diag = make_diag(kind, 0, bad % 27, bad / 27);
        if (!L.frames[f].conceal) L.item_ok[L.frames[f].item] = 0;
    }
}

constexpr int kIdctBlocks = 8;                   // blocks per CTA (1000 NTSC frames at the time: 1.92 ms, with 16 1.96)
constexpr int kIdctThreads = kIdctBlocks * 8;    // eight threads (rows) per block

// Stores the eight bytes of `row` at dst (any alignment).
__device__ __forceinline__ void store_row8(uint8_t *dst, unsigned long long row) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(dst);
    if ((a & 7) == 0) {
        *reinterpret_cast<uint2 *>(dst) = make_uint2((uint32_t)row, (uint32_t)(row >> 32));
    } else if ((a & 3) == 0) {
        reinterpret_cast<uint32_t *>(dst)[0] = (uint32_t)row;
        reinterpret_cast<uint32_t *>(dst)[1] = (uint32_t)(row >> 32);
    } else {
#pragma unroll
        for (int x = 0; x < 8; x++) dst[x] = (uint8_t)(row >> (8 * x));
    }
}

__device__ __forceinline__ void store_row4(uint8_t *dst, uint32_t row) {
    if ((reinterpret_cast<uintptr_t>(dst) & 3) == 0) {
        *reinterpret_cast<uint32_t *>(dst) = row;
    } else {
#pragma unroll
        for (int x = 0; x < 4; x++) dst[x] = (uint8_t)(row >> (8 * x));
    }
}

// Eight threads per block: the fp32 passes with the exact fallback (dv_idct_core.h),
// then placement (decoder.rs:432-505) with 8-byte row stores. A warp holds four blocks
// of one frame (frames start at multiples of 4 blocks: 8100 and 9720 blocks per frame),
// found by one division where all frames are of one system; the eight threads of a
// block synchronise through their warp only. Issue-bound (two thirds) with waits for the
// levels between: 32 registers for 28 CTAs of 64 per SM (1000 NTSC frames: 1.82 ms, with
// 52 registers 1.93; 1.78 with fewer and larger parts).
constexpr int kBlockStride = 72;  // ints or floats per block: four blocks' column accesses on distinct banks

__global__ void __launch_bounds__(kIdctThreads, 28) dv_idct_kernel(DvLaunch L) {
    begin_kernel(L.early);
    __shared__ __align__(16) int32_t s_c[kIdctBlocks][kBlockStride];
    __shared__ __align__(16) float s_h[kIdctBlocks][kBlockStride];
    const int lane = threadIdx.x & 31, lb = threadIdx.x >> 3, r = threadIdx.x & 7;
    const unsigned group_mask = 0xffu << (lane & 24);
    const uint32_t gb = blockIdx.x * kIdctBlocks + lb;
    bool valid = gb < L.n_blocks;
    uint32_t f;
    if (L.frame_blocks) {
        f = min(gb / L.frame_blocks, L.n_frames - 1);
    } else {
        uint32_t lo = 0, hi = L.n_frames;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (L.frames[mid].blk_off <= gb) lo = mid;
            else hi = mid;
        }
        f = lo;
    }
    const DvFrame *F = &L.frames[f];
    bool failed = false, mode = false;
    uint32_t local_blk = 0;
    int4 lv = make_int4(0, 0, 0, 0);
    if (valid) {
        local_blk = gb - (uint32_t)F->blk_off;
        valid = L.item_ok[F->item] != 0;
        if (valid) {
            failed = L.seg_err[F->seg_first + local_blk / 30] != 0;
            mode = L.modes[gb] != 0;
            if (!failed) lv = reinterpret_cast<const int4 *>(L.coef + (uint64_t)gb * 64)[r];  // row r: 8 int16
        }
    }
    int32_t *c = s_c[lb];
    // C1 of the block (at most 2^21, exact as a float too) and whether any AC
    // coefficient is nonzero, over its eight threads
    int32_t c1 = 0;
    {
        const uint32_t w[4] = {(uint32_t)lv.x, (uint32_t)lv.y, (uint32_t)lv.z, (uint32_t)lv.w};
        int32_t row[8];
#pragma unroll
        for (int u = 0; u < 8; u++) {
            row[u] = u & 1 ? (int32_t)w[u >> 1] >> 16 : (int32_t)(int16_t)w[u >> 1];
            c1 += abs(row[u]);
        }
        reinterpret_cast<int4 *>(c + r * 8)[0] = make_int4(row[0], row[1], row[2], row[3]);
        reinterpret_cast<int4 *>(c + r * 8)[1] = make_int4(row[4], row[5], row[6], row[7]);
    }
    const bool ac = ((r ? lv.x : lv.x & (int)0xffff0000) | lv.y | lv.z | lv.w) != 0;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) c1 += __shfl_xor_sync(0xffffffffu, c1, o);
    const bool flat = (__ballot_sync(0xffffffffu, ac) & group_mask) == 0;
    const bool active = valid && !failed;
    __syncwarp();
    if (active && !flat) dv_row_pass8(c, nullptr, mode, r, s_h[lb] + r * 8);
    __syncwarp();
    unsigned long long row = 0;
    uint32_t und = 0;
    if (active)
        und = dv_row_fp32(c, s_h[lb], nullptr, nullptr, mode, r, (float)c1, flat, lane & 24, group_mask, &row);
    dv_resolve_row(und, row, c, mode, r, c1, L.fixw);  // every lane of the warp takes part
    if (!valid) return;
    const uint32_t e = __ldg(L.place + (F->pal ? kDvBlocks525 : 0) + local_blk);
    const bool chroma = (e & kDvPlaceChroma) != 0;
    if (failed) row = 0x0101010101010101ull * (chroma ? 128u : 16u);
    const uint32_t stride = chroma ? F->cw : F->width;
    uint8_t *dst = F->planes + (e & kDvPlaceOffset) + r * stride;
    if (e & kDvPlaceSplit) {
        store_row4(dst, (uint32_t)row);
        store_row4(dst + 8 * stride, (uint32_t)(row >> 32));
    } else {
        store_row8(dst, row);
    }
}

}  // namespace

void launch_dv_decode(const DvLaunch &L, cudaStream_t s) {
    const uint32_t steps = (L.n_segments + kSegWarps - 1) / kSegWarps;
    // (an ordinary launch: what comes before it on the stream may be the caller's)
    if (steps) segment_kernel<<<std::min<uint32_t>(steps, 152 * kSegCtasPerSm), kSegThreads, 0, s>>>(L);
    if (L.n_frames) launch_next(dv_resolve_kernel, (L.n_frames + 127) / 128, 128, s, L);
}

void launch_dv_idct(const DvLaunch &L, cudaStream_t s) {
    if (L.n_blocks == 0) return;
    launch_next(dv_idct_kernel, (unsigned)((L.n_blocks + kIdctBlocks - 1) / kIdctBlocks), kIdctThreads, s, L);
}

}  // namespace mmr
