// Chunked, self-synchronising Huffman decode of baseline JPEG scans (sm_103a).
//
// The reference decodes a scan serially, one restart interval after another
// (crates/codecs/mjpeg/src/decoder.rs:313-410, 495-548; entropy.rs:57-182). A
// thread per interval leaves a GB300 nearly idle (135 intervals per 1080p frame,
// one per scan without DRI), so every interval is cut into fixed-size bit slices
// that decode in parallel. Huffman codes resynchronise: a decode started at a
// wrong bit or in a wrong state soon meets the true decode at a block boundary
// with the same position in the MCU, and from there both are identical.
//
// A slice owns the blocks that start inside it; its start state is the first block
// boundary at or past its nominal start (bit position, block of the MCU), which is
// its predecessor's exit state. Two decodes run over the bits: a lean one that only
// finds the states (code lengths and coefficient advances, two symbols per lookup,
// nothing stored), then one from the true states that writes the levels.
//
//   slice_plan     per frame: interval token ranges, slice counts, slot -> interval map
//   slice_spec     the lean decode of every slice from a guessed state spec_lead(S) bits
//                  before it (the first slice from the true one) to its exit; keeps the
//                  first block boundary past each of eight marks (checkpoints)
//   slice_match    slices whose predecessor's exit is their own first boundary are
//                  settled; the others are listed
//   slice_sync     (kSyncPasses passes) listed slices decode again from their
//                  predecessor's exit until they meet one of their checkpoints (then
//                  the rest is known) or their end; a changed exit lists the next slice
//   slice_fix      per interval with slices still listed: walks its slices in order
//                  until every start equals the previous exit. Then slice 0 starts in
//                  the true state and each exit is the true state at that point, so
//                  every start is the true one.
//   slice_prefix   per interval: block index and DC predictors at each slice start
//   slice_decode   from the true states: quantised AC levels, dequantised DC, and each
//                  slice's first event (an error, or the interval's last block completed)
//   slice_resolve  per interval: the earliest event in stream order becomes the
//                  interval's result, or the restart-marker check (entropy.rs:111-134)
//
// Errors are reported by the owner of the block they occur in, decoded a second time
// with the reference's checks in its order, so the earliest reported event is the one
// the serial decoder stops at.
//
// Both decodes are bound by the instructions per symbol and by how few lanes of a
// warp take the same path: a block ends every 10 to 60 symbols, at a different step
// in each lane, and what happens there (the next tables, the DC difference, 128
// bytes of levels) costs more than a symbol. So lanes take kSteps symbols (or pairs)
// at a time without a branch, a lane whose block has ended standing still (its table
// entry reads as zero), and the block ends are handled once per kSteps.
#include <cuda_runtime.h>

#include <algorithm>

#include "entropy_core.h"
#include "kernels.h"
#include "tables.h"

namespace mmr {
namespace {

constexpr unsigned long long kStErr = ~0ull;        // no state: the decode failed before this point
constexpr unsigned long long kStGuess = ~0ull - 1;  // start not yet derived from the predecessor
constexpr int kStride = 72;  // int16 per staged block: 64 levels, and 64.. for what EOB steps store
constexpr int kKeyBits = 26;
constexpr int kSpecSteps = 4;    // lookups between block-end checks, lean decode
constexpr int kDecodeSteps = 4;  // and final decode
constexpr uint32_t kTab = 1u << kHuffFastBits;
__constant__ uint8_t c_slice_zz[64] = MMR_ZIGZAG_INIT;
constexpr uint32_t kMostShared = 2;  // DC and AC tables a CTA keeps in shared memory, of each

__device__ __forceinline__ unsigned long long pack_state(unsigned long long p, uint32_t si) { return (p << 8) | si; }

// Bit offset of checkpoint q from the nominal slice start (UINT32_MAX past the slice).
__constant__ uint32_t c_slice_marks[kSliceCheckpoints] = {0, 64, 128, 256, 512, 768, 1024, 1536};

__device__ __forceinline__ uint32_t mark_of(uint32_t q, uint32_t S) {
    const uint32_t m = q < (uint32_t)kSliceCheckpoints ? c_slice_marks[q] : 0xffffffffu;
    return m < S ? m : 0xffffffffu;
}

struct SliceRef {
    uint32_t item, j;
    IvInfo v;
    bool last;
};

__device__ __forceinline__ bool slice_ref(const JpegLaunch &L, uint32_t slot, SliceRef &s) {
    s.item = L.slot_item[slot];
    if (s.item == 0xffffffffu) return false;
    s.v = L.ivs[s.item];
    s.j = slot - s.v.slot_first;
    s.last = s.j + 1 == s.v.n_slices;
    return true;
}

__device__ __forceinline__ uint32_t clamp_u32(unsigned long long x) {
    return x > 0xffffffffull ? 0xffffffffu : (uint32_t)x;
}

// ------------------------------------------------------------- reader ---
//
// The window is the 32 bits at offset `off` of two token words; the word after
// them is loaded one refill ahead. A symbol takes at most 27 bits, a pair 21.

struct Window {
    const uint32_t *next;  // the word after pf
    uint32_t w0, w1, pf;   // pf as stored (little-endian)
    uint32_t off;          // 0..31
};

__device__ __forceinline__ void window_init(Window &r, const uint8_t *tok, unsigned long long bit) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(tok) + (bit >> 5);
    r.w0 = bswap32(__ldg(w));
    r.w1 = bswap32(__ldg(w + 1));
    r.pf = __ldg(w + 2);
    r.next = w + 3;
    r.off = (uint32_t)bit & 31;
}

__device__ __forceinline__ uint32_t window_bits(const Window &r) { return __funnelshift_l(r.w1, r.w0, r.off); }

__device__ __forceinline__ void window_take(Window &r, uint32_t n) {
    r.off += n;
    if (r.off >= 32) {
        r.off -= 32;
        r.w0 = r.w1;
        r.w1 = bswap32(r.pf);
        r.pf = __ldg(r.next);
        r.next++;
    }
}

// Bits taken since the reader stood at bit `bit0` of the token stream at `tok`
// (modulo 2^32: a slice and its lead stay far below).
__device__ __forceinline__ uint32_t window_pos(const Window &r, const uint8_t *tok, uint32_t bit0) {
    return (uint32_t)(r.next - 3 - reinterpret_cast<const uint32_t *>(tok)) * 32 + r.off - bit0;
}

// The signed value of `size` magnitude bits at the top of t (receive_extend,
// entropy.rs:168-182); 0 for size 0.
__device__ __forceinline__ int32_t extend(uint32_t t, uint32_t size) {
    const uint32_t neg = (uint32_t)((int32_t)~t >> 31);
    uint32_t w;
    asm("shr.u32 %0, %1, %2;" : "=r"(w) : "r"(t ^ neg), "r"(32 - size));  // (a shift by 32 gives 0)
    return (int32_t)((w ^ neg) - neg);
}

// A code of more than kHuffFastBits bits: its entry (code bits past the first 11,
// magnitude size, advance), or the invalid marker.
__device__ __noinline__ uint32_t sub_entry(const JpegLaunch &L, uint32_t lut, uint32_t e, uint32_t window) {
    if (e == kSymInvalid) return e;
    return __ldg(L.sub + __ldg(L.sub_first + lut) + (e & 0x7fffu) * kSubEntries + ((window >> 16) & (kSubEntries - 1)));
}

// --------------------------------------------------------------- tables ---
//
// Lookup tables of the CTA's frame. Frames with at most two DC and two AC tables
// (all but exotic ones) keep them in shared memory, where 32 lanes' lookups cost a
// few bank conflicts instead of as many L1 lines; offsets count table entries from
// s_tab. Others read the batch's tables.

// What the lean decode needs of an MCU block: its component and tables (the frame's
// own numbers where they are in shared memory, else the batch's).
struct BlockTabs {
    uint32_t comp, dc, ac;
};

// ------------------------------------------------------------------ plan ---

constexpr int kPlanThreads = 512;
constexpr int kPlanPer = 8;  // consecutive intervals per thread and step

// CTA per frame: kPlanThreads * kPlanPer intervals per step, one prefix sum each (a
// warp per frame with 32 intervals per step took 6.0 ms of the 17.1 ms of a mixed
// batch whose 4:4:4 frames have up to 32k intervals).
__global__ void __launch_bounds__(kPlanThreads) slice_plan_kernel(JpegLaunch L) {
    __shared__ uint32_t s_warp[kPlanThreads / 32];
    const uint32_t f = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const JFrame &F = L.frames[f];
    if (!F.decode || F.ncomp > 4) return;
    const JState &st = L.states[f];
    const unsigned long long termv = st.term;
    const bool scan_ok = termv != ~0ull && !((termv >> 8) & 1);
    const uint32_t n_int = F.n_intervals;
    const uint32_t n_rst = min(st.n_rst, n_int), n_tok = st.n_tokens;
    const RstEntry *rst = L.rsts + F.rst_off;
    const uint32_t S = F.slice_bits;
    uint32_t used = 0;
    for (uint32_t c = 0; c < n_int; c += kPlanThreads * kPlanPer) {
        const uint32_t iv0 = c + tid * kPlanPer;
        uint32_t start[kPlanPer], barrier[kPlanPer], n_s[kPlanPer], sum = 0;
        uint32_t prev = iv0 == 0 ? 0 : iv0 - 1 < n_rst ? rst[iv0 - 1].tok : 0xffffffffu;
#pragma unroll
        for (int i = 0; i < kPlanPer; i++) {
            const uint32_t iv = iv0 + i;
            n_s[i] = 0;
            start[i] = prev;
            barrier[i] = prev;
            const uint32_t end = iv < n_rst ? rst[iv].tok : n_tok;
            // an interval that no RST precedes: an earlier one fails its restart check
            if (iv < n_int && scan_ok && prev != 0xffffffffu) {
                barrier[i] = end;
                n_s[i] = max(1u, (uint32_t)(((unsigned long long)(end - prev) * 8 + S - 1) / S));
            }
            prev = iv < n_rst ? end : 0xffffffffu;
            sum += n_s[i];
        }
        uint32_t incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= (uint32_t)d) incl += o;
        }
        __syncthreads();  // (the last step's sums are read)
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        uint32_t first = used + incl - sum, total = 0;
#pragma unroll
        for (uint32_t w = 0; w < kPlanThreads / 32; w++) {
            if (w < warp) first += s_warp[w];
            total += s_warp[w];
        }
        const bool fits = used + total <= F.slot_count;  // always: slot_count bounds the token count
#pragma unroll
        for (int i = 0; i < kPlanPer; i++) {
            const uint32_t iv = iv0 + i;
            if (!fits) n_s[i] = 0;
            if (iv < n_int) {
                const uint32_t mcu0 = iv * F.ri, mcu1 = min(mcu0 + F.ri, F.total_mcus);
                IvInfo v;
                v.start = start[i];
                v.barrier = barrier[i];
                v.slot_first = F.slot_first + first;
                v.n_slices = n_s[i];
                v.blocks = n_s[i] ? (mcu1 - mcu0) * F.sched_len : 0;
                v.flags = n_s[i] && iv < n_rst ? 1u : 0u;
                v.frame = f;
                v.pad = 0;
                L.ivs[F.item_base + iv] = v;
                L.iv_key[F.item_base + iv] = ~0ull;
                L.iv_pend[F.item_base + iv] = 0xffffffffu;
            }
            const bool own = n_s[i] <= 8;
            if (own)
                for (uint32_t x = 0; x < n_s[i]; x++) L.slot_item[F.slot_first + first + x] = F.item_base + iv;
            for (uint32_t m = __ballot_sync(0xffffffffu, !own); m; m &= m - 1) {  // the warp fills long ones
                const int src = __ffs(m) - 1;
                const uint32_t nt = __shfl_sync(0xffffffffu, n_s[i], src), ft = __shfl_sync(0xffffffffu, first, src);
                const uint32_t it = __shfl_sync(0xffffffffu, F.item_base + iv, src);
                for (uint32_t x = lane; x < nt; x += 32) L.slot_item[F.slot_first + ft + x] = it;
            }
            first += n_s[i];
        }
        if (fits) used += total;
    }
    for (uint32_t x = used + tid; x < F.slot_count; x += kPlanThreads) L.slot_item[F.slot_first + x] = 0xffffffffu;
}

// ------------------------------------------------------------ lean decode ---

// Tables as the lean decode reads them: kShared from the CTA's copies, else the batch's.
template <bool kShared>
struct LeanTabs {
    const uint32_t *skip;  // AC: one or two symbols per entry (huffman_lut.h)
    const uint16_t *sym;   // DC
    const uint32_t *local;   // kShared: per MCU block JBlockRec::local
    const uint32_t *ids;     // kShared: batch index of each of the frame's tables, DC then AC
    const JBlockRec *recs;   // the frame's records
    __device__ __forceinline__ uint32_t skip_at(uint32_t i) const { return kShared ? skip[i] : __ldg(skip + i); }
    __device__ __forceinline__ uint32_t sym_at(uint32_t i) const { return kShared ? sym[i] : __ldg(sym + i); }
    __device__ __forceinline__ uint32_t dc_lut(uint32_t t) const { return kShared ? ids[t] : t; }
    __device__ __forceinline__ uint32_t ac_lut(uint32_t t) const { return kShared ? ids[kMostShared + t] : t; }
    __device__ __forceinline__ BlockTabs block(uint32_t si) const {
        if (kShared) {
            const uint32_t p = local[si];
            return BlockTabs{p & 0xff, (p >> 8) & 0xff, p >> 16};
        }
        const JBlockRec &R = recs[si];
        return BlockTabs{R.comp, R.dc_lut, R.ac_lut};
    }
};

// State of a lean decode between block boundaries.
struct Lean {
    Window r;
    int k;           // next coefficient; 64 or 96 and more: the block is complete, 65..95: invalid
    uint32_t si;     // block of the MCU
    uint32_t tab;    // its AC table's first entry
    uint32_t blocks; // blocks started
};

// kSpecSteps lookups (none for a lane whose block has ended).
template <bool kShared>
__device__ __forceinline__ void lean_steps(const JpegLaunch &L, const LeanTabs<kShared> &T, Lean &s) {
#pragma unroll
    for (int u = 0; u < kSpecSteps; u++) {
        const uint32_t w = window_bits(s.r);
        uint32_t e = 0;
        if (s.k < 64) e = T.skip_at(s.tab + (w >> (32 - kHuffFastBits)));
        if (e & kSkipEscape) {
            const uint32_t lut = T.ac_lut(s.tab / kTab);
            const uint32_t x = sub_entry(L, lut, __ldg(L.sym + lut * kTab + (w >> (32 - kHuffFastBits))), w);
            if (x & kSymEscape) {
                e = 0;
                s.k = 80;
            } else {
                const uint32_t one = (kHuffFastBits + (x & 15) + ((x >> 4) & 15)) | ((x >> 8) & 127) << 5;
                e = one | one << 12;
            }
        }
        if (s.k + (int)((e >> 5) & 127) < 64) e >>= 12;  // the pair: its first symbol leaves the block open
        window_take(s.r, e & 31);
        s.k += (int)((e >> 5) & 127);
    }
}

// The DC symbol at a block boundary: counts the block, adds its difference to
// dc[component], and leaves the decode at its first AC symbol. False when invalid.
template <bool kShared>
__device__ __forceinline__ bool lean_dc(const JpegLaunch &L, const LeanTabs<kShared> &T, Lean &s, int32_t *dc) {
    const BlockTabs b = T.block(s.si);
    s.blocks++;
    uint32_t w = window_bits(s.r);
    uint32_t e = T.sym_at(b.dc * kTab + (w >> (32 - kHuffFastBits)));
    if (e & kSymEscape) {
        e = sub_entry(L, T.dc_lut(b.dc), e, w);
        if (e & kSymEscape) return false;
        window_take(s.r, kHuffFastBits);
        w = window_bits(s.r);
    }
    const uint32_t cl = e & 15, size = (e >> 4) & 15;
    dc[b.comp] += extend(w << cl, size);
    window_take(s.r, cl + size);
    s.tab = b.ac * kTab;
    s.k = 1;
    return true;
}

__device__ __forceinline__ bool lean_invalid(const Lean &s) { return s.k > 64 && s.k < 96; }

// Speculative decode of one slice (not its interval's last).
template <bool kShared>
__device__ __forceinline__ void spec_slice(const JpegLaunch &L, const LeanTabs<kShared> &T, const JFrame &F, uint32_t slot,
                           const SliceRef &s, int32_t *dc) {
    const bool guess = s.j != 0;
    const uint32_t S = F.slice_bits;
    const unsigned long long nominal = (unsigned long long)s.j * S;
    const uint32_t lead = guess ? (uint32_t)min((unsigned long long)spec_lead(S), nominal) : 0;
    const unsigned long long p0 = nominal - lead;  // positions below are from p0
    const uint32_t end = S + lead;
    const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
    const unsigned long long base = (unsigned long long)s.v.start * 8 + p0;
    const uint32_t bit0 = (uint32_t)base;
    Lean d;
    window_init(d.r, F.tok, base);
    d.blocks = 0;
    if (guess) {
        d.k = 1;
        d.si = 0;
        d.tab = T.block(0).ac * kTab;
    } else {
        d.k = 64;
        d.si = F.sched_len - 1;
        d.tab = 0;
    }
#pragma unroll
    for (int c = 0; c < 4; c++) dc[c] = 0;
    SliceSpec *sp = L.spec + slot;
    uint32_t q = 0, valid = 0, next_mark = lead;
    unsigned long long exit_state = kStErr;
    for (;;) {
        if (d.k >= 64) {
            const uint32_t pos = window_pos(d.r, F.tok, bit0);
            bool ok = !lean_invalid(d);
            if (ok) {
                d.si = d.si + 1 == F.sched_len ? 0 : d.si + 1;
                if (pos > lim) break;  // past the interval's end: exit_state stays kStErr
                if (pos >= next_mark) {
                    if (pos >= end) {
                        exit_state = pack_state(p0 + pos, d.si);
                        break;
                    }
                    SlicePoint cp;
                    cp.state = pack_state(p0 + pos, d.si);
                    cp.blocks = d.blocks;
                    cp.pad = 0;
#pragma unroll
                    for (int c = 0; c < 4; c++) cp.dc[c] = dc[c];
                    do {
                        if (guess) {
                            sp->cp[q] = cp;
                            valid |= 1u << q;
                        }
                        q++;
                        const uint32_t m = mark_of(q, S);
                        next_mark = m == 0xffffffffu ? end : m + lead;
                    } while (pos >= next_mark && next_mark < end);
                }
                ok = lean_dc(L, T, d, dc);
            }
            if (!ok) {
                if (!guess || pos >= min(lim, end)) break;
                // A decode from a guessed state met an invalid symbol: start again one bit
                // later; what came before cannot lead to the exit, so its checkpoints go.
                valid = 0;
                d.blocks = 0;
#pragma unroll
                for (int c = 0; c < 4; c++) dc[c] = 0;
                window_init(d.r, F.tok, base + pos + 1);
                d.k = 1;
                d.si = 0;
                d.tab = T.block(0).ac * kTab;
            }
        }
        lean_steps(L, T, d);
    }
    SliceSync out;
    out.start = guess ? kStGuess : pack_state(0, 0);
    out.exit = exit_state;
    out.blocks = d.blocks;
    out.q = kMatchStart;
#pragma unroll
    for (int c = 0; c < 4; c++) out.dc[c] = dc[c];
    L.sync[slot] = out;
    if (guess) {
        SlicePoint e;
        e.state = exit_state;
        e.blocks = d.blocks;
        e.pad = valid;
#pragma unroll
        for (int c = 0; c < 4; c++) e.dc[c] = dc[c];
        sp->exit = e;
    }
}

// Shared copies of the lean decode's tables: [kMostShared] DC (16-bit entries), then
// [kMostShared] AC pair tables, of the CTA's frame.
struct LeanSmem {
    uint32_t skip[kMostShared * kTab];
    uint16_t sym[kMostShared * kTab];
    uint32_t local[kMaxSched];
    uint32_t ids[2 * kMostShared];
    int32_t dc[kSliceThreads][4];
};

__device__ __forceinline__ void copy16(void *dst, const void *src, uint32_t bytes) {
    for (uint32_t i = threadIdx.x; i < bytes / 16; i += kSliceThreads)
        reinterpret_cast<uint4 *>(dst)[i] = __ldg(reinterpret_cast<const uint4 *>(src) + i);
}

__global__ void __launch_bounds__(kSliceThreads) slice_spec_kernel(JpegLaunch L) {
    __shared__ __align__(16) LeanSmem S;
    const uint32_t slot = blockIdx.x * kSliceThreads + threadIdx.x;
    SliceRef s;
    const bool used = slice_ref(L, slot, s);
    // the first slot of a CTA is used if any is, and all are of one frame
    const bool work = used && !s.last;
    if (used && s.last && s.j == 0) {  // (the decode pass takes a last slice's start from its predecessor)
        SliceSync y;
        y.start = y.exit = pack_state(0, 0);
        y.blocks = 0;
        y.q = kMatchStart;
#pragma unroll
        for (int c = 0; c < 4; c++) y.dc[c] = 0;
        L.sync[slot] = y;
    }
    if (!__syncthreads_or(work)) return;
    const JFrame &F = L.frames[L.ivs[L.slot_item[blockIdx.x * kSliceThreads]].frame];
    const bool small = F.n_dc <= kMostShared && F.n_ac <= kMostShared;
    if (small) {
        for (uint32_t i = threadIdx.x; i < F.sched_len; i += kSliceThreads) S.local[i] = L.brec[F.sched_off + i].local;
        for (uint32_t t = 0; t < F.n_dc; t++) copy16(S.sym + t * kTab, L.sym + F.dc_id[t] * kTab, 2 * kTab);
        for (uint32_t t = 0; t < F.n_ac; t++) copy16(S.skip + t * kTab, L.skip + F.ac_id[t] * kTab, 4 * kTab);
        if (threadIdx.x < kMostShared) {
            S.ids[threadIdx.x] = F.dc_id[threadIdx.x];
            S.ids[kMostShared + threadIdx.x] = F.ac_id[threadIdx.x];
        }
    }
    __syncthreads();
    if (!work) return;
    int32_t *dc = S.dc[threadIdx.x];
    if (small) {
        const LeanTabs<true> T{S.skip, S.sym, S.local, S.ids, nullptr};
        spec_slice(L, T, F, slot, s, dc);
    } else {
        const LeanTabs<false> T{L.skip, L.sym, nullptr, nullptr, L.brec + F.sched_off};
        spec_slice(L, T, F, slot, s, dc);
    }
}

// ----------------------------------------------------------------- match ---

// Settles a slice whose true start is its speculative decode's boundary at
// checkpoint q, given what lies before it: blocks and DC differences.
__device__ __forceinline__ void settle(const JpegLaunch &L, uint32_t slot, unsigned long long from, uint32_t q,
                                       uint32_t blocks, const int32_t *dc) {
    const SliceSpec *sp = L.spec + slot;
    const SlicePoint cp = sp->cp[q], e = sp->exit;
    SliceSync y;
    y.start = from;
    y.exit = e.state;
    y.blocks = blocks + e.blocks - cp.blocks;
    y.q = q;
#pragma unroll
    for (int c = 0; c < 4; c++) y.dc[c] = dc[c] + e.dc[c] - cp.dc[c];
    L.sync[slot] = y;
}

// Thread per slice: the predecessor's exit is the slice's own first boundary for
// most; the others go to the first list of the sync passes.
__global__ void __launch_bounds__(kSliceThreads) slice_match_kernel(JpegLaunch L) {
    const uint32_t slot = blockIdx.x * kSliceThreads + threadIdx.x, lane = threadIdx.x & 31;
    SliceRef s;
    bool list = false;
    if (slice_ref(L, slot, s) && s.j != 0 && !s.last) {
        const unsigned long long from = L.sync[slot - 1].exit;
        const int32_t none[4] = {0, 0, 0, 0};
        const bool same = (L.spec[slot].exit.pad & 1) && L.spec[slot].cp[0].state == from;
        if (same) settle(L, slot, from, 0, 0, none);
        list = !same;
    }
    const unsigned m = __ballot_sync(0xffffffffu, list);
    uint32_t base = 0;
    if (lane == 0 && m) base = atomicAdd(L.sync_count, (uint32_t)__popc(m));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (list) L.sync_list[base + __popc(m & ((1u << lane) - 1u))] = slot;
}

// ------------------------------------------------------------ sync pass ---

// Re-decodes slice `slot` (not the first, not the last) from state `from`, the
// exit of its predecessor, until it meets one of the slice's speculative
// checkpoints or passes the slice end. Returns whether the exit state changed.
__device__ bool resync_slice(const JpegLaunch &L, uint32_t slot, const SliceRef &s, unsigned long long from,
                             int32_t *dc) {
    const JFrame &F = L.frames[s.v.frame];
    const unsigned long long old_exit = L.sync[slot].exit;
    SliceSync y;
    y.start = from;
    y.exit = kStErr;
    y.blocks = 0;
    y.q = kMatchNone;
#pragma unroll
    for (int c = 0; c < 4; c++) {
        dc[c] = 0;
        y.dc[c] = 0;
    }
    if (from != kStErr) {
        const uint32_t S = F.slice_bits;
        const unsigned long long nominal = (unsigned long long)s.j * S, p0 = from >> 8;
        const uint32_t rel = clamp_u32(p0 - nominal);  // (a block may reach past the slice)
        const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
        const unsigned long long base = (unsigned long long)s.v.start * 8 + p0;
        const LeanTabs<false> T{L.skip, L.sym, nullptr, nullptr, L.brec + F.sched_off};
        const SliceSpec *sp = L.spec + slot;
        const uint32_t valid = sp->exit.pad;
        Lean d;
        window_init(d.r, F.tok, base);
        d.blocks = 0;
        d.k = 64;
        d.si = (uint32_t)(from & 0xff);
        d.tab = 0;
        uint32_t q = 0, next_mark = 0;
        bool first = true;
        for (;;) {
            if (d.k >= 64) {
                if (lean_invalid(d)) break;
                if (!first) d.si = d.si + 1 == F.sched_len ? 0 : d.si + 1;
                first = false;
                const uint32_t pos = window_pos(d.r, F.tok, (uint32_t)base);
                if (pos > lim) break;
                const uint32_t pn = pos + rel;
                if (pn >= S) {
                    y.exit = pack_state(p0 + pos, d.si);
                    break;
                }
                if (pn >= next_mark) {
                    const unsigned long long here = pack_state(p0 + pos, d.si);
                    bool met = false;
                    do {
                        met = (valid >> q & 1) && sp->cp[q].state == here;
                        if (!met) next_mark = mark_of(++q, S);
                    } while (!met && pn >= next_mark);
                    if (met) {  // the rest of the slice is the speculative decode's
                        settle(L, slot, from, q, d.blocks, dc);
                        return sp->exit.state != old_exit;
                    }
                }
                if (!lean_dc(L, T, d, dc)) break;
            }
            lean_steps(L, T, d);
        }
        y.blocks = d.blocks;
#pragma unroll
        for (int c = 0; c < 4; c++) y.dc[c] = dc[c];
    }
    L.sync[slot] = y;
    return y.exit != old_exit;
}

// Persistent threads take listed slots from a counter (re-decode lengths vary a lot;
// the lanes that reach the counter together take consecutive entries with one
// atomic). A changed exit lists the next slice for the pass after; after the last
// pass it is left to slice_fix_kernel, from the interval's first such slice on.
__global__ void __launch_bounds__(kSliceThreads) slice_sync_kernel(JpegLaunch L, uint32_t pass) {
    __shared__ int32_t s_dc[kSliceThreads][4];
    const uint32_t n = L.sync_count[pass];
    const uint32_t *list = L.sync_list + (uint64_t)(pass & 1) * L.n_slots;
    uint32_t *next_list = L.sync_list + (uint64_t)(~pass & 1) * L.n_slots;
    uint32_t *taken = L.sync_count + kSyncPasses + 1 + pass;
    const uint32_t lane = threadIdx.x & 31;
    for (;;) {
        const unsigned act = __activemask();
        const int leader = __ffs(act) - 1;
        uint32_t base = 0;
        if ((int)lane == leader) base = atomicAdd(taken, (uint32_t)__popc(act));
        base = __shfl_sync(act, base, leader);
        const uint32_t at = base + __popc(act & ((1u << lane) - 1u));
        if (at >= n) return;
        const uint32_t slot = list[at];
        SliceRef s;
        slice_ref(L, slot, s);
        const unsigned long long prev = *(volatile const unsigned long long *)&L.sync[slot - 1].exit;
        if (prev == L.sync[slot].start) continue;
        if (!resync_slice(L, slot, s, prev, s_dc[threadIdx.x]) || s.j + 2 >= s.v.n_slices) continue;
        if (pass + 1 < (uint32_t)kSyncPasses) next_list[atomicAdd(L.sync_count + pass + 1, 1u)] = slot + 1;
        else {
            atomicAdd(L.sync_count + kSyncPasses, 1u);
            atomicMin(L.iv_pend + s.item, slot + 1 - s.v.slot_first);
        }
    }
}

// One warp per interval that still has a listed slice.
__global__ void __launch_bounds__(kSliceThreads) slice_fix_kernel(JpegLaunch L) {
    __shared__ int32_t s_dc[kSliceThreads][4];
    if (L.sync_count[kSyncPasses] == 0) return;
    const uint32_t item = blockIdx.x * (kSliceThreads / 32) + threadIdx.x / 32;
    const uint32_t lane = threadIdx.x & 31;
    if (item >= L.n_items_small) return;
    const uint32_t pend = L.iv_pend[item];
    if (pend == 0xffffffffu) return;
    const IvInfo v = L.ivs[item];
    for (uint32_t c = pend; c + 1 < v.n_slices; c += 32) {  // (the last slice has no exit)
        for (;;) {
            const uint32_t j = c + lane;
            bool bad = false;
            if (j + 1 < v.n_slices) {
                const uint32_t slot = v.slot_first + j;
                bad = *(volatile unsigned long long *)&L.sync[slot].start !=
                      *(volatile unsigned long long *)&L.sync[slot - 1].exit;
            }
            const uint32_t m = __ballot_sync(0xffffffffu, bad);
            if (!m) break;
            if (lane == (uint32_t)__ffs(m) - 1) {
                const uint32_t slot = v.slot_first + j;
                SliceRef s;
                slice_ref(L, slot, s);
                resync_slice(L, slot, s, *(volatile unsigned long long *)&L.sync[slot - 1].exit, s_dc[threadIdx.x]);
                __threadfence_block();
            }
            __syncwarp();
        }
    }
}

// ---------------------------------------------------------------- prefix ---

constexpr int kPrefixThreads = 256;
constexpr uint32_t kPrefixLong = 512;  // slices an interval is worth the whole CTA from

struct SliceSums {
    uint32_t blocks;
    long long dc[4];
};

__device__ __forceinline__ void add_slice(const JpegLaunch &L, const IvInfo &v, uint32_t j, SliceSums &a) {
    if (j + 1 >= v.n_slices) return;  // the last slice's counts are never needed
    const SliceSync &y = L.sync[v.slot_first + j];
    a.blocks += y.blocks;
#pragma unroll
    for (int c = 0; c < 4; c++) a.dc[c] += y.dc[c];
}

// Inclusive prefix over the warp.
__device__ __forceinline__ void warp_prefix(SliceSums &a) {
    const uint32_t lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t b = __shfl_up_sync(0xffffffffu, a.blocks, o);
        long long d[4];
#pragma unroll
        for (int c = 0; c < 4; c++) d[c] = __shfl_up_sync(0xffffffffu, a.dc[c], o);
        if (lane >= (uint32_t)o) {
            a.blocks += b;
#pragma unroll
            for (int c = 0; c < 4; c++) a.dc[c] += d[c];
        }
    }
}

__device__ __forceinline__ void write_prefix(const JpegLaunch &L, const IvInfo &v, uint32_t j, const SliceSums &a) {
    SlicePrefix P;
    P.base = a.blocks;
    P.pad = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) P.dc[c] = a.dc[c];
    L.prefix[v.slot_first + j] = P;
}

// Warp per interval; intervals of many slices (scans without restart markers) are
// taken by the whole CTA, a run of slices per thread (a warp per interval took
// 1.5 ms for the 10k slices of 4K scans). One-slice intervals need no prefix.
__global__ void __launch_bounds__(kPrefixThreads) slice_prefix_kernel(JpegLaunch L) {
    __shared__ SliceSums s_warp[kPrefixThreads / 32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t item0 = blockIdx.x * (kPrefixThreads / 32), item = item0 + warp;
    if (item < L.n_items_small) {
        const IvInfo v = L.ivs[item];
        if (v.n_slices > 1 && v.n_slices < kPrefixLong) {
            SliceSums carry{};
            for (uint32_t c = 0; c < v.n_slices; c += 32) {
                SliceSums a{}, own{};
                add_slice(L, v, c + lane, own);
                a = own;
                warp_prefix(a);
                const SliceSums incl = a;
                a.blocks += carry.blocks - own.blocks;
#pragma unroll
                for (int q = 0; q < 4; q++) a.dc[q] += carry.dc[q] - own.dc[q];
                if (c + lane < v.n_slices) write_prefix(L, v, c + lane, a);
                carry.blocks += __shfl_sync(0xffffffffu, incl.blocks, 31);
#pragma unroll
                for (int q = 0; q < 4; q++) carry.dc[q] += __shfl_sync(0xffffffffu, incl.dc[q], 31);
            }
        }
    }
    for (uint32_t i = 0; i < kPrefixThreads / 32 && item0 + i < L.n_items_small; i++) {
        const IvInfo v = L.ivs[item0 + i];
        if (v.n_slices < kPrefixLong) continue;  // uniform over the CTA
        const uint32_t per = (v.n_slices + kPrefixThreads - 1) / kPrefixThreads;
        const uint32_t j0 = min(threadIdx.x * per, v.n_slices), j1 = min(j0 + per, v.n_slices);
        SliceSums own{};
        for (uint32_t j = j0; j < j1; j++) add_slice(L, v, j, own);
        SliceSums a = own;
        warp_prefix(a);
        __syncthreads();
        if (lane == 31) s_warp[warp] = a;
        __syncthreads();
        a.blocks -= own.blocks;
#pragma unroll
        for (int q = 0; q < 4; q++) a.dc[q] -= own.dc[q];
        for (uint32_t w = 0; w < warp; w++) {
            a.blocks += s_warp[w].blocks;
#pragma unroll
            for (int q = 0; q < 4; q++) a.dc[q] += s_warp[w].dc[q];
        }
        for (uint32_t j = j0; j < j1; j++) {
            write_prefix(L, v, j, a);
            add_slice(L, v, j, a);
        }
    }
}

// ---------------------------------------------------------------- decode ---

// Records a slice's first event: an error, or the interval's completion.
__device__ __forceinline__ void report(const JpegLaunch &L, const SliceRef &s, uint32_t slot, unsigned long long pos,
                                       const Diag &d, uint32_t complete) {
    SliceEvent e;
    e.diag = d;
    e.complete = complete;
    L.events[slot] = e;
    atomicMin(&L.iv_key[s.item], (pos << kKeyBits) | s.j);
}

// The block whose DC symbol starts at bit `at` of the interval failed: decodes it
// again with the reference's checks in its order (decoder.rs:501-546; the DC checks of
// :507-515 right after the DC symbol) and reports what the serial decoder stops at.
__device__ __noinline__ void report_bad_block(const JpegLaunch &L, const SliceRef &s, uint32_t slot,
                                              unsigned long long at, uint32_t si, long long pred) {
    const JFrame &F = L.frames[s.v.frame];
    const JBlockRec R = L.brec[F.sched_off + si];
    const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - at);
    Bits r;
    bits_init(r, F.tok, (uint64_t)s.v.start * 8 + at, 0);
    int k = 0;
    uint16_t kind = kDeviceError;  // (never kept: the fast decode only refuses what this one does)
    uint32_t errpos = 0, ev_at = 0;
    while (k < 64) {
        const uint32_t sym_at = r.used;
        const int k0 = k;
        int32_t val;
        uint16_t err;
        uint32_t eb;
        if (!decode_symbol(r, lim > sym_at ? lim - sym_at : 0, L.luts + (k0 == 0 ? R.dc_lut : R.ac_lut), L.symbols, k, val, err, eb)) {
            kind = err;
            errpos = eb;
            ev_at = sym_at;
            break;
        }
        if (k0 != 0) continue;
        const long long pn = pred + val, d = pn * (long long)R.q0;
        const bool pred_bad = pn > INT32_MAX || pn < INT32_MIN;
        if (pred_bad || d > INT32_MAX || d < INT32_MIN) {
            kind = pred_bad ? kJDcPredOverflow : kJDcDeqOverflow;
            errpos = r.used;
            break;
        }
    }
    Diag d;
    if (kind == kBarrierErr) {
        d = (s.v.flags & 1) ? make_diag(kJMarkerInData, s.v.barrier, 0xd0 + L.rsts[F.rst_off + L.items[s.item].y].number)
                            : make_diag(kJEndOfData, L.states[s.v.frame].n_tokens);
    } else {
        d = make_diag(kind, s.v.start + (uint32_t)((at + errpos + 7) / 8));
    }
    report(L, s, slot, at + ev_at, d, 0);
}

struct DecodeSmem {
    __align__(16) int16_t stage[kSliceThreads * kStride];
    __align__(16) uint16_t sym[2 * kMostShared * kTab];  // DC tables, then AC tables
    JBlockRec recs[kMaxSched];
    long long pred[4][kSliceThreads];
    uint32_t ids[2 * kMostShared];
    uint8_t zz[160];  // stage slot of k - 1: natural index, or past the block for EOB (k + 95 at most 158)
};

// What the final decode needs while it is in a slice.
struct Walk {
    Window r;
    int k;
    uint32_t tab;      // table of the next symbol: the block's DC table, then its AC table
    uint32_t ac;       // its AC table
};

// kDecodeSteps symbols (none for a lane whose block has ended): each level into the
// lane's stage; the DC difference at zigzag index 0.
template <bool kShared>
__device__ __forceinline__ void decode_steps(const JpegLaunch &L, const DecodeSmem &S, int16_t *stage, Walk &d) {
#pragma unroll
    for (int u = 0; u < kDecodeSteps; u++) {
        uint32_t w = window_bits(d.r);
        uint32_t e = 0;
        const uint32_t at = d.tab + (w >> (32 - kHuffFastBits));
        if (d.k < 64) e = kShared ? S.sym[at] : __ldg(L.sym + at);
        if (e & kSymEscape) {
            const uint32_t t = d.tab / kTab;
            e = sub_entry(L, kShared ? S.ids[t] : t, e, w);
            if (e & kSymEscape) {
                e = 0;
                d.k = 80;
            } else {
                window_take(d.r, kHuffFastBits);
                w = window_bits(d.r);
            }
        }
        const uint32_t cl = e & 15, size = (e >> 4) & 15;
        const int32_t val = extend(w << cl, size);
        const int k = d.k + (int)(e >> 8);
        if (e) stage[S.zz[k - 1]] = (int16_t)val;
        d.k = k;
        window_take(d.r, cl + size);
        d.tab = d.ac;
    }
}

// Warps stay together: lanes decode kDecodeSteps symbols, then those whose block is
// complete settle it (DC, address, the next block), and the warp writes the completed
// blocks together, eight lanes per block, as whole 128-byte lines.
template <bool kShared>
__device__ __forceinline__ void decode_slices(const JpegLaunch &L, DecodeSmem &S, const JFrame &F, uint32_t slot,
                                              const SliceRef &s, uint32_t n, unsigned long long from, uint32_t base) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    int16_t *stage = S.stage + tid * kStride;
    bool live = n != 0;
    Walk d;
    d.k = 128;
    d.tab = d.ac = 0;
    d.r.w0 = d.r.w1 = d.r.pf = d.r.off = 0;
    d.r.next = reinterpret_cast<const uint32_t *>(F.tok);
    const unsigned long long p0 = from >> 8;
    uint32_t si = (uint32_t)(from & 0xff), lim = 0, bit0 = 0, blk_at = 0;
    uint32_t mx = 0, my = 0, left = n;
    uint64_t blk = 0;
    int32_t q0 = 0;
    uint32_t comp = 0;
    auto setup = [&]() {
        const JBlockRec &R = S.recs[si];
        comp = R.comp;
        q0 = R.q0;
        blk = F.blk_off + R.base_off + mx * R.mul_x + (uint64_t)my * R.mul_y;
        if (kShared) {
            d.tab = ((R.local >> 8) & 0xff) * kTab;
            d.ac = (kMostShared + (R.local >> 16)) * kTab;
        } else {
            d.tab = R.dc_lut * kTab;
            d.ac = R.ac_lut * kTab;
        }
        d.k = 0;
    };
    if (live) {
        const unsigned long long b0 = (unsigned long long)s.v.start * 8 + p0;
        bit0 = (uint32_t)b0;
        lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
        window_init(d.r, F.tok, b0);
        const uint32_t mcu = L.items[s.item].y * F.ri + base / F.sched_len;
        my = mcu / F.mcu_cols;
        mx = mcu - my * F.mcu_cols;
        setup();
    }
    while (__any_sync(0xffffffffu, live)) {
        decode_steps<kShared>(L, S, stage, d);
        bool put = false;
        uint32_t to = 0;  // the completed block (the arena holds less than 2^32)
        if (live && d.k >= 64) {
            const uint32_t pos = window_pos(d.r, F.tok, bit0);
            const long long pn = S.pred[comp][tid] + stage[0], dq = pn * (long long)q0;
            const bool ok = (d.k == 64 || d.k >= 96) && pos <= lim && pn <= INT32_MAX && pn >= INT32_MIN &&
                            dq <= INT32_MAX && dq >= INT32_MIN;
            if (!ok) {
                report_bad_block(L, s, slot, p0 + blk_at, si, S.pred[comp][tid]);
                live = false;
            } else {
                S.pred[comp][tid] = pn;
                L.dc[blk] = (int32_t)dq;
                to = (uint32_t)blk;
                put = true;
                blk_at = pos;
                if (++base == s.v.blocks) {  // the interval's last block
                    const unsigned long long endbit = p0 + pos;
                    report(L, s, slot, endbit, make_diag(kDiagNone, s.v.start + (uint32_t)((endbit + 7) / 8)), 1);
                }
                live = --left != 0;
                if (++si == F.sched_len) {
                    si = 0;
                    if (++mx == F.mcu_cols) {
                        mx = 0;
                        my++;
                    }
                }
                if (live) setup();
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, put);
        while (m) {
            // lanes 8i .. 8i + 7 write the i-th block left
            unsigned mine = m;
            for (uint32_t i = 0; i < lane >> 3; i++) mine &= mine - 1;
            const int src = __ffs(mine) - 1;
            const uint32_t g = __shfl_sync(0xffffffffu, to, src & 31);
            if (src >= 0) {
                int4 *st = reinterpret_cast<int4 *>(S.stage + ((tid & ~31u) + src) * kStride) + (lane & 7);
                reinterpret_cast<int4 *>(L.coef + (uint64_t)g * 64)[lane & 7] = *st;
                *st = make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int i = 0; i < 4; i++) m &= m - 1;
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(kSliceThreads) slice_decode_kernel(JpegLaunch L) {
    extern __shared__ __align__(16) uint8_t s_raw[];
    DecodeSmem &S = *reinterpret_cast<DecodeSmem *>(s_raw);
    const uint32_t tid = threadIdx.x, slot = blockIdx.x * kSliceThreads + tid;
    SliceRef s;
    s.item = 0;
    const bool used = slice_ref(L, slot, s);
    // the blocks this slice decodes
    uint32_t n = 0, base = 0;
    unsigned long long from = 0;
    bool redone = false, whole = false;
    if (used) {
        if (s.v.n_slices > 1) {
            const SlicePrefix P = L.prefix[slot];
            base = P.base;
#pragma unroll
            for (int c = 0; c < 4; c++) S.pred[c][tid] = P.dc[c];
            from = s.j == 0 ? pack_state(0, 0) : L.sync[slot - 1].exit;
            if (!s.last) {
                const SliceSync &y = L.sync[slot];
                n = y.blocks;
                redone = s.j != 0 && y.q != 0;
                whole = y.q == kMatchNone;
            } else {
                n = 0xffffffffu;
            }
            n = from == kStErr || base >= s.v.blocks ? 0 : min(n, s.v.blocks - base);
        } else {
#pragma unroll
            for (int c = 0; c < 4; c++) S.pred[c][tid] = 0;
            from = pack_state(0, 0);
            n = s.v.blocks;
        }
    }
    const int n_used = __syncthreads_count(used), n_redone = __syncthreads_count(redone),
              n_whole = __syncthreads_count(whole);
    if (!n_used) return;
    if (tid == 0) {
        atomicAdd(L.fix_count + 3, (uint32_t)n_used);
        if (n_redone) atomicAdd(L.fix_count + 2, (uint32_t)n_redone);
        if (n_whole) atomicAdd(L.fix_count + 5, (uint32_t)n_whole);
    }
    const JFrame &F = L.frames[L.ivs[L.slot_item[blockIdx.x * kSliceThreads]].frame];
    const bool small = F.n_dc <= kMostShared && F.n_ac <= kMostShared;
    for (uint32_t i = tid; i < kSliceThreads * kStride / 8; i += kSliceThreads)
        reinterpret_cast<int4 *>(S.stage)[i] = make_int4(0, 0, 0, 0);
    for (uint32_t i = tid; i < 160; i += kSliceThreads) S.zz[i] = i < 64 ? c_slice_zz[i] : 64;
    copy16(S.recs, L.brec + F.sched_off, F.sched_len * (uint32_t)sizeof(JBlockRec));
    if (small) {
        for (uint32_t t = 0; t < F.n_dc; t++) copy16(S.sym + t * kTab, L.sym + F.dc_id[t] * kTab, 2 * kTab);
        for (uint32_t t = 0; t < F.n_ac; t++)
            copy16(S.sym + (kMostShared + t) * kTab, L.sym + F.ac_id[t] * kTab, 2 * kTab);
        if (tid < kMostShared) {
            S.ids[tid] = F.dc_id[tid];
            S.ids[kMostShared + tid] = F.ac_id[tid];
        }
    }
    __syncthreads();
    if (small) decode_slices<true>(L, S, F, slot, s, n, from, base);
    else decode_slices<false>(L, S, F, slot, s, n, from, base);
}

// --------------------------------------------------------------- resolve ---

__global__ void slice_resolve_kernel(JpegLaunch L) {
    const uint32_t item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= L.n_items_small) return;
    const IvInfo v = L.ivs[item];
    if (v.n_slices == 0) return;
    const uint2 it = L.items[item];
    const JFrame &F = L.frames[it.x];
    JState *st = L.states + it.x;
    const uint32_t iv = it.y;
    const unsigned long long key = L.iv_key[item];
    Diag out = make_diag(kDiagNone);
    if (key == ~0ull) {
        out = make_diag(kDeviceError);  // every decoded interval ends in an event
    } else {
        const SliceEvent e = L.events[v.slot_first + (uint32_t)(key & ((1u << kKeyBits) - 1))];
        if (!e.complete) {
            out = e.diag;
        } else if (iv + 1 < F.n_intervals) {
            // consume_restart before the next interval (entropy.rs:111-134)
            const uint32_t tend = e.diag.offset, expected = iv & 7, n_tok = st->n_tokens;
            const RstEntry *rst = L.rsts + F.rst_off;
            if ((v.flags & 1) && rst[iv].tok == tend) {
                if (rst[iv].number != expected) out = make_diag(kJRstMismatch, tend, expected, 0xd0 + rst[iv].number);
            } else if (tend < n_tok && F.tok[tend] == 0xff) {
                out = make_diag(kJRstMismatch, tend, expected, 0x00);
            } else {
                out = make_diag(kJExpectRst, tend);
            }
        }
    }
    L.results[item] = out;
    if (out.kind != kDiagNone) atomicMin(&st->bad_interval, iv);
}

}  // namespace

int jpeg_slice_launches(const JpegLaunch &L) { return L.n_items_small ? 7 + kSyncPasses : 0; }

void launch_jpeg_slices(const JpegLaunch &L, cudaStream_t s, cudaEvent_t *marks, bool capturing) {
    auto mark = [&](int k) {
        if (marks) capturing ? cudaEventRecordWithFlags(marks[k], s, cudaEventRecordExternal) : cudaEventRecord(marks[k], s);
    };
    const bool run = L.n_items_small && L.n_slots;
    const uint32_t grid = L.n_slots / kSliceThreads;  // (frames reserve whole CTAs of slots)
    const uint32_t warps = kSliceThreads / 32, pwarps = kPrefixThreads / 32;
    if (run) {
        slice_plan_kernel<<<L.n_frames, kPlanThreads, 0, s>>>(L);
        slice_spec_kernel<<<grid, kSliceThreads, 0, s>>>(L);
    }
    mark(0);
    if (run) {
        slice_match_kernel<<<grid, kSliceThreads, 0, s>>>(L);
        const uint32_t sync_grid = std::min<uint32_t>(grid, 152 * 8);
        for (uint32_t p = 0; p < (uint32_t)kSyncPasses; p++) slice_sync_kernel<<<sync_grid, kSliceThreads, 0, s>>>(L, p);
        slice_fix_kernel<<<(L.n_items_small + warps - 1) / warps, kSliceThreads, 0, s>>>(L);
        slice_prefix_kernel<<<(L.n_items_small + pwarps - 1) / pwarps, kPrefixThreads, 0, s>>>(L);
    }
    mark(1);
    if (run) slice_decode_kernel<<<grid, kSliceThreads, sizeof(DecodeSmem), s>>>(L);
    mark(2);
    if (run) slice_resolve_kernel<<<(L.n_items_small + 127) / 128, 128, 0, s>>>(L);
}

}  // namespace mmr
