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
//   slice_plan     per interval: token range, slices, slots
//   slice_spec     the lean decode of every slice from a guessed state JFrame::lead bits
//                  before it (the first slice from the true one) to its exit; keeps the
//                  first block boundary past each of eight marks (checkpoints). Small
//                  batches decode each slice from several guesses (JFrame::paths)
//   slice_sync     (one to kSyncPasses passes) a slice whose start is not its predecessor's exit
//                  takes it: where that is the first boundary of a speculative decode the
//                  rest is known, else it decodes again from there until it meets one of
//                  the checkpoints or its end; each CTA repeats this over its slices until
//                  nothing changes
//   slice_fix      per interval in which the last pass changed the last exit of a CTA:
//                  walks its slices in order until every start equals the previous exit.
//                  Then slice 0 starts in the true state and each exit is the true state
//                  at that point, so every start is the true one.
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
// warp take the same path: a block ends every 5 to 60 symbols, at a different step
// in each lane, and what happens there (the next tables, the DC difference, 128
// bytes of levels) costs more than a symbol. So lanes take a few symbols (or pairs)
// at a time without a branch, a lane whose block has ended, or whose next bits are no
// valid symbol, standing still (its table entry reads as zero), and what ended is
// handled once per group of steps.
#include <cuda_runtime.h>

#include <algorithm>

#include "entropy_core.h"
#include "kernels.h"
#include "launch.h"
#include "tables.h"

namespace mmr {
namespace {

constexpr unsigned long long kStErr = ~0ull;        // no state: the decode failed before this point
constexpr unsigned long long kStGuess = ~0ull - 1;  // start not yet derived from the predecessor

// Slices only ever take real states from their predecessors. After a true error the
// slices that follow keep what they guessed: they may decode nonsense, within their
// interval (slice_share), but events count by slice, so theirs come after the one that matters.
__device__ __forceinline__ bool is_state(unsigned long long x) { return x < kStGuess; }

constexpr int kStride = 72;  // int16 per staged block: 64 levels, and 64.. for what EOB steps store
constexpr int kSpecSteps = 4;  // lookups per group, lean decode
// Symbols per group, final decode. A group ends with the blocks that it completed, half of
// the instructions with four symbols to one: where warps are many, that is what counts
// (1422 M instructions, 1189 M with eight: 300 1080p frames 5.79 -> 5.67 ms); in small
// calls the wait for the group's other lanes does (320x240: 176 us, with eight 182).
constexpr int kDecodeSteps = 4, kDecodeStepsLong = 8;
__constant__ uint8_t c_slice_zz[64] = MMR_ZIGZAG_INIT;

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

// n < 32. Predicated, so that lanes crossing a word at different steps stay together.
__device__ __forceinline__ void window_take(Window &r, uint32_t n) {
    asm("{\n\t"
        ".reg .pred p;\n\t"
        "add.u32 %0, %0, %5;\n\t"
        "setp.ge.u32 p, %0, 32;\n\t"
        "@p mov.b32 %1, %2;\n\t"
        "@p prmt.b32 %2, %3, 0, 0x0123;\n\t"
        "@p ld.global.nc.u32 %3, [%4];\n\t"
        "@p add.u64 %4, %4, 4;\n\t"
        "and.b32 %0, %0, 31;\n\t"
        "}"
        : "+r"(r.off), "+r"(r.w0), "+r"(r.w1), "+r"(r.pf), "+l"(r.next)
        : "r"(n));
}

// What window_pos subtracts for positions counted from bit `bit0` of the tokens.
__device__ __forceinline__ uint32_t window_zero(const uint8_t *tok, unsigned long long bit0) {
    return (uint32_t)reinterpret_cast<uintptr_t>(tok) * 8 + 96 + (uint32_t)bit0;
}

// Position of the window (modulo 2^32: a slice and its lead stay far below).
__device__ __forceinline__ uint32_t window_pos(const Window &r, uint32_t zero) {
    return (uint32_t)reinterpret_cast<uintptr_t>(r.next) * 8 + r.off - zero;
}

// The signed value of `size` magnitude bits at the top of t (receive_extend,
// entropy.rs:168-182); 0 for size 0.
__device__ __forceinline__ int32_t extend(uint32_t t, uint32_t size) {
    const uint32_t neg = (uint32_t)((int32_t)~t >> 31);
    uint32_t w;
    asm("shr.u32 %0, %1, %2;" : "=r"(w) : "r"(t ^ neg), "r"(32 - size));  // (a shift by 32 gives 0)
    return (int32_t)((w ^ neg) - neg);
}

// --------------------------------------------------------------- tables ---
//
// Lookup tables as a decode reads them. Where a frame's tables fit (JFrame::
// shared_tabs: all but exotic ones) each CTA, whose slots are all of one frame, keeps
// them in shared memory: 32 lanes' lookups there cost a few bank conflicts instead of
// as many L1 lines, and no table byte is fetched from L2 in the middle of a decode.

// A table: its first entry (shared: byte address in shared memory; else entry in the
// batch's tables), and the window limits of lut_entry_index.
struct Tab {
    uint32_t at, first_long, last;
};

// Per MCU block: its component and tables.
struct BlockTabs {
    Tab dc, ac;
    uint32_t comp;
};

__device__ __forceinline__ Tab batch_tab(const JpegLaunch &L, uint32_t lut) {
    const LutMeta m = L.lut_meta[lut];
    return Tab{m.off, m.first_long, m.last};
}

__device__ __forceinline__ BlockTabs batch_tabs(const JpegLaunch &L, const JBlockRec &R) {
    return BlockTabs{batch_tab(L, R.dc_lut), batch_tab(L, R.ac_lut), R.comp};
}

// The sym or skip entry of window w; 0 unless `on`.
template <bool kShared>
__device__ __forceinline__ uint32_t sym_entry(const JpegLaunch &L, const Tab &t, uint32_t w, bool on) {
    uint32_t e = 0;
    if (kShared) {
        const uint32_t a = t.at + 2 * lut_entry_index(w, t.first_long);
        asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.shared.u16 %0, [%1];\n\t}"
            : "+r"(e) : "r"(a), "r"((uint32_t)on));
    } else if (on) {
        e = __ldg(L.sym + t.at + lut_entry_index(min(w, t.last), t.first_long));
    }
    return e;
}

template <bool kShared>
__device__ __forceinline__ uint32_t skip_entry(const JpegLaunch &L, const Tab &t, uint32_t w, int k) {
    uint32_t e = 0;
    if (kShared) {
        const uint32_t a = t.at + 4 * lut_entry_index(w, t.first_long);
        asm("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %2, 64;\n\t@p ld.shared.u32 %0, [%1];\n\t}"
            : "+r"(e) : "r"(a), "r"(k));
    } else if (k < 64) {
        e = __ldg(L.skip + t.at + lut_entry_index(min(w, t.last), t.first_long));
    }
    return e;
}

// (a multiple of 16 bytes; four loads in flight per thread)
__device__ __forceinline__ void copy16(void *dst, const void *src, uint32_t bytes) {
    const uint32_t n = bytes / 16;
    for (uint32_t i0 = threadIdx.x; i0 < n; i0 += 4 * kSliceThreads) {
        uint4 v[4];
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i0 + u * kSliceThreads < n) v[u] = __ldg(reinterpret_cast<const uint4 *>(src) + i0 + u * kSliceThreads);
#pragma unroll
        for (int u = 0; u < 4; u++)
            if (i0 + u * kSliceThreads < n) reinterpret_cast<uint4 *>(dst)[i0 + u * kSliceThreads] = v[u];
    }
}

__device__ __forceinline__ uint32_t shared_address(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ------------------------------------------------------------------ plan ---

// Thread per restart interval. An interval's slots start at its first token's bits / S
// plus its number: such ranges never overlap (floor(a) + ceil(b) <= floor(a + b) + 1)
// and need no prefix sum over the frame; slots between them stay unused. (A warp per
// frame, 32 intervals per step, took 6.0 of the 17.1 ms of a mixed batch whose 4:4:4
// frames have up to 32k intervals; a CTA per frame 0.36 ms.)
constexpr int kPlanThreads = 128;

// The last n_luts CTAs make the skip tables (host code took 13 us for one).
__global__ void __launch_bounds__(kPlanThreads) slice_plan_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    if (blockIdx.x + L.n_luts >= gridDim.x) {
        const LutMeta m = L.lut_meta[gridDim.x - 1 - blockIdx.x];
        for (uint32_t x = threadIdx.x; x < m.len; x += kPlanThreads)
            L.skip[m.off + x] = skip_entry_of(L.sym + m.off, m.first_long, x);
        return;
    }
    const uint32_t item = blockIdx.x * kPlanThreads + threadIdx.x, lane = threadIdx.x & 31;
    uint32_t first = 0, n_s = 0, limit = 0;  // slots [first, first + n_s) used, up to limit unused
    if (item < L.n_items_small) {
        const uint32_t f = L.items[item].x, iv = L.items[item].y;
        const JFrame &F = L.frames[f];
        const JState &st = L.states[f];
        const unsigned long long termv = st.term;
        const bool scan_ok = termv != ~0ull && !((termv >> 8) & 1);
        const uint32_t n_rst = min(st.n_rst, F.n_intervals), S = F.slice_bits;
        const RstEntry *rst = L.rsts + F.rst_off;
        uint32_t start = 0, end = 0;
        // an interval that no RST precedes: an earlier one fails its restart check
        const bool dec = scan_ok && iv <= n_rst;
        if (dec) {
            start = iv ? rst[iv - 1].tok : 0;
            end = iv < n_rst ? rst[iv].tok : st.n_tokens;
            n_s = max(1u, (uint32_t)(((unsigned long long)(end - start) * 8 + S - 1) / S));
            first = F.slot_first + (uint32_t)((unsigned long long)start * 8 / S) + iv;
            limit = iv == n_rst || iv + 1 == F.n_intervals
                        ? F.slot_first + F.slot_count
                        : F.slot_first + (uint32_t)((unsigned long long)end * 8 / S) + iv + 1;
        } else if (iv == 0) {
            first = F.slot_first;
            limit = first + F.slot_count;
        }
        const uint32_t mcu0 = iv * F.ri, mcu1 = min(mcu0 + F.ri, F.total_mcus);
        IvInfo v;
        v.start = start;
        v.barrier = end;
        v.slot_first = first;
        v.n_slices = n_s;
        v.blocks = (mcu1 - mcu0) * F.sched_len;
        v.flags = iv < n_rst ? 1u : 0u;
        v.frame = f;
        v.pad = 0;
        L.ivs[item] = v;
        L.iv_key[item] = ~0ull;
        L.iv_pend[item] = 0xffffffffu;
    }
    const bool own = limit - first <= 4;
    if (own)
        for (uint32_t x = first; x < limit; x++) L.slot_item[x] = x - first < n_s ? item : 0xffffffffu;
    for (uint32_t m = __ballot_sync(0xffffffffu, !own); m; m &= m - 1) {  // the warp fills longer ones
        const int src = __ffs(m) - 1;
        const uint32_t ft = __shfl_sync(0xffffffffu, first, src), nt = __shfl_sync(0xffffffffu, n_s, src);
        const uint32_t lt = __shfl_sync(0xffffffffu, limit, src), it = __shfl_sync(0xffffffffu, item, src);
        for (uint32_t x = ft + lane; x < lt; x += 32) L.slot_item[x] = x - ft < nt ? it : 0xffffffffu;
    }
}

// ------------------------------------------------------------ lean decode ---

// The lean decode's tables in shared memory: DC and AC (pair) tables of the CTA's
// frame, then per MCU block its BlockTabs.
struct LeanSmem {
    __align__(16) uint32_t skip[kSharedTabs][kSharedTab];
    __align__(16) uint16_t sym[kSharedTabs][kSharedTab];
    BlockTabs tabs[kMaxSched];
    int32_t dc[4][kSliceThreads];  // DC sums of the slice, per component
    uint32_t frame;
};

__device__ __forceinline__ void lean_load(const JpegLaunch &L, const JFrame &F, LeanSmem &S) {
    if (F.shared_tabs) {
        for (uint32_t t = 0; t < F.n_dc; t++) {
            const LutMeta m = L.lut_meta[F.dc_id[t]];
            copy16(S.sym[t], L.sym + m.off, 2 * m.len);
        }
        for (uint32_t t = 0; t < F.n_ac; t++) {
            const LutMeta m = L.lut_meta[F.ac_id[t]];
            copy16(S.skip[t], L.skip + m.off, 4 * m.len);
        }
    }
    for (uint32_t i = threadIdx.x; i < F.sched_len; i += kSliceThreads) {
        const JBlockRec &R = L.brec[F.sched_off + i];
        BlockTabs b = batch_tabs(L, R);
        if (F.shared_tabs) {
            b.dc.at = shared_address(S.sym[(R.local >> 8) & 0xff]);
            b.ac.at = shared_address(S.skip[R.local >> 16]);
        }
        S.tabs[i] = b;
    }
}

// State of a lean decode.
struct Lean {
    Window r;
    int k;            // next coefficient; 64 or from 96 on: the block is complete, 65..95: overrun
    uint32_t si;      // block of the MCU
    Tab ac;           // its AC table
    uint32_t blocks;  // blocks started
};

// kSpecSteps lookups (none for a lane whose block has ended). Returns 0 when the last
// one found no valid symbol (or the block has ended).
template <bool kShared>
__device__ __forceinline__ uint32_t lean_steps(const JpegLaunch &L, Lean &s) {
    uint32_t e = 0;
#pragma unroll
    for (int u = 0; u < kSpecSteps; u++) {
        e = skip_entry<kShared>(L, s.ac, window_bits(s.r), s.k);
        if (s.k + (int)(e >> 24) >= 64) e >>= 16;  // the first symbol ends the block: it alone
        window_take(s.r, e & 0xff);
        s.k += (int)((e >> 8) & 0xff);
    }
    return e;
}

__device__ __forceinline__ bool lean_complete(const Lean &s) { return s.k == 64 || s.k >= 96; }

// The DC symbol at a block boundary: counts the block, adds its difference to its
// component's sum, and leaves the decode at its first AC symbol. False when invalid.
template <bool kShared>
__device__ __forceinline__ bool lean_dc(const JpegLaunch &L, LeanSmem &S, Lean &s) {
    const BlockTabs &b = S.tabs[s.si];
    s.blocks++;
    const uint32_t w = window_bits(s.r);
    const uint32_t e = sym_entry<kShared>(L, b.dc, w, true), cl = e & 31, size = (e >> 5) & 15;
    S.dc[b.comp][threadIdx.x] += extend(w << cl, size);
    window_take(s.r, cl + size);
    s.ac = b.ac;
    s.k = 1;
    return e != 0;
}

__device__ __forceinline__ void lean_clear(LeanSmem &S, Lean &s) {
    s.blocks = 0;
#pragma unroll
    for (int c = 0; c < 4; c++) S.dc[c][threadIdx.x] = 0;
}

__device__ __forceinline__ void lean_point(const LeanSmem &S, const Lean &s, unsigned long long state, SlicePoint &p) {
    p.state = state;
    p.blocks = s.blocks;
#pragma unroll
    for (int c = 0; c < 4; c++) p.dc[c] = S.dc[c][threadIdx.x];
}

// Speculative decode `path` of one slice (not its interval's last).
template <bool kShared>
__device__ __forceinline__ void spec_slice(const JpegLaunch &L, LeanSmem &S, const JFrame &F, uint32_t slot,
                                           const SliceRef &s, uint32_t path) {
    const bool guess = s.j != 0;
    const uint32_t bits = F.slice_bits, sched_len = F.sched_len;
    const unsigned long long nominal = (unsigned long long)s.j * bits;
    const uint32_t lead = guess ? (uint32_t)min((unsigned long long)F.lead, nominal) : 0;
    const unsigned long long p0 = nominal - lead;  // positions below are from p0
    const uint32_t end = bits + lead;              // (less than lim: the next slice has a bit at least)
    const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
    const unsigned long long base = (unsigned long long)s.v.start * 8 + p0;
    const uint32_t zero = window_zero(F.tok, base);
    Lean d;
    window_init(d.r, F.tok, base);
    lean_clear(S, d);
    const uint32_t si0 = path * sched_len / F.paths;  // paths guess different blocks of the MCU
    d.ac = S.tabs[si0].ac;
    d.k = guess ? 1 : 64;
    d.si = guess ? si0 : sched_len - 1;
    SliceSpec *sp = L.spec + (uint64_t)path * L.n_slots + slot;
    uint32_t q = 0, valid = 0, next_mark = lead, e = 1;
    unsigned long long exit_state = kStErr;
    for (;;) {
        if (d.k >= 64 || e == 0) {
            const uint32_t pos = window_pos(d.r, zero);
            bool ok = lean_complete(d);
            if (ok) {
                d.si = d.si + 1 == sched_len ? 0 : d.si + 1;
                if (pos >= next_mark) {
                    const unsigned long long here = pack_state(p0 + pos, d.si);
                    if (pos >= end) {
                        if (pos <= lim) exit_state = here;  // (else past the interval's end)
                        break;
                    }
                    do {
                        if (guess) {
                            SlicePoint cp;
                            lean_point(S, d, here, cp);
                            cp.pad = 0;
                            sp->cp[q] = cp;
                            valid |= 1u << q;
                        }
                        const uint32_t m = mark_of(++q, bits);
                        next_mark = m == 0xffffffffu ? end : m + lead;
                    } while (pos >= next_mark && next_mark < end);
                }
                ok = lean_dc<kShared>(L, S, d);
            }
            if (!ok) {
                if (!guess || pos >= min(lim, end)) break;
                // A decode from a guessed state met an invalid symbol: start again one bit
                // later; what came before cannot lead to the exit, so its checkpoints go.
                valid = 0;
                lean_clear(S, d);
                window_init(d.r, F.tok, base + pos + 1);
                d.k = 1;
                d.si = si0;
                d.ac = S.tabs[si0].ac;
            }
        }
        e = lean_steps<kShared>(L, d);
    }
    SlicePoint x;
    lean_point(S, d, exit_state, x);
    x.pad = valid;
    if (guess) sp->exit = x;
    if (path != 0) return;
    SliceSync out;
    out.start = guess ? kStGuess : pack_state(0, 0);
    out.exit = exit_state;
    out.blocks = x.blocks;
    out.q = kMatchStart;
#pragma unroll
    for (int c = 0; c < 4; c++) out.dc[c] = x.dc[c];
    L.sync[slot] = out;
}

__global__ void __launch_bounds__(kSliceThreads) slice_spec_kernel(JpegLaunch L, uint32_t spread) {
    begin_kernel(L.early);
    __shared__ LeanSmem S;
    const uint32_t at = blockIdx.x * kSliceThreads + threadIdx.x, slot = at >> spread;
    SliceRef s;
    // (a last slice has no exit, and the decode pass takes its start from its predecessor)
    const uint32_t path = blockIdx.y;
    bool work = slot << spread == at && slice_ref(L, slot, s) && !s.last;
    if (work) {
        S.frame = s.v.frame;  // the same for all
        work = path == 0 || (s.j != 0 && path < L.frames[s.v.frame].paths);
    }
    if (!__syncthreads_or(work)) return;
    const JFrame &F = L.frames[S.frame];
    lean_load(L, F, S);
    __syncthreads();
    if (!work) return;
    if (F.shared_tabs) spec_slice<true>(L, S, F, slot, s, path);
    else spec_slice<false>(L, S, F, slot, s, path);
}

// ------------------------------------------------------------------ sync ---

// Settles a slice whose true decode, from `from`, is its speculative decode from
// checkpoint q on, given what lies before it; y.blocks and y.dc hold that.
__device__ __forceinline__ void settle(const SliceSpec *sp, uint32_t q, SliceSync &y) {
    const SlicePoint cp = sp->cp[q], e = sp->exit;
    y.exit = e.state;
    y.q = q;
    y.blocks += e.blocks - cp.blocks;
#pragma unroll
    for (int c = 0; c < 4; c++) y.dc[c] += e.dc[c] - cp.dc[c];
}

// The speculative decode of the slice that passes checkpoint q in state `here`.
__device__ __forceinline__ const SliceSpec *meets(const JpegLaunch &L, uint32_t slot, uint32_t paths, uint32_t q,
                                                  unsigned long long here) {
    const SliceSpec *found = nullptr;
    for (uint32_t h = 0; h < paths; h++) {
        const SliceSpec *sp = L.spec + (uint64_t)h * L.n_slots + slot;
        if ((sp->exit.pad >> q & 1) && sp->cp[q].state == here) found = sp;
    }
    return found;
}

// What slice `slot` (not the first, not the last) gives from state `from`, the exit of
// its predecessor: it decodes until it meets one of its speculative checkpoints or
// passes its end.
template <bool kShared>
__device__ __forceinline__ void resync_slice(const JpegLaunch &L, LeanSmem &S, const JFrame &F, uint32_t slot,
                                             const SliceRef &s, unsigned long long from, SliceSync &y) {
    y.start = from;
    y.exit = kStErr;
    y.blocks = 0;
    y.q = kMatchNone;
#pragma unroll
    for (int c = 0; c < 4; c++) y.dc[c] = 0;
    const uint32_t bits = F.slice_bits, sched_len = F.sched_len;
    const unsigned long long nominal = (unsigned long long)s.j * bits, p0 = from >> 8;
    const uint32_t rel = clamp_u32(p0 - nominal);  // (a block may reach past the slice)
    const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
    const unsigned long long base = (unsigned long long)s.v.start * 8 + p0;
    const uint32_t zero = window_zero(F.tok, base);
    const uint32_t paths = F.paths;
    Lean d;
    window_init(d.r, F.tok, base);
    lean_clear(S, d);
    d.ac = S.tabs[0].ac;
    d.k = 64;
    const uint32_t si0 = (uint32_t)(from & 0xff);
    d.si = si0 == 0 ? sched_len - 1 : si0 - 1;
    uint32_t q = 0, next_mark = 0, e = 1;
    const SliceSpec *met = nullptr;
    for (;;) {
        if (d.k >= 64 || e == 0) {
            if (!lean_complete(d)) break;
            d.si = d.si + 1 == sched_len ? 0 : d.si + 1;
            const uint32_t pos = window_pos(d.r, zero), pn = pos + rel;
            if (pn >= min(next_mark, bits)) {
                const unsigned long long here = pack_state(p0 + pos, d.si);
                if (pn >= bits) {
                    if (pos <= lim) y.exit = here;
                    break;
                }
                do {
                    met = meets(L, slot, paths, q, here);
                    if (!met) next_mark = mark_of(++q, bits);
                } while (!met && pn >= next_mark);
                if (met) break;
            }
            if (!lean_dc<kShared>(L, S, d)) break;
        }
        e = lean_steps<kShared>(L, d);
    }
    y.blocks = d.blocks;
#pragma unroll
    for (int c = 0; c < 4; c++) y.dc[c] = S.dc[c][threadIdx.x];
    if (met) settle(met, q, y);
}

// A CTA's slices take their predecessors' exits until nothing changes. A slice whose
// predecessor's exit is the first boundary of one of its speculative decodes takes that
// one's exit, from registers: these steps are repeated until none changes anything
// (wrong exits die out within a few slices), and only then do the slices that no
// speculative decode fits decode again, from tables loaded for them. (Decoding again
// at once, half of it from exits that were still wrong, took 1.3 ms of the 1.9 ms of
// 30 restart-less 4:2:0 VGA frames.) The slice before the CTA's first is read once:
// what another CTA still changes there is the next pass's, and after the last pass
// slice_fix_kernel's, from the interval's first such slice on.
__global__ void __launch_bounds__(kSliceThreads) slice_sync_kernel(JpegLaunch L, bool first_pass, bool last_pass) {
    begin_kernel(L.early);
    __shared__ LeanSmem S;
    __shared__ unsigned long long s_exit[kSliceThreads + 1];  // of the slice before the CTA's first, then of each
    const uint32_t tid = threadIdx.x, slot = blockIdx.x * kSliceThreads + tid;
    SliceRef s;
    bool work = slice_ref(L, slot, s) && !s.last;
    unsigned long long start = 0, exit = 0, entry[kMostPaths], leave[kMostPaths];
    unsigned long long stored = 0;  // the exit that the next CTA finds in L.sync
    if (work) {
        S.frame = s.v.frame;
        const uint32_t paths = L.frames[s.v.frame].paths;
        start = L.sync[slot].start;
        exit = stored = L.sync[slot].exit;
#pragma unroll
        for (uint32_t h = 0; h < kMostPaths; h++) {
            entry[h] = leave[h] = kStGuess;  // (never an exit)
            if (s.j == 0 || h >= paths) continue;
            const SliceSpec *sp = L.spec + (uint64_t)h * L.n_slots + slot;
            leave[h] = sp->exit.state;
            if (sp->exit.pad & 1) entry[h] = sp->cp[0].state;
        }
        if (start == kStGuess) {  // to begin with, the exit most decodes agree on
            uint32_t most = 0;
#pragma unroll
            for (uint32_t h = 0; h < kMostPaths; h++) {
                uint32_t n = 0;
#pragma unroll
                for (uint32_t i = 0; i < kMostPaths; i++) n += leave[i] == leave[h];
                if (is_state(leave[h]) && n > most) {
                    most = n;
                    exit = leave[h];
                }
            }
        }
        if (tid == 0 && s.j != 0) s_exit[0] = *(volatile const unsigned long long *)&L.sync[slot - 1].exit;
    }
    work = work && s.j != 0;
    s_exit[tid + 1] = exit;
    __syncthreads();
    if (!first_pass && !__syncthreads_or(work && is_state(s_exit[tid]) && s_exit[tid] != start)) return;
    bool loaded = false, told = false;         // (whether another exit than `stored` was ever in L.sync)
    uint32_t met = kMostPaths;                 // the speculative decode the slice takes, if it changes
    unsigned long long refused = kStGuess;     // an exit no speculative decode fits
    for (;;) {
        for (;;) {
            const unsigned long long from = work ? s_exit[tid] : 0;
            bool take = false;
            if (work && is_state(from) && from != start && from != refused) {
                uint32_t m = kMostPaths;
#pragma unroll
                for (uint32_t h = 0; h < kMostPaths; h++)
                    if (entry[h] == from) m = h;
                if (m < kMostPaths) {
                    take = true;
                    met = m;
                    start = from;
#pragma unroll
                    for (uint32_t h = 0; h < kMostPaths; h++)
                        if (m == h) exit = leave[h];
                } else {
                    refused = from;
                }
            }
            if (!__syncthreads_or(take)) break;  // (everyone has read the exits)
            if (take) s_exit[tid + 1] = exit;
            __syncthreads();
        }
        const unsigned long long from = work ? s_exit[tid] : 0;
        const bool go = work && is_state(from) && from != start;
        if (!__syncthreads_or(go)) break;
        const JFrame &F = L.frames[S.frame];
        if (!loaded) {
            lean_load(L, F, S);
            loaded = true;
            __syncthreads();
        }
        if (go) {
            SliceSync y;
            if (F.shared_tabs) resync_slice<true>(L, S, F, slot, s, from, y);
            else resync_slice<false>(L, S, F, slot, s, from, y);
            L.sync[slot] = y;
            told |= y.exit != stored;
            met = kMostPaths;
            start = from;
            exit = y.exit;
            s_exit[tid + 1] = exit;
        }
        __syncthreads();
    }
    if (met < kMostPaths) {
        const SliceSpec *sp = L.spec + (uint64_t)met * L.n_slots + slot;
        SliceSync y;
        y.start = start;
        y.blocks = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) y.dc[c] = 0;
        settle(sp, 0, y);
        L.sync[slot] = y;
    }
    // (`stored` is path 0's exit where the slice had no start yet, whatever most guesses agree on)
    if (last_pass && tid == kSliceThreads - 1 && work && (told || exit != stored) && s.j + 2 < s.v.n_slices) {
        atomicAdd(L.sync_left, 1u);
        atomicMin(L.iv_pend + s.item, s.j + 1);
    }
}

// One warp per interval that the sync passes left unsettled.
__global__ void __launch_bounds__(kSliceThreads) slice_fix_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    __shared__ LeanSmem S;
    if (*L.sync_left == 0) return;
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = 0; i < kSliceThreads / 32; i++) {  // (one interval of the CTA's four at a time: they share the tables)
        const uint32_t item = blockIdx.x * (kSliceThreads / 32) + i;
        if (item >= L.n_items_small) return;
        const uint32_t pend = L.iv_pend[item];
        if (pend == 0xffffffffu) continue;
        const IvInfo v = L.ivs[item];
        const JFrame &F = L.frames[v.frame];
        __syncthreads();
        lean_load(L, F, S);
        __syncthreads();
        if (threadIdx.x >= 32) continue;
        for (uint32_t c = pend; c + 1 < v.n_slices; c += 32) {  // (the last slice has no exit)
            for (;;) {
                const uint32_t j = c + lane, slot = v.slot_first + j;
                unsigned long long from = 0;
                bool bad = false;
                if (j + 1 < v.n_slices) {
                    from = *(volatile unsigned long long *)&L.sync[slot - 1].exit;
                    bad = is_state(from) && *(volatile unsigned long long *)&L.sync[slot].start != from;
                }
                const uint32_t m = __ballot_sync(0xffffffffu, bad);
                if (!m) break;
                if (lane == (uint32_t)__ffs(m) - 1) {
                    SliceRef s;
                    slice_ref(L, slot, s);
                    SliceSync y;
                    if (F.shared_tabs) resync_slice<true>(L, S, F, slot, s, from, y);
                    else resync_slice<false>(L, S, F, slot, s, from, y);
                    L.sync[slot] = y;
                    __threadfence_block();
                }
                __syncwarp();
            }
        }
    }
}

// ---------------------------------------------------------------- prefix ---

constexpr int kPrefixThreads = 512;
constexpr uint32_t kPrefixCtas = 4 * 152;      // as many as run at a time
constexpr uint32_t kPrefixLong = 192;  // slices an interval is worth the whole CTA from

struct SliceSums {
    uint32_t blocks;
    long long dc[4];
};

__device__ __forceinline__ void add_slice(const JpegLaunch &L, const IvInfo &v, uint32_t j, SliceSums &a) {
    if (j + 1 >= v.n_slices) return;  // the last slice's counts are never needed
    const SliceSync &y = L.sync[v.slot_first + j];
    a.blocks += __ldg(&y.blocks);
#pragma unroll
    for (int c = 0; c < 4; c++) a.dc[c] += __ldg(&y.dc[c]);
}

// Inclusive prefix over the warp's first n lanes.
__device__ __forceinline__ void warp_prefix(SliceSums &a, uint32_t n) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t o = 1; o < n; o <<= 1) {
        const uint32_t b = __shfl_up_sync(0xffffffffu, a.blocks, o);
        long long d[4];
#pragma unroll
        for (int c = 0; c < 4; c++) d[c] = __shfl_up_sync(0xffffffffu, a.dc[c], o);
        if (lane >= o) {
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

// Prefixes of slices [j0, j1) after the sums `carry`, by one warp.
__device__ __forceinline__ void prefix_run(const JpegLaunch &L, const IvInfo &v, uint32_t j0, uint32_t j1, SliceSums carry) {
    for (uint32_t c = j0; c < j1; c += 32) {
        const uint32_t j = c + (threadIdx.x & 31);
        SliceSums own{};
        if (j < j1) add_slice(L, v, j, own);
        SliceSums a = own;
        warp_prefix(a, min(j1 - c, 32u));
        const SliceSums incl = a;
        a.blocks += carry.blocks - own.blocks;
#pragma unroll
        for (int q = 0; q < 4; q++) a.dc[q] += carry.dc[q] - own.dc[q];
        if (j < j1) write_prefix(L, v, j, a);
        if (c + 32 >= j1) break;
        carry.blocks += __shfl_sync(0xffffffffu, incl.blocks, 31);
#pragma unroll
        for (int q = 0; q < 4; q++) carry.dc[q] += __shfl_sync(0xffffffffu, incl.dc[q], 31);
    }
}

// Warp per interval; intervals of many slices (scans without restart markers) are
// taken by the whole CTA, a run of slices per warp: its sum, then its prefixes (a warp per
// interval took 1.5 ms for the 10k slices of 4K scans). One-slice intervals need no prefix.
//
// A chain of loads and shuffles. A CTA takes `per_cta` intervals, up to one a warp: long
// ones are taken one after another, so a CTA takes one while they fit on the GPU at a time
// (30 VGA scans without markers in two CTAs: 37 us, in thirty: 7). Consecutive lanes take
// consecutive slices (a run of slices per thread touched a line per lane and load: 250 us
// against 147 in a step of 64 mixed frames).
__global__ void __launch_bounds__(kPrefixThreads) slice_prefix_kernel(JpegLaunch L, uint32_t per_cta) {
    begin_kernel(L.early);
    constexpr uint32_t kWarps = kPrefixThreads / 32;
    __shared__ SliceSums s_warp[kWarps];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t item0 = blockIdx.x * per_cta, n = min(per_cta, L.n_items_small - item0);
    bool any_long = false;
    if (warp < n) {
        const IvInfo v = L.ivs[item0 + warp];
        any_long = v.n_slices >= kPrefixLong;
        if (v.n_slices > 1 && !any_long) prefix_run(L, v, 0, v.n_slices, SliceSums{});
    }
    if (!__syncthreads_or(any_long)) return;
    for (uint32_t i = 0; i < n; i++) {
        const IvInfo v = L.ivs[item0 + i];
        if (v.n_slices < kPrefixLong) continue;  // uniform over the CTA
        const uint32_t run = (v.n_slices + kPrefixThreads - 1) / kPrefixThreads * 32;
        const uint32_t j0 = min(warp * run, v.n_slices), j1 = min(j0 + run, v.n_slices);
        SliceSums a{};
#pragma unroll 4
        for (uint32_t j = j0 + lane; j < j1; j += 32) add_slice(L, v, j, a);
        warp_prefix(a, 32);
        __syncthreads();  // (the last interval's sums are read)
        if (lane == 31) s_warp[warp] = a;
        __syncthreads();
        SliceSums carry{};
        for (uint32_t w = 0; w < warp; w++) {
            carry.blocks += s_warp[w].blocks;
#pragma unroll
            for (int q = 0; q < 4; q++) carry.dc[q] += s_warp[w].dc[q];
        }
        prefix_run(L, v, j0, j1, carry);
    }
}

// ---------------------------------------------------------------- decode ---

// Records a slice's first event: an error, or the interval's completion.
__device__ __forceinline__ void report(const JpegLaunch &L, const SliceRef &s, uint32_t slot, const Diag &d,
                                       uint32_t complete) {
    SliceEvent e;
    e.diag = d;
    e.complete = complete;
    L.events[slot] = e;
    atomicMin(&L.iv_key[s.item], (unsigned long long)s.j);
}

// The block whose DC symbol starts at bit `at` of the interval failed: decodes it
// again with the reference's checks in its order (decoder.rs:501-546; the DC checks of
// :507-515 right after the DC symbol) and reports what the serial decoder stops at.
__device__ __noinline__ void report_bad_block(const JpegLaunch &L, const SliceRef &s, uint32_t slot,
                                              unsigned long long at, uint32_t si, int32_t pred) {
    const JFrame &F = L.frames[s.v.frame];
    const JBlockRec R = L.brec[F.sched_off + si];
    const uint32_t lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - at);
    Bits r;
    bits_init(r, F.tok, (uint64_t)s.v.start * 8 + at, 0);
    int k = 0;
    uint16_t kind = kDeviceError;  // (never kept: the fast decode only refuses what this one does)
    uint32_t errpos = 0;
    while (k < 64) {
        const uint32_t sym_at = r.used;
        const int k0 = k;
        int32_t val;
        uint16_t err;
        uint32_t eb;
        refill(r);
        if (!checked_symbol(r, lim > sym_at ? lim - sym_at : 0, L.canon + (k0 == 0 ? R.dc_lut : R.ac_lut), L.symbols, k,
                            val, err, eb)) {
            kind = err;
            errpos = eb;
            break;
        }
        if (k0 != 0) continue;
        const long long pn = (long long)pred + val, d = pn * (long long)R.q0;
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
    report(L, s, slot, d, 0);
}

struct DecodeSmem {
    __align__(16) int16_t stage[kSliceThreads * kStride];
    __align__(16) uint16_t sym[2 * kSharedTabs][kSharedTab];  // DC tables, then AC tables
    BlockTabs tabs[kMaxSched];
    uint32_t base_off[kMaxSched], mul_x[kMaxSched], mul_y[kMaxSched];
    int32_t q0[kMaxSched];
    int32_t pred[4][kSliceThreads];
    uint32_t frame;
    uint8_t zz[160];  // stage slot of k - 1: natural index, or past the block for EOB (k + 95 at most 158)
};

// Warps stay together: lanes decode kSteps AC symbols, then those whose block is
// complete settle it and decode the next block's DC symbol, and the warp writes the
// completed blocks together, eight lanes per block, as whole 128-byte lines.
template <bool kShared, int kSteps>
__device__ __forceinline__ void decode_slices(const JpegLaunch &L, DecodeSmem &S, const JFrame &F, uint32_t slot,
                                              const SliceRef &s, uint32_t n, unsigned long long from, uint32_t base) {
    const uint32_t tid = threadIdx.x, lane = tid & 31;
    const uint32_t stage = shared_address(S.stage + tid * kStride), zz = shared_address(S.zz);
    const uint32_t sched_len = F.sched_len, mcu_cols = F.mcu_cols, blk_off = (uint32_t)F.blk_off;
    bool live = n != 0;
    Window r;
    r.w0 = r.w1 = r.pf = r.off = 0;
    r.next = reinterpret_cast<const uint32_t *>(F.tok);
    Tab ac{0, 0xffffffffu, 0};
    int k = 128;  // (no block yet, nothing to step)
    const unsigned long long p0 = from >> 8;
    uint32_t si = (uint32_t)(from & 0xff), lim = 0, zero = 0, blk_at = 0, left = n;
    uint32_t mx = 0, my = 0, blk = 0, e = 1;
    int32_t diff = 0;
    bool bad_dc = false;
    // the DC symbol of block si of MCU (mx, my), at bit blk_at
    auto begin = [&]() {
        const BlockTabs &b = S.tabs[si];
        blk = blk_off + S.base_off[si] + mx * S.mul_x[si] + my * S.mul_y[si];
        const uint32_t w = window_bits(r);
        const uint32_t x = sym_entry<kShared>(L, b.dc, w, true), cl = x & 31, size = (x >> 5) & 15;
        diff = extend(w << cl, size);
        window_take(r, cl + size);
        ac = b.ac;
        bad_dc = x == 0;
        k = 1;
    };
    if (live) {
        const unsigned long long b0 = (unsigned long long)s.v.start * 8 + p0;
        zero = window_zero(F.tok, b0);
        lim = clamp_u32((unsigned long long)(s.v.barrier - s.v.start) * 8 - p0);
        window_init(r, F.tok, b0);
        const uint32_t mcu = L.items[s.item].y * F.ri + base / sched_len;
        my = mcu / mcu_cols;
        mx = mcu - my * mcu_cols;
        begin();
    }
    while (__any_sync(0xffffffffu, live)) {
#pragma unroll
        for (int u = 0; u < kSteps; u++) {
            const uint32_t w = window_bits(r);
            e = sym_entry<kShared>(L, ac, w, k < 64);
            const uint32_t cl = e & 31, size = (e >> 5) & 15;
            const int32_t val = extend(w << cl, size);
            k += (int)(e >> 9);
            asm volatile("{\n\t"
                         ".reg .pred p;\n\t"
                         ".reg .u32 z, a;\n\t"
                         "setp.ne.u32 p, %0, 0;\n\t"
                         "@p ld.shared.u8 z, [%1];\n\t"
                         "@p mad.lo.u32 a, z, 2, %2;\n\t"
                         "@p st.shared.u16 [a], %3;\n\t"
                         "}" ::"r"(e), "r"(zz + (uint32_t)k - 1), "r"(stage), "h"((short)val)
                         : "memory");
            window_take(r, cl + size);
        }
        bool put = false;
        uint32_t to = 0;
        if (live && (k >= 64 || e == 0 || bad_dc)) {
            const uint32_t pos = window_pos(r, zero), comp = S.tabs[si].comp;
            const int32_t q0 = S.q0[si], pred = S.pred[comp][tid], pn = (int32_t)((uint32_t)pred + (uint32_t)diff);
            const int32_t dq = (int32_t)((uint32_t)pn * (uint32_t)q0);
            const bool over = ((pn ^ pred) & (pn ^ diff)) < 0 || __mulhi(pn, q0) != dq >> 31;
            if ((k != 64 && k < 96) || bad_dc || pos > lim || over) {
                report_bad_block(L, s, slot, p0 + blk_at, si, pred);
                live = false;
                k = 128;
            } else {
                S.pred[comp][tid] = pn;
                L.dc[blk] = dq;
                to = blk;
                put = true;
                blk_at = pos;
                if (++base == s.v.blocks) {  // the interval's last block
                    const unsigned long long endbit = p0 + pos;
                    report(L, s, slot, make_diag(kDiagNone, s.v.start + (uint32_t)((endbit + 7) / 8)), 1);
                }
                live = --left != 0;
                if (++si == sched_len) {
                    si = 0;
                    if (++mx == mcu_cols) {
                        mx = 0;
                        my++;
                    }
                }
                if (live) begin();
            }
        }
        unsigned m = __ballot_sync(0xffffffffu, put);
        while (m) {  // lanes 8i .. 8i + 7 write the i-th block left
            const unsigned m1 = m & (m - 1), m2 = m1 & (m1 - 1), m3 = m2 & (m2 - 1);
            const unsigned mine = lane < 16 ? lane < 8 ? m : m1 : lane < 24 ? m2 : m3;
            const int src = __ffs(mine) - 1;
            const uint32_t g = __shfl_sync(0xffffffffu, to, src & 31);
            if (src >= 0) {
                int4 *st = reinterpret_cast<int4 *>(S.stage + ((tid & ~31u) + src) * kStride) + (lane & 7);
                reinterpret_cast<int4 *>(L.coef + (uint64_t)g * 64)[lane & 7] = *st;
                *st = make_int4(0, 0, 0, 0);
            }
            m = m3 & (m3 - 1);
        }
        __syncwarp();
    }
}

template <int kSteps>
__global__ void __launch_bounds__(kSliceThreads) slice_decode_kernel(JpegLaunch L, uint32_t spread) {
    begin_kernel(L.early);
    __shared__ DecodeSmem S;
    const uint32_t tid = threadIdx.x, at = blockIdx.x * kSliceThreads + tid, slot = at >> spread;
    SliceRef s;
    s.item = 0;
    const bool used = slot << spread == at && slice_ref(L, slot, s);
    // the blocks this slice decodes
    uint32_t n = 0, base = 0;
    unsigned long long from = pack_state(0, 0);
    bool redone = false, whole = false;
#pragma unroll
    for (int c = 0; c < 4; c++) S.pred[c][tid] = 0;
    if (used) {
        S.frame = s.v.frame;  // the same for all
        n = s.v.blocks;
        if (s.v.n_slices > 1) {
            const SlicePrefix P = L.prefix[slot];
            base = P.base;
            bool over = false;  // (then a DC check fails in an earlier slice, which reports it)
#pragma unroll
            for (int c = 0; c < 4; c++) {
                S.pred[c][tid] = (int32_t)P.dc[c];
                over |= P.dc[c] != (int32_t)P.dc[c];
            }
            if (s.j != 0) from = L.sync[slot - 1].exit;
            if (!s.last) {
                const SliceSync &y = L.sync[slot];
                n = y.blocks;
                redone = s.j != 0 && y.q != 0;
                whole = y.q == kMatchNone;
            }
            n = !is_state(from) || over
                    ? 0 : slice_share(n, base, s.v.blocks, (uint32_t)(from & 0xff), L.frames[s.v.frame].sched_len);
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
    const JFrame &F = L.frames[S.frame];
    for (uint32_t i = tid; i < kSliceThreads * kStride / 8; i += kSliceThreads)
        reinterpret_cast<int4 *>(S.stage)[i] = make_int4(0, 0, 0, 0);
    for (uint32_t i = tid; i < 160; i += kSliceThreads) S.zz[i] = i < 64 ? c_slice_zz[i] : 64;
    if (F.shared_tabs) {
        for (uint32_t t = 0; t < F.n_dc; t++) {
            const LutMeta m = L.lut_meta[F.dc_id[t]];
            copy16(S.sym[t], L.sym + m.off, 2 * m.len);
        }
        for (uint32_t t = 0; t < F.n_ac; t++) {
            const LutMeta m = L.lut_meta[F.ac_id[t]];
            copy16(S.sym[kSharedTabs + t], L.sym + m.off, 2 * m.len);
        }
    }
    for (uint32_t i = tid; i < F.sched_len; i += kSliceThreads) {
        const JBlockRec &R = L.brec[F.sched_off + i];
        BlockTabs b = batch_tabs(L, R);
        if (F.shared_tabs) {
            b.dc.at = shared_address(S.sym[(R.local >> 8) & 0xff]);
            b.ac.at = shared_address(S.sym[kSharedTabs + (R.local >> 16)]);
        }
        S.tabs[i] = b;
        S.base_off[i] = R.base_off;
        S.mul_x[i] = R.mul_x;
        S.mul_y[i] = R.mul_y;
        S.q0[i] = R.q0;
    }
    __syncthreads();
    if (F.shared_tabs) decode_slices<true, kSteps>(L, S, F, slot, s, n, from, base);
    else decode_slices<false, kSteps>(L, S, F, slot, s, n, from, base);
}

// --------------------------------------------------------------- resolve ---

__global__ void slice_resolve_kernel(JpegLaunch L) {
    begin_kernel(L.early);
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
        const SliceEvent e = L.events[v.slot_first + (uint32_t)key];
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

// One CTA of slots has no neighbours to settle with.
static uint32_t jpeg_sync_passes(const JpegLaunch &L) { return L.n_slots > (uint32_t)kSliceThreads ? kSyncPasses : 1; }

int jpeg_slice_launches(const JpegLaunch &L) {
    if (!L.n_items_small) return 0;
    const uint32_t passes = jpeg_sync_passes(L);
    return 5 + (int)passes + (passes > 1 ? 1 : 0);
}

// Small grids leave most of the GPU idle while each warp settles and writes its 32 lanes'
// blocks one group after another: there one thread in 2^spread takes a slice, as long as
// that makes no more than two CTAs per SM (320x240: one thread in four, 174 -> 164 us; 30 VGA
// frames: one in two, 347 -> 342; with up to four CTAs per SM a single 1080p frame gains
// nothing and 60 720p ones lose 3 %).
constexpr uint32_t kSpreadCtas = 2 * 152, kMostSpread = 2;

static uint32_t slice_spread(uint32_t ctas) {
    uint32_t spread = 0;
    while (spread < kMostSpread && ctas << (spread + 1) <= kSpreadCtas) spread++;
    return spread;
}

void launch_jpeg_slices(const JpegLaunch &L, cudaStream_t s, cudaEvent_t *marks, bool capturing) {
    auto mark = [&](int k) {
        if (marks) capturing ? cudaEventRecordWithFlags(marks[k], s, cudaEventRecordExternal) : cudaEventRecord(marks[k], s);
    };
    const bool run = L.n_items_small && L.n_slots;
    const uint32_t grid = L.n_slots / kSliceThreads;  // (frames reserve whole CTAs of slots)
    auto per_item = [&](uint32_t items) { return (L.n_items_small + items - 1) / items; };
    if (run) {
        launch_next(slice_plan_kernel, per_item(kPlanThreads) + L.n_luts, kPlanThreads, s, L);
        const uint32_t spread = slice_spread(grid * L.paths);
        launch_next(slice_spec_kernel, dim3(grid << spread, L.paths), kSliceThreads, s, L, spread);
    }
    mark(0);
    if (run) {
        const uint32_t passes = jpeg_sync_passes(L);
        for (uint32_t p = 0; p < passes; p++) launch_next(slice_sync_kernel, grid, kSliceThreads, s, L, p == 0, p + 1 == passes);
        if (passes > 1) launch_next(slice_fix_kernel, per_item(kSliceThreads / 32), kSliceThreads, s, L);
        const uint32_t per_cta = std::min<uint32_t>((L.n_items_small + kPrefixCtas - 1) / kPrefixCtas, kPrefixThreads / 32);
        launch_next(slice_prefix_kernel, per_item(per_cta), kPrefixThreads, s, L, per_cta);
    }
    mark(1);
    // (one path per slice: the long slices of a large batch)
    const uint32_t spread = slice_spread(grid);
    if (run) launch_next(L.paths == 1 ? slice_decode_kernel<kDecodeStepsLong> : slice_decode_kernel<kDecodeSteps>, grid << spread, kSliceThreads, s, L, spread);
    mark(2);
    if (run) launch_next(slice_resolve_kernel, per_item(128), 128, s, L);
}

}  // namespace mmr
