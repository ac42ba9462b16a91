// MJPEG decode kernels for sm_103a.
//
//   scan_count / scan_emit  marker scan of the entropy-coded data
//       (crates/codecs/mjpeg/src/parser.rs:373-414 and the byte-unstuffing of
//       entropy.rs:143-165), parallel over 4 KiB tiles: finds the terminating
//       marker, lists RSTn markers in order and writes the unstuffed bytes.
//   entropy  one restart interval per thread (decoder.rs:313-410, 495-548):
//       Huffman decode, DC prediction, run/level expansion; writes quantised AC
//       levels (natural order) and the dequantised DC of every block, and the
//       interval's restart-marker check (entropy.rs:111-134).
//   resolve  picks each frame's first failing interval (sequential semantics).
//   idct     planar output: dequantisation + the IDCT in fp32 with a proven error
//       bound (idct_core.h), +128, round-half-away, clamp, clipped block write
//       (decoder.rs:550-565); idct_fixup settles the samples the bound leaves
//       undecided, a warp per block, in exact fixed point or the reference's
//       binary64 order (transform.rs:86-109).
#include <cuda_runtime.h>

#include "entropy_core.h"
#include "idct_core.h"
#include "kernels.h"
#include "launch.h"
#include "tables.h"

namespace mmr {

__constant__ int c_zigzag[64] = MMR_ZIGZAG_INIT;

namespace {

constexpr int kEntropyThreads = 128;
constexpr int kStageStride = 72;              // int16 per staged block (144 B: conflict-free 16 B rows)

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        T n = __shfl_up_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) >= (unsigned)o) v += n;
    }
    return v;
}

// ---------------------------------------------------------- marker scan ---
//
// One warp per 4 KiB tile of a packet, eight 16-byte chunks per lane (chunk c of lane l
// starts 512 c + 16 l bytes into the tile, so that each load of the warp is 512 bytes in a
// row, all eight in flight). A tile starts on a 16-byte address whatever the packet's own
// alignment is; the packet's first and last chunk are read by byte. Both kernels work on
// 16-bit masks, a bit per byte of a chunk: a loop runs only for runs of 0xFF that are not
// a stuffed data byte (a marker, fill bytes) and for the bytes that a chunk drops.
//
// Latency- and issue-bound (55 % issue, 33 % of the copy rate): 142 and 275 instructions
// per 512 bytes against 364 and 590 with a byte loop per group that holds an 0xFF, two
// CTA-wide scans and byte stores to shared memory. 330 MB of 300 1080p scans, eight parts:
// count 331 -> 167 us, emit 694 -> 307 us, and no kernel between them (the prefix over a
// frame's tiles, 44 us there and 5 of a single frame's call: each emit warp sums the counts
// before its tile, by groups of 64 tiles).

constexpr int kScanThreads = 128;
constexpr int kScanChunks = kScanTile / 512;

struct Tile {
    uint32_t frame, t, j;  // tile, and its index in the frame
    long long base;        // packet-relative first byte: below data_start in a frame's first tile
};

// The warp's tile. (32 probes a step: the search's loads are a chain.)
__device__ __forceinline__ bool warp_tile(const JpegLaunch &L, Tile &T) {
    T.t = (blockIdx.x * kScanThreads + threadIdx.x) >> 5;
    if (T.t >= L.n_tiles) return false;
    uint32_t lo = 0, hi = L.n_frames;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, at = lo + (threadIdx.x & 31) * step;
        const uint32_t below = __ballot_sync(0xffffffffu, at < hi && L.tile_first[at] <= T.t);
        lo += (uint32_t)(31 - __clz(below)) * step;  // (lane 0's probe always holds)
        hi = min(lo + step, hi);
    }
    T.frame = lo;
    T.j = T.t - L.tile_first[lo];
    const JFrame &F = L.frames[lo];
    T.base = scan_base(F.in, F.data_start) + (long long)T.j * kScanTile;
    return true;
}

// Bytes of a 16-byte chunk that are zero: bit i for byte i in address order.
__device__ __forceinline__ uint32_t zero_mask(uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
    const uint32_t v[4] = {x, y, z, w};
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 4; i++) m |= (((zero_bytes(v[i]) >> 7) * 0x10204080u) >> 28) << (4 * i);  // (flags to one nibble)
    return m;
}

// Bits of the chunk at p whose bytes lie in [first, limit).
__device__ __forceinline__ uint32_t range_mask(long long p, uint32_t first, uint32_t limit) {
    if (p >= first && p + 16 <= limit) return 0xffffu;
    const long long lo = max(first - p, 0ll), hi = min((long long)limit - p, 16ll);
    return lo < hi ? (0xffffu >> (16 - (hi - lo))) << lo : 0;
}

// The tile's chunks, bytes outside [data_start, limit) read as 0.
__device__ __forceinline__ void load_chunks(const uint8_t *in, long long p0, uint32_t ds, uint32_t limit,
                                            uint4 (&v)[kScanChunks]) {
#pragma unroll
    for (int c = 0; c < kScanChunks; c++) {
        const long long p = p0 + 512 * c;
        v[c] = make_uint4(0, 0, 0, 0);
        if (p >= ds && p + 16 <= limit) {
            v[c] = *reinterpret_cast<const uint4 *>(in + p);
        } else if (p + 16 > ds && p < limit) {
            uint32_t w[4] = {0, 0, 0, 0};
#pragma unroll
            for (int i = 0; i < 16; i++)
                if (p + i >= ds && p + i < limit) w[i >> 2] |= (uint32_t)in[p + i] << (8 * (i & 3));
            v[c] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

// Which bytes of a chunk are data (*keep) and which start a run of 0xFF that is not one
// stuffed byte (returned: settled one by one). A maximal run of 0xFF starts a marker
// sequence whose code is the next byte (parser.rs:385-391): 0x00 = the run is one data
// byte, D0-D7 = RSTn, anything else ends the scan; its other bytes are dropped.
__device__ __forceinline__ uint32_t chunk_tokens(const uint8_t *in, long long p, uint32_t limit, const uint4 &v,
                                                 uint32_t prev_ff, uint32_t valid, uint32_t *keep) {
    const uint32_t ff = zero_mask(~v.x, ~v.y, ~v.z, ~v.w);
    *keep = valid;
    if (!(ff | prev_ff)) return 0;
    const uint32_t after = (ff << 1) | prev_ff, start = ff & ~after;
    uint32_t next_zero = (zero_mask(v.x, v.y, v.z, v.w) & valid) >> 1;
    if (start & 0x8000u && p + 16 < limit && in[p + 16] == 0) next_zero |= 0x8000u;
    *keep = valid & ((~ff & ~after) | (start & next_zero));
    return valid & start & ~next_zero;
}

// The code that ends the run of 0xFF at p; 256 when the packet ends first.
__device__ __forceinline__ uint32_t run_code(const uint8_t *in, uint32_t len, long long p) {
    do p++;
    while (p < len && in[p] == 0xff);
    return p < len ? in[p] : 256u;
}

// Index of the first sum of frame f's tile groups (64 tiles each): frames take separate
// groups.
__device__ __forceinline__ uint32_t group_base(const JpegLaunch &L, uint32_t f) {
    return (L.tile_first[f] >> 6) + f;
}

__global__ void __launch_bounds__(kScanThreads) scan_count_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    Tile T;
    if (!warp_tile(L, T)) return;
    const JFrame &F = L.frames[T.frame];
    const uint8_t *in = F.in;
    const uint32_t len = F.in_len, ds = F.data_start, lane = threadIdx.x & 31;
    const long long p0 = T.base + lane * 16;
    uint4 v[kScanChunks];
    load_chunks(in, p0, ds, len, v);
    uint32_t prev_tile = T.base > ds && in[T.base - 1] == 0xff ? 1u : 0u;  // the byte before the tile is 0xFF
    uint32_t tokens = 0, rsts = 0;
    unsigned long long term = ~0ull;
#pragma unroll
    for (int c = 0; c < kScanChunks; c++) {
        const long long p = p0 + 512 * c;
        const uint32_t ends = __ballot_sync(0xffffffffu, v[c].w >= 0xff000000u);
        uint32_t keep;
        uint32_t other = chunk_tokens(in, p, len, v[c], ((ends << 1 | prev_tile) >> lane) & 1,
                                      range_mask(p, ds, len), &keep);
        prev_tile = ends >> 31;
        while (other) {
            const long long q = p + __ffs(other) - 1;
            other &= other - 1;
            const uint32_t code = run_code(in, len, q);
            if (code == 0) tokens++;
            else if (code >= 0xd0 && code <= 0xd7) rsts++;
            else term = min(term, (unsigned long long)q << 9 | code);
        }
        tokens += __popc(keep);
    }
    tokens = __reduce_add_sync(0xffffffffu, tokens);
    rsts = __reduce_add_sync(0xffffffffu, rsts);
    if (term != ~0ull) atomicMin(&L.states[T.frame].term, term);
    if (lane == 0) {
        const unsigned long long cnt = (unsigned long long)rsts << 32 | tokens;
        L.tile_cnt[T.t] = cnt;
        atomicAdd(&L.tile_group[group_base(L, T.frame) + (T.j >> 6)], cnt);
    }
}

// Counts of the frame's tiles before the warp's: whole groups of 64 by their sums.
__device__ __forceinline__ void tiles_before(const JpegLaunch &L, const Tile &T, uint32_t *tokens, uint32_t *rsts) {
    const uint32_t lane = threadIdx.x & 31, t0 = T.t - (T.j & 63), g0 = group_base(L, T.frame), g = T.j >> 6;
    unsigned long long sum = 0;
    for (uint32_t i = lane; i < g; i += 32) sum += L.tile_group[g0 + i];
    for (uint32_t t = t0 + lane; t < T.t; t += 32) sum += L.tile_cnt[t];
    *tokens = __reduce_add_sync(0xffffffffu, (uint32_t)sum);
    *rsts = __reduce_add_sync(0xffffffffu, (uint32_t)(sum >> 32));
}

// Takes byte i out of the chunk's 16; a zero follows the last.
__device__ __forceinline__ uint4 drop_byte(const uint4 &v, uint32_t i) {
    // selector per word: bytes from the dropped one on come from one place further
    const unsigned long long m = 0x1111111111111111ull << (4 * i);
    const uint32_t lo = (uint32_t)m, hi = (uint32_t)(m >> 32);
    uint4 r;
    r.x = __byte_perm(v.x, v.y, 0x3210u + (lo & 0xffffu));
    r.y = __byte_perm(v.y, v.z, 0x3210u + (lo >> 16));
    r.z = __byte_perm(v.z, v.w, 0x3210u + (hi & 0xffffu));
    r.w = __byte_perm(v.w, 0u, 0x3210u + (hi >> 16));
    return r;
}

__global__ void __launch_bounds__(kScanThreads) scan_emit_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    // a warp's tokens, staged at their destination's offset within a 16-byte line
    constexpr uint32_t kLines = kScanTile / 16 + 1;
    __shared__ uint4 s_line[kScanThreads / 32][kLines + 1];  // (one more: a chunk is written as five words)
    Tile T;
    if (!warp_tile(L, T)) return;
    const JFrame &F = L.frames[T.frame];
    const unsigned long long termv = L.states[T.frame].term;
    if (termv == ~0ull || ((termv >> 8) & 1)) return;  // parse error: no usable scan end
    const uint32_t term = (uint32_t)(termv >> 9), lane = threadIdx.x & 31;
    if (T.base >= term) return;
    const uint8_t *in = F.in;
    const uint32_t ds = F.data_start;
    const long long p0 = T.base + lane * 16;
    uint4 v[kScanChunks];
    load_chunks(in, p0, ds, term, v);
    uint32_t prev_tile = T.base > ds && in[T.base - 1] == 0xff ? 1u : 0u;
    uint4 *lines = s_line[threadIdx.x >> 5];
    uint32_t *words = reinterpret_cast<uint32_t *>(lines);
    for (uint32_t l = lane; l < kLines + 1; l += 32) lines[l] = make_uint4(0, 0, 0, 0);
    uint32_t tok0, rst0;
    tiles_before(L, T, &tok0, &rst0);

    uint32_t keep[kScanChunks], rst[kScanChunks], any_rst = 0;
    uint32_t sums[(kScanChunks + 2) / 3] = {};  // the lane's counts, three 10-bit fields a word
#pragma unroll
    for (int c = 0; c < kScanChunks; c++) {
        const long long p = p0 + 512 * c;
        const uint32_t ends = __ballot_sync(0xffffffffu, v[c].w >= 0xff000000u);
        rst[c] = chunk_tokens(in, p, term, v[c], ((ends << 1 | prev_tile) >> lane) & 1,
                              range_mask(p, ds, term), &keep[c]);
        prev_tile = ends >> 31;
        for (uint32_t other = rst[c]; other;) {  // before the terminator: RSTn, or fill bytes and a stuffed one
            const uint32_t bit = other & -other;
            other ^= bit;
            if (run_code(in, F.in_len, p + __ffs(bit) - 1) == 0) {
                keep[c] |= bit;
                rst[c] ^= bit;
            }
        }
        any_rst |= rst[c];
        sums[c / 3] += __popc(keep[c]) << (10 * (c % 3));
    }
    __syncwarp();
    // (a field holds at most 512: the fields' prefixes over the warp do not meet)
    uint32_t incl[(kScanChunks + 2) / 3];
#pragma unroll
    for (int i = 0; i < (kScanChunks + 2) / 3; i++) incl[i] = warp_incl_scan(sums[i]);

    const uint32_t mis = (uint32_t)((uintptr_t)(F.tok + tok0) & 15);
    uint32_t at[kScanChunks], total = 0;  // first token of the lane's chunks within the tile
#pragma unroll
    for (int c = 0; c < kScanChunks; c++) {
        const int sh = 10 * (c % 3);
        at[c] = total + (((incl[c / 3] - sums[c / 3]) >> sh) & 1023u);
        total += (__shfl_sync(0xffffffffu, incl[c / 3], 31) >> sh) & 1023u;
        uint32_t drop = ~keep[c] & 0xffffu;
        const uint32_t n = 16 - __popc(drop);
        while (drop) {
            const uint32_t i = 31 - __clz(drop);
            drop ^= 1u << i;
            v[c] = drop_byte(v[c], i);
        }
        // the chunk's bytes are v's first n, zeros after them; words that another chunk
        // has bytes in are combined
        const uint32_t o = mis + at[c], sl = 8 * (o & 3);
        uint32_t *w = words + (o >> 2);
        const uint32_t x1 = __funnelshift_l(v[c].x, v[c].y, sl), x2 = __funnelshift_l(v[c].y, v[c].z, sl),
                       x3 = __funnelshift_l(v[c].z, v[c].w, sl), x4 = __funnelshift_l(v[c].w, 0u, sl);
        if (n) atomicOr(w, v[c].x << sl);
        if (n >= 12) {
            w[1] = x1;
            w[2] = x2;
        } else {
            if (x1) atomicOr(w + 1, x1);
            if (x2) atomicOr(w + 2, x2);
        }
        if (x3) atomicOr(w + 3, x3);
        if (x4) atomicOr(w + 4, x4);
    }
    uint32_t n_rst = 0;
    if (__any_sync(0xffffffffu, any_rst)) {
        RstEntry *out = L.rsts + F.rst_off;
#pragma unroll
        for (int c = 0; c < kScanChunks; c++) {
            const uint32_t mine = __popc(rst[c]), upto = warp_incl_scan(mine);
            uint32_t idx = rst0 + n_rst + upto - mine;
            for (uint32_t left = rst[c]; left; idx++) {
                const uint32_t i = __ffs(left) - 1;
                left &= left - 1;
                if (idx < F.n_intervals) {
                    RstEntry e;
                    e.tok = tok0 + at[c] + __popc(keep[c] & ((1u << i) - 1));
                    e.number = run_code(in, F.in_len, p0 + 512 * c + i) - 0xd0;
                    out[idx] = e;
                }
            }
            n_rst += __shfl_sync(0xffffffffu, upto, 31);
        }
    }
    __syncwarp();
    // copy out: whole 16-byte lines as vectors, the partial first and last lines by byte
    uint8_t *dst = F.tok + tok0 - mis;  // 16-byte aligned
    const uint32_t span = mis + total, whole0 = mis ? 1 : 0, whole1 = span >> 4;
    for (uint32_t l = whole0 + lane; l < whole1; l += 32) reinterpret_cast<uint4 *>(dst)[l] = lines[l];
    const uint8_t *bytes = reinterpret_cast<const uint8_t *>(lines);
    const uint32_t b = lane < 16 ? lane : (whole1 << 4) + lane - 16;
    if (lane < 16 ? whole0 && b >= mis && b < span : (whole1 || !whole0) && b < span) dst[b] = bytes[b];
    // The last tile that starts before the terminator publishes the totals (the
    // terminator may sit exactly on the next tile's first byte).
    if (lane == 0 && term <= T.base + kScanTile) {
        L.states[T.frame].n_tokens = tok0 + total;
        L.states[T.frame].n_rst = rst0 + n_rst;
    }
}

// ------------------------------------------------------------ entropy -----
//
// Frames with more than four components (their DC predictors do not fit the
// chunked decoder's per-slice sums): one restart interval per thread, a flat
// loop decoding one Huffman symbol per iteration (entropy_core.h).

template <int MAXC>
__device__ void decode_interval(const JpegLaunch &L, uint32_t item, int16_t *stage, const uint8_t *s_zz) {
    uint2 it = L.items[item];
    const uint32_t f = it.x, iv = it.y;
    const JFrame *Fp = L.frames + f;
    JState *st = L.states + f;
    unsigned long long termv = st->term;
    if (!Fp->decode || termv == ~0ull || ((termv >> 8) & 1)) return;
    const uint32_t n_int = Fp->n_intervals, ri = Fp->ri, total_mcus = Fp->total_mcus, mcu_cols = Fp->mcu_cols;
    const uint32_t sched_len = Fp->sched_len;
    const uint64_t blk_off = Fp->blk_off;
    const uint32_t n_rst = min(st->n_rst, n_int), n_tok = st->n_tokens;
    const RstEntry *rst = L.rsts + Fp->rst_off;
    uint32_t start;
    if (iv == 0) start = 0;
    else if (iv - 1 < n_rst) start = rst[iv - 1].tok;
    else return;  // no RST precedes this interval: an earlier interval fails its restart check
    const bool barrier_rst = iv < n_rst;
    const uint32_t barrier = barrier_rst ? rst[iv].tok : n_tok;
    const uint32_t limit = (barrier - start) * 8;

    Bits r;
    bits_init(r, Fp->tok, (unsigned long long)start * 8, 0);
    int32_t pred[MAXC];
#pragma unroll
    for (int c = 0; c < MAXC; c++) pred[c] = 0;
    int4 *stage4 = reinterpret_cast<int4 *>(stage);

    uint32_t mcu = iv * ri;
    const uint32_t mcu1 = min(mcu + ri, total_mcus);
    if (mcu >= mcu1 || sched_len == 0) return;
    uint32_t si = 0, comp = 0;
    const HuffLut *dcl = nullptr, *acl = nullptr;
    int32_t q0 = 0, dq = 0;
    uint64_t blk = 0;
    const JBlockRec *recs = L.brec + Fp->sched_off;
    auto setup_block = [&]() {
        const JBlockRec R = recs[si];
        comp = R.comp;
        const uint32_t mx = mcu % mcu_cols, my = mcu / mcu_cols;
        blk = blk_off + R.base_off + mx * R.mul_x + (uint64_t)my * R.mul_y;
        q0 = R.q0;
        dcl = L.luts + R.dc_lut;
        acl = L.luts + R.ac_lut;
    };
    setup_block();
    int k = 0;
    uint16_t kind = kDiagNone;
    uint32_t errpos = 0;
    for (;;) {
        int32_t val;
        uint16_t err;
        uint32_t eb;
        const int k0 = k;
        if (!decode_symbol(r, limit - r.used, k0 == 0 ? dcl : acl, L.symbols, k, val, err, eb)) {
            kind = err;
            errpos = eb;
            break;
        }
        if (k0 == 0) {  // decoder.rs:507-515
            int64_t p = (int64_t)pred[comp] + val;
            if (p > INT32_MAX || p < INT32_MIN) {
                kind = kJDcPredOverflow;
                errpos = r.used;
                break;
            }
            pred[comp] = (int32_t)p;
            int64_t d = p * (int64_t)q0;
            if (d > INT32_MAX || d < INT32_MIN) {
                kind = kJDcDeqOverflow;
                errpos = r.used;
                break;
            }
            dq = (int32_t)d;
            continue;
        }
        stage[s_zz[k - 1]] = (int16_t)val;
        if (k < 64) continue;
        // block complete: levels + dequantised DC out, staging cleared
        int4 *dst = reinterpret_cast<int4 *>(L.coef + blk * 64);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            dst[q] = stage4[q];
            stage4[q] = make_int4(0, 0, 0, 0);
        }
        L.dc[blk] = dq;
        if (++si == sched_len) {
            si = 0;
            if (++mcu == mcu1) break;
        }
        setup_block();
        k = 0;
    }

    Diag out = make_diag(kDiagNone);
    if (kind != kDiagNone) {
        if (kind == kBarrierErr)
            out = barrier_rst ? make_diag(kJMarkerInData, barrier, 0xd0 + rst[iv].number) : make_diag(kJEndOfData, n_tok);
        else out = make_diag(kind, start + (errpos + 7) / 8);
    } else if (iv + 1 < n_int) {
        // consume_restart before the next interval (entropy.rs:111-134)
        uint32_t tend = start + (r.used + 7) / 8;
        uint32_t expected = iv & 7;
        if (barrier_rst && rst[iv].tok == tend) {
            if (rst[iv].number != expected) out = make_diag(kJRstMismatch, tend, expected, 0xd0 + rst[iv].number);
        } else if (tend < n_tok && Fp->tok[tend] == 0xff) {
            out = make_diag(kJRstMismatch, tend, expected, 0x00);
        } else {
            out = make_diag(kJExpectRst, tend);
        }
    }
    L.results[item] = out;
    if (out.kind != kDiagNone) atomicMin(&st->bad_interval, iv);
}

template <int MAXC>
__global__ void __launch_bounds__(kEntropyThreads) entropy_kernel(JpegLaunch L, uint32_t first, uint32_t count) {
    begin_kernel(L.early);
    __shared__ __align__(16) int16_t s_stage[kEntropyThreads * kStageStride];
    __shared__ uint8_t s_zz[64];
    int4 *mine = reinterpret_cast<int4 *>(s_stage + threadIdx.x * kStageStride);
#pragma unroll
    for (int q = 0; q < 8; q++) mine[q] = make_int4(0, 0, 0, 0);
    if (threadIdx.x < 64) s_zz[threadIdx.x] = (uint8_t)c_zigzag[threadIdx.x];
    __syncthreads();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    decode_interval<MAXC>(L, first + i, s_stage + threadIdx.x * kStageStride, s_zz);
}

__global__ void resolve_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    uint32_t f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= L.n_frames) return;
    const JFrame &F = L.frames[f];
    JState *st = &L.states[f];
    unsigned long long termv = st->term;
    bool ok = F.decode && termv != ~0ull && !((termv >> 8) & 1);
    if (st->bad_interval != 0xffffffffu) {
        st->diag = L.results[F.item_base + st->bad_interval];
        ok = false;
    }
    if (!ok) L.item_ok[F.item] = 0;
}

// ---------------------------------------------------------------- IDCT ----
// (the transform core and its exactness bound live in idct_core.h)

constexpr int kIdctBlocks = 64;  // blocks per CTA, all of one (frame, component) range
constexpr int kIdctThreads = kIdctBlocks * 4;
constexpr int kIdctStride = 68;     // floats per staged block: 16-byte rows, 8 blocks on distinct banks

__device__ __forceinline__ uint32_t find_range(const JpegLaunch &L, uint64_t g) {
    uint32_t lo = 0, hi = L.n_ranges;
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) >> 1;
        if (L.ranges[mid].first <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Planar output: a CTA transforms up to L.idct_tiles times 64 blocks of one (frame,
// component) range, four threads per block, the next tile's levels on their way to shared
// memory meanwhile, and writes each block row as one 8-byte store.
// Per CTA and tile it waited for a search over the ranges, four more dependent loads and the
// levels; now once for up to four tiles (60 720p frames: 218 -> 154 us, 30 VGA frames 34 -> 26).
__global__ void __launch_bounds__(kIdctThreads, 4) idct_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    __shared__ __align__(16) float s_f[kIdctBlocks * kIdctStride];
    __shared__ __align__(16) float s_q[64];
    __shared__ float4 s_m[16];
    __shared__ int4 s_row[2 * kIdctThreads];
    __shared__ int32_t s_dc[kIdctThreads];
    uint32_t r = 0;
    for (uint32_t n = L.n_ranges; n > 1;) {  // the CTA's range, 32 probes a step
        const uint32_t step = (n + 31) / 32, lane = threadIdx.x & 31;
        const uint32_t m = __ballot_sync(0xffffffffu, lane * step < n && L.idct_cta_first[r + lane * step] <= blockIdx.x);
        const uint32_t k = 31 - __clz(m);  // (lane 0's probe always holds)
        r += k * step;
        n = min(step, n - k * step);
    }
    const JBlockRange R = L.ranges[r];
    const JFrame &F = L.frames[R.frame];
    if (!L.item_ok[F.item]) return;
    const JComp &C = L.comps[F.comp_off + R.comp];
    const uint32_t nblk = C.bw * C.bh;
    const uint32_t lb = threadIdx.x >> 2, q = threadIdx.x & 3;
    uint32_t local = (blockIdx.x - L.idct_cta_first[r]) * L.idct_tiles * kIdctBlocks + lb;
    const uint32_t end = min(local - lb + L.idct_tiles * kIdctBlocks, nblk);
    const RowSlots slots{s_row, s_dc};
    if (local < end) copy_rows(L.coef, L.dc, R.first + local, q, slots, threadIdx.x, kIdctThreads);
    idct_fill_rows(s_m, threadIdx.x);
    if (threadIdx.x < 64) s_q[threadIdx.x] = (float)L.quant[F.quant_off + C.q * 64 + threadIdx.x];
    __syncthreads();
    float *blk = s_f + lb * kIdctStride;
    uint8_t *plane = F.planes + C.out_off;
    for (; local - lb < end; local += kIdctBlocks) {  // (a block's threads share a warp: no more barriers)
        const bool valid = local < end;
        const uint64_t g = R.first + local;
        float l1 = valid ? stage_rows(staged_rows(slots, threadIdx.x, kIdctThreads), q, s_q, blk) : 0.0f;
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) l1 += __shfl_xor_sync(0xffffffffu, l1, o);
        __syncwarp();
        if (local + kIdctBlocks < end) copy_rows(L.coef, L.dc, g + kIdctBlocks, q, slots, threadIdx.x, kIdctThreads);
        const uint32_t gx = local % C.bw, gy = local / C.bw;
        unsigned long long mask = 0, rows[2];  // rows q and 7 - q
        if (valid) mask = idct_rows(blk, s_m + 4 * q, q, l1, rows);
        if (mask) {
            // only samples inside the plane are written, and only those go to the exact pass
            const uint32_t vis_w = gx * 8 >= C.plane_w ? 0 : min(8u, C.plane_w - gx * 8);
            const uint32_t vis_h = gy * 8 >= C.plane_h ? 0 : min(8u, C.plane_h - gy * 8);
            const unsigned long long colm = 0x0101010101010101ull * ((1u << vis_w) - 1u);
            const unsigned long long rowm = vis_h >= 8 ? ~0ull : ((1ull << (8 * vis_h)) - 1ull);
            mask &= colm & rowm;
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) mask |= __shfl_xor_sync(0xffffffffu, mask, o);
        if (q == 0 && mask) {  // one entry per block: the queue holds n_blocks entries
            const uint32_t slot = atomicAdd(L.fix_count, 1u);
            L.fix[slot] = make_ulonglong2(g, mask);
            atomicAdd(L.fix_count + 1, (uint32_t)__popcll(mask));
        }
        __syncwarp();  // (the staged block is read)
        // 8 bytes a row, clipped to the plane (blocks of the MCU padding may lie wholly
        // outside it)
        const uint32_t col0 = gx * 8;
        if (!valid || col0 >= C.plane_w) continue;
        const uint32_t ncol = min(8u, C.plane_w - col0);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const uint32_t prow = gy * 8 + (h ? 7 - q : q);
            if (prow >= C.plane_h) continue;
            uint8_t *dst = plane + (uint64_t)prow * C.plane_w + col0;
            if (ncol == 8 && (((uintptr_t)dst) & 7) == 0) {
                *reinterpret_cast<uint2 *>(dst) = make_uint2((uint32_t)rows[h], (uint32_t)(rows[h] >> 32));
            } else {
                for (uint32_t c = 0; c < ncol; c++) dst[c] = (uint8_t)(rows[h] >> (8 * c));
            }
        }
    }
}

// The queued samples the fp32 transform could not decide, a warp per queued
// block: its exact coefficients into shared memory, then settle_samples
// (fixed-point value, or the reference order for genuine near-ties).
__global__ void __launch_bounds__(256) idct_fixup_kernel(JpegLaunch L) {
    begin_kernel(L.early);
    __shared__ int32_t s_c[8][64];
    const uint32_t n = *L.fix_count;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t *c = s_c[w];
    for (uint32_t i = blockIdx.x * 8 + w; i < n; i += gridDim.x * 8) {
        const ulonglong2 e = L.fix[i];
        const uint64_t g = e.x;
        const uint32_t r = find_range(L, g);
        const JFrame *F = &L.frames[L.ranges[r].frame];
        const JComp *C = &L.comps[F->comp_off + L.ranges[r].comp];
        const uint16_t *Q = L.quant + F->quant_off + C->q * 64;
        const int16_t *lv = L.coef + g * 64;
        c[lane] = lane == 0 ? L.dc[g] : (int32_t)lv[lane] * (int32_t)Q[lane];
        c[lane + 32] = (int32_t)lv[lane + 32] * (int32_t)Q[lane + 32];
        __syncwarp();
        const uint32_t local = (uint32_t)(g - L.ranges[r].first);
        const uint32_t gx = local % C->bw, gy = local / C->bw;
        uint8_t *plane = F->planes + C->out_off;
        settle_samples(L.fixw, c, e.y, [&](int y, int x, uint8_t v) {
            plane[(uint64_t)(gy * 8 + y) * C->plane_w + gx * 8 + x] = v;
        });
        __syncwarp();
    }
}

}  // namespace

void launch_jpeg_scan(const JpegLaunch &L, cudaStream_t s) {
    if (L.n_tiles == 0) return;
    const uint32_t ctas = (L.n_tiles + kScanThreads / 32 - 1) / (kScanThreads / 32);
    scan_count_kernel<<<ctas, kScanThreads, 0, s>>>(L);  // (after the uploads)
    launch_next(scan_emit_kernel, ctas, kScanThreads, s, L);
}

void launch_jpeg_entropy(const JpegLaunch &L, cudaStream_t s) {
    uint32_t big = L.n_items - L.n_items_small;
    if (big)
        launch_next(entropy_kernel<256>, (big + kEntropyThreads - 1) / kEntropyThreads, kEntropyThreads, s, L, L.n_items_small, big);
    if (L.n_frames) launch_next(resolve_kernel, (L.n_frames + 127) / 128, 128, s, L);
}

uint32_t idct_ctas(uint32_t blocks, uint32_t tiles) { return (blocks + tiles * kIdctBlocks - 1) / (tiles * kIdctBlocks); }

void launch_jpeg_idct(const JpegLaunch &L, cudaStream_t s) {
    if (L.n_blocks == 0 || L.n_idct_ctas == 0) return;
    launch_next(idct_kernel, L.n_idct_ctas, kIdctThreads, s, L);
    launch_next(idct_fixup_kernel, L.fixup_grid, 256, s, L);
}

}  // namespace mmr
