// Batch JPEG encoder on the GPU (sm_103a): the reference encoder's forward DCT,
// quantisation and Huffman coding (crates/codecs/mjpeg/src/encoder.rs:341-545,
// transform.rs:111-134), byte-identical to it, for many frames per pass.
//
//   fdct_kernel        8 threads per 8x8 block: edge-replicated samples, fp32 row and
//                      column passes, quantisation; coefficients whose quotient lies
//                      within the error bound of a half-integer are listed and
//                      recomputed packed, a thread each, in binary64 in the
//                      reference's operation order
//   bits_kernel        thread per block: Huffman bit count (DC difference against the
//                      previous block of the component in its restart interval)
//   scans              exclusive prefix of the bit counts of 128 blocks each, of the segment
//                      chunks, and of the 0xFF counts of segments and of 256 chunks each
//                      (two launches each)
//   segment_kernel     warp per restart interval ("segment"): its bits and 16-byte chunks
//   write_bits_kernel  thread per block: its codes into the segment's bit buffer
//                      (interior words stored, the two shared edge words OR-ed)
//   ff_count_kernel    thread per 16-byte chunk: 0xFF bytes (each gets a stuffed 0x00)
//   layout_kernel      CTA per frame: where each segment lands after stuffing, the
//                      frame's size, its header; the last CTA places the frames that are
//                      staged for host buffers
//   emit_kernel        thread per chunk: stuffed bytes, then RSTn or EOI after the
//                      segment's last chunk, straight into device buffers
// The header bytes (SOI .. SOS) are the host plan's (plan_jpeg_encode).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "block_source.h"
#include "common.h"
#include "encode.h"
#include "encode_gpu.h"
#include "fdct_core.h"
#include "launch.h"
#include "plane_uploads.h"
#include "tables.h"

namespace mmr {
namespace {


struct EncFrame {
    const uint8_t *plane[3];
    uint32_t pw[3], ph[3];
    size_t stride[3];
    uint32_t mcu_cols, mcus, bpm, ri;  // MCUs per row, MCUs, blocks per MCU, restart interval (0: none)
    uint64_t block_base;               // first block of the frame (scan order, batch-wide)
    uint32_t seg_base, nseg;           // first segment, segments (restart intervals)
    uint8_t *out;                      // device buffer of `cap` bytes, nullptr: staged for a host one
    uint64_t cap;
    uint32_t hdr_off, hdr_len;         // header bytes
    uint8_t sched_comp[10], sched_bx[10], sched_by[10];
    uint8_t comp_first[3], comp_count[3], comp_h[3], comp_v[3], comp_tq[3], comp_tab[3];
};

struct EncLaunch {
    const EncFrame *frames;
    uint32_t n_frames;
    uint64_t n_blocks;
    uint32_t n_segs;
    const uint8_t *qt;        // [2][64] natural order
    const uint32_t *codes;    // [dc 0, dc 1, ac 0, ac 1][256]: bits | length << 16
    const float *rq;          // [2][64] fp32 reciprocals of qt
    const uint8_t *nat2zz;    // [64] zigzag position of each natural index
    int16_t *coef;            // 64 per block, zigzag order
    const uint8_t *headers;
    uint32_t *block_bits;     // per block
    uint32_t *tile_bits;      // per kSymThreads blocks (scanned into tile_off)
    uint64_t *tile_off;       // tiles + 1
    uint64_t *seg_off;        // per segment: its first block's bit offset in the batch
    uint32_t *seg_chunks;     // per segment (scanned into seg_chunk_off)
    uint64_t *seg_bits;       // per segment
    uint64_t *seg_chunk_off;  // n_segs + 1
    uint32_t *raw;            // segment bit buffers, big-endian words, four per chunk
    uint8_t *chunk_ff;        // per chunk: its 0xFF bytes
    uint32_t *ff_sums;        // of them, per segment, then per kEmitThreads chunks
    uint64_t *ff_off;         // their exclusive prefix
    uint32_t *seg_out;        // per segment: its offset in the frame's entropy bytes
    uint32_t *frame_len;      // per frame: entropy bytes, markers and EOI
    uint64_t *frame_off;      // per frame staged for a host buffer: its entropy bytes in `out`
    uint8_t *out;
    uint32_t *done;           // CTAs of layout_kernel that are through (zeroed)
    unsigned long long *exact;  // coefficients recomputed in binary64
};

// frame holding global block b (frames sorted by block_base)
__device__ __forceinline__ uint32_t frame_of_block(const EncLaunch &L, uint64_t b) {
    uint32_t lo = 0, hi = L.n_frames - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (L.frames[mid].block_base <= b) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

__device__ __forceinline__ uint32_t frame_of_segment(const EncLaunch &L, uint32_t s) {
    uint32_t lo = 0, hi = L.n_frames - 1;
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (L.frames[mid].seg_base <= s) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// lo, hi: segments it lies between
__device__ __forceinline__ uint32_t segment_of_chunk(const EncLaunch &L, uint64_t c, uint32_t lo, uint32_t hi) {
    while (lo < hi) {
        const uint32_t mid = (lo + hi + 1) >> 1;
        if (L.seg_chunk_off[mid] <= c) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// ----------------------------------------------------------------- FDCT ---

constexpr int kEncBlocksPerTile = 32;                    // blocks per CTA step, eight threads each
constexpr int kEncThreads = 8 * kEncBlocksPerTile;
constexpr int kTieQueue = kEncThreads;                   // packed binary64 work: a thread per entry
constexpr int kRowStride = 12;                           // floats per row: 16-byte stores of 8 rows hit all banks
constexpr int kOutStride = 80;                           // int16 per block: four blocks' scattered stores least alike
constexpr int kTileStride = 8 * kRowStride + 8;          // per block: four blocks' column loads on distinct banks

// Where block blk's samples come from.
__device__ __forceinline__ BlockSource block_source(const EncFrame &F, uint64_t blk) {
    const uint32_t i = (uint32_t)(blk - F.block_base);
    const uint32_t mcu = i / F.bpm, k = i - mcu * F.bpm;
    const uint32_t c = F.sched_comp[k];
    const uint32_t my = mcu / F.mcu_cols, mx = mcu - my * F.mcu_cols;
    BlockSource B;
    B.plane = F.plane[c];
    B.stride = F.stride[c];
    B.x0 = (mx * F.comp_h[c] + F.sched_bx[k]) * 8;
    B.y0 = (my * F.comp_v[c] + F.sched_by[k]) * 8;
    B.pw = F.pw[c];
    B.ph = F.ph[c];
    B.tq = F.comp_tq[c];
    return B;
}

__device__ __forceinline__ uint2 source_row(const BlockSource &B, uint32_t r) {
    return plane_row<uint2>(
        B, r, [](const uint2 *p) { return *p; }, [](const uint8_t *p) { return *p; });
}

// Persistent CTAs, 32 blocks per step. Quotients too close to a half-integer (exact
// ties of the DC and of the (0, 4), (4, 0), (4, 4) coefficients, a few per cent of
// the blocks, and what the fp32 bound leaves open) are not recomputed where they
// turn up: a binary64 warp instruction holds GB300's FP64 pipe for tens of cycles
// whatever its active lanes, and one or two lanes per warp cost 5.6 of the 7.0 ms
// of an encode of 60 1080p 4:2:2 frames of integer content. They are listed in
// shared memory instead and recomputed a thread each once about 256 are waiting
// (363k of 249 M coefficients): 0.73 ms against 5.67 ms, with the even/odd passes.
//
// A tile's samples are loaded while the one before it is transformed, and whether enough
// coefficients are listed is agreed on at its one barrier; scattered 2-byte stores of a
// warp's four blocks go to rows 40 words apart (with 32 each bank was taken four times):
// 735 -> 598 us for those 60 frames, issue-bound now (63 % of the slots).
__global__ void __launch_bounds__(kEncThreads, 4) fdct_kernel(EncLaunch L, uint64_t n_tiles) {
    __shared__ __align__(16) float s_t[kEncBlocksPerTile * kTileStride];
    __shared__ __align__(16) int16_t s_out[kEncBlocksPerTile][kOutStride];  // blocks in zigzag order
    __shared__ double s_m64[64];
    __shared__ float s_rq[2][64];
    __shared__ unsigned long long s_tie[kTieQueue + 64 * kEncBlocksPerTile];  // block << 6 | v * 8 + u
    __shared__ uint32_t s_ties;
    const int lb = threadIdx.x >> 3, r = threadIdx.x & 7;
    if (threadIdx.x < 64) s_m64[threadIdx.x] = c_m64[threadIdx.x];
    if (threadIdx.x < 128) s_rq[threadIdx.x >> 6][threadIdx.x & 63] = L.rq[threadIdx.x];
    if (threadIdx.x == 0) s_ties = 0;
    uint32_t zzcol[2];  // zigzag positions of this thread's column, byte v of the pair
    {
        uint32_t w[2] = {0, 0};
#pragma unroll
        for (int v = 0; v < 8; v++) w[v >> 2] |= (uint32_t)L.nat2zz[v * 8 + r] << (8 * (v & 3));
        zzcol[0] = w[0];
        zzcol[1] = w[1];
    }
    // row r of the thread's block of a tile, and the block's quantisation table
    uint64_t blk = (uint64_t)blockIdx.x * kEncBlocksPerTile + lb;
    uint32_t f = blk < L.n_blocks ? frame_of_block(L, blk) : 0, next_tq = 0;
    uint2 next = make_uint2(0, 0);
    auto fetch = [&](uint64_t at) {
        if (at >= L.n_blocks) return;
        while (f + 1 < L.n_frames && L.frames[f + 1].block_base <= at) f++;
        const BlockSource B = block_source(L.frames[f], at);
        next_tq = B.tq;
        next = source_row(B, r);
    };
    fetch(blk);
    __syncthreads();
    // recomputes the listed coefficients, a thread each
    auto settle = [&]() {
        const uint32_t n = s_ties;
        for (uint32_t i = threadIdx.x; i < n; i += kEncThreads) {
            const uint64_t eb = s_tie[i] >> 6;
            const int nat = (int)(s_tie[i] & 63);
            const BlockSource B = block_source(L.frames[frame_of_block(L, eb)], eb);
            uint2 rows[8];
#pragma unroll
            for (int y = 0; y < 8; y++) rows[y] = source_row(B, y);
            int k = exact_coefficient(s_m64, rows, nat & 7, nat >> 3, L.qt[B.tq * 64 + nat]);
            if (nat) k = min(max(k, -1023), 1023);
            L.coef[eb * 64 + L.nat2zz[nat]] = (int16_t)k;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            if (n) atomicAdd(L.exact, (unsigned long long)n);
            s_ties = 0;
        }
        __syncthreads();
    };
    for (uint64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        const bool valid = blk < L.n_blocks;
        float *tb = s_t + lb * kTileStride;
        float mag = 0.0f;
        const uint32_t tq = next_tq;
        const uint2 w = next;
        fetch(blk + (uint64_t)gridDim.x * kEncBlocksPerTile);
        if (valid) {  // row pass: t[r][u] = sum_x M[x][u] S[r][x]
            float s[8], t[8];
#pragma unroll
            for (int x = 0; x < 8; x++) {  // 2^23 + sample as a float, then centred
                const uint32_t b = __byte_perm(x < 4 ? w.x : w.y, 0x4B00u, 0x5440 | (x & 3));
                s[x] = __uint_as_float(b) - 8388736.0f;
                mag += fabsf(s[x]);
            }
#pragma unroll
            for (int u = 0; u < 8; u++) t[u] = fdct_row(s, u);
            reinterpret_cast<float4 *>(tb + r * kRowStride)[0] = make_float4(t[0], t[1], t[2], t[3]);
            reinterpret_cast<float4 *>(tb + r * kRowStride)[1] = make_float4(t[4], t[5], t[6], t[7]);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) mag += __shfl_xor_sync(0xffffffffu, mag, o);
        __syncwarp();  // a warp's blocks are its own
        bool full = false;
        if (valid) {   // column pass of column u = r, quantisation
            const int u = r;
            const float *rq = s_rq[tq];
            const float b = mag * kFdctBound;
            float t[8];
#pragma unroll
            for (int y = 0; y < 8; y++) t[y] = tb[y * kRowStride + u];
            uint32_t open = 0;
#pragma unroll
            for (int v = 0; v < 8; v++) {
                bool unsure;
                int k = fdct_round(fdct_column(t, v), b, rq[v * 8 + u], unsure);
                open |= (unsure ? 1u : 0u) << v;
                if (v | u) k = min(max(k, -1023), 1023);  // encode_scan (encoder.rs:372-374)
                s_out[lb][(zzcol[v >> 2] >> (8 * (v & 3))) & 63] = (int16_t)k;
            }
            if (open) {
                const uint32_t more = (uint32_t)__popc(open);
                uint32_t at = atomicAdd(&s_ties, more);
                full = at + more >= (uint32_t)kTieQueue;
                for (; open; open &= open - 1) s_tie[at++] = blk << 6 | (uint32_t)((__ffs(open) - 1) * 8 + u);
            }
        }
        __syncwarp();
        if (valid)  // 16 bytes per thread: the block's 128 bytes in one coalesced row
            reinterpret_cast<uint4 *>(L.coef + blk * 64)[r] = reinterpret_cast<const uint4 *>(s_out[lb])[r];
        blk += (uint64_t)gridDim.x * kEncBlocksPerTile;
        // (the same answer for all: the entry that fills the queue is added once)
        if (__syncthreads_or(full)) settle();  // the list is complete, the coefficients are written
    }
    settle();
}

// ------------------------------------------------------------- Huffman ---

__device__ __forceinline__ uint32_t category(int v) { return 32u - __clz(v < 0 ? -v : v); }

// A CTA's blocks and the code tables in shared memory: the blocks come in as whole
// lines, and a thread then visits its block's nonzero coefficients only, at any index.
// (A thread reading its own 128 bytes from global memory and testing all 64
// coefficients took 0.28 ms to count and 0.57 ms to write 3.9 M blocks of 18 nonzeros.)
constexpr int kSymThreads = 128;

// kLengths: the tables hold, a byte each, a code's bits and its amplitude's, which is all
// that counting needs (and four entries to a word: fewer lanes at a time want one bank).
template <bool kLengths>
struct SymSmem {
    __align__(16) uint4 blk[kSymThreads * 9];  // eight per block, the ninth spreads the banks
    __align__(16) uint32_t codes[kLengths ? 256 : 4 * 256];
    uint32_t frame;
    uint32_t sum[kSymThreads / 32];
};

template <bool kLengths>
__device__ __forceinline__ void load_symbols(const EncLaunch &L, SymSmem<kLengths> &S) {
    const uint64_t b0 = (uint64_t)blockIdx.x * kSymThreads;
    if (threadIdx.x == 0) S.frame = frame_of_block(L, b0);
    const uint4 *src = reinterpret_cast<const uint4 *>(L.coef + b0 * 64);
    const uint64_t n = min((uint64_t)kSymThreads, L.n_blocks - b0) * 8;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const uint32_t i = threadIdx.x + u * kSymThreads;
        if (i < n) S.blk[(i >> 3) * 9 + (i & 7)] = src[i];
    }
#pragma unroll
    for (int u = 0; u < 2; u++) {
        const uint32_t i = threadIdx.x + u * kSymThreads;  // entries 4 i .. 4 i + 3
        const uint4 c = __ldg(reinterpret_cast<const uint4 *>(L.codes) + i);
        if (kLengths) {  // entry e is for a magnitude of e & 15 bits: 4 i & 12, the next three
            const uint32_t sz = 4 * (i & 3) * 0x01010101u + 0x03020100u;
            S.codes[i] = (c.x >> 16 | c.y >> 16 << 8 | c.z >> 16 << 16 | c.w >> 16 << 24) + sz;
        } else {
            reinterpret_cast<uint4 *>(S.codes)[i] = c;
        }
    }
    __syncthreads();
}

// Bits 2i and 2i + 1: whether the halves of word i of 16 are nonzero, given as the
// low-half flags in bits 0..15 and the high-half flags in bits 16..31.
__device__ __forceinline__ uint32_t interleave16(uint32_t x) {
    uint32_t t = (x ^ (x >> 8)) & 0x0000ff00u;
    x ^= t ^ (t << 8);
    t = (x ^ (x >> 4)) & 0x00f000f0u;
    x ^= t ^ (t << 4);
    t = (x ^ (x >> 2)) & 0x0c0c0c0cu;
    x ^= t ^ (t << 2);
    t = (x ^ (x >> 1)) & 0x22222222u;
    return x ^ t ^ (t << 1);
}

// Walks the symbols of block blk of frame F (encode_block, encoder.rs:404-425) and
// hands each to emit(table, entry, value): a code of the 256-entry table (DC, then AC ones)
// and an amplitude of entry & 15 bits of value; at most 27 bits together.
template <bool kLengths, class Emit>
__device__ __forceinline__ void block_symbols(const EncLaunch &L, const SymSmem<kLengths> &S, const EncFrame &F,
                                              uint64_t blk, uint32_t mcu, uint32_t k, Emit emit) {
    const uint4 *row = S.blk + threadIdx.x * 9;
    const int16_t *coef = reinterpret_cast<const int16_t *>(row);
    const uint32_t c = F.sched_comp[k];
    // the DC prediction: the previous block of the component in this restart interval
    const bool interval_start = F.ri ? mcu % F.ri == 0 : mcu == 0;
    int pred = 0;
    if (k != F.comp_first[c]) pred = L.coef[(blk - 1) * 64];
    else if (!interval_start) pred = L.coef[(blk - F.bpm + F.comp_count[c] - 1) * 64];
    const uint32_t dc = F.comp_tab[c] * 256, ac = dc + 512;
    // nonzero coefficients, in zigzag order
    uint32_t mask[2];
#pragma unroll
    for (int h = 0; h < 2; h++) {
        uint32_t flags = 0;
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const uint4 v = row[4 * h + q];
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; j++)
                flags = flags >> 1 | ((((w[j] & 0x7fff7fffu) + 0x7fff7fffu) | w[j]) & 0x80008000u);
        }
        mask[h] = interleave16(flags);
    }
    const int diff = (int)coef[0] - pred;
    emit(dc, category(diff), diff);
    mask[0] &= ~1u;
    uint32_t next = 1;  // the coefficient after the last coded one
#pragma unroll
    for (int h = 0; h < 2; h++)
        for (uint32_t m = mask[h]; m; m &= m - 1) {
            const uint32_t i = (uint32_t)(__ffs(m) - 1) + 32 * h;
            const int v = coef[i];
            uint32_t run = i - next;
            next = i + 1;
            for (; run >= 16; run -= 16) emit(ac, 0xf0, 0);
            emit(ac, run << 4 | category(v), v);
        }
    if (next < 64) emit(ac, 0, 0);
}

// Frame of block blk, from the CTA's first block's on.
__device__ __forceinline__ const EncFrame &frame_from(const EncLaunch &L, uint32_t f, uint64_t blk) {
    while (f + 1 < L.n_frames && L.frames[f + 1].block_base <= blk) f++;
    return L.frames[f];
}

__global__ void __launch_bounds__(kSymThreads) bits_kernel(EncLaunch L) {
    begin_kernel(false);
    __shared__ SymSmem<true> S;
    load_symbols(L, S);
    const uint64_t blk = (uint64_t)blockIdx.x * kSymThreads + threadIdx.x;
    uint32_t bits = 0;
    if (blk < L.n_blocks) {
        const EncFrame &F = frame_from(L, S.frame, blk);
        const uint32_t i = (uint32_t)(blk - F.block_base), mcu = i / F.bpm;
        const uint8_t *len = reinterpret_cast<const uint8_t *>(S.codes);
        block_symbols(L, S, F, blk, mcu, i - mcu * F.bpm,
                      [&](uint32_t table, uint32_t entry, int) { bits += len[table + entry]; });
        L.block_bits[blk] = bits;
    }
    __syncwarp();
    const uint32_t sum = __reduce_add_sync(0xffffffffu, bits);
    if ((threadIdx.x & 31) == 0) S.sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
#pragma unroll
        for (int w = 0; w < kSymThreads / 32; w++) all += S.sum[w];
        L.tile_bits[blockIdx.x] = all;
    }
}

// first block (batch-wide) of segment j of frame F, j <= nseg
__device__ __forceinline__ uint64_t segment_block(const EncFrame &F, uint32_t j) {
    const uint32_t mcu = F.ri ? min(j * F.ri, F.mcus) : (j ? F.mcus : 0u);
    return F.block_base + (uint64_t)mcu * F.bpm;
}

// Bits before block b (up to n_blocks) of the batch, by one warp.
__device__ __forceinline__ uint64_t bits_before(const EncLaunch &L, uint64_t b) {
    const uint64_t tile = b / kSymThreads;
    const uint32_t n = (uint32_t)(b - tile * kSymThreads), lane = threadIdx.x & 31;
    uint32_t sum = 0;
    for (uint32_t i = lane; i < n; i += 32) sum += L.block_bits[tile * kSymThreads + i];
    return L.tile_off[tile] + __reduce_add_sync(0xffffffffu, sum);
}

// Warp per segment. (Offsets are kept per tile of the symbol kernels' blocks: with one per
// block a scan read and wrote 60 MB more for 3.9 M blocks: 1.458 ms an encode, now 1.429.)
__global__ void __launch_bounds__(256) segment_kernel(EncLaunch L) {
    begin_kernel(false);
    const uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (s >= L.n_segs) return;
    const EncFrame &F = L.frames[frame_of_segment(L, s)];
    const uint32_t j = s - F.seg_base;
    const uint64_t at = bits_before(L, segment_block(F, j)), bits = bits_before(L, segment_block(F, j + 1)) - at;
    if (threadIdx.x & 31) return;
    L.seg_off[s] = at;
    L.seg_bits[s] = bits;
    // the last byte is padded with 1 bits; whole 16-byte chunks, so that every chunk's
    // 16-byte load is aligned and inside its segment
    L.seg_chunks[s] = (uint32_t)(((bits + 7) / 8 + 15) / 16);
}

// Shifts by 32 or more give 0.
__device__ __forceinline__ uint32_t shl_clamp(uint32_t x, uint32_t n) {
    uint32_t r;
    asm("shl.b32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}

__device__ __forceinline__ uint32_t shr_clamp(uint32_t x, uint32_t n) {
    uint32_t r;
    asm("shr.u32 %0, %1, %2;" : "=r"(r) : "r"(x), "r"(n));
    return r;
}

// Writes block blk's codes at its bit offset in its segment's big-endian word
// buffer (zeroed): the words after the first are stored as they fill, by a predicated
// store; the first, which the blocks before may share, and the last partial one are OR-ed
// at the end. The segment's last block pads its final byte with 1 bits
// (EntropyWriter::finish, encoder.rs:530-543).
//
// Issue-bound (78 % of the slots, 19 of 32 lanes: blocks have different numbers of
// symbols). 60 1080p frames: 384 -> 351 us, with a 64-bit accumulator and a branch per word;
// counting, from byte tables, 232 -> 197 us.
__global__ void __launch_bounds__(kSymThreads) write_bits_kernel(EncLaunch L) {
    __shared__ SymSmem<false> S;
    // bits of the tile's blocks before the thread's
    const uint64_t blk = (uint64_t)blockIdx.x * kSymThreads + threadIdx.x;
    if (blk < L.n_segs) L.ff_sums[blk] = 0;  // (for ff_count_kernel; a segment has a block at least)
    const uint32_t mine = blk < L.n_blocks ? L.block_bits[blk] : 0, warp = threadIdx.x >> 5;
    uint32_t before = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
        if ((threadIdx.x & 31) >= (uint32_t)o) before += v;
    }
    if ((threadIdx.x & 31) == 31) S.sum[warp] = before;
    before -= mine;
    load_symbols(L, S);  // (a barrier)
    if (blk >= L.n_blocks) return;
#pragma unroll
    for (uint32_t w = 0; w + 1 < kSymThreads / 32; w++)
        if (w < warp) before += S.sum[w];
    const EncFrame &F = frame_from(L, S.frame, blk);
    const uint32_t i = (uint32_t)(blk - F.block_base), mcu = i / F.bpm;
    const uint32_t j = F.ri ? mcu / F.ri : 0u, seg = F.seg_base + j;
    const uint64_t p = L.tile_off[blockIdx.x] + before - L.seg_off[seg];
    uint32_t *const first_word = L.raw + 4 * L.seg_chunk_off[seg] + (p >> 5);
    uint32_t *word = first_word;
    uint32_t acc = 0, first = 0;             // the word's bits so far; the first word
    uint32_t nacc = (uint32_t)(p & 31);      // how many, the earlier blocks' counted as zeros
    auto put = [&](uint32_t value, uint32_t n) {  // n < 32
        const uint32_t total = nacc + n;
        acc |= shl_clamp(value, 32 - total) | shr_clamp(value, total - 32);  // (one of them, but for the same at 32)
        if (total >= 32) {
            if (word == first_word) first = acc;
            else *word = acc;
            word++;
            acc = shl_clamp(value, 64 - total);
        }
        nacc = total & 31;
    };
    block_symbols(L, S, F, blk, mcu, i - mcu * F.bpm, [&](uint32_t table, uint32_t entry, int v) {
        const uint32_t code = S.codes[table + entry], sz = entry & 15;
        put((code & 0xffffu) << sz | ((uint32_t)(v + (v >> 31)) & ((1u << sz) - 1)), (code >> 16) + sz);
    });
    if (blk + 1 == segment_block(F, j + 1)) {
        const uint32_t pad = (8u - (uint32_t)(L.seg_bits[seg] & 7)) & 7u;
        if (pad) put((1u << pad) - 1, pad);
    }
    if (first) atomicOr(first_word, first);
    if (acc) atomicOr(word, acc);
}

// big-endian word: stream byte b of the word is bits 31 - 8b .. 24 - 8b; the first
// nv bytes as a mask of their top bits
__device__ __forceinline__ uint32_t lead_bytes_mask(int nv) {
    return nv >= 4 ? 0x80808080u : nv <= 0 ? 0u : (0x80808080u << (8 * (4 - nv)));
}

// A CTA's chunks lie between two segments, found once.
struct ChunkSmem {
    uint32_t lo, hi;
};

__device__ __forceinline__ void chunk_range(const EncLaunch &L, uint64_t n_chunks, ChunkSmem &S) {
    if (threadIdx.x < 2) {
        const uint64_t first = (uint64_t)blockIdx.x * blockDim.x;
        const uint64_t c = threadIdx.x ? min(first + blockDim.x, n_chunks) - 1 : first;
        (threadIdx.x ? S.hi : S.lo) = segment_of_chunk(L, c, 0, L.n_segs - 1);
    }
    __syncthreads();
}

// Segment s of chunk c, its number k in it, and its bytes.
__device__ __forceinline__ void chunk_of(const EncLaunch &L, const ChunkSmem &S, uint64_t c, uint32_t *s, uint64_t *k,
                                         uint32_t *n) {
    *s = segment_of_chunk(L, c, S.lo, S.hi);
    *k = c - L.seg_chunk_off[*s];
    const uint64_t bytes = (L.seg_bits[*s] + 7) / 8;
    *n = (uint32_t)min((uint64_t)16, bytes - 16 * *k);
}

constexpr int kEmitThreads = 256;  // chunks per CTA of ff_count_kernel and emit_kernel

// (Sums per segment and per CTA: a scan over all chunks' counts read and wrote 68 MB for
// the 4.2 M chunks of 60 1080p frames, which emit_kernel read again: 1.429 ms an encode, now 1.403.)
__global__ void __launch_bounds__(kEmitThreads) ff_count_kernel(EncLaunch L, uint64_t n_chunks) {
    begin_kernel(false);
    __shared__ ChunkSmem S;
    __shared__ uint32_t s_sum[kEmitThreads / 32];
    chunk_range(L, n_chunks, S);
    const uint64_t c = (uint64_t)blockIdx.x * kEmitThreads + threadIdx.x;
    uint32_t s = 0, count = 0;
    if (c < n_chunks) {
        uint32_t n;
        uint64_t k;
        chunk_of(L, S, c, &s, &k, &n);
        const uint4 v = *reinterpret_cast<const uint4 *>(L.raw + 4 * c);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; q++) count += __popc(zero_bytes(~w[q]) & lead_bytes_mask((int)n - 4 * q));
        L.chunk_ff[c] = (uint8_t)count;
    }
    __syncwarp();
    const uint32_t lane = threadIdx.x & 31, sum = __reduce_add_sync(0xffffffffu, count);
    const uint32_t s0 = __shfl_sync(0xffffffffu, s, 0);
    if (__all_sync(0xffffffffu, s == s0 || !count)) {
        if (lane == 0 && sum) atomicAdd(L.ff_sums + s0, sum);
    } else if (count) {
        atomicAdd(L.ff_sums + s, count);
    }
    if (lane == 0) s_sum[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
#pragma unroll
        for (int w = 0; w < kEmitThreads / 32; w++) all += s_sum[w];
        L.ff_sums[L.n_segs + blockIdx.x] = all;
    }
}

// Exclusive prefix of v over a CTA of NT threads; *total = the CTA's sum.
template <int NT>
__device__ __forceinline__ uint64_t cta_exclusive(uint64_t v, uint64_t *total) {
    __shared__ uint64_t s_warp[NT / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint64_t incl = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint64_t o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint64_t w = lane < NT / 32 ? s_warp[lane] : 0, wi = w;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint64_t o = __shfl_up_sync(0xffffffffu, wi, d);
            if (lane >= d) wi += o;
        }
        if (lane < NT / 32) s_warp[lane] = wi - w;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    const uint64_t r = s_warp[warp] + incl - v;
    __syncthreads();
    return r;
}

constexpr int kLayoutThreads = 256;

// Where frame f's entropy bytes go; nullptr when its buffer is too small.
__device__ __forceinline__ uint8_t *frame_dst(const EncLaunch &L, uint32_t f) {
    const EncFrame &F = L.frames[f];
    if (!F.out) return L.out + L.frame_off[f];
    return F.hdr_len + (uint64_t)L.frame_len[f] <= F.cap ? F.out + F.hdr_len : nullptr;
}

// CTA per frame: each segment's offset in the frame's entropy bytes, each segment
// followed by its marker (RSTn, or EOI after the last); the frame's header into a
// device buffer. The last CTA to finish lays out the frames staged for host buffers.
__global__ void __launch_bounds__(kLayoutThreads) layout_kernel(EncLaunch L) {
    begin_kernel(false);
    __shared__ uint64_t s_total;
    __shared__ bool s_last;
    const uint32_t f = blockIdx.x;
    const EncFrame &F = L.frames[f];
    uint64_t pos = 0;
    for (uint32_t j0 = 0; j0 < F.nseg; j0 += kLayoutThreads) {
        const uint32_t j = j0 + threadIdx.x, s = F.seg_base + j;
        uint64_t bytes = 0;
        if (j < F.nseg)
            bytes = (L.seg_bits[s] + 7) / 8 + L.ff_sums[s] + 2;
        const uint64_t ex = cta_exclusive<kLayoutThreads>(bytes, &s_total);
        if (j < F.nseg) L.seg_out[s] = (uint32_t)(pos + ex);
        pos += s_total;
        __syncthreads();
    }
    if (F.out && F.hdr_len + pos <= F.cap)
        for (uint32_t i = threadIdx.x; i < F.hdr_len; i += kLayoutThreads) F.out[i] = L.headers[F.hdr_off + i];
    if (threadIdx.x == 0) {
        L.frame_len[f] = (uint32_t)pos;
        __threadfence();
        s_last = atomicAdd(L.done, 1u) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    uint64_t carry = 0;
    for (uint32_t g0 = 0; g0 < L.n_frames; g0 += kLayoutThreads) {
        const uint32_t g = g0 + threadIdx.x;
        const uint64_t len = g < L.n_frames && !L.frames[g].out ? *(volatile uint32_t *)&L.frame_len[g] : 0;
        const uint64_t ex = cta_exclusive<kLayoutThreads>(len, &s_total);
        if (g < L.n_frames) L.frame_off[g] = carry + ex;
        carry += s_total;
        __syncthreads();
    }
}

// thread per chunk: its bytes with a 0x00 after each 0xFF (EntropyWriter::push,
// encoder.rs:519-528), then the segment's marker after its last chunk. A CTA whose
// chunks are of one frame collects its run of bytes in shared memory and stores it as
// 16-byte vectors; byte stores took 0.20 ms for the 67 MB of 60 1080p frames.

__global__ void __launch_bounds__(kEmitThreads) emit_kernel(EncLaunch L, uint64_t n_chunks) {
    begin_kernel(false);
    __shared__ ChunkSmem S;
    __shared__ __align__(16) uint8_t s_out[kEmitThreads * 34 + 32];
    __shared__ uint8_t *s_dst;
    __shared__ uint32_t s_frame[2], s_len, s_ff[kEmitThreads / 32];
    const uint64_t c = (uint64_t)blockIdx.x * kEmitThreads + threadIdx.x;
    const bool valid = c < n_chunks;
    // 0xFF bytes of the CTA's chunks before the thread's
    const uint32_t mine = valid ? L.chunk_ff[c] : 0, warp = threadIdx.x >> 5;
    uint32_t before = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, before, o);
        if ((threadIdx.x & 31) >= (uint32_t)o) before += v;
    }
    if ((threadIdx.x & 31) == 31) s_ff[warp] = before;
    before -= mine;
    chunk_range(L, n_chunks, S);  // (a barrier)
#pragma unroll
    for (uint32_t w = 0; w + 1 < kEmitThreads / 32; w++)
        if (w < warp) before += s_ff[w];
    if (threadIdx.x < 2) s_frame[threadIdx.x] = frame_of_segment(L, threadIdx.x ? S.hi : S.lo);
    __syncthreads();
    const bool one = s_frame[0] == s_frame[1];
    uint32_t f = s_frame[0];
    uint8_t *base = frame_dst(L, f);
    if (one && !base) return;  // (uniform: the frame's buffer is too small)
    uint8_t *dst = base;
    uint32_t s = 0, n = 0;
    uint64_t k = 0;
    if (valid) {
        chunk_of(L, S, c, &s, &k, &n);
        if (!one) {
            f = frame_of_segment(L, s);
            base = frame_dst(L, f);
        }
        dst = base + L.seg_out[s] + 16 * k + (L.ff_off[L.n_segs + blockIdx.x] - L.ff_off[L.n_segs] + before - L.ff_off[s]);
    }
    if (threadIdx.x == 0) s_dst = dst;
    __syncthreads();
    uint8_t *first = s_dst;  // the CTA's first byte
    const uint32_t mis = (uint32_t)(reinterpret_cast<uintptr_t>(first) & 15);
    uint8_t *p = one ? s_out + mis + (dst - first) : dst;
    if (valid && base) {
        const uint4 v = *reinterpret_cast<const uint4 *>(L.raw + 4 * c);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int b = 0; b < 16; b++) {
            if (b >= (int)n) break;
            const uint8_t x = (uint8_t)(w[b >> 2] >> (24 - 8 * (b & 3)));
            *p++ = x;
            if (x == 0xff) *p++ = 0x00;
        }
        const uint64_t bytes = (L.seg_bits[s] + 7) / 8;
        if (16 * k + n == bytes) {
            const EncFrame &F = L.frames[f];
            const uint32_t j = s - F.seg_base;
            p[0] = 0xff;
            p[1] = j + 1 < F.nseg ? (uint8_t)(0xd0 + (j & 7)) : (uint8_t)0xd9;
            p += 2;
        }
        if (one && (threadIdx.x == kEmitThreads - 1 || c + 1 == n_chunks)) s_len = (uint32_t)(p - s_out);
    }
    if (!one) return;
    __syncthreads();
    const uint32_t end = s_len;  // bytes [mis, end) of s_out
    uint8_t *line = first - mis;
    for (uint32_t b0 = threadIdx.x * 16; b0 < end; b0 += kEmitThreads * 16) {
        if (b0 >= mis && b0 + 16 <= end) {
            *reinterpret_cast<uint4 *>(line + b0) = *reinterpret_cast<const uint4 *>(s_out + b0);
        } else {
            for (uint32_t b = max(b0, mis); b < min(b0 + 16, end); b++) line[b] = s_out[b];
        }
    }
}

// ----------------------------------------------------------------- scan ---

constexpr int kScanThreads = 1024;
constexpr int kScanItems = 4;  // consecutive values per thread
constexpr uint64_t kScanTile = (uint64_t)kScanThreads * kScanItems;

// Tile sums; the last CTA to finish turns them into their exclusive prefix in place and
// writes the grand total.
__global__ void __launch_bounds__(kScanThreads) scan_reduce_kernel(const uint32_t *in, uint64_t n, uint64_t *part,
                                                                   uint64_t *total, uint32_t *done) {
    begin_kernel(false);
    __shared__ uint64_t s_total;
    __shared__ bool s_last;
    const uint64_t base = blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint64_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n) sum += in[base + k];
    cta_exclusive<kScanThreads>(sum, &s_total);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s_total;
        __threadfence();
        s_last = atomicAdd(done, 1u) + 1 == gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    uint64_t carry = 0;
    for (uint64_t b = 0; b < gridDim.x; b += kScanThreads) {
        const uint64_t i = b + threadIdx.x;
        const uint64_t v = i < gridDim.x ? *(volatile uint64_t *)&part[i] : 0;
        const uint64_t ex = cta_exclusive<kScanThreads>(v, &s_total);
        if (i < gridDim.x) part[i] = carry + ex;
        carry += s_total;
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void __launch_bounds__(kScanThreads) scan_apply_kernel(const uint32_t *in, uint64_t n,
                                                                    const uint64_t *part, uint64_t *out) {
    begin_kernel(false);
    __shared__ uint64_t s_total;
    const uint64_t base = blockIdx.x * kScanTile + (uint64_t)threadIdx.x * kScanItems;
    uint32_t v[kScanItems];
    uint64_t sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
        v[k] = base + k < n ? in[base + k] : 0u;
        sum += v[k];
    }
    uint64_t run = (part ? part[blockIdx.x] : 0) + cta_exclusive<kScanThreads>(sum, &s_total);
    if (!part && threadIdx.x == 0) out[n] = s_total;
#pragma unroll
    for (int k = 0; k < kScanItems; k++)
        if (base + k < n) {
            out[base + k] = run;
            run += v[k];
        }
}

// out[0, n) = exclusive prefix of in, out[n] = the sum (part: ceil(n / 4096) scratch,
// done: a zeroed counter); n > 0
void exclusive_scan(const uint32_t *in, uint64_t n, uint64_t *out, uint64_t *part, uint32_t *done, cudaStream_t s) {
    const unsigned tiles = (unsigned)((n + kScanTile - 1) / kScanTile);
    if (tiles == 1) {  // (12 719x405 frames: three launches less: 196.4 us a call, now 192.8)
        launch_next(scan_apply_kernel, 1u, kScanThreads, s, in, n, nullptr, out);
        return;
    }
    launch_next(scan_reduce_kernel, tiles, kScanThreads, s, in, n, part, out + n, done);
    launch_next(scan_apply_kernel, tiles, kScanThreads, s, in, n, part, out);
}

}  // namespace

// ---------------------------------------------------------------- host ---

size_t jpeg_encode_bound(uint32_t format, size_t width, size_t height, uint16_t restart_interval) {
    size_t hmax = 1, vmax = 1, bpm = 1;
    switch (format) {
    case kYuv420: hmax = vmax = 2; bpm = 6; break;
    case kYuv422: hmax = 2; bpm = 4; break;
    case kYuv444: bpm = 3; break;
    default: break;
    }
    const size_t mcus = ((width + 8 * hmax - 1) / (8 * hmax)) * ((height + 8 * vmax - 1) / (8 * vmax));
    const size_t segs = restart_interval ? (mcus + restart_interval - 1) / restart_interval : 1;
    // DC: code <= 16 + amplitude 11 bits; 63 AC coefficients: code <= 16 + amplitude 10
    // bits: 1665 bits < 209 bytes, each possibly stuffed; per segment a padded byte
    // (stuffed) and a marker
    return 1024 + mcus * bpm * 418 + segs * 4 + 2;
}

namespace {

struct DBuf {
    void *p = nullptr;
    size_t cap = 0;
    void ensure(size_t bytes) {
        if (bytes <= cap) return;
        const size_t want = std::max(bytes, cap + cap / 2);
        if (p) cudaFree(p);
        p = nullptr;
        cap = 0;
        if (cudaMalloc(&p, want) != cudaSuccess) {
            cudaGetLastError();
            throw std::runtime_error("GPU encoder: out of device memory");
        }
        cap = want;
    }
    template <class T>
    T *as() const {
        return static_cast<T *>(p);
    }
    ~DBuf() {
        if (p) cudaFree(p);
    }
};

struct PBuf {
    void *p = nullptr;
    size_t cap = 0;
    void ensure(size_t bytes) {
        if (bytes <= cap) return;
        const size_t want = std::max(bytes, cap + cap / 2);
        if (p) cudaFreeHost(p);
        p = nullptr;
        cap = 0;
        if (cudaHostAlloc(&p, want, cudaHostAllocDefault) != cudaSuccess) {
            cudaGetLastError();
            throw std::runtime_error("GPU encoder: out of pinned memory");
        }
        cap = want;
    }
    ~PBuf() {
        if (p) cudaFreeHost(p);
    }
};

// The range that a host address was pinned or registered in.
HostRange host_range(const uint8_t *p) {
    using Query = CUresult(CUDAAPI *)(void *, CUpointer_attribute, CUdeviceptr);
    static const Query query = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuPointerGetAttribute", &f, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            f = nullptr;
        }
        return reinterpret_cast<Query>(f);
    }();
    cudaPointerAttributes at;
    if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
        cudaGetLastError();
        return HostRange{p, p};  // unknown: continued by nothing
    }
    if (at.type == cudaMemoryTypeUnregistered) return HostRange{};
    CUdeviceptr lo = 0;
    size_t size = 0;
    const CUdeviceptr at_p = reinterpret_cast<CUdeviceptr>(p);
    if (!query || query(&lo, CU_POINTER_ATTRIBUTE_RANGE_START_ADDR, at_p) != CUDA_SUCCESS ||
        query(&size, CU_POINTER_ATTRIBUTE_RANGE_SIZE, at_p) != CUDA_SUCCESS || at_p < lo || at_p >= lo + size)
        return HostRange{p, p};
    return HostRange{reinterpret_cast<const uint8_t *>(lo), reinterpret_cast<const uint8_t *>(lo + size)};
}

void flush(PlaneUploads &up, cudaStream_t s) {
    if (up.bytes && cudaMemcpyAsync(up.dst, up.src, up.bytes, cudaMemcpyHostToDevice, s) != cudaSuccess)
        throw std::runtime_error("GPU encoder: upload failed");
    up.bytes = 0;
}

}  // namespace

struct GpuJpegEncoder::Impl {
    int device = 0;
    cudaStream_t s = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
    std::mutex mu;
    DBuf plan, in, coef, block_bits, tile_bits, tile_off, part, seg_bits, seg_off, seg_chunks, seg_chunk_off, raw, chunk_ff, ff_sums, ff_off, seg_out,
        frame_len, frame_off, out, counters;
    PBuf up, back;
};

GpuJpegEncoder::GpuJpegEncoder(int device) : impl_(new Impl) {
    impl_->device = device;
    if (cudaSetDevice(device) != cudaSuccess || cudaStreamCreateWithFlags(&impl_->s, cudaStreamNonBlocking) != cudaSuccess ||
        cudaEventCreate(&impl_->ev0) != cudaSuccess || cudaEventCreate(&impl_->ev1) != cudaSuccess) {
        if (impl_->ev0) cudaEventDestroy(impl_->ev0);
        if (impl_->ev1) cudaEventDestroy(impl_->ev1);
        if (impl_->s) cudaStreamDestroy(impl_->s);
        cudaGetLastError();
        delete impl_;
        throw std::runtime_error("GPU encoder: cannot create its stream");
    }
}

GpuJpegEncoder::~GpuJpegEncoder() {
    cudaSetDevice(impl_->device);
    cudaStreamSynchronize(impl_->s);
    cudaStreamDestroy(impl_->s);
    cudaEventDestroy(impl_->ev0);
    cudaEventDestroy(impl_->ev1);
    delete impl_;
}

int32_t GpuJpegEncoder::encode(EncodeItem *items, size_t n, const JpegEncodeOptions &opt) {
    Impl &I = *impl_;
    std::lock_guard<std::mutex> g(I.mu);
    stats_ = EncodeStats();
    if (cudaSetDevice(I.device) != cudaSuccess) {
        cudaGetLastError();
        return kInternal;
    }
    // host plans: validation and geometry per frame; tables and header bytes per format
    struct Live {
        size_t item;
        uint32_t plan;
    };
    JpegEncodePlan plans[5], scratch;  // by pixel format - 1 (validation refuses 4:1:1)
    bool have[5] = {};
    std::vector<Live> live;
    std::vector<EncFrame> fr;
    std::vector<uint8_t> headers;
    uint64_t blocks = 0, in_bytes = 0;
    uint32_t segs = 0;
    for (size_t i = 0; i < n; i++) {
        EncodeItem &it = items[i];
        it.status = kOk;
        it.message.clear();
        it.out_len = 0;
        const uint32_t form = it.frame.format - kGray8;
        JpegEncodePlan &P = form < 5 ? plans[form] : scratch;
        if (!plan_jpeg_frame(it.frame, opt, &P) || (!have[form] && !plan_jpeg_tables(it.frame, opt, &P))) {
            it.status = P.status;
            it.message = P.message;
            continue;
        }
        have[form] = true;
        EncFrame F;
        memset(&F, 0, sizeof F);
        F.mcu_cols = (uint32_t)P.mcu_cols;
        F.mcus = (uint32_t)(P.mcu_cols * P.mcu_rows);
        F.ri = P.restart_interval;
        uint32_t bpm = 0;
        for (uint32_t c = 0; c < P.ncomp; c++) {
            F.comp_first[c] = (uint8_t)bpm;
            F.comp_count[c] = (uint8_t)(P.comp_h[c] * P.comp_v[c]);
            F.comp_h[c] = P.comp_h[c];
            F.comp_v[c] = P.comp_v[c];
            F.comp_tq[c] = P.comp_tq[c];
            F.comp_tab[c] = P.comp_table[c];
            for (uint32_t by = 0; by < P.comp_v[c]; by++)
                for (uint32_t bx = 0; bx < P.comp_h[c]; bx++) {
                    F.sched_comp[bpm] = (uint8_t)c;
                    F.sched_bx[bpm] = (uint8_t)bx;
                    F.sched_by[bpm] = (uint8_t)by;
                    bpm++;
                }
            const PlaneIn &pl = it.frame.planes[c];
            F.pw[c] = (uint32_t)pl.width;
            F.ph[c] = (uint32_t)pl.height;
            if (!it.in_on_device) in_bytes += (pl.width * pl.height + 255) / 256 * 256;
        }
        F.bpm = bpm;
        F.block_base = blocks;
        F.seg_base = segs;
        F.nseg = F.ri ? (F.mcus + F.ri - 1) / F.ri : 1;
        F.out = it.out_on_device ? it.out : nullptr;
        F.cap = it.out && it.out_on_device ? it.out_capacity : 0;
        F.hdr_off = (uint32_t)headers.size();
        F.hdr_len = (uint32_t)P.header.size();
        headers.insert(headers.end(), P.header.begin(), P.header.end());
        uint8_t *size = headers.data() + F.hdr_off + P.size_at;
        size[0] = (uint8_t)(it.frame.height >> 8);
        size[1] = (uint8_t)it.frame.height;
        size[2] = (uint8_t)(it.frame.width >> 8);
        size[3] = (uint8_t)it.frame.width;
        blocks += (uint64_t)F.mcus * bpm;
        segs += F.nseg;
        fr.push_back(F);
        live.push_back({i, form});
    }
    if (live.empty()) return kOk;
    // the tables depend on the options only; a gray frame's plan lacks the second ones
    const JpegEncodePlan *P0 = &plans[live[0].plan];
    for (const Live &l : live)
        if (plans[l.plan].ncomp > P0->ncomp) P0 = &plans[l.plan];
    // device tables: qt [2][64] | codes [4][256] | fp32 reciprocals of qt [2][64] | zigzag
    // position of each natural index [64]
    constexpr size_t kTabBytes = 128 + 4 * 256 * 4 + 2 * 64 * 4 + 64;
    uint8_t tab[kTabBytes];
    memcpy(tab, P0->qt, 128);
    float *rq = reinterpret_cast<float *>(tab + 128 + 4096);
    for (int t = 0; t < 2; t++)
        for (int i = 0; i < 64; i++) {
            const float r = 1.0f / (float)P0->qt[t][i];
            memcpy(rq + t * 64 + i, &r, 4);
        }
    static const int kZigzagOrder[64] = MMR_ZIGZAG_INIT;
    for (int k = 0; k < 64; k++) tab[128 + 4096 + 512 + kZigzagOrder[k]] = (uint8_t)k;
    uint32_t *codes = reinterpret_cast<uint32_t *>(tab + 128);
    for (int t = 0; t < 2; t++)
        for (int sym = 0; sym < 256; sym++) {
            const uint32_t d = P0->dc[t][sym].bits | (uint32_t)P0->dc[t][sym].length << 16;
            const uint32_t a = P0->ac[t][sym].bits | (uint32_t)P0->ac[t][sym].length << 16;
            memcpy(codes + t * 256 + sym, &d, 4);
            memcpy(codes + (2 + t) * 256 + sym, &a, 4);
        }
    stats_.blocks = blocks;
    try {
        cudaEventRecord(I.ev0, I.s);
        I.in.ensure(std::max<uint64_t>(in_bytes, 256));
        uint64_t at = 0;
        PlaneUploads up;
        for (size_t k = 0; k < live.size(); k++) {
            const EncodeItem &it = items[live[k].item];
            for (uint32_t c = 0; c < plans[live[k].plan].ncomp; c++) {
                const PlaneIn &pl = it.frame.planes[c];
                if (it.in_on_device) {
                    fr[k].plane[c] = pl.data;
                    fr[k].stride[c] = pl.stride;
                    continue;
                }
                const size_t bytes = pl.width * pl.height;
                fr[k].stride[c] = pl.width;
                const uint8_t *before = up.src;
                if (pl.stride == pl.width && up.append(pl.data, bytes, host_range)) {  // packed right behind the last one
                    fr[k].plane[c] = up.dst + (pl.data - before);
                    at += bytes;
                    continue;
                }
                flush(up, I.s);
                at = (at + 255) / 256 * 256;
                uint8_t *dst = I.in.as<uint8_t>() + at;
                fr[k].plane[c] = dst;
                at += bytes;
                if (pl.stride == pl.width) {
                    up.start(pl.data, dst, bytes, host_range);
                } else if (cudaMemcpy2DAsync(dst, pl.width, pl.data, pl.stride, pl.width, pl.height,
                                             cudaMemcpyHostToDevice, I.s) != cudaSuccess) {  // row by row
                    throw std::runtime_error("GPU encoder: upload failed");
                }
            }
        }
        flush(up, I.s);
        // the plan: frames | tables | headers, one copy
        const uint32_t nf = (uint32_t)live.size();
        const size_t o_tab = (nf * sizeof(EncFrame) + 255) / 256 * 256, o_hdr = o_tab + (kTabBytes + 255) / 256 * 256;
        I.plan.ensure(o_hdr + headers.size());
        I.up.ensure(o_hdr + headers.size());
        uint8_t *hp = static_cast<uint8_t *>(I.up.p);
        memcpy(hp, fr.data(), nf * sizeof(EncFrame));
        memcpy(hp + o_tab, tab, kTabBytes);
        memcpy(hp + o_hdr, headers.data(), headers.size());
        cudaMemcpyAsync(I.plan.p, hp, o_hdr + headers.size(), cudaMemcpyHostToDevice, I.s);
        // read back: two totals, then the frames' sizes and places and the tie count
        const size_t b_len = 16, b_off = b_len + (nf * 4 + 15) / 16 * 16, b_exact = b_off + nf * 8;
        I.back.ensure(b_exact + 8);
        uint8_t *hb = static_cast<uint8_t *>(I.back.p);
        I.coef.ensure(blocks * 128);
        I.block_bits.ensure(blocks * 4);
        const uint64_t sym_tiles = (blocks + kSymThreads - 1) / kSymThreads;
        I.tile_bits.ensure(sym_tiles * 4);
        I.tile_off.ensure((sym_tiles + 1) * 8);
        I.seg_off.ensure(segs * 8);
        I.part.ensure(((std::max<uint64_t>(sym_tiles, segs) + kScanTile - 1) / kScanTile + 1) * 8);
        I.seg_bits.ensure(segs * 8);
        I.seg_chunks.ensure(segs * 4);
        I.seg_chunk_off.ensure((segs + 1) * 8);
        I.seg_out.ensure(segs * 4);
        I.frame_len.ensure(nf * 4);
        I.frame_off.ensure(nf * 8);
        I.counters.ensure(32);
        EncLaunch L;
        memset(&L, 0, sizeof L);
        L.frames = I.plan.as<EncFrame>();
        const uint8_t *dt = I.plan.as<uint8_t>() + o_tab;
        L.headers = I.plan.as<uint8_t>() + o_hdr;
        L.n_frames = nf;
        L.n_blocks = blocks;
        L.n_segs = segs;
        L.qt = dt;
        L.codes = reinterpret_cast<const uint32_t *>(dt + 128);
        L.rq = reinterpret_cast<const float *>(dt + 128 + 4096);
        L.nat2zz = dt + 128 + 4096 + 512;
        L.coef = I.coef.as<int16_t>();
        L.block_bits = I.block_bits.as<uint32_t>();
        L.tile_bits = I.tile_bits.as<uint32_t>();
        L.tile_off = I.tile_off.as<uint64_t>();
        L.seg_off = I.seg_off.as<uint64_t>();
        L.seg_chunks = I.seg_chunks.as<uint32_t>();
        L.seg_bits = I.seg_bits.as<uint64_t>();
        L.seg_chunk_off = I.seg_chunk_off.as<uint64_t>();
        L.seg_out = I.seg_out.as<uint32_t>();
        L.frame_len = I.frame_len.as<uint32_t>();
        L.frame_off = I.frame_off.as<uint64_t>();
        L.exact = I.counters.as<unsigned long long>();
        uint32_t *done = I.counters.as<uint32_t>() + 2;  // of three scans and the layout
        L.done = done + 3;
        cudaMemsetAsync(I.counters.p, 0, 32, I.s);
        const unsigned bgrid = (unsigned)((blocks + kSymThreads - 1) / kSymThreads);
        const uint64_t tiles = (blocks + kEncBlocksPerTile - 1) / kEncBlocksPerTile;
        // one wave of resident CTAs (64 registers: four per SM)
        fdct_kernel<<<(unsigned)std::min<uint64_t>(tiles, 152 * 4), kEncThreads, 0, I.s>>>(L, tiles);
        launch_next(bits_kernel, bgrid, kSymThreads, I.s, L);
        exclusive_scan(L.tile_bits, sym_tiles, L.tile_off, I.part.as<uint64_t>(), done, I.s);
        launch_next(segment_kernel, (unsigned)((segs + 7) / 8), 256, I.s, L);
        exclusive_scan(L.seg_chunks, segs, L.seg_chunk_off, I.part.as<uint64_t>(), done + 1, I.s);
        cudaMemcpyAsync(hb, L.seg_chunk_off + segs, 8, cudaMemcpyDeviceToHost, I.s);
        if (cudaStreamSynchronize(I.s) != cudaSuccess) throw std::runtime_error("GPU encoder: device failure");
        const uint64_t chunks = *reinterpret_cast<const uint64_t *>(hb), words = 4 * chunks;
        I.raw.ensure(std::max<uint64_t>(words, 4) * 4);
        const unsigned cgrid = (unsigned)((chunks + kEmitThreads - 1) / kEmitThreads);
        const uint64_t ff_sums = segs + (uint64_t)cgrid;
        I.chunk_ff.ensure(std::max<uint64_t>(chunks, 1));
        I.ff_sums.ensure(ff_sums * 4);
        I.ff_off.ensure((ff_sums + 1) * 8);
        I.part.ensure(((ff_sums + kScanTile - 1) / kScanTile + 1) * 8);
        I.out.ensure(std::max<uint64_t>(chunks * 32 + (uint64_t)segs * 2, 16));
        L.raw = I.raw.as<uint32_t>();
        L.chunk_ff = I.chunk_ff.as<uint8_t>();
        L.ff_sums = I.ff_sums.as<uint32_t>();
        L.ff_off = I.ff_off.as<uint64_t>();
        L.out = I.out.as<uint8_t>();
        cudaMemsetAsync(L.raw, 0, words * 4, I.s);
        write_bits_kernel<<<bgrid, kSymThreads, 0, I.s>>>(L);
        launch_next(ff_count_kernel, cgrid, kEmitThreads, I.s, L, chunks);
        exclusive_scan(L.ff_sums, ff_sums, L.ff_off, I.part.as<uint64_t>(), done + 2, I.s);
        launch_next(layout_kernel, nf, kLayoutThreads, I.s, L);
        launch_next(emit_kernel, cgrid, kEmitThreads, I.s, L, chunks);
        if (cudaGetLastError() != cudaSuccess) throw std::runtime_error("GPU encoder: launch failed");
        cudaMemcpyAsync(hb + b_len, L.frame_len, nf * 4, cudaMemcpyDeviceToHost, I.s);
        cudaMemcpyAsync(hb + b_off, L.frame_off, nf * 8, cudaMemcpyDeviceToHost, I.s);
        cudaMemcpyAsync(hb + b_exact, L.exact, 8, cudaMemcpyDeviceToHost, I.s);
        cudaEventRecord(I.ev1, I.s);
        if (cudaStreamSynchronize(I.s) != cudaSuccess) throw std::runtime_error("GPU encoder: device failure");
        const uint32_t *len = reinterpret_cast<const uint32_t *>(hb + b_len);
        const uint64_t *off = reinterpret_cast<const uint64_t *>(hb + b_off);
        stats_.exact_coefficients = *reinterpret_cast<const uint64_t *>(hb + b_exact);
        // host buffers: header, then the staged entropy bytes
        bool copied = false;
        for (size_t k = 0; k < live.size(); k++) {
            EncodeItem &it = items[live[k].item];
            const size_t total = (size_t)fr[k].hdr_len + len[k];
            if (!it.out || total > it.out_capacity) {
                it.status = kInvalidArgument;
                it.message = "output buffer is smaller than the encoded frame";
                continue;
            }
            if (!it.out_on_device) {
                memcpy(it.out, headers.data() + fr[k].hdr_off, fr[k].hdr_len);
                cudaMemcpyAsync(it.out + fr[k].hdr_len, L.out + off[k], len[k], cudaMemcpyDeviceToHost, I.s);
                copied = true;
            }
            it.out_len = total;
            stats_.bytes_out += total;
        }
        if (copied) {
            cudaEventRecord(I.ev1, I.s);
            if (cudaStreamSynchronize(I.s) != cudaSuccess) throw std::runtime_error("GPU encoder: device failure");
        }
        cudaEventElapsedTime(&stats_.device_ms, I.ev0, I.ev1);
    } catch (const std::exception &) {
        cudaGetLastError();
        for (const Live &l : live) {
            items[l.item].status = kInternal;
            items[l.item].message = "CUDA device failure during encode";
            items[l.item].out_len = 0;
        }
        return kInternal;
    }
    return kOk;
}

}  // namespace mmr
