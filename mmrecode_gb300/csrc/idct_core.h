// The reference's 8x8 inverse DCT reproduced exactly (crates/codecs/mjpeg/src/transform.rs:86-109).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "exact_fixed.h"
#include "kernels.h"
#include "packed.h"
#include "rounding.h"
#include "tables.h"

namespace mmr {

// transform.rs:86-109 computes, in binary64 and in this order,
//   t[v][x] = sum_u M[x][u] * c[v][u]            (from 0.0, u = 0..7)
//   s[y][x] = sum_v M[y][v] * t[v][x]            (from 0.0, v = 0..7)
//   sample  = clamp(round_half_away(s + 128.0), 0, 255)
// GB300 issues binary64 at a small fraction of its fp32 rate, so every sample
// is first computed in fp32 and kept only when it provably rounds like the
// binary64 value:
//   S  = sum_v sum_u M[y][v] M[x][u] c[v][u]   (exact real value, double M)
//   B  = sum_v sum_u |M[y][v]| |M[x][u]| |c[v][u]|  <=  Mmax^2 * C1,
//        C1 = sum |c|, Mmax = max |M| = 0.49039264 (Mmax^2 < 0.2405)
//   fp32 path (idct_block; M and c rounded to fp32, u = 2^-24): each pass output
//        is fl(E +- O) with E, O chains of four FMAs, so it carries at most 5
//        roundings over its sum of |terms| (Higham ch. 3: gamma_5), plus u each
//        for rounding M and c to fp32:
//          pass 1   |t32 - t| <= 7u A,   A = sum_u |M[x][u]| |c[v][u]|
//          pass 2   |s32 - S| <= 5u B + u B + 7u B = 13u B   (+ O(u^2) B)
//   binary64 reference: |s64 - S| <= 16 * 2^-53 * B, and its +128.0 rounds
//        by at most 2^-53 |s + 128|.
// With delta = 2^-22 * C1 + 2^-40 |s32| + 2^-30 (2^-22 * C1 = 4u C1 >=
// 13u * 0.2405 C1 = 3.13u C1, margin 1.28 over the bound; |s32| <= C1 / 4 turns
// the middle term into 2^-42 C1), if no half-integer lies within delta of s32
// (+128 shifts by an integer) both values round to the same integer, and so
// clamp to the same sample.
// Every other sample is recomputed in the exact reference order. Zero
// coefficients are skipped in the exact path: a zero term adds +-0.0, which
// leaves any sum that is not -0.0 unchanged, and these sums are never -0.0.

namespace {

__constant__ double c_idct[64] = MMR_IDCT_MATRIX_INIT;
__constant__ float c_idct32[64] = MMR_IDCT_MATRIX_INIT;

// Pass 1 of the reference order for one row: t[v][x] = sum_u M[x][u] c[v][u].
__device__ __forceinline__ double exact_row(const int32_t *crow, int x) {
    double acc = 0.0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const int32_t cv = crow[u];
        if (cv) acc = __dadd_rn(acc, __dmul_rn(c_idct[x * 8 + u], (double)cv));
    }
    return acc;
}

// + 128, round half away from zero, clamp.
__device__ __forceinline__ uint8_t exact_pixel(double s) {
    const double px = __dadd_rn(s, 128.0);
    if (!(px > 0.0)) return 0;
    if (px >= 255.0) return 255;
    const int n = __double2int_rd(px);
    return (uint8_t)(n + (__dsub_rn(px, (double)n) >= 0.5 ? 1 : 0));
}

// A block with at least this many undecided samples ties in them: they take the reference
// order without trying the fixed-point value first.
constexpr int kManyTies = 12;

// Settles the samples in `mask` of one block whose exact dequantised coefficients
// are in c (shared memory; all 32 lanes of the warp call this together). First the exact fixed-point value of each (exact_fixed.h, offset +128), four
// samples at a time, lane v of eight taking row v of the coefficients; what is still too
// close to a half-integer takes the reference order, four columns at a time: lane v
// forms t[v][x], then sample (v, x) from the eight of them. A block with no nonzero AC
// coefficient is evaluated once. put(y, x, sample) may run on any lane.
//
// Bound by the binary64 pipe (16 cycles per warp instruction and SM) where samples tie, by
// the chains' latency elsewhere. By columns, a block's ties cost 8 row terms and 8 column
// terms per four columns; a lane per sample cost every nonzero coefficient's term and the
// column's (the fused 4:4:4 transform of 64 mixed frames: 1367 us, 57 % of it waiting for
// that pipe; now 693). Of a 320x240 frame's call the fixup takes 14 us instead of 24.
template <class Put>
__device__ __forceinline__ void settle_samples(const long long *fixw, const int32_t *c, unsigned long long mask,
                                               Put put) {
    const uint32_t lane = threadIdx.x & 31, v = lane & 7, g = lane >> 3;
    long long c1 = llabs((long long)c[lane]) + llabs((long long)c[lane + 32]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c1 += __shfl_xor_sync(0xffffffffu, c1, o);
    if (c1 == llabs((long long)c[0])) {  // every M[x][0] is the same literal: all 64 samples are equal
        int s = -1;
        if (c1 < kFixMaxC1) s = fixed_round(fixw[0] * (long long)c[0], (int32_t)c1, 128);
        // (the other terms of both passes are zeros, and 0.0 + x = x)
        if (s < 0) s = exact_pixel(__dmul_rn(c_idct[0], __dmul_rn(c_idct[0], (double)c[0])));
        for (int b = lane; b < 64; b += 32)
            if (mask >> b & 1) put(b >> 3, b & 7, (uint8_t)s);
        return;
    }
    unsigned long long left = mask;  // samples for the reference order
    if (c1 < kFixMaxC1 && __popcll(mask) < kManyTies) {
        left = 0;
        while (mask) {
            if (!(mask & (mask - 1))) {  // one sample: over all lanes
                const int b = __ffsll((long long)mask) - 1;
                const int s = fixed_round(fixed_sum(fixw + b * 64, c), (int32_t)c1, 128);
                if (s < 0) left |= mask;
                else if (lane == 0) put(b >> 3, b & 7, (uint8_t)s);
                break;
            }
            int b = -1;  // of the lane's group of eight
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) {
                if (k == g && mask) b = __ffsll((long long)mask) - 1;
                mask &= mask - 1;
            }
            long long t = 0;
            if (b >= 0) {
                const longlong2 *w = reinterpret_cast<const longlong2 *>(fixw + b * 64 + v * 8);
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const longlong2 ww = __ldg(w + u);
                    t += ww.x * c[v * 8 + 2 * u] + ww.y * c[v * 8 + 2 * u + 1];
                }
            }
#pragma unroll
            for (int o = 1; o < 8; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            const int s = b >= 0 ? fixed_round(t, (int32_t)c1, 128) : 0;
            if (s >= 0 && b >= 0 && v == 0) put(b >> 3, b & 7, (uint8_t)s);
            for (uint32_t m = __ballot_sync(0xffffffffu, s < 0 && v == 0); m; m &= m - 1)
                left |= 1ull << __shfl_sync(0xffffffffu, b, __ffs(m) - 1);
        }
    }
    uint32_t cols = (uint32_t)(left | left >> 32);
    cols |= cols >> 16;
    cols = (cols | cols >> 8) & 0xffu;
    while (cols) {
        int x = -1;  // the group's column
#pragma unroll
        for (uint32_t k = 0; k < 4; k++) {
            if (k == g && cols) x = __ffs(cols) - 1;
            cols &= cols - 1;
        }
        const double t = x >= 0 ? exact_row(c + v * 8, x) : 0.0;
        double acc = 0.0;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const double ti = __shfl_sync(0xffffffffu, t, (lane & 24) | i);
            if (__double_as_longlong(ti) << 1 != 0) acc = __dadd_rn(acc, __dmul_rn(c_idct[v * 8 + i], ti));
        }
        if (x >= 0 && left >> (v * 8 + x) & 1) put(v, x, exact_pixel(acc));
    }
}

// What thread q of a block reads of it: level rows q and q + 4, and the DC.
struct BlockRows {
    int4 row[2];
    int32_t dc;
};

// They come by way of shared memory, asynchronously: slot of thread tid of nt, whose copies
// begin with copy_rows (once what the slot held has been used) and are waited for by
// staged_rows. Only the thread itself reads what it copied. (The transforms waited longest
// for their levels; loads a tile ahead into registers spilled.)
struct RowSlots {
    int4 *row;    // 2 * nt
    int32_t *dc;  // nt
};

__device__ __forceinline__ void copy_rows(const int16_t *levels, const int32_t *dc, uint64_t g, uint32_t q,
                                          const RowSlots &to, uint32_t tid, uint32_t nt) {
    const int4 *src = reinterpret_cast<const int4 *>(levels + g * 64) + q;
    const uint32_t a = (uint32_t)__cvta_generic_to_shared(to.row + tid), d = (uint32_t)__cvta_generic_to_shared(to.dc + tid);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a), "l"(src) : "memory");
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(a + 16 * nt), "l"(src + 4) : "memory");
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(dc + g) : "memory");
}

__device__ __forceinline__ BlockRows staged_rows(const RowSlots &from, uint32_t tid, uint32_t nt) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    BlockRows b;
    b.row[0] = from.row[tid];
    b.row[1] = from.row[tid + nt];
    b.dc = from.dc[tid];
    return b;
}

// Dequantises them into fp32 rows q and q+4 of `blk` (the product of an
// int16 level and an 8-bit quantiser is exact in fp32; the DC is the decoder's
// dequantised int32, rounded to fp32 like every c in the bound). Returns the
// sum of |c| over the two rows.
__device__ __forceinline__ float stage_rows(const BlockRows &b, uint32_t q, const float *Qf, float *blk) {
    float l1 = 0.0f;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const int row = q + 4 * h;
        const int4 v = b.row[h];
        const int16_t *lv = reinterpret_cast<const int16_t *>(&v);
        const float4 qa = reinterpret_cast<const float4 *>(Qf + row * 8)[0];
        const float4 qb = reinterpret_cast<const float4 *>(Qf + row * 8)[1];
        const float qv[8] = {qa.x, qa.y, qa.z, qa.w, qb.x, qb.y, qb.z, qb.w};
        float f[8];
#pragma unroll
        for (int j = 0; j < 8; j++) f[j] = (float)lv[j] * qv[j];
        if (row == 0) f[0] = (float)b.dc;
#pragma unroll
        for (int j = 0; j < 8; j++) l1 += fabsf(f[j]);
        reinterpret_cast<float4 *>(blk + row * 8)[0] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4 *>(blk + row * 8)[1] = make_float4(f[4], f[5], f[6], f[7]);
    }
    return l1;
}

// Rounding an fp32 transform value provably equals rounding the binary64 value when no
// half-integer lies within delta of acc, i.e. when acc is closer than near = 0.5 -
// delta to its nearest integer (with delta >= 0.5 nothing is certain); the exact pass
// settles the rest, ties included, so the rounding mode's ties-to-even never decides a
// sample. Clamping after an agreed rounding agrees.
//
// round_nearest (rounding.h) avoids conversion instructions and is exact for
// |acc| < 2^22. Larger values need no check of their own: |s| <= C1/4 and
// |acc - s| <= delta give C1 > 2^24 for |acc| >= 2^22, so near < 0 and the
// rounding is unsure already.

// A value so far beyond the clamp limits (s + 128 > 255.5 or < -0.5 whatever the
// rounding; 129 and -130 leave room for the fp32 rounding of the bounds) is decided by
// the clamp.
__device__ __forceinline__ bool clamped(float acc, float near) {
    const float delta = 0.5f - near;
    return acc > 129.0f + delta || acc < -130.0f - delta;
}

// Transform of one staged block by its four threads; thread q produces output rows
// q and 7 - q as eight bytes each (the first sample in the low byte). Both passes use
// the even/odd split of the basis: M[7-x][u] = (-1)^u M[x][u] holds for the fp32
// roundings of the reference's literals (the literals themselves differ from exact
// symmetry by < 2e-15, far inside the fp32 rounding), so
//   s[x] = E + O, s[7-x] = E - O,  E = sum_{u even} M[x][u] c[u], O = sum_{u odd}.
// The vertical pass comes first, two columns to a packed FMA, so that a thread has whole
// rows of samples; the horizontal one keeps E and O side by side over the pairs (t[0],
// t[1]), (t[2], t[3]), ... Per output this is 4 FMAs per half and one add: each pass's
// error is <= 5u of the sum of |terms|, plus u for each rounded M and c, <= 13u B after
// both passes (the bound above, which is the same in either order of the passes). |s| <=
// Mmax^2 C1 < C1/4, so the relative term 2^-40 |s| of the bound is folded into 2^-42 C1.
// One comparison of the largest distance to an integer decides the eight outputs of a
// row, but for one in a hundred.
// Returns the samples left to the exact pass as bits (row * 8 + column).
//
// Shared memory's wavefronts are the scarcest: rows leave as two 8-byte stores where
// columns took sixteen of a byte, and eight in a hundred instructions less (a step of 300
// 1080p frames with RGB output: 5.92 -> 5.85 ms).
// mrow: M[q][0..7], each twice.
__device__ __forceinline__ unsigned long long idct_rows(const float *blk, const float4 *mrow, uint32_t q, float c1,
                                                        unsigned long long (&row)[2]) {
    F2 e[4], o[4];  // even and odd sums of the columns (0, 1), (2, 3), ...
#pragma unroll
    for (int v = 0; v < 8; v++) {
        const float4 mm = mrow[v >> 1];
        const F2 m = v & 1 ? f2(mm.z, mm.w) : f2(mm.x, mm.y);
        const float4 a = reinterpret_cast<const float4 *>(blk + v * 8)[0];
        const float4 b = reinterpret_cast<const float4 *>(blk + v * 8)[1];
        const F2 c[4] = {f2(a.x, a.y), f2(a.z, a.w), f2(b.x, b.y), f2(b.z, b.w)};
#pragma unroll
        for (int p = 0; p < 4; p++) {
            F2 &s = v & 1 ? o[p] : e[p];
            s = v < 2 ? mul2(c[p], m) : fma2(c[p], m, s);
        }
    }
    // delta = 2^-22 C1 >= 13u Mmax^2 C1 (margin 1.28), see the bound above
    const float near = 0.5f - (c1 * (0x1p-22f + 0x1p-42f) + 0x1p-30f);
    unsigned long long mask = 0;
#pragma unroll
    for (int p = 0; p < 4; p++) {
        const F2 sum = add2(e[p], o[p]);
        o[p] = sub2(e[p], o[p]);
        e[p] = sum;
    }
    float all[2][8];
#pragma unroll
    for (int x = 0; x < 4; x++) {  // (both rows at a time: the factors take registers)
        const float *f = c_idct32 + x * 8;
        const F2 m[4] = {f2(f[0], f[1]), f2(f[2], f[3]), f2(f[4], f[5]), f2(f[6], f[7])};
#pragma unroll
        for (int side = 0; side < 2; side++) {
            const F2 *t = side ? o : e;
            F2 s = mul2(t[0], m[0]);
            s = fma2(t[1], m[1], s);
            s = fma2(t[2], m[2], s);
            s = fma2(t[3], m[3], s);
            float ev, od;
            split2(s, ev, od);
            all[side][x] = ev + od;
            all[side][7 - x] = ev - od;
        }
    }
#pragma unroll
    for (int side = 0; side < 2; side++) {
        const float (&acc)[8] = all[side];
        float far = 0.0f;
        const uint32_t y = side ? 7 - q : q;
        int32_t n[8];
#pragma unroll
        for (int x = 0; x < 8; x++) {
            float r;
            n[x] = round_nearest(acc[x], r) + 128;
            far = fmaxf(far, fabsf(acc[x] - r));
        }
        row[side] = (unsigned long long)sat_quad_u8(n[4], n[5], n[6], n[7]) << 32 | sat_quad_u8(n[0], n[1], n[2], n[3]);
        if (far < near) continue;
#pragma unroll
        for (int x = 0; x < 8; x++) {
            float r;
            round_nearest(acc[x], r);
            if (fabsf(acc[x] - r) < near) continue;
            if (clamped(acc[x], near)) {
                const unsigned long long byte = 0xffull << (8 * x);
                row[side] = acc[x] > 0.0f ? row[side] | byte : row[side] & ~byte;
            } else {
                mask |= 1ull << (y * 8 + x);
            }
        }
    }
    return mask;
}

// The factors of thread q's vertical pass are rows[4 * q .. 4 * q + 3].
__device__ __forceinline__ void idct_fill_rows(float4 *rows, uint32_t tid) {
    if (tid < 16) {
        const float a = c_idct32[2 * tid], b = c_idct32[2 * tid + 1];
        rows[tid] = make_float4(a, a, b, b);
    }
}

// The samples into out[row * stride + column] (rows 8-byte aligned).
__device__ __forceinline__ unsigned long long idct_block(const float *blk, const float4 *mrow, uint32_t q, float c1,
                                                         uint8_t *out, int stride) {
    unsigned long long row[2];
    const unsigned long long mask = idct_rows(blk, mrow, q, c1, row);
    *reinterpret_cast<uint2 *>(out + q * stride) = make_uint2((uint32_t)row[0], (uint32_t)(row[0] >> 32));
    *reinterpret_cast<uint2 *>(out + (7 - q) * stride) = make_uint2((uint32_t)row[1], (uint32_t)(row[1] >> 32));
    return mask;
}

// With the factors in registers.
__device__ __forceinline__ unsigned long long idct_block(const float *blk, uint32_t q, float c1, uint8_t *out,
                                                         int stride) {
    float4 mrow[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float a = c_idct32[q * 8 + 2 * i], b = c_idct32[q * 8 + 2 * i + 1];
        mrow[i] = make_float4(a, a, b, b);
    }
    return idct_block(blk, mrow, q, c1, out, stride);
}

}  // namespace

}  // namespace mmr
