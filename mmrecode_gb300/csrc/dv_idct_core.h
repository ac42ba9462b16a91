// The reference's DV25 inverse DCTs reproduced exactly
// (crates/codecs/dv/src/decoder.rs:520-548 inverse_88, 555-602 inverse_248).
//
// Both transforms are first evaluated in fp32 as separable sums (8 + 8 terms for
// 8-8; butterfly, 8 + 4 terms for 2-4-8), each factor cu * cos the fp32 product
// of the fp32 roundings (3u, u = 2^-24), every eight-term sum as two four-term FMA
// chains (even and odd terms) added and subtracted for two outputs (the fp32 factors
// are exactly symmetric). Against the exact real value of the reference's terms (its
// doubles: FRAC_1_SQRT_2, the cos table, the integer c) the fp32 sum is off by at most
// (3u + 5u) + (3u + 5u) = 16u B for 8-8 and (u + 3u + 4u) + (3u + 5u) = 16u B for 2-4-8
// (the bounds below take 22u); the
// binary64 sequence by < 70 * 2^-53 B. B = sum |terms| <= C1 = sum |c| for 8-8 (|cos| <= 1, cu cv <= 1) and
// <= C1 / 2 per 2-4-8 field (a butterfly output is at most |c1| + |c2|); after the
// final / 4.0 or / 2.0, |value32 - value64| <= 5.5u C1 < delta = 2^-21 C1 + 2^-30
// (= 8u C1 + 2^-30, margin 1.45). If no half-integer lies within delta of value32
// both round (half away from zero) and clamp alike; the rest are recomputed in
// the reference order.
//
// Used by dv_idct_kernel (eight threads per block, the row-parallel form at the
// end of this file) and, with the same functions, by the block-level transform
// tests.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "exact_fixed.h"
#include "packed.h"
#include "rounding.h"

namespace mmr {
namespace {

__constant__ double c_cos16[128] = {
#include "cos_table.inc"
};

constexpr double kFrac = 0.7071067811865476;  // FRAC_1_SQRT_2

// The reference's binary64 8-8 direct sum for sample (y, x) (decoder.rs:520-548):
// terms ((((cu*cv)*c)*cos_u)*cos_v) accumulated in (v, u) order, then / 4.0. Zero
// coefficients are skipped: their term is +-0.0, which leaves any sum that is not
// -0.0 unchanged, and these sums are never -0.0. (c: 16-byte aligned rows.)
__device__ __noinline__ double exact_88(const int32_t *c, int y, int x) {
    const double kk00 = __dmul_rn(kFrac, kFrac);
    double sum = 0.0;
    for (int v = 0; v < 8; v++) {
        const int4 lo = reinterpret_cast<const int4 *>(c + v * 8)[0], hi = reinterpret_cast<const int4 *>(c + v * 8)[1];
        const int32_t row[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        if (!(lo.x | lo.y | lo.z | lo.w | hi.x | hi.y | hi.z | hi.w)) continue;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if (row[u] == 0) continue;
            const double k = (u == 0 && v == 0) ? kk00 : (u == 0 || v == 0) ? kFrac : 1.0;
            double t = __dmul_rn(k, (double)row[u]);
            t = __dmul_rn(t, c_cos16[(2 * x + 1) * u]);
            t = __dmul_rn(t, c_cos16[(2 * y + 1) * v]);
            sum = __dadd_rn(sum, t);
        }
    }
    return sum / 4.0;
}

// The reference's binary64 2-4-8 transform for sample (y, x) (decoder.rs:555-602):
// butterfly of row pairs, horizontal pass per row (/ 2.0), four-term field pass (/ 2.0).
__device__ __noinline__ double exact_248(const int32_t *c, int y, int x) {
    const int field = y & 1, yy = y >> 1;
    double sum = 0.0;
    for (int v = 0; v < 4; v++) {
        const int4 *p = reinterpret_cast<const int4 *>(c + v * 16);
        const int4 a0 = p[0], a1 = p[1], b0 = p[2], b1 = p[3];
        const int32_t first[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
        const int32_t second[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
        double hs = 0.0;
#pragma unroll
        for (int u = 0; u < 8; u++) {
            if ((first[u] | second[u]) == 0) continue;
            const double b = field ? __dsub_rn((double)first[u], (double)second[u])
                                   : __dadd_rn((double)first[u], (double)second[u]);
            if (b != 0.0) hs = __dadd_rn(hs, __dmul_rn(__dmul_rn(u == 0 ? kFrac : 1.0, b), c_cos16[(2 * x + 1) * u]));
        }
        const double h = hs / 2.0;
        if (h != 0.0) sum = __dadd_rn(sum, __dmul_rn(__dmul_rn(v == 0 ? kFrac : 1.0, h), c_cos16[2 * (2 * yy + 1) * v]));
    }
    return sum / 2.0;
}

// Rounds half away from zero and clamps to 0..255.
__device__ __forceinline__ int dv_round_clamp(double e) {
    if (!(e > 0.0)) return 0;
    if (e >= 255.0) return 255;
    const int n = __double2int_rd(e);
    return n + (__dsub_rn(e, (double)n) >= 0.5 ? 1 : 0);
}

// The reference order for sample (y, x), rounded and clamped.
__device__ __forceinline__ uint8_t dv_exact_sample(const int32_t *c, bool mode248, int y, int x) {
    return (uint8_t)dv_round_clamp(mode248 ? exact_248(c, y, x) : exact_88(c, y, x));
}

// The sample of every position of a block whose only nonzero coefficient is the
// DC: all 64 are equal (cos16[0] = cos8[0] = 1.0, and only the u = v = 0 terms
// are nonzero: their factors of 1.0 and the sums with 0.0 change nothing). These
// blocks are common in smooth content, and with an odd DC level their exact value is
// a half-integer.
__device__ __forceinline__ uint8_t dv_flat_sample(const int32_t *c, bool mode248) {
    const double dc = (double)c[0];
    const double h = mode248 ? __dmul_rn(kFrac, __dmul_rn(kFrac, dc) * 0.5) * 0.5
                             : __dmul_rn(__dmul_rn(kFrac, kFrac), dc) * 0.25;
    return (uint8_t)dv_round_clamp(h);
}

// ---------------------------------------------------------------------------
// Eight threads per block: thread r takes column r in the vertical pass (with the
// 2-4-8 butterfly, exact), then row r in the horizontal pass. The factors are fp32
// products of the fp32 roundings, W[u][x] = (u ? 1 : FRAC) * cos16[(2x+1)u] and
// V4[yy][v] = (v ? 1 : FRAC) * cos16[2(2yy+1)v]. Where the outputs x and 7 - x share
// an eight-term sum (W[u][7-x] = (-1)^u W[u][x]), one packed FMA per pair of terms
// keeps the even and the odd sum side by side; a 2-4-8 column keeps its two fields
// side by side. All in all 32 packed FMAs a thread in either mode.

// The factors, as operands of the FMAs straight from constant memory (from shared memory
// they were 16 vector loads a thread: 1000 NTSC frames took 2.53 ms instead of 2.34). Row
// x < 4 holds W[0..7][x], then row yy < 4 (of four) V4[yy][0..3].
constexpr int kDvTable = 48;
constexpr int kDvV4 = 32;  // offset of V4 in it

struct DvFactors {
    float w[kDvTable];
};

constexpr DvFactors dv_factors() {
    constexpr double cs[128] = {
#include "cos_table.inc"
    };
    DvFactors t{};
    for (int i = 0; i < kDvV4; i++) t.w[i] = ((i & 7) == 0 ? (float)kFrac : 1.0f) * (float)cs[(2 * (i >> 3) + 1) * (i & 7)];
    for (int i = 0; i < 16; i++)
        t.w[kDvV4 + i] = ((i & 3) == 0 ? (float)kFrac : 1.0f) * (float)cs[2 * (2 * (i >> 2) + 1) * (i & 3)];
    return t;
}

__constant__ DvFactors c_dv_factors = dv_factors();

// (The passes take tables no more: for callers that have some.)
__device__ __forceinline__ void dv_fill_tables(float *, float * = nullptr) {}

// The eight-point sums out[i] = sum_u W[u][i] b[u], b as the pairs (b[0], b[1]), ...
__device__ __forceinline__ void dv_eight_point(const F2 (&b)[4], float (&out)[8]) {
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const float *w = c_dv_factors.w + i * 8;
        F2 s;  // (even, odd) terms
        s = fma2(f2(w[0], w[1]), b[0], s);
        s = fma2(f2(w[2], w[3]), b[1], s);
        s = fma2(f2(w[4], w[5]), b[2], s);
        s = fma2(f2(w[6], w[7]), b[3], s);
        float e, o;
        split2(s, e, o);
        out[i] = e + o;
        out[7 - i] = e - o;
    }
}

// First pass, thread r: the vertical sums of column r, outputs y = 0..7 into hcol
// (16-byte aligned). c: the block's 64 coefficients (natural order).
__device__ __forceinline__ void dv_row_pass8(const int32_t *c, const float *, bool mode248, int r, float *hcol) {
    float b[8], out[8];
#pragma unroll
    for (int v = 0; v < 8; v++) b[v] = (float)c[v * 8 + r];
    if (mode248) {
        F2 s[4];  // (field 0, field 1) of row yy
#pragma unroll
        for (int yy = 0; yy < 4; yy++) {
            const float *w = c_dv_factors.w + kDvV4 + yy * 4;
            // the butterfly of each row pair is exact: |c| < 2^23
            s[yy] = fma2(f2(w[0], w[0]), f2(b[0] + b[1], b[0] - b[1]), s[yy]);
            s[yy] = fma2(f2(w[1], w[1]), f2(b[2] + b[3], b[2] - b[3]), s[yy]);
            s[yy] = fma2(f2(w[2], w[2]), f2(b[4] + b[5], b[4] - b[5]), s[yy]);
            s[yy] = fma2(f2(w[3], w[3]), f2(b[6] + b[7], b[6] - b[7]), s[yy]);
            split2(s[yy], out[2 * yy], out[2 * yy + 1]);
        }
    } else {
        const F2 p[4] = {f2(b[0], b[1]), f2(b[2], b[3]), f2(b[4], b[5]), f2(b[6], b[7])};
        dv_eight_point(p, out);
    }
    reinterpret_cast<float4 *>(hcol)[0] = make_float4(out[0], out[1], out[2], out[3]);
    reinterpret_cast<float4 *>(hcol)[1] = make_float4(out[4], out[5], out[6], out[7]);
}

// Second pass, thread y: the samples of row y that the fp32 evaluation decides, packed
// little-endian (x = 0 in the low byte) into *row; returns the undecided ones as bits
// (x). h: the first pass's outputs, column u's at h + 8 * u. For a flat block (no nonzero
// AC coefficient) lane `flat_src` of the warp computes the one reference-order value and
// broadcasts it (all eight lanes of the block's group call this together).
__device__ __forceinline__ uint32_t dv_row_fp32(const int32_t *c, const float *h, const float *, const float *,
                                                bool mode248, int y, float c1, bool flat, int flat_src,
                                                unsigned group_mask, unsigned long long *row) {
    if (flat) {
        uint32_t v = 0;
        if ((int)(threadIdx.x & 31) == flat_src) v = dv_flat_sample(c, mode248);
        v = __shfl_sync(group_mask, v, flat_src);
        *row = 0x0101010101010101ull * v;
        return 0;
    }
    const F2 p[4] = {f2(h[y], h[8 + y]), f2(h[16 + y], h[24 + y]), f2(h[32 + y], h[40 + y]), f2(h[48 + y], h[56 + y])};
    float value[8];
    dv_eight_point(p, value);
#pragma unroll
    for (int x = 0; x < 8; x++) value[x] *= 0.25f;  // (exact; 8-8's / 4.0, 2-4-8's two / 2.0)
    // A value is certain when no half-integer lies within delta = 2^-21 C1 + 2^-30 of
    // it. (round_nearest holds below 2^22; |value| <= C1 / 4 + delta beyond that makes
    // delta more than a half.) Values past 256 + delta or below -1 - delta are clamped
    // whatever their rounding.
    const float delta = c1 * 0x1p-21f + 0x1p-30f, near = 0.5f - delta;
    int32_t n[8];
    uint32_t und = 0;
#pragma unroll
    for (int x = 0; x < 8; x++) {
        float r;
        n[x] = round_nearest(value[x], r);
        und |= (fabsf(value[x] - r) < near ? 0u : 1u) << x;
    }
    if (und) {
#pragma unroll
        for (int x = 0; x < 8; x++) {
            if (!(und >> x & 1)) continue;
            const bool over = value[x] > 256.0f + delta, under = value[x] < -1.0f - delta;
            if (over || under) und &= ~(1u << x);
            n[x] = over ? 255 : 0;  // (an undecided one is filled in later)
        }
    }
    *row = (unsigned long long)sat_quad_u8(n[4], n[5], n[6], n[7]) << 32 | sat_quad_u8(n[0], n[1], n[2], n[3]);
    return und;
}

constexpr int kDvManyTies = 12;

// Settles the undecided samples of every lane of the warp (all 32 lanes call
// this; und = 0 for lanes with none, whose bytes of row are 0). One sample at a time
// the whole warp forms its exact fixed-point value (exact_fixed.h); those too close to
// a half-integer for that take the reference order, each lane its own. (A block whose
// few coefficients have rational factors ties in all its samples: one after another
// they made one frame's transform wait 0.1 ms for one warp.)
// c: the lane's block coefficients (shared), c1i = sum |c| exactly, fix: the
// 8-8 table followed by the 2-4-8 table.
__device__ __forceinline__ void dv_resolve_row(uint32_t und, unsigned long long &row, const int32_t *c,
                                               bool mode248, int y, int32_t c1i, const long long *fix) {
    const int lane = threadIdx.x & 31;
    uint32_t m, left = 0;
    if (__ballot_sync(0xffffffffu, und != 0) == 0) return;
    // a block with many undecided samples ties in them: straight to the reference order
    int open = __popc(und);
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) open += __shfl_xor_sync(0xffffffffu, open, o);
    if (open >= kDvManyTies) {
        left = und;
        und = 0;
    }
    while ((m = __ballot_sync(0xffffffffu, und != 0)) != 0) {
        const int src = __ffs(m) - 1;
        const uint32_t sund = __shfl_sync(0xffffffffu, und, src);
        const int x = __ffs(sund) - 1;
        const int sy = __shfl_sync(0xffffffffu, y, src);
        const int smode = __shfl_sync(0xffffffffu, mode248 ? 1 : 0, src);
        const int32_t sc1 = __shfl_sync(0xffffffffu, c1i, src);
        const int32_t *sc = reinterpret_cast<const int32_t *>(
            __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(c), src));
        int smp = -1;
        if (sc1 < kFixMaxC1) smp = fixed_round(fixed_sum(fix + smode * kFixEntries + (sy * 8 + x) * 64, sc), sc1, 0);
        if (lane == src) {
            if (smp < 0) left |= 1u << x;
            else row |= (unsigned long long)smp << (8 * x);
            und &= und - 1;
        }
    }
    for (; left; left &= left - 1) {
        const int x = __ffs(left) - 1;
        row |= (unsigned long long)dv_exact_sample(c, mode248, y, x) << (8 * x);
    }
}

}  // namespace
}  // namespace mmr
