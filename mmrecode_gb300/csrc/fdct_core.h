// The reference's forward DCT and quantisation reproduced exactly
// (crates/codecs/mjpeg/src/transform.rs:111-134 forward_dct_quantize): an fp32
// evaluation with an error bound, and the binary64 reference
// order for quotients within that bound of a half-integer. fdct_kernel (8 threads per
// block) takes one bound per block (fdct_row, fdct_column, fdct_round, kFdctBound,
// exact_coefficient), as does a block-level test; fdct_row_pass and fdct_quantise take the
// tighter bound per coefficient and are the other block-level test's alone.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "rounding.h"
#include "tables.h"

namespace mmr {
namespace {

__constant__ float c_m32[64] = MMR_IDCT_MATRIX_INIT;   // IDCT_MATRIX[x][u] at x * 8 + u, rounded to fp32
__constant__ double c_m64[64] = MMR_IDCT_MATRIX_INIT;  // the reference's binary64 values

// The quantised coefficient (v, u) of a block exactly as forward_dct_quantize
// (transform.rs:111-134) computes it: binary64, every product and sum rounded
// separately, rows accumulated over x, then the column over y, both from 0.0,
// the quotient rounded half away from zero. m: the reference's matrix (c_m64, or a
// copy in shared memory, where lanes index it freely); rows: the samples, row y's
// sample x in bits 8x of rows[y].
__device__ __forceinline__ int exact_coefficient(const double *m, const uint2 (&rows)[8], int u, int v, int q) {
    double mu[8], value = 0.0;
#pragma unroll
    for (int x = 0; x < 8; x++) mu[x] = m[x * 8 + u];
#pragma unroll
    for (int y = 0; y < 8; y++) {
        double t = 0.0;
#pragma unroll
        for (int x = 0; x < 8; x++) {
            const int s = (int)(((x < 4 ? rows[y].x : rows[y].y) >> (8 * (x & 3))) & 0xff) - 128;
            t = __dadd_rn(t, __dmul_rn(mu[x], (double)s));
        }
        value = __dadd_rn(value, __dmul_rn(m[y * 8 + v], t));
    }
    return (int)round(__ddiv_rn(value, (double)q));
}

// Error bound of the fp32 path, per coefficient. With S = sample - 128 and the
// coefficient's magnitude sum B = sum_y |M[y][v]| sum_x |M[x][u]| |S[y][x]|: both
// passes use the basis' symmetry M[7-x][u] = (-1)^u M[x][u] (the fp32 roundings of
// the reference's literals are exactly symmetric, the literals themselves to less
// than 2e-15), so a pass is a four-term FMA chain over M[x][u] (a[x] +- a[7-x]).
// In the row pass the sums of samples are exact: 4 roundings and the fp32 matrix
// entry, 5 * 2^-24 of its magnitude sum; the column pass adds one rounding for the
// sum, 4 for the chain and one for the entry: |V32 - V64| <= 11 * 2^-24 * B +
// 2^-46 * B (second-order terms and the binary64 chains) < 6.6e-7 * B. The fp32
// quotient is V32 times the rounded reciprocal of q (two roundings of 2^-24 each:
// within 1.2e-7 |q32| of V32 / q, and |q32| <= 1.001 B / q) and the binary64 one is
// within 2^-53 |V64 / q|, so |q32 - q64| < 7.9e-7 * B / q + 1e-12. The guard takes
// 1.1e-6 and 1e-9 for these, B being an upper bound computed in fp32 (within 2^-20
// relative): a fp32 quotient farther than that from the nearest half-integer rounds
// to the reference's integer; the rest are recomputed in binary64. (B <= 1970 for
// the whole-block bound below, so the guard never exceeds 3e-3.)
__device__ __forceinline__ float tie_guard(float b, float rq) { return fmaf(1.1e-6f * b, rq, 1e-9f); }

// B of every coefficient of a block is at most Mmax^2 sum |S| = 0.2405 sum |S|:
// one bound for the block costs a row sum and three shuffles instead of a second
// transform over magnitudes.
constexpr float kFdctBound = 0.2406f;

// Row pass output (r, u): t = sum_x M[x][u] S[r][x] over the row's centred
// samples srow[x] = sample - 128.
__device__ __forceinline__ float fdct_row(const float *srow, int u) {
    const float sg = u & 1 ? -1.0f : 1.0f;
    float a = c_m32[u] * fmaf(sg, srow[7], srow[0]);
#pragma unroll
    for (int x = 1; x < 4; x++) a = fmaf(c_m32[x * 8 + u], fmaf(sg, srow[7 - x], srow[x]), a);
    return a;
}

// Column pass: the coefficient (v, u) from its column's row-pass outputs t[y].
__device__ __forceinline__ float fdct_column(const float *t, int v) { return fdct_row(t, v); }

// The quotient of a coefficient rounded to the nearest integer, and whether it lies
// too close to a half-integer for that to be certain (b: an upper bound of its B).
__device__ __forceinline__ int fdct_round(float acc, float b, float rq, bool &unsure) {
    const float quot = acc * rq;  // |quot| <= 1025
    float r;
    const int k = round_nearest(quot, r);
    unsure = !(fabsf(quot - r) < 0.5f - tie_guard(b, rq));
    return k;
}

// Row pass output and its magnitude sum sum_x |M[x][u]| |S[r][x]|.
__device__ __forceinline__ void fdct_row_pass(const float *srow, int u, float &acc, float &mag) {
    float m = 0.0f;
#pragma unroll
    for (int x = 0; x < 8; x++) m = fmaf(fabsf(c_m32[x * 8 + u]), fabsf(srow[x]), m);
    acc = fdct_row(srow, u);
    mag = m;
}

// Quantised coefficient (v, u) from the row-pass outputs rows[y * stride + u]
// and their magnitude sums mags[..] (raw: the block's 64 samples, q the
// quantiser, rq its fp32 reciprocal). exact reports whether the binary64
// reference order decided it. Unclamped.
__device__ __forceinline__ int fdct_quantise(const float *rows, const float *mags, int stride, const uint8_t *raw,
                                            int u, int v, int q, float rq, bool &exact) {
    float t[8], mag = 0.0f;
#pragma unroll
    for (int y = 0; y < 8; y++) {
        t[y] = rows[y * stride + u];
        mag = fmaf(fabsf(c_m32[y * 8 + v]), mags[y * stride + u], mag);
    }
    const int k = fdct_round(fdct_column(t, v), mag * (1.0f + 1.0f / 1048576.0f), rq, exact);
    if (!exact) return k;
    uint2 w[8];
#pragma unroll
    for (int y = 0; y < 8; y++) {
        w[y] = make_uint2(0, 0);
#pragma unroll
        for (int x = 0; x < 4; x++) {
            w[y].x |= (uint32_t)raw[y * 8 + x] << (8 * x);
            w[y].y |= (uint32_t)raw[y * 8 + 4 + x] << (8 * x);
        }
    }
    return exact_coefficient(c_m64, w, u, v, q);
}

}  // namespace
}  // namespace mmr
