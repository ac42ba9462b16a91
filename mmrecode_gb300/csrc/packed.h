// Packed operations: two fp32 FMAs in one instruction (each rounded as its scalar
// form), and saturating byte packs.
#pragma once

#include <stdint.h>

#include <cuda_runtime.h>

namespace mmr {

struct F2 {
    unsigned long long v = 0;  // two floats, the first in the low half (0: both +0.0)
};

__device__ __forceinline__ F2 f2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
    return r;
}

__device__ __forceinline__ void split2(const F2 &x, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}

__device__ __forceinline__ F2 fma2(const F2 &a, const F2 &b, const F2 &c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

__device__ __forceinline__ F2 mul2(const F2 &a, const F2 &b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

__device__ __forceinline__ F2 add2(const F2 &a, const F2 &b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}

// a - b (as a + -1.0 * b: one rounding)
__device__ __forceinline__ F2 sub2(const F2 &a, const F2 &b) { return fma2(b, f2(-1.0f, -1.0f), a); }

// Four values saturated to 0..255 and packed, b0 in the low byte
// (cvt.pack.sat: d = c << 16 | sat(a) << 8 | sat(b)).
__device__ __forceinline__ uint32_t sat_quad_u8(int32_t b0, int32_t b1, int32_t b2, int32_t b3) {
    uint32_t hi, d;
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(hi) : "r"(b3), "r"(b2), "r"(0));
    asm("cvt.pack.sat.u8.s32.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(b1), "r"(b0), "r"(hi));
    return d;
}

}  // namespace mmr
