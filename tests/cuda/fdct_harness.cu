// Block-level harness for the forward DCT as the encoder decides it: fdct_kernel's functions
// (fdct_core.h) with its thread mapping (8 threads per block) and its one error bound per
// block; coefficients it leaves open in the reference's binary64 order. Built by the tests
// with nvcc; not part of the library.
#include <cuda_runtime.h>
#include <stdint.h>

#include "fdct_core.h"

namespace mmr {
namespace {

constexpr int kBlocks = 32, kStride = 9;

__global__ void __launch_bounds__(kBlocks * 8) fdct_block_bound(const uint8_t *samples, const uint8_t *qt,
                                                                const float *rq, uint64_t n, int32_t *out,
                                                                unsigned long long *exact) {
    __shared__ float s_t[kBlocks][8 * kStride];
    const int lb = threadIdx.x >> 3, r = threadIdx.x & 7;
    const uint64_t b = (uint64_t)blockIdx.x * kBlocks + lb;
    const bool valid = b < n;
    float mag = 0.0f;
    if (valid) {
        float s[8];
        for (int x = 0; x < 8; x++) {
            s[x] = (float)samples[b * 64 + r * 8 + x] - 128.0f;
            mag += fabsf(s[x]);
        }
        for (int u = 0; u < 8; u++) s_t[lb][r * kStride + u] = fdct_row(s, u);
    }
    for (int o = 1; o < 8; o <<= 1) mag += __shfl_xor_sync(0xffffffffu, mag, o);
    __syncwarp();
    if (!valid) return;
    const int u = r;
    float t[8];
    for (int y = 0; y < 8; y++) t[y] = s_t[lb][y * kStride + u];
    uint2 rows[8];
    for (int y = 0; y < 8; y++) rows[y] = *reinterpret_cast<const uint2 *>(samples + b * 64 + y * 8);
    uint32_t open = 0;
    for (int v = 0; v < 8; v++) {
        bool unsure;
        const uint64_t at = b * 64 + v * 8 + u;
        int k = fdct_round(fdct_column(t, v), mag * kFdctBound, rq[at], unsure);
        if (unsure) {
            k = exact_coefficient(c_m64, rows, u, v, qt[at]);
            open++;
        }
        out[at] = k;
    }
    if (open) atomicAdd(exact, (unsigned long long)open);
}

}  // namespace
}  // namespace mmr

// n blocks of 64 samples with a quantiser table (and its fp32 reciprocals) each; host arrays
// in and out. Returns a CUDA error code (0 = success); *exact: coefficients left open.
extern "C" int harness_fdct_block_bound(const uint8_t *samples, const uint8_t *qt, const float *rq, uint64_t n,
                                        int32_t *out, unsigned long long *exact) {
    uint8_t *d = nullptr;
    const size_t o_qt = n * 64, o_rq = 2 * n * 64, o_out = o_rq + n * 256, o_exact = o_out + n * 256;
    cudaError_t e = cudaMalloc((void **)&d, o_exact + 8);
    if (e == cudaSuccess) e = cudaMemcpy(d, samples, n * 64, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + o_qt, qt, n * 64, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(d + o_rq, rq, n * 256, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(d + o_exact, 0, 8);
    if (e == cudaSuccess && n) {
        mmr::fdct_block_bound<<<(unsigned)((n + mmr::kBlocks - 1) / mmr::kBlocks), mmr::kBlocks * 8>>>(
            d, d + o_qt, reinterpret_cast<const float *>(d + o_rq), n, reinterpret_cast<int32_t *>(d + o_out),
            reinterpret_cast<unsigned long long *>(d + o_exact));
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, d + o_out, n * 256, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(exact, d + o_exact, 8, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return (int)e;
}
