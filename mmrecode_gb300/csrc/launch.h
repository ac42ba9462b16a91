// Launches of a pipeline's kernels, one after another on a stream.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace mmr {

#if defined(__CUDACC__)
// First statement of every kernel that launch_next launches: waits for the kernel before it
// on the stream to end (its writes are visible then); `early` lets the next kernel's CTAs
// take their places, and wait there, from now on.
__device__ __forceinline__ void begin_kernel(bool early) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (early) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Blocks of a batch up to which that pays (320x240: 174 -> 169 us; a 1080p frame loses 3 us,
// and 64 mixed frames 4 %: CTAs wait where others could run).
constexpr uint64_t kEarlyBlocks = 32 << 10;

// Launches a kernel that is made ready while the kernel before it on the stream, one of the
// pipeline's own, runs and starts when its last CTA ends. A single frame's call is a dozen kernels of 2 to 25 us: 320x240
// 206 -> 180 us, 1080p 281 -> 266, 30 VGA frames 356 -> 350; 12 719x405 frames encoded from
// and to the host 233 -> 206, 60 1080p ones 1486 -> 1458.
template <class... P, class... A>
inline void launch_next(void (*kernel)(P...), dim3 grid, unsigned block, cudaStream_t s, A &&...args) {
    cudaLaunchAttribute early{};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = dim3(block);
    c.stream = s;
    c.attrs = &early;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, P(std::forward<A>(args))...);
}
#endif

}  // namespace mmr
