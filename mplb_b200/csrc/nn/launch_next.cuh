// The network's launches: the kernels of a pass are queued one behind the other,
// each with programmatic stream serialisation.  No kernel triggers its successor
// early, so the next one's CTAs come in when the last CTA has ended, and their
// set-up (arguments, barriers, tensor memory) runs beside the flush of the
// results, which GridWait waits for.  A pass of 32 images is 30 to 80 launches of
// 5 to 90 us: 256 predictions take 4.42 ms so and 4.85 in plain launches, four
// training steps of 32 6.47 and 7.14.
#pragma once

#include <cuda_runtime.h>

namespace mplb {
namespace nn {

// Waits until everything queued before this kernel has ended; nothing that
// another launch writes or reads is touched in front of it.
__device__ __forceinline__ void GridWait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches a kernel that calls GridWait; errors are left for cudaGetLastError.
template <typename... P, typename... A>
void LaunchNext(void (*kernel)(P...), dim3 grid, unsigned threads, int smem,
                cudaStream_t s, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

}  // namespace nn
}  // namespace mplb
