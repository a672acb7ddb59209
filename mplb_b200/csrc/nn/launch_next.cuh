// The network's launches: kernels of a pass are queued one behind the other, and
// each sets itself up (arguments, barriers, tensor memory, clearing) while the
// last CTAs of the one before it run.  32 images' passes are 30 to 80 launches of
// 5 to 90 us: 256 predictions 4.85 -> 4.42 ms,
// four training steps of 32 7.14 -> 6.47.
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
