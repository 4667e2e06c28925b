// Launches that are set up while the kernel in front of them still runs, and
// kernels with more than 48 KB of dynamic shared memory.
#pragma once
#include <cuda_runtime.h>

#include "once_per_device.h"

namespace hbl {

// Launches in a chain: every kernel waits for the one in front of it at its
// first instruction, so it may be set up while that one still runs. A launch
// then costs 1.4 us instead of 4.1 (152 to 1216 blocks, measured back to back).
// A kernel that is launched chained waits before anything else, in every block:
// what stands behind it relies on that.
__device__ __forceinline__ void wait_for_launch() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline cudaError_t launch(bool chained, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s,
                          A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <class... P, class... A>
inline cudaError_t chain(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
    return launch(true, kernel, grid, block, smem, s, args...);
}

// Lets `kernel` take `bytes` of dynamic shared memory on the current device (from
// 48 KB on a device refuses the launch otherwise). `once` is the kernel's own.
template <class... P>
inline cudaError_t allow_shared(OncePerDevice& once, void (*kernel)(P...), size_t bytes) {
    int device = -1;
    const cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    return (cudaError_t)once(device, [&] {
        return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    });
}

}  // namespace hbl
