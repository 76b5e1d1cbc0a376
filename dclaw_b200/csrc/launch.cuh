// launch.cuh -- programmatic dependent launch of a chain of kernels.
#pragma once
#include <cuda_runtime.h>

namespace dclaw {

// A kernel launched with launch_pdl calls pdl_wait before it reads or writes
// anything: the kernel before it on the stream has then completed and its
// writes are visible (pdl_wait returns at once in a kernel launched the
// ordinary way). The launch itself no longer waits for the stream: with
// ordinary launches ten 64^2 steps took 0.69 ms and four 1000 x 731 steps
// 1.036 ms, with these 0.585 and 0.993 ms. No kernel lets the next one start
// while it runs (griddepcontrol.launch_dependents): CTAs of the next kernel
// then hold places on the SMs while they wait, which took back the gain
// (0.617 and 1.055 ms when every kernel did so at its start, 0.609 and
// 1.001 ms at the end of its work).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... KArgs, typename... Args>
inline void launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace dclaw
