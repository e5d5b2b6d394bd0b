// dependent_launch.cuh -- programmatic dependent launch: a kernel launched
// with it is made ready while the one before it in the stream still runs, starts
// as that one's last blocks end, and waits (grid_wait) until its writes are
// visible before it reads them.  Every kernel of a chain waits, so the end of
// one implies the end of all before it.
//
// No kernel lets the next one start earlier (griddepcontrol.launch_dependents):
// blocks that start while others still hold most of the SMs crowd onto the few
// free ones, and a grid that does not fill the GPU then stays there (the
// recursion's vertical walk after prep: 168 -> 280 us a call; a 256x192 pair's
// tile pass: 34.3 -> 36.7).
#pragma once
#include <cuda_runtime.h>

namespace dep {

__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with (early) or without programmatic dependence on the kernel before it.
template <typename... Params, typename... Args>
cudaError_t launch(bool early, void (*kernel)(Params...), dim3 grid, int block, size_t smem, cudaStream_t st,
                   Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace dep
