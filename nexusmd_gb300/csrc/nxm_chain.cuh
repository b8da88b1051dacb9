// Kernels that follow one another in a stream and are short: each may be placed
// on the GPU while the one before it still runs, and waits there for its end
// (programmatic dependent launch), which takes launch latency out of a chain of
// five-microsecond kernels.  For the no-allocation PME on one stream: 77 -> 72
// us.  Not in the engine: as nodes of its step graph, beside the other branch,
// the same links made the step slower (2,700 atoms 44 -> 56 us, 94,100 235 ->
// 264), and blocks that wait take the place of running ones.
#pragma once

#include <cuda_runtime.h>

namespace nxm {

// At the start of a kernel of such a chain: the next may be placed; the one
// before has ended and its writes are seen.  Nothing that the kernels before
// wrote is read, and nothing is written, ahead of this.
__device__ __forceinline__ void chain_link() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// kernel<<<grid, block, smem, st>>>(args...), as a link behind the kernel
// before it in the stream when `chained` is set.
template <typename... P, typename... A>
inline void launch_link(bool chained, void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t st,
                        const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace nxm
