// Programmatic dependent launch of the iteration-body kernels.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace dphd {

bool pdl_enabled();  // process-wide switch (set_pdl), read when a kernel is launched or captured

// Each kernel launched by launch_k may start while its predecessor in the stream drains.  It begins with
// pdl_enter: it lets its own successor launch, then waits (griddepcontrol.wait) until the predecessor grid has
// completed and its memory is visible, before reading anything.  Launched without the attribute, the wait returns
// at once.  Every such kernel then reads ctrl->done with an ordinary load (ordered after the wait's memory
// clobber) and branches on it before it touches data a predecessor wrote: loads through the read-only path
// (ld.global.nc, which the compiler may treat as invariant and move across the wait) stay behind that branch, so
// none is issued before the wait.  A kernel without that branch (k_noalloc_prepare) reads what a predecessor may have
// written through pointers that are not __restrict__.
__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// Launches `kern` with programmatic stream serialization when the switch is on; inside stream capture this becomes
// a programmatic edge of the graph.
template <typename... KArgs, typename... Args>
void launch_k(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...);
}

}  // namespace dphd
