// Programmatic dependent launch.
#pragma once

#include <cuda_runtime.h>

namespace gbds {

// Programmatic dependent launch: the next kernel launched on the stream with
// the programmatic-serialisation attribute may start its blocks once every
// block of this grid has started; it waits (griddepcontrol.wait) for this
// grid's completion and memory before its first global read.  Without the
// attribute both instructions are no-ops.
__device__ __forceinline__ void pdl_allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_prev() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launch with the programmatic-serialisation attribute (see pdl_wait_prev).
template <typename... P, typename... A>
void launch_pdl_smem(void (*kernel)(P...), dim3 grid, int block, size_t smem, cudaStream_t stream, const A &...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    // a failed launch also sets the runtime's last error, which every
    // launcher returns through cudaGetLastError()
    (void)cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <typename... P, typename... A>
void launch_pdl(void (*kernel)(P...), dim3 grid, int block, cudaStream_t stream, const A &...args) {
    launch_pdl_smem(kernel, grid, block, 0, stream, args...);
}

}  // namespace gbds
