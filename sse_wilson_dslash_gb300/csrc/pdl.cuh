// Programmatic dependent launch.
#pragma once

#include <cuda_runtime.h>

namespace gbds {

// Programmatic dependent launch: the next kernel launched on the stream with
// the programmatic-serialisation attribute may start its blocks once every
// block of this grid has started; it waits (griddepcontrol.wait) for this
// grid's completion and memory before its first global read.  Without the
// attribute both instructions are no-ops.  Where all blocks of a grid are
// resident at once, those of the next come up right away and sit beside it for
// its whole run, their shared memory taken out of its L1 cache; kernels that
// live on that cache only allow it from a second wave on, or not at all (the
// next grid is then launched, its parameters in place, when this one ends).  us
// with the early start / without: FP64 on 12^2x16x20 22.5 / 16.6 (16^3x32, two
// waves: 38.2 / 38.7); 12 rhs on 8^3x16 9.2 / 6.2; 2 rhs on 10x14x12x20 6.9 /
// 5.3; FP32 on 32^3x40 78.2 / 79.6.  The multi-RHS kernels never allow it: on large
// lattices it makes no difference (24^3x48: FP32 12 rhs 260.9 / 260.7, bfloat16 32
// rhs 406.6 / 406.5), on 16^3x32 FP32 with 4 rhs takes 20.3 / 19.7.
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
