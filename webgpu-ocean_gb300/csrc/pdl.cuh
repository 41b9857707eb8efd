// pdl.cuh -- programmatic dependent launch: a kernel's blocks may be placed,
// and run up to pdl_wait(), while the kernel before it in the stream finishes.
//
// For chains of short kernels launched one by one.  A kernel calls pdl_begin()
// first, which lets in the blocks of the next one (if launch_pdl() launched it)
// once all of its own have started.  A kernel that launch_pdl() launches calls
// pdl_wait() in every thread before it touches memory that any kernel of the
// chain writes or still reads: that returns when the kernel before it has
// finished and its writes are visible.  Every kernel of a chain waits, so a
// finished one implies that all before it have finished too.
//
//   - The chain's first kernel is launched plainly: what came before the chain,
//     of any kind and on any stream that was joined, has then finished, so
//     its inputs are read-only for the life of every kernel of the chain.
//   - A buffer that the chain itself writes is not read through a const
//     __restrict__ pointer: the compiler may take such loads for invariant and
//     move them above the wait.
//
// Captured into a graph, the dependency becomes a programmatic edge between the
// two kernels.
#pragma once
#include <cuda_runtime.h>

namespace mpm {

__device__ __forceinline__ void pdl_begin() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Errors are left for cudaGetLastError(), as with <<<>>>.
template <class... P, class... A>
void launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                const A&... args) {
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    (void)cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace mpm
