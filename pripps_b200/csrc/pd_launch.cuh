// Dependent launches: a solve is a chain of short kernels on one stream (a 3,000-atom
// one 7 kernels in 75 µs), and the launch of a kernel costs 1 to 2 µs between the end
// of one and the first instruction of the next. A kernel launched with `after_kernel`
// may start while the previous one of its stream ends: its blocks take their places
// and wait in chain_enter for the previous kernel to be complete, its writes visible.
#pragma once

#include <cuda_runtime.h>

namespace pd {

// First statement of every kernel of the chain, before any access to memory. The
// next kernel's blocks may be scheduled as soon as all of this kernel's have started;
// each kernel waits, so a kernel that is complete has complete predecessors.
__device__ __forceinline__ void chain_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// after_kernel: the operation before it on the stream is a kernel of the chain, with
// no event, copy or memset between.
template <class... P, class... A>
inline cudaError_t chain_launch(bool after_kernel, void (*kernel)(P...), dim3 grid, dim3 block,
                                size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = after_kernel ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace pd
