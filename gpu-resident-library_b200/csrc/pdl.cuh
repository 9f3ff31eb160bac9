// Dependent launches within one call's chain of kernels (programmatic
// dependent launch). A kernel launched with `after_kernel` may be launched
// before the kernel ahead of it on the stream has ended; chain_begin() at its
// start waits until that kernel has finished and its writes are visible, so
// nothing is read or written early. Every kernel of a chain waits, so the
// order is that of plain launches, transitively. The first kernel of a chain,
// and one that follows an event or another stream's work, is launched plainly.
// What is bound here is the gap between small kernels: one product at N = 2^15
// (10 kernels) 108.5 -> 89.1 us, a 3 + 3 rotation transform at N = 2^13 404 ->
// 373 us, 5 products at N = 2^16 463 -> 461 us. No kernel releases its
// successor early: its blocks then fill whichever SMs run dry first instead of
// spreading (one product 105-111 us, the transform 410 us), and a release
// before a kernel's last round gave 91 and 372 us.
#pragma once
#include <cuda_runtime.h>

namespace gfx {

__device__ __forceinline__ void chain_begin() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t chain_launch(void (*kernel)(P...), bool after_kernel, dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                         A&&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = after_kernel ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace gfx
