// Launches of kernels that follow one another (the multigrid's, the network's).
#pragma once
#include <cuda_runtime.h>

namespace lica {

// Chained launches.  The kernels of a solve are a chain of short launches, each of which needs all
// of the one before it, and between two of them the chip stood idle for the launch, the CTAs' start
// and their first loads.  A kernel launched by launch_next may start early, set itself up and read
// what no kernel since the set-up writes (the weights); it waits in after_previous() until the one
// before has ended, which itself waited for the one before it, and its stores can be seen.  What the
// kernels before wrote is read through pointers that are not both const and __restrict__, so that no
// read of it can be moved above the wait.
//
// EARLY: the next kernel may start once all CTAs of this one have, otherwise once they have all
// passed the wait.  A kernel starts only after every CTA of the one before it has, so those that
// wait take no room from one that must still start.  Early is better where the CTAs are large and
// their weights many (red-black, 1024 x 1024 cells: a solve 1.57 -> 1.49 ms chained, 1.45 early;
// two 512 x 1536 film steps 9.9 -> 9.66, 9.50), late where a launch is a few small CTAs (y-lines,
// 256 x 256: 12.1 -> 11.0 ms, 11.6 early).
// The network (early): the guess of a 1024 x 1024 image 709 -> 680 us, four 256 x 256 images'
// gradient 1115 -> 998.  A kernel that takes tensor memory takes it after the wait: the one before,
// whose CTAs may only just have started, must find it free.
template <bool EARLY = true>
__device__ __forceinline__ void after_previous() {
    if (EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (!EARLY) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... P, typename... A>
cudaError_t launch_next(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace lica
