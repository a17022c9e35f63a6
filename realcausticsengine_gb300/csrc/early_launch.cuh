// Launches that start while the launch before them in the stream ends (programmatic stream
// serialisation): the kernel's CTAs set up what depends on nothing, then wait.
#pragma once
#include <cuda_runtime.h>

namespace rc {

// In a kernel launched with launch_early: waits until the launch before has ended and its
// memory is visible, then lets the next such launch start.  Above it nothing may be touched
// that the launch before writes, and nothing written that it reads; what the launch before
// that one wrote is complete (read past L1: __ldcg), because the launch before let this one
// start after its own wait.  The kernel's pointers carry no __restrict__: a load through a
// const restrict pointer may be taken for a read of constant memory, past the wait's clobber
// and past L1 coherence.
__device__ __forceinline__ void early_launch_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <class... P, class... A>
void launch_early(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &at;
    c.numAttrs = 1;
    cudaLaunchKernelEx(&c, kernel, static_cast<P>(args)...);
}

}  // namespace rc
