// Launches that start while the launch before them in the stream ends (programmatic stream
// serialisation): the kernel's CTAs set up what depends on nothing, then wait.
#pragma once
#include <cuda_runtime.h>

namespace rc {

// In a kernel launched with launch_early: lets the next such launch start, then waits until
// the launch before has ended and its memory is visible.  Nothing that launch reads or
// writes may be touched above.
__device__ __forceinline__ void early_launch_wait() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
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
