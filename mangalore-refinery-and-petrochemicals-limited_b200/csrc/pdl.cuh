// Programmatic dependent launch: a kernel of an iteration may be scheduled while its
// predecessor still runs, does what does not depend on it, and waits for it here.  What a
// kernel reads before pdl_wait must be older than the predecessor's own predecessor, or never
// change between the two.
#pragma once

#include <cuda_runtime.h>

namespace b2p {

// Everything the preceding kernels of the stream wrote is visible after this.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel may be scheduled from here on (its own pdl_wait still waits for this one to end).
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches fn so that it may overlap the end of the kernel before it.
template <typename... P, typename... A>
cudaError_t pdl_launch(void (*fn)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s, A... args) {
    cudaLaunchConfig_t lc{};
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.gridDim = dim3(grid);
    lc.blockDim = dim3(block);
    lc.dynamicSmemBytes = smem;
    lc.stream = s;
    lc.attrs = &at;
    lc.numAttrs = 1;
    return cudaLaunchKernelEx(&lc, fn, static_cast<P>(args)...);
}

}  // namespace b2p
