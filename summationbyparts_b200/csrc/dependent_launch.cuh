// Programmatic dependent launch: a kernel may start while its predecessor in the stream drains, so
// that launch latency, barrier set-up and index arithmetic overlap the predecessor's last wave.
#pragma once

#include <cuda_runtime.h>

namespace sbp {

// Returns once every earlier kernel of the stream has completed and its writes are visible; only then
// does the kernel let its own successor start, so that what a successor does before its wait sees
// finished work up to its predecessor's predecessor.  Every CTA that touches global memory calls it.
__device__ __forceinline__ void dependency_wait() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Dependent launch of a kernel that calls dependency_wait.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

}  // namespace sbp
