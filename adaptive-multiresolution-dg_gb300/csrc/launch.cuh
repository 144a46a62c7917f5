// Launch of kernels that may begin before the previous kernel of their stream has ended.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace amdg {

// Programmatic stream serialisation: the kernel's CTAs may be scheduled once every CTA of the
// previous kernel has executed griddepcontrol.launch_dependents or ended.  The kernel executes
// griddepcontrol.wait before it reads or writes anything a kernel of the stream writes, and
// launch_dependents after that wait, so that what it does before the wait can rely on every kernel
// but the previous one.
template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
}

#ifdef __CUDACC__
// wait until the previous kernel of the stream has ended and its writes are visible, then let the next
// kernel begin
__device__ __forceinline__ void wait_for_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif

}  // namespace amdg
