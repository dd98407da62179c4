// Launches of the step's kernels on one stream, each able to start while the one before drains.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace lbmh {

// First statement of every kernel that a step launches with launch_next (before it touches memory
// another kernel writes): lets the next kernel of the stream be set up on the SMs as this one's last
// blocks start, then waits until the kernel before has finished and its writes are visible.  Without
// the launch attribute both instructions do nothing.
__device__ __forceinline__ void step_begin() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// kernel<<<grid, block, smem, stream>>>(args...); `follows`: the stream's work just before this launch is
// a kernel, whose completion the new kernel awaits itself (step_begin) instead of being launched after
// it.  A gap between dependent kernels is some 2 us of idle SMs otherwise, which is what small
// lattices spend their steps on (16^3 single component: 10.4 -> 8.3 us a step, 64^3 80 -> 74 us).
template <class... P, class... A>
cudaError_t launch_next(bool follows, void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t stream,
                        A &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = follows ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

}  // namespace lbmh
