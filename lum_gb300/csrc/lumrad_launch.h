// lumrad_launch.h — kernel launches, plain or as programmatic dependents of the stream's previous kernel.
#pragma once
#include <cuda_runtime.h>
#include <utility>

namespace lumrad {

// A launch of `kern`; dependent: as a programmatic dependent of the stream's previous kernel.  It may
// start once every CTA of that kernel has called grid_launch_dependents (or ended); what it reads
// or overwrites of earlier work waits in grid_dependency_wait, which returns when that kernel has
// ended.  Every kernel launched so waits before it ends itself: the end of a kernel then is the
// end of all work before it in the stream.
template <class... P, class... A>
cudaError_t launch_kernel(void (*kern)(P...), dim3 blocks, dim3 threads, size_t smem, cudaStream_t stream, bool dependent,
                          A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, P(std::forward<A>(args))...);
}

}  // namespace lumrad
