// fem_launch.cuh -- kernel launches that may begin before the previous kernel of the
// stream has ended (programmatic dependent launch).
//
// The kernel must call cudaGridDependencySynchronize() before it touches what earlier
// kernels write, and, if it triggers a dependent launch itself, only after that (or it is
// never launched with overlap): a later kernel may then take everything before its
// predecessor as complete.  Data that the predecessor writes is read with plain loads,
// not __ldg or const __restrict__, which may move ahead of the wait.  overlap
// is set only where the previous operation of the stream is a kernel of this library,
// one of another library may trigger before its inputs are complete.
#pragma once

#include <cuda_runtime.h>

namespace fem {

template <class... P, class... A>
cudaError_t launch_kernel(void (*f)(P...), dim3 blocks, unsigned threads, size_t smem, cudaStream_t st, bool overlap,
                          const A&... args) {
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = blocks;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = overlap ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, f, P(args)...);
}

}  // namespace fem
