// Launch with programmatic stream serialisation.
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace sblas {

// The kernel may start while the previous kernel of the stream finishes, and
// waits for it (ptx::griddep_wait) before it touches global memory.  Every
// thread of a kernel launched this way must execute that wait: a kernel's
// completion then implies its predecessors' completion, however long the
// chain of such launches.
template <class... KArgs, class... Args>
cudaError_t launch_pdl(void (*kfn)(KArgs...), dim3 grid, dim3 block, size_t smem,
                       cudaStream_t stream, Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kfn, std::forward<Args>(args)...);
}

}  // namespace sblas
