// mgr_launch.hh — kernel launches with programmatic stream serialisation.
#pragma once

#include <cuda_runtime.h>

#include <stdexcept>
#include <string>

namespace mgr {

// A launch that may start while the kernel before it in the stream is still
// running (the kernel waits in pdl_wait before it reads that kernel's
// outputs), or a plain stream-ordered launch.  A launch that fails is reported
// at once: no kernel after it runs on what it would have written.
template <typename... KArgs, typename... Args>
inline void launch_pdl(bool pdl, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                       Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string("kernel launch: ") + cudaGetErrorString(e));
    }
}

}  // namespace mgr
