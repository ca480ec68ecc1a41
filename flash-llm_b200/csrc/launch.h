// Kernel launches of this library.
//
// Every kernel is launched with the programmatic-serialisation attribute and executes griddepcontrol.wait before it
// touches global memory (an SpMM with launch overlap on: before it touches anything but its weights), so a call keeps
// plain stream order, while the launch itself and the kernel's set-up no longer wait for the predecessor to drain.
// How early that is, the predecessor says with griddepcontrol.launch_dependents; the kernels that write an encoding
// do not, so that an SpMM with launch overlap on, which reads its weights before it waits, starts when they have ended.
// What that is worth: on B200 with driver 580.159 a chain of plain launches advances in steps of 2.048 us (a kernel of
// 1.0 us takes 4.1 us per launch, one of 2.5 us takes 6.1 us); with the attribute the same kernels take 2.05 and 2.6 us.
#pragma once
#include <cuda_runtime.h>

#include "tiled_csl_host.h"

namespace flashllm {

template<typename... Params, typename... Args>
inline cudaError_t launch_in_stream_order(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream,
                                          int cluster_x, Args&&... args)
{
    cudaLaunchConfig_t  cfg{};
    cudaLaunchAttribute attr[2];
    cfg.gridDim                                        = grid;
    cfg.blockDim                                       = block;
    cfg.dynamicSmemBytes                               = smem;
    cfg.stream                                         = stream;
    attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id                                         = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x                           = static_cast<unsigned>(cluster_x);
    attr[1].val.clusterDim.y                           = 1;
    attr[1].val.clusterDim.z                           = 1;
    cfg.attrs                                          = attr;
    cfg.numAttrs                                       = cluster_x > 1 ? 2 : 1;
    count_launch();
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

}  // namespace flashllm
