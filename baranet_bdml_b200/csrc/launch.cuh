// How kernels are launched with attributes (host code alone)
#pragma once

#include <cuda_runtime.h>

namespace bn {

// Launches with the attributes of `cfg`; where that is refused, with the first `needed` of them alone: a kernel cannot do without its
// cluster's size, but without being a programmatic dependent it only starts later.
template <typename... P, typename... A>
inline cudaError_t launch_config(cudaLaunchConfig_t cfg, unsigned needed, void (*kernel)(P...), A... args) {
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (e != cudaSuccess && cfg.numAttrs > needed) {
        (void)cudaGetLastError();
        cfg.numAttrs = needed;
        e = cudaLaunchKernelEx(&cfg, kernel, args...);
    }
    return e;
}

// Launches `kernel` as a programmatic dependent of the stream's previous kernel: it may be scheduled while that
// kernel is still running, so the kernel must execute griddepcontrol.wait before its first access to global memory
// that depends on earlier work (everything but constant weights).  What this buys is the launch latency and the
// kernel's own prologue, hidden under the predecessor's tail - the decode step is a chain of ~180 short kernels.
// Falls back to an ordinary launch if the attribute is refused.
template <typename... P, typename... A>
inline void launch_dependent(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    (void)launch_config(cfg, 0, kernel, args...);              // (an error is launch_status's to find)
}

}  // namespace bn
