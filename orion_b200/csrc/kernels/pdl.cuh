// Programmatic dependent launch.  A kernel launched with the programmatic-stream-serialization attribute may start
// while the kernel before it in the stream is still running; pdl_wait() blocks the calling thread until that kernel
// has completed and its writes are visible (a no-op for a normally launched kernel).  pdl_launch_dependents() tells the
// device that, as far as this CTA is concerned, the next kernel of the stream may begin to start: its CTAs become
// resident where there is room and run up to their own pdl_wait().  Only kernels that call pdl_wait() before they touch
// global memory are ever launched with the attribute; every kernel may call pdl_launch_dependents().
#pragma once
#include <cuda_runtime.h>
#include <stdlib.h>
#include <string.h>

namespace ob200 {

// Launches a kernel that begins with pdl_wait() as a programmatic dependent of the kernel before it in the stream: launch and
// set-up overlap that kernel's tail, about 2 us per launch of a chain of short kernels.  ORION_PDL=0: plain stream order.
template <typename... KArgs, typename... Args>
inline int launch_pdl(void (*kernel)(KArgs...), unsigned grid, unsigned block, cudaStream_t stream, Args... args) {
    static const bool pdl = [] {
        const char* e = getenv("ORION_PDL");
        return !(e && e[0] == '0');
    }();
    cudaLaunchConfig_t cfg;
    memset(&cfg, 0, sizeof cfg);
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl ? 1 : 0;
    return (int)cudaLaunchKernelEx(&cfg, kernel, (KArgs)args...);
}

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

}  // namespace ob200
