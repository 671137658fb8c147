// Programmatic dependent launch for every kernel of the step list.
//
// A step list is a chain of short kernels in one stream; launched the plain way, each kernel's launch
// latency and prologue (index arithmetic, barrier and tensor-memory set-up) start only when the previous
// grid has drained.  With the programmatic-stream-serialisation attribute the next grid is scheduled as
// soon as every CTA of the previous one has called `griddepcontrol.launch_dependents` (or exited), and it
// blocks in `griddepcontrol.wait` until the previous grid has completed and its writes are visible.  Every
// kernel therefore calls `pdl_enter()` before its first access to global memory; kernels with a set-up
// phase that touches no global memory call it after that phase.  The attribute is kept under stream
// capture: the captured graph carries programmatic edges between consecutive kernel nodes.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <utility>

namespace kn {

__device__ __forceinline__ void pdl_enter() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <typename... Params, typename... Args>
inline void launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args&&... args) {
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
    (void)cudaLaunchKernelEx(&cfg, kernel, Params(std::forward<Args>(args))...);   // a failure stays in cudaGetLastError()
}

// Dynamic shared memory above 48 KB is opted in to once per device and kernel.
template <class Kernel>
int allow_shared(Kernel kernel, int bytes, bool (&done)[64], std::mutex& mu) {
    int device = 0;
    cudaGetDevice(&device);
    std::lock_guard<std::mutex> lock(mu);
    if (device >= 0 && device < 64 && !done[device]) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return (int)e;
        done[device] = true;
    }
    return 0;
}

// Two multiply-adds in one instruction (fma.rn.f32x2).
__device__ __forceinline__ float2 fma_pair(float2 a, float2 b, float2 c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(*(uint64_t*)&a), "l"(*(uint64_t*)&b), "l"(*(uint64_t*)&c));
    return *(float2*)&d;
}

}  // namespace kn
