// Small transfers between the arena and pinned host memory, by a kernel instead of by copy-engine operations.
//
// A copy-engine node inside a CUDA graph costs some 3 us of hand-over on either side; a kernel that reads or writes the
// pinned pages over PCIe is a kernel node like the others.  Measured (graph of four empty kernels, launch to
// synchronise): 18.9 us with one upload and two downloads as memcpy nodes, 12.3 us with two of these kernels.  From
// about 64 KB on the copy engine is as fast, and it leaves the SMs alone.
#include <cuda_runtime.h>

#include "../kernels.h"
#include "launch.cuh"

namespace kn {

namespace {

// 16 bytes per thread and turn where both ends allow it, else one byte; every range is walked by the whole grid
__global__ void __launch_bounds__(256) host_copy_kernel(const __grid_constant__ HostCopyParams p) {
    pdl_enter();
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int r = 0; r < p.n; r++) {
        const uint8_t* s = (const uint8_t*)p.src[r];
        uint8_t* d = (uint8_t*)p.dst[r];
        int64_t vectors = 0;
        if ((((uintptr_t)s | (uintptr_t)d) & 15) == 0) {
            vectors = p.bytes[r] >> 4;
            for (int64_t i = first; i < vectors; i += step) ((uint4*)d)[i] = ((const uint4*)s)[i];
        }
        for (int64_t i = (vectors << 4) + first; i < p.bytes[r]; i += step) d[i] = s[i];
    }
}

}  // namespace

int launch_host_copy(const HostCopyParams& p, cudaStream_t stream) {
    int64_t most = 0;
    for (int r = 0; r < p.n; r++) most = p.bytes[r] > most ? p.bytes[r] : most;
    // four 16-byte accesses per thread: a 64 KB range is in flight as a whole on 4 SMs
    const int64_t blocks = (most + 256 * 64 - 1) / (256 * 64);
    launch_pdl(host_copy_kernel, dim3((unsigned)(blocks < 1 ? 1 : (blocks > 64 ? 64 : blocks))), dim3(256), (size_t)0, stream, p);
    return (int)cudaGetLastError();
}

}  // namespace kn
