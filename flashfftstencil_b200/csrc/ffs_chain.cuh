// Launches whose start-up overlaps the end of the kernel before them in the stream (programmatic
// dependent launch).  The kernel calls chain_wait() before it touches global memory that another
// kernel reads or writes: it returns when every earlier kernel has finished and its writes are visible.
// Passes of a solve are chains of short kernels, and the gap between two of them in a stream is
// 2 to 3 us otherwise.
#pragma once
#include <cuda_runtime.h>

namespace ffst {

__device__ __forceinline__ void chain_wait()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

template <class Kernel, class... Args>
cudaError_t launch_chained(Kernel kernel, unsigned grid, unsigned block, size_t smem, cudaStream_t s, const Args &...args)
{
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    cudaLaunchAttribute a{};
    a.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    a.val.programmaticStreamSerializationAllowed = 1;
    c.attrs = &a;
    c.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&c, kernel, args...);
    return e != cudaSuccess ? e : cudaGetLastError();
}

} // namespace ffst
