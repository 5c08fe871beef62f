// Kernel launches that overlap the end of the kernel before them on the stream (programmatic dependent launch).
//
// A kernel launched with launch_chained() may start while its predecessor is still running: its blocks set up their
// barriers and tensor memory meanwhile and then wait in wait_for_predecessor() until the predecessor has completed and its
// writes are visible. EVERY thread of such a kernel calls it before it reads or writes global memory, so the kernels of a
// stream still complete in order. release_successor() lets the next kernel's blocks be scheduled; a kernel that allocates
// tensor memory calls it after the allocation, so that a waiting successor never holds the columns its predecessor needs.
// What it buys is the launch latency and the set-up between two kernels, 2 to 4 us each: a call is a chain of three to five
// kernels that may take 5 us each.
#pragma once
#include <cuda_runtime.h>

namespace kutacc {
namespace dev {

#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_predecessor() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }
__device__ __forceinline__ void release_successor() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }

template <typename... Params, typename... Args>
cudaError_t launch_chained(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
#endif

}  // namespace dev
}  // namespace kutacc
