// Programmatic dependent launch: a kernel whose blocks may start while the
// kernel before it on the stream ends.  pdl_trigger lets the next one start
// once every block of this one has; pdl_wait returns when the kernel before
// is complete and its writes are visible.  Every block of a kernel launched
// with launch_overlapped calls pdl_wait before it reads what an earlier kernel
// wrote, and before it ends (so that its end means the end of the earlier
// ones too).
#pragma once

#include "internal.hpp"

namespace virs {
namespace {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kern)(P...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
                              const A &...args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

} // namespace
} // namespace virs
