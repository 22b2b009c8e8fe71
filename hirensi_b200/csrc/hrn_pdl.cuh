// hrn_pdl.cuh -- programmatic dependent launch: a kernel of a chain starts while the
// launch before it drains, loads what no launch of the chain writes, then waits for that
// launch's results.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace hrn {

__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with or without programmatic dependence on the launch before.
template <typename... P, typename... A>
static void chain_start(void (*kern)(P...), int blocks, int threads, size_t smem, cudaStream_t st, bool pdl, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(unsigned(blocks));
    cfg.blockDim = dim3(unsigned(threads));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
}

}  // namespace hrn
