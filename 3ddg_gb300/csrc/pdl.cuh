// Programmatic dependent launch: a kernel launched by launch_pdl may start
// while the kernel before it in the stream drains.  Its blocks come up, find
// their tasks and read tables that no kernel writes, and wait (pdl_wait) for
// the kernel before to complete before they touch anything it or an earlier
// one writes.  pdl_next, called after that wait, lets the next kernel of the
// stream come up in turn: at most one kernel waits at a time, and its blocks
// take only the room that the running kernel leaves.
//
// What earlier kernels write is read by plain loads after pdl_wait, not by
// __ldg: the compiler may move a read-only load across the wait.
//
// On short launches the gap between two kernels is half of the time: figures at
// Solver::short_launches and launch_batch.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace dg {

__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// A load of what earlier kernels wrote, in a kernel launched by launch_pdl or
// not.
template <bool PDL, typename T>
__device__ __forceinline__ T pdl_load(const T* p)
{
    if constexpr (PDL) return *p;
    else return __ldg(p);
}

template <typename... P, typename... A>
inline cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, cudaStream_t stream, A&&... args)
{
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(std::forward<A>(args))...);
}

}  // namespace dg
