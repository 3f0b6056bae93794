// hydro_chain.cuh -- programmatic dependent launch for the kernels of a call.
//
// A call that launches several short kernels spends a few microseconds
// between two of them: the first one's tail, its memory flush, the launch and
// the second one's set-up.  A chained kernel is placed while the one before it
// runs (from that one's launch_dependents(), or its end) and waits in
// dependency_wait() until that one has ended and its writes are visible.
//
// Two rules keep this correct.  A chained kernel reads nothing that an earlier
// kernel writes, and writes nothing, before dependency_wait(); as every link
// waits so, a kernel's end implies the end of all before it.  And the first
// kernel of a call is launched as usual, so that what a call finds in memory
// (weights, tables, counters of the call before) is complete when its first
// kernel starts.  Where a first kernel is chained all the same, none of the
// call's kernels reads anything before its wait.
#pragma once

#include <cuda_runtime.h>

namespace sfh {

__device__ __forceinline__ void dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launches k behind the stream's last kernel; chained false: as usual.
inline cudaError_t launch_chained(const void* k, unsigned grid, unsigned block, size_t smem, cudaStream_t s, void** args,
                                  bool chained = true)
{
    cudaLaunchAttribute chain{};
    chain.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    chain.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = dim3(grid);
    c.blockDim = dim3(block);
    c.dynamicSmemBytes = smem;
    c.stream = s;
    c.attrs = &chain;
    c.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelExC(&c, k, args);
}

}  // namespace sfh
