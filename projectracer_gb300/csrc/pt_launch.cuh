// pt_launch.cuh -- programmatic dependent launches.
#pragma once
#include <utility>

#include "pt_internal.h"

namespace pt {

// Programmatic dependent launch: every kernel of a cycle that is launched so starts by waiting for its
// predecessor grid (griddepcontrol.wait returns once that grid has completed and its writes are
// visible; it is a no-op for a kernel launched without the attribute) and then lets its own
// successor be scheduled.  The successor's launch latency hides behind this kernel's run, which
// matters on the coarse levels where each stage kernel lasts a couple of microseconds.
__device__ __forceinline__ void pdl_begin() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

template <typename... KArgs, typename... Args>
static int launch_pdl(const char* what, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                      Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PT_COUNT();
    return cuda_check(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...), what);
}

}  // namespace pt
