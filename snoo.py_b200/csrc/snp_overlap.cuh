// Launches that may overlap the end of the previous kernel on their stream (programmatic dependent
// launch).  The later kernel starts once every block of the earlier one has called
// allow_next_kernel() or ended; wait_for_previous_kernel() returns when the earlier kernel is
// complete and its writes are visible.  Every kernel launched so waits in each block before it
// ends, so that its own completion implies that of all kernels before it.  What a kernel still
// running may write is not read through the read-only path (const __restrict__, __ldg).
#pragma once

#include <cuda_runtime.h>

namespace snp {

__device__ __forceinline__ void wait_for_previous_kernel() { cudaGridDependencySynchronize(); }
__device__ __forceinline__ void allow_next_kernel() { cudaTriggerProgrammaticLaunchCompletion(); }

// overlap = false: an ordinary launch.  Errors are left for the caller's launch check.
template <typename... P, typename... A>
void launch_overlapping(bool overlap, void (*kern)(P...), int grid, int block, size_t smem, cudaStream_t s,
                        const A &...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = overlap ? 1 : 0;
    (void)cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
}

}  // namespace snp
