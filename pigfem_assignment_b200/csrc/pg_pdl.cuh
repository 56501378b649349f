// Programmatic dependent launch.
#pragma once

#include <cuda_runtime.h>

namespace pgb {

// Programmatic dependent launch (sm_90 and later).  A kernel launched with
// launch_pdl may start while the kernel before it on the stream is still
// running, once every CTA of that one has called pdl_trigger (or exited);
// pdl_wait blocks until the kernel before has completed and its writes are
// visible.  Both are no-ops for a kernel launched the ordinary way.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Launches kern with the programmatic-stream-serialization attribute (see
// pdl_trigger / pdl_wait).
template <typename... KArgs, typename... Args>
void launch_pdl(void (*kern)(KArgs...), int grid, int block, size_t smem, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

}  // namespace pgb
