// Launching kernels: clusters, programmatic stream serialisation, counting and timing.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "ep_kernels.cuh"

namespace mcep {

// Lets `kernel` use `smem` bytes of dynamic shared memory on the current device
// (asked of the runtime once per kernel, device and larger size).
cudaError_t allow_shared_memory(const void* kernel, size_t smem);

// Prepares `kernel` for clusters of `blocks` blocks of this shape; `fits`: whether the
// current device can run them (asked of the runtime once per device and shape).
cudaError_t cluster_fits(const void* kernel, int blocks, int threads, size_t smem, bool* fits);

// While per-kernel timing is on, kernels run one after the other.
bool kernel_timing_on();

template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(const char* name, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, int cluster,
                          const LaunchCtx& ctx, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute attr[2];
    cfg.attrs = attr;
    if (cluster > 1) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeClusterDimension;
        attr[cfg.numAttrs].val.clusterDim.x = cluster;
        attr[cfg.numAttrs].val.clusterDim.y = attr[cfg.numAttrs].val.clusterDim.z = 1;
        ++cfg.numAttrs;
    }
    if (ctx.pdl && !kernel_timing_on()) {
        attr[cfg.numAttrs].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[cfg.numAttrs].val.programmaticStreamSerializationAllowed = 1;
        ++cfg.numAttrs;
    }
    LaunchScope scope(name, ctx.stream);
    return scope.done(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

}  // namespace mcep
