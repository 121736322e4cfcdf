// Kernel launches with programmatic dependent launch, clusters and cooperation.
#pragma once

#include <cstring>

#include "device.cuh"

namespace tpa {

// Kernel launch on `s`, with programmatic dependent launch when `pdl`: the
// next kernel of the cycle is scheduled while this one drains and waits in
// pdl_entry() for its results, which hides the launch gap between the short,
// dependent kernels of a V-cycle.
struct Launch {
    cudaStream_t s;
    bool pdl;
    int cluster = 1;     // CTAs per thread-block cluster (grid must be a multiple)
    bool coop = false;   // cooperative launch (every CTA resident at once)
    template <typename... KArgs, typename... Args>
    void operator()(void (*kernel)(KArgs...), int grid, int block, size_t smem, Args... args) const {
        cudaLaunchConfig_t cfg;
        std::memset(&cfg, 0, sizeof(cfg));
        cfg.gridDim = dim3(unsigned(grid));
        cfg.blockDim = dim3(unsigned(block));
        cfg.dynamicSmemBytes = smem;
        cfg.stream = s;
        cudaLaunchAttribute at[3];
        unsigned na = 0;
        if (coop) {
            at[na].id = cudaLaunchAttributeCooperative;
            at[na].val.cooperative = 1;
            ++na;
        }
        if (pdl) {
            at[na].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[na].val.programmaticStreamSerializationAllowed = 1;
            ++na;
        }
        if (cluster > 1) {
            at[na].id = cudaLaunchAttributeClusterDimension;
            at[na].val.clusterDim.x = unsigned(cluster);
            at[na].val.clusterDim.y = 1;
            at[na].val.clusterDim.z = 1;
            ++na;
        }
        cfg.attrs = at;
        cfg.numAttrs = na;
        TPA_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...));
    }
};

}  // namespace tpa
