// Launches shared by the kernels' host code.
#pragma once
#include <type_traits>

#include "backend.h"
#include "trellis_decode.cuh"

namespace st {

// The launch of clusters of `cluster` CTAs below, with programmatic start or without.
template <class... Params, class... Args>
inline cudaError_t launch_clusters(void (*kernel)(Params...), int cluster, dim3 grid, int block, size_t smem, bool programmatic,
                                   cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[programmatic].id = cudaLaunchAttributeClusterDimension;
    attr[programmatic].val.clusterDim.x = cluster;
    attr[programmatic].val.clusterDim.y = 1;
    attr[programmatic].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}
// One launch; `programmatic`: it may start while the launch before it in the stream still runs (the
// kernel then waits with griddepcontrol.wait).
template <class... Params, class... Args>
inline cudaError_t launch_pdl(void (*kernel)(Params...), dim3 grid, int block, size_t smem, bool programmatic, cudaStream_t stream,
                              Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = programmatic ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...);
}

// use(std::integral_constant<int, K>) for rate code K of the weights; half-integer rates exist for mul1 only.
template <int CB, class Use>
inline cudaError_t for_rate(int bits, Use&& use) {
    switch (bits) {
    case 1: return use(std::integral_constant<int, 1>{});
    case 2: return use(std::integral_constant<int, 2>{});
    case 3: return use(std::integral_constant<int, 3>{});
    case 4: return use(std::integral_constant<int, 4>{});
    case 5: return use(std::integral_constant<int, 5>{});
    case 6: return use(std::integral_constant<int, 6>{});
    case 7: return use(std::integral_constant<int, 7>{});
    case 8: return use(std::integral_constant<int, 8>{});
    default:
        if constexpr (CB == CB_MUL1) {
            if (bits == 9) return use(std::integral_constant<int, 9>{});
            if (bits == 10) return use(std::integral_constant<int, 10>{});
            if (bits == 11) return use(std::integral_constant<int, 11>{});
        }
        return cudaErrorInvalidValue;
    }
}

// use(std::integral_constant<int, CB>) for a codebook.
template <class Use>
inline cudaError_t for_codebook(int codebook, Use&& use) {
    switch (codebook) {
    case CB_3INST: return use(std::integral_constant<int, CB_3INST>{});
    case CB_MCG: return use(std::integral_constant<int, CB_MCG>{});
    case CB_MUL1: return use(std::integral_constant<int, CB_MUL1>{});
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace st
