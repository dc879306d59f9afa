// Kernel launch with programmatic stream serialisation (programmatic dependent launch): the
// kernel may begin launching while the previous kernel on the stream drains; every kernel launched
// this way calls pdl_wait() before its first global access, and most call pdl_trigger() before their
// last stores (fft_core.cuh).
// BFLY_PDL=0 in the environment launches them plainly instead (read once per process).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdlib>

namespace bfly {
namespace backend {

inline bool pdlEnabled() {
    static const bool on = [] {
        const char* env = std::getenv("BFLY_PDL");
        return !(env && env[0] == '0');
    }();
    return on;
}

// `args` must have exactly the kernel's parameter types.  `cluster` CTAs (dividing the grid) form
// a thread-block cluster.
template <typename... Args>
cudaError_t launchPdlCluster(const void* fn, unsigned grid, int block, int smem, unsigned cluster, cudaStream_t stream,
                             Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdlEnabled() ? 2 : 1;
    void* argv[] = {static_cast<void*>(&args)...};
    return cudaLaunchKernelExC(&cfg, fn, argv);
}

template <typename... Args>
cudaError_t launchPdl(const void* fn, unsigned grid, int block, int smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = (size_t)smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdlEnabled() ? 1 : 0;
    void* argv[] = {static_cast<void*>(&args)...};
    return cudaLaunchKernelExC(&cfg, fn, argv);
}

// The same for a typed kernel: the arguments convert to its parameters.
template <typename T>
struct SameType {
    using type = T;
};
template <typename... P>
cudaError_t launchPdlKernel(void (*fn)(P...), uint64_t grid, int block, int smem, void* stream,
                            typename SameType<P>::type... args) {
    return launchPdl((const void*)fn, (unsigned)grid, block, smem, reinterpret_cast<cudaStream_t>(stream), args...);
}

}  // namespace backend
}  // namespace bfly
