// Programmatic dependent launch for the kernels of a decode step. A kernel launched through
// launch_pdl may start (set up barriers, allocate tensor memory, prefetch WEIGHTS) while the kernel
// before it in the stream is still running; it must execute griddep_wait() before it reads anything
// an earlier kernel wrote or writes anything an earlier kernel may still read. griddep_launch() at
// its top lets the kernel after it do the same. Kernels launched the ordinary way keep the ordinary
// stream order on both sides. TLB_NO_PDL=1 turns the attribute off (the device-side calls are then
// no-ops). A product's weights may be copied in front of the wait only if no kernel writes them (weights_settled in
// lower.cu): launch_pdl_if(false, ...) is the ordinary launch that other operands take.
#pragma once
#include <cuda_runtime.h>
#include <cstdlib>
#include <utility>

namespace tlb {

__device__ __forceinline__ void griddep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void griddep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

inline bool pdl_enabled() {
    static const bool on = [] {
        const char *e = getenv("TLB_NO_PDL");
        return !(e && e[0] == '1');
    }();
    return on;
}

// cluster: CTAs of one (1: none)
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_cluster(bool early, int cluster, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    unsigned n = 0;
    if (early && pdl_enabled()) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n++].val.clusterDim = {(unsigned)cluster, 1, 1};
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl_if(bool early, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    return launch_pdl_cluster(early, 1, kernel, grid, block, smem, st, std::forward<Args>(args)...);
}
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args &&...args) {
    return launch_pdl_if(true, kernel, grid, block, smem, st, std::forward<Args>(args)...);
}

}  // namespace tlb
