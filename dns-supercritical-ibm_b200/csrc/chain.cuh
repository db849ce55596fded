// chain.cuh -- programmatic dependent launch of a small grid's kernels.
//
// A kernel of a step reads what the one before it wrote, so each waits for the whole of its
// predecessor; launched with launch_chained, its CTAs are placed as soon as the predecessor's
// last ones are (chain_trigger) and run their set-up -- barriers, plan tables -- up to
// chain_wait, which returns when the predecessor has completed and its writes are visible.  That
// takes launch latency and set-up off a step of a few microseconds per kernel: 24.6 -> 23.1 us at
// 48 x 32 x 24, a Poisson solve 45.6 -> 39.4 us at 128 x 96 x 64.  Large grids lose by it (CTAs that
// wait take the places of CTAs that work: 3.60 -> 4.28 ms at 768 x 384 x 384, 231 -> 278 us at
// 256 x 128 x 128), so launch_chained sets the attribute up to 2^20 points.
// Every kernel launched this way calls chain_wait before it touches memory that another kernel of
// a step reads or writes; plan tables are written with the device synchronised, so they may be
// read before it.
#pragma once
#include <cuda_runtime.h>

namespace prj {

__device__ __forceinline__ void chain_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

constexpr long long kChainPoints = 1ll << 20;

// chained: the launch attribute (a grid of up to kChainPoints points); cluster > 1: clusters of
// that many CTAs along x
template <typename... P, typename... A>
inline cudaError_t launch_chained(bool chained, void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem,
                                  cudaStream_t st, unsigned cluster, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2]{};
    unsigned n = 0;
    if (chained) {
        at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    if (cluster > 1) {
        at[n].id = cudaLaunchAttributeClusterDimension;
        at[n].val.clusterDim.x = cluster;
        at[n].val.clusterDim.y = at[n].val.clusterDim.z = 1;
        n++;
    }
    cfg.attrs = at;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// Are `count` clusters of C CTAs along x resident at once, of a kernel of which `slots` CTAs are?
// A cluster's CTAs share one GPC, so fewer are than slots / C (15 clusters of 8 at one CTA per SM
// of 148), and the runtime is asked, which takes some 40 us; but not for what the slots cannot
// hold, for single CTAs, or for clusters on half of the slots, which always fit: a GPC of g >= C
// slots uses C floor(g / C) >= g / 2 of them.  Kernels asked about here are launched with the limit set here, the
// device's: one value for all callers, so a thread that creates a plan takes nothing from one
// that launches.
constexpr int kSmemLimit = 227 * 1024;
template <typename K>
inline bool clusters_resident(K kernel, unsigned threads, size_t smem, unsigned C, int count, int slots) {
    const long long need = (long long)count * C;
    if (need > slots) return false;
    if (C == 1 || 2 * need <= slots) return true;
    int most = 0;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(C);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = C;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return most >= count;
}

}  // namespace prj
