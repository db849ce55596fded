// cluster_util.cuh -- thread-block cluster primitives for sm_100a, inline PTX: the cluster
// barrier, and stores into a neighbour CTA's shared memory that complete on that CTA's
// mbarrier.  Waits on such an mbarrier are bounded by a clock budget (tma_util.cuh).
#pragma once
#include "tma_util.cuh"

namespace prj {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// arrive / wait of the hardware cluster barrier; exited threads count as arrived
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// the address, in the cluster's window, of this CTA's shared address `p` in CTA `rank`
__device__ __forceinline__ uint32_t cluster_map(const void* p, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
    return r;
}

// 16 bytes into a CTA's shared memory (cluster_map addresses), counted on its mbarrier
__device__ __forceinline__ void st_async(uint32_t dst, double2 v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "d"(v.x), "d"(v.y), "r"(bar)
                 : "memory");
}

// mbar_wait_bounded that also acquires another CTA's stores
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t phase,
                                                  long long budget = kWaitBudgetCycles) {
    const long long t0 = clock64();
    for (;;) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(phase)
            : "memory");
        if (ok) return true;
        if (clock64() - t0 > budget) return false;
    }
}

// The way out of a CTA that gave up a wait (every thread calls it): its own copy on `copy_bar`
// (phase 0; null: none was issued) must not land after it has left, so thread 0 waits for that
// within the limit first; then the cluster barrier, so that no CTA leaves while a neighbour can
// still write to it.
__device__ __forceinline__ void cluster_leave(uint64_t* copy_bar) {
    if (copy_bar && threadIdx.x == 0) mbar_wait_bounded(copy_bar, 0);
    __syncthreads();
    cluster_arrive();
    cluster_wait();
}

}  // namespace prj
