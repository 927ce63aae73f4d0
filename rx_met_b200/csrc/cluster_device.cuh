// Device helpers of the recurrences that run over a thread-block cluster: distributed shared memory addresses,
// asynchronous copies into a peer that count their bytes on its mbarrier, and the hardware cluster barrier.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "umma_device.cuh"

namespace rxmet {
namespace cluster {

__device__ __forceinline__ uint32_t rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The shared::cluster address of the same shared-memory location in CTA `cta` of the cluster.
__device__ __forceinline__ uint32_t remote(uint32_t sharedAddr, uint32_t cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(sharedAddr), "r"(cta));
    return r;
}

// Copies shared memory of this CTA into another CTA of the cluster; the bytes complete on the mbarrier `bar` of the CTA they
// go to (dst and bar in shared::cluster, 16-byte aligned).  One such copy costs the receiver's barrier one update,
// where a store that completes on it by itself costs one per lane.
__device__ __forceinline__ void copyTo(uint32_t dst, uint32_t src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void initBarrier(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(umma::smemAddr(bar)), "r"(count) : "memory");
}
// One arrival that announces the bytes the phase waits for.
__device__ __forceinline__ void arriveExpect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}

__device__ __forceinline__ void barrierAll() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Dynamic shared memory that a CTA with `tmemCols` columns of tensor memory asks for at the least: its share of an SM's 228 kB (1 kB of
// which every CTA takes by itself) is that of the tensor memory.  CTAs that fit an SM together then fit its tensor memory as well.  One too many waits in
// tcgen05.alloc until another ends, which costs a short kernel its overlap and would stop clusters for good that wait crosswise for one
// another's SMs.
inline size_t leastShared(uint32_t tmemCols) { return static_cast<size_t>(228 * 1024) * tmemCols / 512 - 1024 - 512; }   // 512: the static part

}  // namespace cluster
}  // namespace rxmet
