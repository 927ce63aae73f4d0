// Device pieces shared by the reverse recurrences over thread-block clusters (gru_backward_cluster.cu, lstm_backward_cluster.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace rxmet {
namespace bwdcluster {

template <int COUNT>
__device__ __forceinline__ void tmemLoad(uint32_t addr, uint32_t (&r)[COUNT]) {
    static_assert(COUNT == 2 || COUNT == 4 || COUNT == 8, "row spans of the tiles below");
    if constexpr (COUNT == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
    else if constexpr (COUNT == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
    else
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                     : "r"(addr));
}
__device__ __forceinline__ void tmemStore4(uint32_t addr, const uint4 &v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
__device__ __forceinline__ void tmemStore8(uint32_t addr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n" ::"r"(addr), "r"(v[0]), "r"(v[1]), "r"(v[2]),
                 "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
// D += A B with A in tensor memory: lane = row of A, a 32-bit column holds two consecutive bf16 along K
__device__ __forceinline__ void mmaBf16TmemA(uint32_t tmemD, uint32_t tmemA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n"
        :
        : "r"(tmemD), "r"(tmemA), "l"(descB), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
template <int BYTES>
__device__ __forceinline__ void copyAsync(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst), "l"(src), "n"(BYTES) : "memory");
}

constexpr uint32_t powerOfTwoFrom(uint32_t n) {
    uint32_t p = 32;
    while (p < n) p *= 2;
    return p;
}

}  // namespace bwdcluster
}  // namespace rxmet
