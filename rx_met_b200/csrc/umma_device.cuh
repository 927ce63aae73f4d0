// Device helpers shared by the tcgen05 kernels: operand and instruction descriptors, commits, bounded mbarrier waits, rings of
// chunks, tensor-memory loads.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace rxmet {
namespace umma {

constexpr int kTileM = 128;             // accumulator rows = tensor-memory lanes
constexpr uint32_t kCore = 128;         // bytes of one core matrix: 8 rows of 16 bytes
constexpr uint32_t kSpinLimit = 1u << 20;  // about 0.13 s of polling; a legitimate wait lasts microseconds

// True in one lane of a converged warp.  Issue loops of tcgen05.mma belong behind this and a warp-uniform branch, not behind
// a test of the thread index: the compiler then keeps descriptors and addresses in uniform registers.  Measured for 24
// MMAs of 128 x 16 x 16: 274 cycles to issue against 1136.
__device__ __forceinline__ bool electOne() {
    uint32_t elected;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(elected));
    return elected != 0;
}
// The warp's index in its block, as a value the compiler knows to be the same in every lane.
__device__ __forceinline__ int warpIndex() { return __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0); }

__device__ __forceinline__ uint32_t smemAddr(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ uint32_t packBf16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float bf16Lo(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float bf16Hi(uint32_t v) { return __uint_as_float(v & 0xffff0000u); }

// Shared-memory operand descriptor, no swizzle, 16-bit elements.  A core matrix is 128
// contiguous bytes: 8 rows of 16 bytes.
//   MN-major operand: element (mn, k) lives at
//     (mn / 8) * mnGroupStride + (k / 8) * kGroupStride + (k % 8) * 16 + (mn % 8) * 2   bytes,
//   K-major operand:  element (mn, k) lives at
//     (mn / 8) * mnGroupStride + (k / 8) * kGroupStride + (mn % 8) * 16 + (k % 8) * 2   bytes.
// Bits: start address >> 4 in [0,14), k-group stride >> 4 in [16,30) ("leading byte offset"),
// mn-group stride >> 4 in [32,46) ("stride byte offset"), descriptor version 1 in [46,48).
__device__ __forceinline__ uint64_t operandDescriptor(uint32_t addr, uint32_t kGroupStride, uint32_t mnGroupStride) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (static_cast<uint64_t>((kGroupStride >> 4) & 0x3fffu) << 16) |
           (static_cast<uint64_t>((mnGroupStride >> 4) & 0x3fffu) << 32) | (1ull << 46);
}

// Instruction descriptor of kind::f16 for a 128-row accumulator tile: fp32 accumulator (bits
// [4,6) = 1), bf16 A and B ([7,10) = [10,13) = 1), A K-major (bit 15 clear), the major of B in bit 16,
// 1 = MN-major, N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t instructionDescriptor(int n, bool bMnMajor) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (bMnMajor ? (1u << 16) : 0u) |
           (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
}

__device__ __forceinline__ void commitTo(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// Whether the barrier's phase of the given parity is over.
__device__ __forceinline__ bool testPhase(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}
// Polls the barrier phase of the given parity; false when the limit ran out.  `polls`
// (optional) receives the number of polls made.
__device__ __forceinline__ bool waitPhase(uint32_t bar, uint32_t parity, uint32_t *polls = nullptr) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (testPhase(bar, parity)) {
            if (polls) *polls = i + 1;
            return true;
        }
    }
    if (polls) *polls = kSpinLimit;
    return false;
}

// The same for warps that wait beside others that compute: suspended by the hardware for up to kSuspendNs a try.  Eight warps of a
// scheduler that poll take all of its issue slots (LSTM inference, H = 256, two CTAs of eight rows on an SM: 151 us alone, 1665 us together).
// About 0.13 s in all.
constexpr uint32_t kSuspendNs = 2000, kSuspendLimit = 1u << 16;
__device__ __forceinline__ bool waitSuspended(uint32_t bar, uint32_t parity) {
    for (uint32_t i = 0; i < kSuspendLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t"
            ".reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t"
            "}\n"
            : "=r"(done)
            : "r"(bar), "r"(parity), "r"(kSuspendNs)
            : "memory");
        if (done) return true;
    }
    return false;
}

// Walks a ring of mbarriers: place and phase parity of the current use.  Counters, not divisions: a division by a value known at run time costs
// a lone thread more than issuing the products of a chunk.
struct Turn {
    int at = 0;
    uint32_t parity = 0;
    bool again = false;   // the place was used before
    __device__ __forceinline__ void step(int size, int by = 1) {
        at += by;
        if (at >= size) {
            at -= size;
            parity ^= 1u;
            again = true;
        }
    }
};

// Walks a ring whose chunks two groups of warps take in turn.  A place has two "full" barriers, chunk i that of index i mod 2 ring, so that
// each barrier belongs to one group.  With one a place, a ring of an odd number of places handed it from group to group, and a group that came for
// chunk i + ring before chunk i had landed was let through by the phase before it, which has the parity that it waits for.
struct RingTurn {
    int ring;
    Turn full;
    __device__ __forceinline__ RingTurn(int places, int first) : ring(places) { step(first); }
    __device__ __forceinline__ void step(int by) { full.step(2 * ring, by); }
    __device__ __forceinline__ int place() const { return full.at < ring ? full.at : full.at - ring; }
};

// The loop of a copy warp: ask(i, place, bar) issues the copies of chunk i, which complete on `bar`, one of full[2 ring] (RingTurn); a place is asked
// for again once its chunk was read (`wait` on freed[place]).  After a wait of the CTA that gave up (`failed`) the warp leaves by vote, all lanes after the same
// chunk: `failed` may change between the reads of two lanes.  Nothing is left in flight when it returns the number of chunks asked for.
template <class Wait, class Ask>
__device__ __forceinline__ int fillRing(int chunks, int ring, uint64_t *full, uint64_t *freed, const volatile int &failed, Wait wait, Ask ask) {
    RingTurn turn(ring, 0);
    Turn slot;
    int issued = 0;
    for (; issued < chunks; ++issued, turn.step(1), slot.step(ring)) {
        if (slot.again) wait(&freed[slot.at], slot.parity ^ 1u);
        if (__any_sync(0xffffffffu, failed)) break;
        ask(issued, slot.at, &full[turn.full.at]);
    }
    for (int i = max(0, issued - ring); i < issued; ++i) waitPhase(smemAddr(&full[i % (2 * ring)]), (i / (2 * ring)) & 1);
    return issued;
}

__device__ __forceinline__ void tmemLoad32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

}  // namespace umma
}  // namespace rxmet
