// Reverse recurrence of a QAT backward inside one CTA, up to 128 hidden units, the product of the gate gradients with the recurrent
// weights on tcgen05 kind::f16, a thread per hidden unit and row.
//
// A lane of tensor memory is the unit whose dh the product gives; K runs over the channels of all gates.  The weight codes (exact in
// bf16) stay in tensor memory as the A operand; the gradients of a step, times the channels' scales, are the B operand as three bf16
// terms that carry all of their 24 bits, term i of row r in column 4 r + i.  The sums over the channels of 64 units (32 where 64 do
// not divide the width) have accumulators of their own that are added in fp32: a tcgen05 accumulator truncates each addition, and the sums are bit for
// bit those of the cluster kernels, whose CTAs own 64 (32) units.  Layers of 32 units (up to 256 rows) and 64 (up to 128) had an accumulator
// for every gate and term of mma.sync added in fp32 before; against 64-bit sums their gradient of the initial state after 60 steps is as near as
// it was (7.1e-8 of its norm then, 6.2e-8 now).  Where a layer leaves lanes free, copies of its weights serve other rows.
// Per step and thread:
//   sums of the step before -> dh -> gate gradients -> B operand (the warps only arrive at the barrier behind it) -> control warp starts the
//   product; under it the gradients are stored, the factors of the next step formed from operands that were asked for four steps ahead,
//   and the next operands asked for (asynchronous copies into a ring that only the thread itself reads: a wait for registers that are
//   loaded steps ahead is one for those that were asked for last as well).
// Bound: the chain of a step, of which 24 (GRU) or 32 (LSTM) MMAs are about half.  The cluster kernels it replaced up to 128 units sent partial sums
// between two CTAs: T = 100, H = 128, GRU 45 rows 79 -> 49 us, 256 rows 82 -> 62, 1100 rows 175 -> 164; LSTM 45 rows 84 -> 55 us, 256 rows 87 -> 68;
// H = 64, GRU 45 rows 81 -> 44 us.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "backward_cluster_device.cuh"
#include "cluster_device.cuh"
#include "common.h"
#include "dependent_launch.cuh"
#include "umma_device.cuh"

namespace rxmet {
namespace unitrev {

using namespace umma;

struct Problem {
    int T, B;
};

// A tile of weights in shared memory: 32 output units x 32 channels in bf16.  Rows are 16 bytes apart and change the order of their 16-byte pieces every
// eight units, so that a warp reads a piece of each row, and writes a pair of channels of every fourth unit, without bank conflicts.
constexpr uint32_t kTileStride = 64 + 16;
__device__ __forceinline__ uint8_t *tilePlace(uint8_t *tile, int unit, int channel) {
    return tile + unit * kTileStride + (((channel >> 3) ^ (unit >> 3)) << 4) + (channel & 7) * 2;
}

template <class Cell, int H, int ROWS>
struct Geometry {
    static_assert(H % 32 == 0 && H <= 128, "tiles of 32 units inside one CTA");
    static constexpr int kGates = Cell::kGates, kPart = H % 64 == 0 ? 64 : 32, kParts = H / kPart;
    static constexpr int kUnits = H <= 32 ? 32 : H <= 64 ? 64 : 128, kCopies = 128 / kUnits;   // lanes of a copy of the weights
    static constexpr int kGroups = ROWS / kCopies < 2 ? 1 : 2;                                    // warps of a quarter
    static constexpr int kWarps = 4 * kGroups, kThreads = 32 * (kWarps + 1);                     // and the control warp
    static constexpr int kRows = ROWS / (kCopies * kGroups);                                      // rows of a thread
    static_assert(kRows >= 1 && kRows * kCopies * kGroups == ROWS, "rows divide");
    static constexpr int kSlots = 4;                                                               // steps whose operands are under way or there
    static constexpr int kGroupsPart = kGates * kPart / 8, kGroupsK = kParts * kGroupsPart;        // 16-byte k-groups
    static constexpr int kCols = (4 * ROWS + 15) / 16 * 16;                                       // accumulator columns of a part
    static constexpr uint32_t kTmemCols = bwdcluster::powerOfTwoFrom(kParts * kCols + kGroupsK * 4);
    static_assert(kTmemCols <= 512, "tensor memory has 512 columns");
    static constexpr int kResident = kTmemCols <= 256 ? 2 : 1;
    static constexpr uint32_t kStrideB = kCols * 16 + 16;   // 16 bytes more than its rows spread a warp's units over the banks
    static constexpr uint32_t kOperandBytes = kGroupsK * kStrideB;
    static constexpr uint32_t kWordStride = kWarps * 32 * 4, kSlotBytes = kRows * Cell::kWords * kWordStride;   // a word per thread, the operands of a step
    static constexpr uint32_t kTileBytes = 32 * kTileStride;                                                  // weights on their way
    static constexpr size_t kSharedBytes = kOperandBytes + std::max(kSlots * kSlotBytes, kWarps * 2 * kTileBytes);
};

// Cell contract (device functions; t descends):
//   kGates
//   void tile<H>(at, lane, m, gate, unit)         a warp: bf16 weights of output units m .. m + 31 (any values beyond H) and the channels of `gate` of units
//                                                 unit .. unit + 31 as a tile at `at`
//   State begin(row, unit)                        State::dh: what flows into the last step beside its own gradient
//   kWords, void fetch(dst, t, row, unit)         copies the kWords words of a step's operands to shared memory, kWordStride bytes apart
//   Factors factors<STRIDE>(const uint8_t *, unit)   what a step does to dh, formed from them before dh is there
//   void advance(Unit, Factors, State &, alive, float (&b)[kGates], Out &)   gradients times scales; State::dh without the product's sums
//   Unit unitOf(unit)
//   void store(Out, t, row, unit), void finish(State, row, unit, alive)
template <class Cell, int H, int ROWS>
__global__ void __launch_bounds__(Geometry<Cell, H, ROWS>::kThreads, Geometry<Cell, H, ROWS>::kResident)
unitReverse(const __grid_constant__ Problem p, const __grid_constant__ Cell c) {
    using G = Geometry<Cell, H, ROWS>;
    constexpr int kGates = G::kGates, kRows = G::kRows, kSlots = G::kSlots;
    extern __shared__ __align__(128) uint8_t bTile[];   // [kGroupsK][kCols + 1][16]
    uint8_t *ring = bTile + G::kOperandBytes;           // [kSlots][kRows][kWords][threads] words
    __shared__ __align__(8) uint64_t productBar;
    __shared__ uint32_t tmemSlot;

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex(), quarter = warp & 3, group = warp >> 2;
    const int unit = quarter % (G::kUnits / 32) * 32 + lane;
    const int b0 = static_cast<int>(blockIdx.x) * ROWS, rowInCta = (group * G::kCopies + quarter / (G::kUnits / 32)) * kRows;
    const bool live = warp < G::kWarps && unit - lane < H;   // uniform in the warp

    if (tid == 0) {
        cluster::initBarrier(&productBar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (uint32_t i = tid; i < G::kOperandBytes / 16; i += G::kThreads) reinterpret_cast<uint4 *>(bTile)[i] = make_uint4(0u, 0u, 0u, 0u);
    waitForPredecessor();   // what is above needs nothing from earlier kernels
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0), tmemWeights = tmem + G::kParts * G::kCols;
    const uint32_t quarterBase = static_cast<uint32_t>(32 * quarter) << 16;
    // The weights, shared out among the warps of a quarter.  Tiles through shared memory: a lane needs the channels of one output unit, which in
    // memory are rows or columns of 4-byte codes; read lane by lane they took a third of a call of four steps (GRU, H = 128, 290 rows: 14.1 -> 9.5 us).
    if (warp < G::kWarps) {
        uint8_t *tiles = ring + warp * (2 * G::kTileBytes);
#pragma unroll (G::kGroups == 1 ? 4 : 2)
        for (int n = group, turn = 0; n < kGates * (H / 32); n += G::kGroups, ++turn) {
            const int gate = n / (H / 32), of = n % (H / 32) * 32;
            uint8_t *tile = tiles + (turn & 1) * G::kTileBytes;
            c.template tile<H>(tile, lane, unit - lane, gate, of);
            __syncwarp();   // also parts the reads of a tile from the writes of the next but one
            const uint32_t to = tmemWeights + quarterBase + (of / G::kPart * G::kGroupsPart + gate * (G::kPart / 8) + of % G::kPart / 8) * 4;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint4 w = *reinterpret_cast<const uint4 *>(tilePlace(tile, lane, 8 * j));
                bwdcluster::tmemStore4(to + j * 4, unit < H ? w : make_uint4(0u, 0u, 0u, 0u));
            }
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    if (warp == G::kWarps) {
        constexpr uint32_t kIdesc = instructionDescriptor(G::kCols, false);
        const uint64_t descB = operandDescriptor(smemAddr(bTile), G::kStrideB, kCore);
#pragma unroll 1
        for (int n = 0; n < p.T; ++n) {
            asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");   // the gradients of step n are written
            if (electOne()) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int part = 0; part < G::kParts; ++part)
#pragma unroll
                    for (int ks = 0; ks < G::kGroupsPart / 2; ++ks)
                        bwdcluster::mmaBf16TmemA(tmem + part * G::kCols, tmemWeights + (part * G::kGroupsPart + 2 * ks) * 4,
                                                 descB + static_cast<uint64_t>(((part * G::kGroupsPart + 2 * ks) * G::kStrideB) >> 4), kIdesc, ks > 0 ? 1u : 0u);
                commitTo(smemAddr(&productBar));
            }
            __syncwarp();
        }
    } else if (!live) {
        for (int n = 0; n < p.T; ++n) asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");
    } else {
        bool alive = true;   // false once a wait of this warp gave up: it waits no more and its values become NaN
        const typename Cell::Unit mine = c.unitOf(unit);
        int row[kRows];
        typename Cell::State state[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {   // rows beyond the last one repeat it: the same values to the same places
            row[r] = min(b0 + rowInCta + r, p.B - 1);
            state[r] = c.begin(row[r], unit);
        }
        const uint32_t column = tmem + quarterBase + rowInCta * 4;
        uint8_t *to = bTile + (unit / G::kPart * G::kGroupsPart + unit % G::kPart / 8) * G::kStrideB + rowInCta * 64 + (unit & 7) * 2;
        typename Cell::Factors factors[kRows];
        uint8_t *mySlot = ring + tid * 4;
        auto fetch = [&](int n) {   // of step n, counted from the last one; every call is one group of copies
            if (n < p.T) {
                const uint32_t dst = smemAddr(mySlot) + static_cast<uint32_t>(n % kSlots) * G::kSlotBytes;
#pragma unroll
                for (int r = 0; r < kRows; ++r) c.template fetch<G::kWordStride>(dst + r * (Cell::kWords * G::kWordStride), p.T - 1 - n, row[r], unit);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto prepare = [&](int n) {   // the factors of step n, of which at most kSlots - 1 later groups are under way
            asm volatile("cp.async.wait_group %0;" ::"n"(kSlots - 1) : "memory");
            if (n < p.T) {
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    factors[r] = c.template factors<G::kWordStride>(mySlot + static_cast<uint32_t>(n % kSlots) * G::kSlotBytes + r * (Cell::kWords * G::kWordStride), unit);
            }
            fetch(n + kSlots);
        };
        auto collect = [&](int n) {   // the sums of step n
            if (alive) alive = __all_sync(0xffffffffu, waitPhase(smemAddr(&productBar), n & 1));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t v[kRows][G::kParts][4];
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int part = 0; part < G::kParts; ++part) bwdcluster::tmemLoad<4>(column + part * G::kCols + 4 * r, v[r][part]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
#pragma unroll
            for (int r = 0; r < kRows; ++r)
#pragma unroll
                for (int part = 0; part < G::kParts; ++part)
                    state[r].dh += (__uint_as_float(v[r][part][2]) + __uint_as_float(v[r][part][1])) + __uint_as_float(v[r][part][0]);
        };
#pragma unroll
        for (int n = 0; n < kSlots; ++n) fetch(n);
        prepare(0);
#pragma unroll 1
        for (int n = 0; n < p.T; ++n) {
            if (n > 0) collect(n - 1);
            typename Cell::Out out[kRows];
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                float b[kGates];
                c.advance(mine, factors[r], state[r], alive, b, out[r]);
#pragma unroll
                for (int g = 0; g < kGates; g += 2) {   // two gates share a conversion
                    float x = b[g], y = g + 1 < kGates ? b[g + 1 < kGates ? g + 1 : g] : 0.0f;
                    uint8_t *at = to + g * (G::kPart / 8) * G::kStrideB + r * 64;
#pragma unroll
                    for (int term = 0; term < 3; ++term) {
                        const uint32_t word = packBf16(x, y);
                        x -= bf16Lo(word);
                        y -= bf16Hi(word);
                        *reinterpret_cast<uint16_t *>(at + term * 16) = static_cast<uint16_t>(word);
                        if (g + 1 < kGates) *reinterpret_cast<uint16_t *>(at + G::kPart / 8 * G::kStrideB + term * 16) = static_cast<uint16_t>(word >> 16);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            // a warp whose wait gave up must not run ahead of the others: it waits here
            if (alive) asm volatile("bar.arrive 1, %0;" ::"n"(G::kThreads) : "memory");
            else asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");
#pragma unroll
            for (int r = 0; r < kRows; ++r) c.store(out[r], p.T - 1 - n, row[r], unit);
            prepare(n + 1);
        }
        collect(p.T - 1);
#pragma unroll
        for (int r = 0; r < kRows; ++r) c.finish(state[r], row[r], unit, alive);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols) : "memory");
}

template <int ROWS, class Cell, int H>
void launch(const char *name, const Problem &p, const Cell &cell, cudaStream_t st) {
    using G = Geometry<Cell, H, ROWS>;
    const auto kernel = unitReverse<Cell, H, ROWS>;
    // no more CTAs on an SM than its tensor memory holds: one more would wait there for the whole sequence of another
    const size_t smem = std::max(G::kSharedBytes, static_cast<size_t>(currentDevice().smemMax) / (512 / G::kTmemCols + 1) + 1024);
    ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
    {
        KernelTimer timer__(name, st);
        launchDependent(kernel, (p.B + ROWS - 1) / ROWS, G::kThreads, smem, st, p, cell);
    }
    afterLaunch(name);
}

// Rows of a CTA: as few as let all of them run at the same time.
template <int H, class Cell>
void launchRows(const char *name, const Problem &p, const Cell &cell, cudaStream_t st) {
    constexpr int kLeast = H > 64 ? 1 : H > 32 ? 2 : 4;
    const int sms = smsPerPass();
    if ((p.B + kLeast - 1) / kLeast <= (kLeast == 1 ? 1 : Geometry<Cell, H, kLeast>::kResident) * sms) launch<kLeast, Cell, H>(name, p, cell, st);
    else if ((p.B + 2 * kLeast - 1) / (2 * kLeast) <= Geometry<Cell, H, 2 * kLeast>::kResident * sms) launch<2 * kLeast, Cell, H>(name, p, cell, st);
    else launch<4 * kLeast, Cell, H>(name, p, cell, st);
}

}  // namespace unitrev
}  // namespace rxmet
