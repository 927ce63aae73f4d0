// Reverse recurrence of the LSTM QAT backward over thread-block clusters, dh = G_hh W_hh per step on tcgen05.
//
// The plan is that of gru_backward_cluster.cu, where the choices are measured: the H / U CTAs of a cluster advance a tile of
// batch rows; a CTA owns U hidden units, whose pointwise derivative yields exactly the 4 U columns of G_hh that are ITS
// slice of the contraction.  Its rows of W_hh stay in tensor memory as exact bf16 codes (lane = hidden unit), G_hh, scaled
// per channel and split into three bf16 terms (exact products, fp32 accumulation), is the B operand, the terms three groups of
// accumulator columns.  Partial sums [units][rows] travel as bulk copies to the CTA that owns the units, which adds them in
// a fixed order.  A wait is bounded; one that gives up ends all further waiting of the CTA and turns its outputs into NaN.
//
// Everything of a step that does not depend on the incoming dh and dc is formed while the partial sums are under way: with
// them every gate gradient is one product, F[g] mdc for the input, forget and cell gate and F[3] dh for the output gate.
//
// Up to 256 units a CTA owns 64 (32 where 64 do not divide H) of them and a cluster has at most eight CTAs.  Beyond, nine to
// sixteen CTAs own 32 units each: the weights of 64 would fill tensor memory.  Seven such clusters are resident at once.
// Their shared memory takes twenty rows where sixteen would need another round of clusters: a step of 2.7 instead of 2.2 us (T = 100, H = 512, 256 rows
// 618 -> 505 us in two rounds instead of three, 128 rows 413 -> 257 in one).
// Up to 128 units: unit_reverse_umma.cuh.  T = 100, B = 100, H = 160: about 1 ms -> 91 us (FP32 FMA);
// T = 1000, B = 256, H = 512: 10.2 -> 6.0 ms, T = 100, B = 112: 1067 -> 213 us (partial sums through L2 and a grid-wide counter per step).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "backward_cluster_device.cuh"
#include "cluster_device.cuh"
#include "common.h"
#include "lstm_backward_cluster.h"
#include "umma_device.cuh"

namespace rxmet {
namespace lstm {
namespace reverse {

using namespace bwdcluster;

constexpr int kOperands = 8;   // 8-byte pieces of a pair of cells: four gates, tanh(cell), previous cell, incoming gradient, flags

// Geometry of a cluster of H / U CTAs that advances ROWS batch rows.
template <int H, int U, int ROWS>
struct Tile {
    static constexpr int kCtas = H / U, kTiles = (H + 127) / 128, kSliceK = 4 * U, kGroupsK = kSliceK / 8;
    // Twenty rows of 32 units are 320 pairs of cells: a thread each, two warps without a tile to read out.
    static constexpr int kThreads = ROWS == 20 ? 320 : 256, kReadWarps = 8;
    static constexpr int kPairs = U / 2, kRowPass = kThreads / kPairs, kRowsPerThread = (ROWS + kRowPass - 1) / kRowPass;
    static constexpr int kCols = (3 * ROWS + 15) / 16 * 16;          // accumulator columns of one tile of 128 units
    static constexpr uint32_t kColsA = kSliceK / 2;                   // tensor-memory columns of one weight tile
    static constexpr uint32_t kTmemCols = powerOfTwoFrom(kTiles * (kCols + kColsA));
    static_assert(kTmemCols <= 512, "tensor memory has 512 columns");
    static constexpr uint32_t kStrideB = kCols * 16 + 16;            // K-group stride: 16 bytes more spread a warp over the banks
    static constexpr uint32_t kOperandBytes = kGroupsK * kStrideB;
    static constexpr uint32_t kPartBytes = static_cast<uint32_t>(ROWS) * H * 4;
    static constexpr uint32_t kRowBytes = kOperands * kThreads * 8;
    static constexpr uint32_t kSlotBytes = kRowsPerThread * kRowBytes;   // operands of one step
    static constexpr size_t kSharedBytes = kOperandBytes + 4 * kPartBytes + 2 * kSlotBytes + 128;
};

template <int H, int U, int ROWS>
__global__ void __launch_bounds__(Tile<H, U, ROWS>::kThreads, 1) recurrentBackwardCluster(const __grid_constant__ BackwardClusterArgs a) {
    using namespace umma;
    using G = Tile<H, U, ROWS>;
    constexpr int C = 4 * H, NC = G::kCtas, MT = G::kTiles, RPT = G::kRowsPerThread, kThreads = G::kThreads;
    extern __shared__ __align__(128) uint8_t smemC[];
    __shared__ __align__(8) uint64_t productBar[2], partBar[2];
    __shared__ uint32_t tmemSlot;
    uint8_t *bTile = smemC;                                                    // [kGroupsK][kCols (+1)][16 bytes]
    float *part = reinterpret_cast<float *>(bTile + G::kOperandBytes);         // [2][NC sources][U / 32][ROWS][32 units]
    float *outS = part + 2 * ROWS * H;                                         // [2][H / 32 unit tiles][ROWS][32 units], to be sent
    uint8_t *ring = reinterpret_cast<uint8_t *>(outS + 2 * ROWS * H);          // [2 slots][RPT][kOperands][threads] x 8 bytes

    const int tid = threadIdx.x, lane = tid & 31, warp = umma::warpIndex();
    const uint32_t rank = cluster::rank();
    const int ul = tid % G::kPairs * 2, rowOf = tid / G::kPairs;   // pointwise role: units ul, ul + 1 of rows rowOf + i kRowPass
    const int j = static_cast<int>(rank) * U + ul;
    const int b0 = static_cast<int>(blockIdx.x) / NC * ROWS;

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) cluster::initBarrier(&productBar[i], 1);
        for (int i = 0; i < 2; ++i) cluster::initBarrier(&partBar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < 2; ++i) cluster::arriveExpect(smemAddr(&partBar[i]), G::kPartBytes);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (uint32_t i = tid; i < G::kOperandBytes / 16; i += kThreads) reinterpret_cast<uint4 *>(bTile)[i] = make_uint4(0u, 0u, 0u, 0u);
    float2 scale[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) scale[g] = *reinterpret_cast<const float2 *>(a.channelScale + g * H + j);
    float2 dhBase[RPT], dc[RPT];
    bool live[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = rowOf + G::kRowPass * i;
        live[i] = row < ROWS && b0 + row < a.B;
        const size_t o = live[i] ? static_cast<size_t>(b0 + row) * H + j : 0;
        dhBase[i] = *reinterpret_cast<const float2 *>(a.gradFinalHidden + o);
        dc[i] = *reinterpret_cast<const float2 *>(a.gradFinalCell + o);
    }
    // Operands of a step travel two steps ahead through shared memory (a thread reads back what it copied itself): those of step n + 2 replace
    // the operands of step n, of which only the factors are left then.
    const size_t first = (static_cast<size_t>(a.T - 1) * a.B + b0 + rowOf) * H + j;   // element of the last step
    const size_t stepH = static_cast<size_t>(a.B) * H;
    const float *gateFrom = a.gateOutputs + (first - j) * 4 + j, *tanhFrom = a.cellTanh + first, *gradFrom = a.gradOutput + first;
    const uint32_t *bitsFrom = a.stepMasks ? a.stepMasks + first : nullptr;
    const uint32_t mySlot = smemAddr(ring) + tid * 8;
    auto fetch = [&](int t, uint32_t slotBase) {   // steps in descending order, each once
        const float *cellFrom = t > 0 ? a.cellStates + (static_cast<size_t>(t - 1) * a.B + b0 + rowOf) * H + j
                                      : a.c0 + static_cast<size_t>(b0 + rowOf) * H + j;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const uint32_t dst = mySlot + slotBase + i * G::kRowBytes;
            const float *gate = gateFrom + i * (G::kRowPass * C);
#pragma unroll
            for (int g = 0; g < 4; ++g) copyAsync<8>(dst + g * (kThreads * 8), gate + g * H);
            copyAsync<8>(dst + 4 * (kThreads * 8), tanhFrom + i * (G::kRowPass * H));
            copyAsync<8>(dst + 5 * (kThreads * 8), cellFrom + i * (G::kRowPass * H));
            copyAsync<8>(dst + 6 * (kThreads * 8), gradFrom + i * (G::kRowPass * H));
            if (bitsFrom) copyAsync<8>(dst + 7 * (kThreads * 8), bitsFrom + i * (G::kRowPass * H));
        }
        gateFrom -= 4 * stepH;
        tanhFrom -= stepH;
        gradFrom -= stepH;
        if (bitsFrom) bitsFrom -= stepH;
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
#pragma unroll 1
    for (int n = 0; n < 2; ++n) {
        if (n < a.T) fetch(a.T - 1 - n, n * G::kSlotBytes);
        commit();
    }
    float *ihTo = a.gIh + (first - j) * 4 + j, *hhTo = a.gHh + (first - j) * 4 + j;
    __syncthreads();
    const uint32_t tmem = tmemSlot, tmemWeights = tmem + MT * G::kCols;
    // weights: lane = hidden unit m, column = two of this CTA's 4 U channels
    for (int tile = warp >> 2; tile < MT && warp < G::kReadWarps; tile += G::kReadWarps / 4) {
        const int m = tile * 128 + 32 * (warp & 3) + lane;
        for (int kg = 0; kg < G::kGroupsK; ++kg) {
            const int gate = kg / (U / 8), within = kg % (U / 8) * 8;
            uint32_t packed[4] = {0u, 0u, 0u, 0u};
            if (m < H) {
                const float *src = a.weightCodes + (static_cast<size_t>(gate) * H + rank * U + within) * H + m;
#pragma unroll
                for (int e = 0; e < 4; ++e) packed[e] = packBf16(__ldg(src + 2 * e * H), __ldg(src + (2 * e + 1) * H));
            }
            tmemStore4(tmemWeights + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + tile * G::kColsA + kg * 4,
                       make_uint4(packed[0], packed[1], packed[2], packed[3]));
        }
    }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    cluster::barrierAll();   // every CTA's barriers are armed before anyone sends
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    constexpr uint32_t kIdesc = instructionDescriptor(G::kCols, false);
    const uint64_t descB0 = operandDescriptor(smemAddr(bTile), G::kStrideB, kCore);
    bool alive = true;   // false once one of this thread's waits gave up: it waits no more and its values become NaN
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (alive) alive = waitPhase(bar, parity);
    };
    // the partial sums of step index n (counted from the last step) for this thread's elements, added to its dhBase
    const float *partMine = part + (ul & ~31) * ROWS + rowOf * 32 + (ul & 31);
    auto collect = [&](int n) {
        const uint32_t bar = smemAddr(&partBar[0]) + (n & 1) * 8;
        wait(bar, (n >> 1) & 1);
        if (tid == 0) cluster::arriveExpect(bar, G::kPartBytes);   // for step n + 2
        const float *src = partMine + (n & 1) * (ROWS * H);
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            float2 v[NC];
#pragma unroll
            for (int s = 0; s < NC; ++s) v[s] = live[i] ? *reinterpret_cast<const float2 *>(src + s * ROWS * U + i * G::kRowPass * 32) : make_float2(0.0f, 0.0f);
#pragma unroll
            for (int s = 0; s < NC; ++s) {
                dhBase[i].x += v[s].x;
                dhBase[i].y += v[s].y;
            }
        }
    };
    // What a step does to dh and dc, apart from dh and dc: mdc = (dc + dh intoCell) keepCell, gate gradient g = F[g] mdc
    // (F[3] dh), dc of the step before = mdc forget.  The flags 11..18 pick where a gate gradient goes.
    struct Factors {
        float f[4], intoCell, keepCell, forget, keepH, grad;
        uint32_t bits;
    };
    auto factorsOf = [&](const float (&gate)[4], float ctCode, float cellCode, float grad, uint32_t bits) {
        auto keep = [&](int pos) { return (bits >> pos) & 1u ? 0.0f : 1.0f; };
        auto real = [](float v, const Dequant &d) { return (v - d.zeroPoint) * d.scale; };
        const float ig = real(gate[0], a.dqGate[0]), fg = real(gate[1], a.dqGate[1]), cg = real(gate[2], a.dqGate[2]), og = real(gate[3], a.dqGate[3]);
        const float ct = real(ctCode, a.dqTanh), cPrev = real(cellCode, a.dqC);
        Factors r;
        r.f[0] = cg * ig * (1.0f - ig) * (keep(3) * keep(7));
        r.f[1] = cPrev * fg * (1.0f - fg) * (keep(4) * keep(8));
        r.f[2] = ig * (1.0f - cg * cg) * (keep(5) * keep(9));
        r.f[3] = ct * og * (1.0f - og) * (keep(6) * keep(10));
        r.intoCell = og * (1.0f - ct * ct) * keep(1);
        r.keepCell = keep(2);
        r.forget = fg;
        r.keepH = keep(0);
        r.grad = grad;
        r.bits = bits;
        return r;
    };
    // role in the product's read-out: a warp carries tiles of 32 units, up to two, and kSpan of the rows of each
    constexpr int kSpan = MT == 1 ? ROWS / 2 : ROWS, kReadouts = (MT + 1) / 2;
    const int quarter = warp & 3, half = min(warp >> 2, 1), row0 = MT == 1 ? half * kSpan : 0;
    uint32_t column[kReadouts], sendTo[kReadouts], sendBar[kReadouts];
    float *outMine[kReadouts];
    bool tileReal[kReadouts];
#pragma unroll
    for (int i = 0; i < kReadouts; ++i) {
        const int tile = MT == 1 ? 0 : half + 2 * i, unit0 = tile * 128 + 32 * quarter;
        tileReal[i] = unit0 < H && warp < G::kReadWarps;
        column[i] = tmem + (static_cast<uint32_t>(32 * quarter) << 16) + static_cast<uint32_t>(tile * G::kCols + row0);
        const uint32_t owner = min(static_cast<uint32_t>(unit0) / U, static_cast<uint32_t>(NC - 1));
        sendTo[i] = cluster::remote(smemAddr(part), owner) + ((rank * U + static_cast<uint32_t>(unit0) % U) * ROWS + row0 * 32) * 4;
        sendBar[i] = cluster::remote(smemAddr(&partBar[0]), owner);
        outMine[i] = outS + (tileReal[i] ? unit0 : 0) * ROWS + row0 * 32 + lane;
    }

    Factors fx[RPT], fy[RPT];
    // the next step's factors from ring slot `slot`
    auto prepare = [&](uint32_t slot) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const uint8_t *src = ring + slot + i * G::kRowBytes + tid * 8;
            auto operand = [&](int k) { return *reinterpret_cast<const float2 *>(src + k * (kThreads * 8)); };
            const float2 g0 = operand(0), g1 = operand(1), g2 = operand(2), g3 = operand(3), ct = operand(4), cell = operand(5), grad = operand(6);
            const uint2 bits = a.stepMasks ? *reinterpret_cast<const uint2 *>(src + 7 * (kThreads * 8)) : make_uint2(0u, 0u);
            fx[i] = factorsOf({g0.x, g1.x, g2.x, g3.x}, ct.x, cell.x, grad.x, bits.x);
            fy[i] = factorsOf({g0.y, g1.y, g2.y, g3.y}, ct.y, cell.y, grad.y, bits.y);
        }
    };
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    prepare(0);
    if (a.T > 2) fetch(a.T - 3, 0);
    commit();
    uint32_t slot = 0;   // of the current step
#pragma unroll 1
    for (int n = 0; n < a.T; ++n) {
        if (n > 0) collect(n - 1);   // the B operand is free as well: every thread has waited for the whole product of step n - 1
        float2 gate[RPT][4];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const float bad = __int_as_float(0x7fc00000);
            auto advance = [&](const Factors &f, float dhIn, float &cell, float (&out)[4]) {
                const float dh = alive ? (dhIn + f.grad) * f.keepH : bad;
                const float mdc = (cell + dh * f.intoCell) * f.keepCell;
#pragma unroll
                for (int g = 0; g < 3; ++g) out[g] = f.f[g] * mdc;
                out[3] = f.f[3] * dh;
                cell = mdc * f.forget;
            };
            float gx[4], gy[4];
            advance(fx[i], dhBase[i].x, dc[i].x, gx);
            advance(fy[i], dhBase[i].y, dc[i].y, gy);
            dhBase[i] = make_float2(0.0f, 0.0f);
            uint8_t *dst = bTile + static_cast<uint32_t>(ul >> 3) * G::kStrideB + (ul & 7) * 2 + (rowOf + G::kRowPass * i) * 16;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                gate[i][g] = make_float2(gx[g], gy[g]);
                float x = (fx[i].bits >> (15 + g)) & 1u ? 0.0f : gx[g] * scale[g].x, y = (fy[i].bits >> (15 + g)) & 1u ? 0.0f : gy[g] * scale[g].y;
#pragma unroll
                for (int term = 0; term < 3; ++term) {
                    const uint32_t word = packBf16(x, y);
                    x -= bf16Lo(word);
                    y -= bf16Hi(word);
                    *reinterpret_cast<uint32_t *>(dst + g * (U / 8) * G::kStrideB + term * ROWS * 16) = word;
                }
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (warp == 0) {
            if (electOne()) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int tile = 0; tile < MT; ++tile) {
#pragma unroll
                    for (int ks = 0; ks < G::kSliceK / 16; ++ks)
                        mmaBf16TmemA(tmem + tile * G::kCols, tmemWeights + tile * G::kColsA + ks * 8,
                                     descB0 + static_cast<uint64_t>(ks * ((2 * G::kStrideB) >> 4)), kIdesc, ks > 0 ? 1u : 0u);
                    if (tile + 1 == MT || tile % 2 == 1) commitTo(smemAddr(&productBar[tile / 2]));   // a pair of tiles is read while the next runs
                }
            }
            __syncwarp();
        }
        // the step's gate gradients leave while the product runs
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float2 v = gate[i][g];
                auto masked = [&](int pos) {
                    return make_float2((fx[i].bits >> pos) & 1u ? 0.0f : v.x, (fy[i].bits >> pos) & 1u ? 0.0f : v.y);
                };
                *reinterpret_cast<float2 *>(ihTo + i * (G::kRowPass * C) + g * H) = masked(11 + g);
                *reinterpret_cast<float2 *>(hhTo + i * (G::kRowPass * C) + g * H) = masked(15 + g);
            }
        }
        ihTo -= 4 * stepH;
        hhTo -= 4 * stepH;
        const uint32_t nextSlot = G::kSlotBytes - slot;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (n + 1 < a.T) prepare(nextSlot);
        // partial sums -> the CTAs that own the units.  A warp without a tile in some pair waits for that pair too: the next step
        // overwrites the B operand, and the sums that collect() waits for may all come from the first pair.
#pragma unroll
        for (int i = 0; i < kReadouts; ++i) {
            wait(smemAddr(&productBar[i]), n & 1);
            if (!tileReal[i]) continue;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            constexpr int kLoad = kSpan % 8 == 0 ? 8 : kSpan < 4 ? kSpan : 4;
            float *out = outMine[i] + (n & 1) * (ROWS * H);
#pragma unroll
            for (int r = 0; r < kSpan; r += kLoad) {
                uint32_t v[3][kLoad];
#pragma unroll
                for (int term = 0; term < 3; ++term) tmemLoad<kLoad>(column[i] + term * ROWS + r, v[term]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < kLoad; ++e)
                    out[(r + e) * 32] = (__uint_as_float(v[2][e]) + __uint_as_float(v[1][e])) + __uint_as_float(v[0][e]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) cluster::copyTo(sendTo[i] + (n & 1) * G::kPartBytes, smemAddr(out), kSpan * 128, sendBar[i] + (n & 1) * 8);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (n + 3 < a.T) fetch(a.T - 1 - (n + 3), nextSlot);   // while the partial sums travel
        commit();
        slot = nextSlot;
    }
    collect(a.T - 1);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        if (!live[i]) continue;
        const size_t o = static_cast<size_t>(b0 + rowOf + G::kRowPass * i) * H + j;
        auto keep = [&](const uint8_t *mask, int e) { return mask == nullptr || mask[o + e] == 0 ? 1.0f : 0.0f; };
        const float bad = alive ? 0.0f : __int_as_float(0x7fc00000);
        *reinterpret_cast<float2 *>(a.dh0 + o) = make_float2(dhBase[i].x * keep(a.maskH0, 0) + bad, dhBase[i].y * keep(a.maskH0, 1) + bad);
        *reinterpret_cast<float2 *>(a.dc0 + o) = make_float2(dc[i].x * keep(a.maskC0, 0) + bad, dc[i].y * keep(a.maskC0, 1) + bad);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols) : "memory");
    cluster::barrierAll();   // nobody leaves while a peer may still copy into its shared memory
}

struct Variant {
    void (*kernel)(BackwardClusterArgs);
    size_t smem;
    int ctas, threads;
};
template <int H, int U, int ROWS>
Variant variant() {
    return Variant{recurrentBackwardCluster<H, U, ROWS>, Tile<H, U, ROWS>::kSharedBytes, H / U, Tile<H, U, ROWS>::kThreads};
}
// The variants beyond 256 hidden units, built in lstm_backward_cluster_wide.cu.
Variant wideVariant(int H, int rows);

}  // namespace reverse
}  // namespace lstm
}  // namespace rxmet
