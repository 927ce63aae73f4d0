// dh of the GRU backward through time with the per-step product on tcgen05 and the hidden units spread over a
// thread-block cluster.
//
// The step is a chain: pointwise derivative -> dh += R dq -> next step.  The H / U CTAs of a cluster advance a tile of
// batch rows together.  A CTA owns U hidden units: their pointwise derivative yields exactly the 3 U columns of dq that
// form ITS slice of the contraction, so nothing has to be gathered for the product.  Its columns of R stay in tensor
// memory for the whole sequence as exact bf16 codes (A operand; all H units are accumulator lanes); dq, scaled per
// column and split into three bf16 terms (products exact, fp32 accumulation), is the B operand in shared memory.  The
// three terms are three groups of accumulator COLUMNS of one product, so the weights are read once per step.  The partial
// sums [units][rows] leave through shared memory as one bulk copy per 32 units into the CTA that owns them, which adds
// the H / U partial sums in a fixed order (reproducible) at the start of its next step.
//
// What bounds it and what that chose (H = 256, 8 rows, cycle counters per step): 0.55 k cycles of tcgen05 (24 MMAs of
// 128 x 32 x 16; weights in shared memory would make that 1.1 k, the operand read is then the bound), 0.4 k of one-way copy
// latency, 0.2 k of barriers, the rest is the pointwise chain.  Hence: operands of later steps and everything that does not
// depend on the incoming dh are handled while product or copy are under way; the loop body is kept small and rolled
// (unrolled by three it ran at half the speed: the warps pass it once per step and instruction fetch showed); the
// MMA issue loop is warp-uniform; the partial sums leave as one bulk copy per warp (a store that completes on the
// barrier by itself costs the receiver one barrier update per lane).  Distributed shared memory carries about 16 bytes
// per clock and SM, so a CTA takes U = 64 units where it can and a cluster as few rows as fill the GPU.
// T = 100, B = 128, H = 256, both directions of a layer at a time: 713 -> 130 us per pass (recurrentBackwardCodes on
// FP32 FMA).  Up to 128 units: unit_reverse_umma.cuh.
//
// Synchronisation: the receiver's mbarrier counts the bytes, two partial-sum buffers by step parity.  A CTA
// sends step t only after it has the partial sums of step t + 1 of every peer, and a peer sends those only after it
// has read the buffer of step t + 2: the buffer of step t is free by then.  No cluster-wide barrier inside the loop;
// every wait is bounded, and one that gives up ends all further waiting of the CTA and turns its outputs into NaN.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "backward_cluster_device.cuh"
#include "cluster_device.cuh"
#include "common.h"
#include "gru_backward_cluster.h"
#include "umma_device.cuh"

namespace rxmet {
namespace gru {
namespace {

using namespace bwdcluster;

constexpr int kThreads = 256, kWarps = kThreads / 32;

struct ClusterArgs {
    BackwardQArgs q;
    const int32_t *Rq;
};

// Geometry of a cluster of H / U CTAs that advances ROWS batch rows.
template <int H, int U, int ROWS>
struct Tile {
    static constexpr int kCtas = H / U, kTiles = (H + 127) / 128, kSliceK = 3 * U, kGroupsK = kSliceK / 8;
    static constexpr int kPairs = U / 2, kRowPass = kThreads / kPairs, kRowsPerThread = (ROWS + kRowPass - 1) / kRowPass;
    static constexpr int kCols = (3 * ROWS + 15) / 16 * 16;          // accumulator columns of one tile of 128 units
    static constexpr uint32_t kColsA = kSliceK / 2;                   // tensor-memory columns of one weight tile
    static constexpr uint32_t kTmemCols = powerOfTwoFrom(kTiles * (kCols + kColsA));
    // K-group stride of the B operand: 16 bytes more than its rows, so that the lanes of a warp (two neighbouring k
    // each) spread over the banks when they store one row
    static constexpr uint32_t kStrideB = kCols * 16 + 16;
    static constexpr uint32_t kOperandBytes = kGroupsK * kStrideB;
    static constexpr uint32_t kPartBytes = static_cast<uint32_t>(ROWS) * H * 4;
    static constexpr uint32_t kSlotBytes = kRowsPerThread * kThreads * (6 * 8 + 4);   // operands of one step
    static constexpr size_t kSharedBytes = kOperandBytes + 4 * kPartBytes + 3 * kSlotBytes + 128;
};

template <int H, int U, int ROWS>
__global__ void __launch_bounds__(kThreads, 1) recurrentBackwardUmma(const __grid_constant__ ClusterArgs ca) {
    using namespace umma;
    using G = Tile<H, U, ROWS>;
    constexpr int C = 3 * H, NC = G::kCtas, MT = G::kTiles, RPT = G::kRowsPerThread;
    const BackwardQArgs &a = ca.q;
    extern __shared__ __align__(128) uint8_t smemC[];
    __shared__ __align__(8) uint64_t productBar, partBar[2];
    __shared__ uint32_t tmemSlot;
    uint8_t *bTile = smemC;                                                    // [kGroupsK][kCols (+1)][16 bytes]
    float *part = reinterpret_cast<float *>(bTile + G::kOperandBytes);         // [2][NC sources][U / 32][ROWS][32 units]
    float *outS = part + 2 * ROWS * H;                                         // [2][H / 32 unit tiles][ROWS][32 units], to be sent
    uint8_t *ring = reinterpret_cast<uint8_t *>(outS + 2 * ROWS * H);          // [3 slots][RPT][6 x float2, 1 x 2 flag words][threads]

    const int tid = threadIdx.x, lane = tid & 31, warp = umma::warpIndex();
    const uint32_t rank = cluster::rank();
    const int ul = tid % G::kPairs * 2, rowOf = tid / G::kPairs;   // pointwise role: units ul, ul + 1 of rows rowOf + i kRowPass
    const int j = static_cast<int>(rank) * U + ul;
    const int b0 = static_cast<int>(blockIdx.x) / NC * ROWS;

    if (tid == 0) {
        cluster::initBarrier(&productBar, 1);
        for (int i = 0; i < 2; ++i) cluster::initBarrier(&partBar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int i = 0; i < 2; ++i) cluster::arriveExpect(smemAddr(&partBar[i]), G::kPartBytes);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (uint32_t i = tid; i < G::kOperandBytes / 16; i += kThreads) reinterpret_cast<uint4 *>(bTile)[i] = make_uint4(0u, 0u, 0u, 0u);
    float2 scale[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) scale[g] = *reinterpret_cast<const float2 *>(a.scaleR + g * H + j);
    float2 dhBase[RPT];
    bool live[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = rowOf + G::kRowPass * i;
        live[i] = row < ROWS && b0 + row < a.B;
        dhBase[i] = (live[i] && a.dhIn) ? *reinterpret_cast<const float2 *>(a.dhIn + static_cast<size_t>(b0 + row) * H + j) : make_float2(0.0f, 0.0f);
    }
    // Operands of a step travel two steps ahead through shared memory (a thread reads back what it copied itself): they come
    // from HBM, and a ring in registers would need the loop unrolled by three - the instruction cache feels that.
    const size_t first = (static_cast<size_t>(a.T - 1) * a.B + b0 + rowOf) * H + j;   // element of the last step
    const size_t stepH = static_cast<size_t>(a.B) * H;
    const float *vFrom = a.v + (first - j) * 4 + j, *hFrom = a.h + first, *dhFrom = a.dhNew + first + stepH;
    const uint16_t *bitsFrom = a.stepBits ? a.stepBits + first : nullptr;
    const uint32_t mySlot = smemAddr(ring) + tid * 8, myBits = smemAddr(ring) + RPT * 6 * kThreads * 8 + tid * 4;
    auto fetch = [&](uint32_t slotBase) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const uint32_t dst = mySlot + slotBase + i * (6 * kThreads * 8);
            const float *v = vFrom + i * (G::kRowPass * 4 * H);
            copyAsync<8>(dst, v);
            copyAsync<8>(dst + kThreads * 8, v + H);
            copyAsync<8>(dst + kThreads * 16, v + 2 * H);
            copyAsync<8>(dst + kThreads * 24, v + 3 * H);
            copyAsync<8>(dst + kThreads * 32, hFrom + i * (G::kRowPass * H));
            copyAsync<8>(dst + kThreads * 40, dhFrom + i * (G::kRowPass * H));
            if (bitsFrom) copyAsync<4>(myBits + slotBase + i * (kThreads * 4), bitsFrom + i * (G::kRowPass * H));
        }
        vFrom -= 4 * stepH;
        hFrom -= stepH;
        dhFrom -= stepH;
        if (bitsFrom) bitsFrom -= stepH;
    };
    auto commit = [] { asm volatile("cp.async.commit_group;" ::: "memory"); };
#pragma unroll 1
    for (int n = 0; n < 3; ++n) {
        if (n < a.T) fetch(n * G::kSlotBytes);
        commit();
    }
    float *dpTo = a.dp + (first - j) * 3 + j, *dqTo = a.dq + (first - j) * 3 + j;
    __syncthreads();
    const uint32_t tmem = tmemSlot, tmemWeights = tmem + MT * G::kCols;
    // weights: lane = hidden unit m, column = two of this CTA's 3 U channels
    for (int tile = warp >> 2; tile < MT; tile += kWarps / 4) {
        const int m = tile * 128 + 32 * (warp & 3) + lane;
        for (int kg = 0; kg < G::kGroupsK; ++kg) {
            const int gate = kg / (U / 8), within = kg % (U / 8) * 8;
            uint4 packed = make_uint4(0u, 0u, 0u, 0u);
            if (m < H) {
                const int4 *src = reinterpret_cast<const int4 *>(ca.Rq + static_cast<size_t>(m) * C + gate * H + rank * U + within);
                const int4 x = __ldg(src), y = __ldg(src + 1);
                packed.x = packBf16(static_cast<float>(x.x), static_cast<float>(x.y));
                packed.y = packBf16(static_cast<float>(x.z), static_cast<float>(x.w));
                packed.z = packBf16(static_cast<float>(y.x), static_cast<float>(y.y));
                packed.w = packBf16(static_cast<float>(y.z), static_cast<float>(y.w));
            }
            tmemStore4(tmemWeights + (static_cast<uint32_t>(32 * (warp & 3)) << 16) + tile * G::kColsA + kg * 4, packed);
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
    // Every gradient of a step is linear in the incoming dh: the factors do not depend on it and are formed while the
    // partial sums are under way.  p: gate-input gradients of the input branch, q: of the recurrent branch.
    struct Factors {
        float p[3], q[3], z, keep;
    };
    auto factorsOf = [](float z, float r, float g, float qg, float hOld, uint32_t bits) {
        auto keep = [&](int pos) { return static_cast<float>((bits >> pos) & 1u); };
        Factors f;
        f.z = z;
        f.keep = keep(12);
        const float fn = ((1.0f - g * g) * (1.0f - z)) * (keep(2) * keep(5));
        const float fr = ((r * (1.0f - r)) * (fn * qg)) * (keep(1) * keep(4));
        const float fz = ((z * (1.0f - z)) * (hOld - g)) * (keep(0) * keep(3));
        f.p[0] = fz * keep(9); f.p[1] = fr * keep(10); f.p[2] = fn * keep(11);
        f.q[0] = fz * keep(6); f.q[1] = fr * keep(7); f.q[2] = (fn * r) * keep(8);
        return f;
    };
    // role in the product's read-out: a warp carries one tile of 32 units and kSpan of the rows
    constexpr int kSpan = MT == 2 ? ROWS : ROWS / 2;
    const int quarter = warp & 3, tileOf = MT == 2 ? warp >> 2 : 0, unit0 = tileOf * 128 + 32 * quarter, row0 = MT == 2 ? 0 : (warp >> 2) * kSpan;
    const uint32_t column = tmem + (static_cast<uint32_t>(32 * quarter) << 16) + static_cast<uint32_t>(tileOf * G::kCols + row0);
    const uint32_t owner = min(static_cast<uint32_t>(unit0) / U, static_cast<uint32_t>(NC - 1));
    const uint32_t sendTo = cluster::remote(smemAddr(part), owner) + ((rank * U + static_cast<uint32_t>(unit0) % U) * ROWS + row0 * 32) * 4;
    const uint32_t sendBar = cluster::remote(smemAddr(&partBar[0]), owner);
    float *outMine = outS + unit0 * ROWS + row0 * 32 + lane;

    Factors fx[RPT], fy[RPT];
    float2 dhNew[RPT];
    // the next step's factors from ring slot `slot`
    auto prepare = [&](uint32_t slot) {
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const uint8_t *src = ring + slot + i * (6 * kThreads * 8) + tid * 8;
            auto operand = [&](int k) { return *reinterpret_cast<const float2 *>(src + k * (kThreads * 8)); };
            const float2 z = operand(0), r = operand(1), g = operand(2), qg = operand(3), hOld = operand(4);
            dhNew[i] = operand(5);
            const uint32_t bits = a.stepBits ? *reinterpret_cast<const uint32_t *>(ring + slot + RPT * 6 * kThreads * 8 + i * (kThreads * 4) + tid * 4) : 0x1fff1fffu;
            fx[i] = factorsOf(z.x, r.x, g.x, qg.x, hOld.x, bits & 0xffffu);
            fy[i] = factorsOf(z.y, r.y, g.y, qg.y, hOld.y, bits >> 16);
        }
    };
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    prepare(0);
    uint32_t slot = 0;   // of the current step
#pragma unroll 1
    for (int n = 0; n < a.T; ++n) {
        if (n > 0) collect(n - 1);   // this CTA's own sums among them: the product of that step has read the B operand
        float2 dh[RPT];
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
            const float bad = __int_as_float(0x7fc00000);
            dh[i] = make_float2(alive ? (dhNew[i].x + dhBase[i].x) * fx[i].keep : bad, alive ? (dhNew[i].y + dhBase[i].y) * fy[i].keep : bad);
            dhBase[i] = make_float2(fx[i].z * dh[i].x, fy[i].z * dh[i].y);
            uint8_t *dst = bTile + static_cast<uint32_t>(ul >> 3) * G::kStrideB + (ul & 7) * 2 + (rowOf + G::kRowPass * i) * 16;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                float x = fx[i].q[g] * dh[i].x * scale[g].x, y = fy[i].q[g] * dh[i].y * scale[g].y;
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
                for (int tile = 0; tile < MT; ++tile)
#pragma unroll
                    for (int ks = 0; ks < G::kSliceK / 16; ++ks)
                        mmaBf16TmemA(tmem + tile * G::kCols, tmemWeights + tile * G::kColsA + ks * 8,
                                     descB0 + static_cast<uint64_t>(ks * ((2 * G::kStrideB) >> 4)), kIdesc, ks > 0 ? 1u : 0u);
                commitTo(smemAddr(&productBar));
            }
            __syncwarp();
        }
        // the step's gate gradients leave while the product runs
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (!live[i]) continue;
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                *reinterpret_cast<float2 *>(dpTo + i * (G::kRowPass * C) + g * H) = make_float2(fx[i].p[g] * dh[i].x, fy[i].p[g] * dh[i].y);
                *reinterpret_cast<float2 *>(dqTo + i * (G::kRowPass * C) + g * H) = make_float2(fx[i].q[g] * dh[i].x, fy[i].q[g] * dh[i].y);
            }
        }
        dpTo -= 3 * stepH;
        dqTo -= 3 * stepH;
        const uint32_t nextSlot = slot == 2 * G::kSlotBytes ? 0 : slot + G::kSlotBytes;
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (n + 1 < a.T) prepare(nextSlot);
        // partial sums -> the CTAs that own the units
        if (unit0 < H) {
            wait(smemAddr(&productBar), n & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            constexpr int kLoad = kSpan < 8 ? kSpan : 8;
            float *out = outMine + (n & 1) * (ROWS * H);
#pragma unroll
            for (int r = 0; r < kSpan; r += kLoad) {
                uint32_t v[3][kLoad];
#pragma unroll
                for (int term = 0; term < 3; ++term) tmemLoad<kLoad>(column + term * ROWS + r, v[term]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int e = 0; e < kLoad; ++e)
                    out[(r + e) * 32] = (__uint_as_float(v[2][e]) + __uint_as_float(v[1][e])) + __uint_as_float(v[0][e]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) cluster::copyTo(sendTo + (n & 1) * G::kPartBytes, smemAddr(out), kSpan * 128, sendBar + (n & 1) * 8);
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        if (n + 3 < a.T) fetch(slot);   // while the partial sums travel
        commit();
        slot = nextSlot;
    }
    collect(a.T - 1);
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        if (!live[i]) continue;
        const size_t o = static_cast<size_t>(b0 + rowOf + G::kRowPass * i) * H + j;
        float2 keep = make_float2(1.0f, 1.0f);
        if (!a.carryOut && a.mH0) keep = make_float2(static_cast<float>(a.mH0[o]), static_cast<float>(a.mH0[o + 1]));
        const float bad = alive ? 0.0f : __int_as_float(0x7fc00000);
        *reinterpret_cast<float2 *>(a.dh0 + o) = make_float2(dhBase[i].x * keep.x + bad, dhBase[i].y * keep.y + bad);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols) : "memory");
    cluster::barrierAll();   // nobody leaves while a peer may still copy into its shared memory
}

using Kernel = void (*)(ClusterArgs);
struct Variant {
    Kernel kernel;
    size_t smem;
    int ctas;
};
template <int H, int ROWS>
Variant variant() {
    constexpr int U = H % 64 == 0 ? 64 : 32;
    return Variant{recurrentBackwardUmma<H, U, ROWS>, Tile<H, U, ROWS>::kSharedBytes, H / U};
}
template <int ROWS>
Variant variantFor(int H) {
    switch (H) {
        case 160: return variant<160, ROWS>();
        case 192: return variant<192, ROWS>();
        case 224: return variant<224, ROWS>();
        default: return variant<256, ROWS>();
    }
}
Variant variantFor(int H, int rows) { return rows == 4 ? variantFor<4>(H) : rows == 8 ? variantFor<8>(H) : variantFor<16>(H); }

}  // namespace

bool backwardClusterTakes(const BackwardQArgs &q, const int32_t *Rq) {
    auto aligned = [](const void *p, uintptr_t n) { return (reinterpret_cast<uintptr_t>(p) & (n - 1)) == 0; };
    return q.H % 32 == 0 && q.H >= 32 && q.H <= 256 && aligned(Rq, 16) && aligned(q.h, 8) && aligned(q.v, 8) && aligned(q.dhNew, 8) &&
           aligned(q.dp, 8) && aligned(q.dq, 8) && aligned(q.dh0, 8) && aligned(q.stepBits, 4) && aligned(q.scaleR, 8);
}

void backwardCluster(const BackwardQArgs &q, const int32_t *Rq, cudaStream_t st) {
    if (q.H <= 128) return backwardUnits(q, Rq, st);   // inside one CTA
    ClusterArgs args{};
    args.q = q;
    args.Rq = Rq;
    // Rows of a cluster: as few as let all clusters of the pass run at the same time (a step costs about 1 + rows / 32
    // of the chain of a one-row step, a second wave costs the whole chain again).
    int best = 4;
    double bestCost = 1e30;
    for (int rows : {4, 8, 16}) {
        if (1.0 + rows / 32.0 >= bestCost) break;   // not even in a single wave: leave the variant unloaded
        const Variant v = variantFor(q.H, rows);
        const int resident = std::max(1, residentClusters(reinterpret_cast<const void *>(v.kernel), v.ctas, kThreads, v.smem) / concurrentPasses());
        const int clusters = (q.B + rows - 1) / rows, waves = (clusters + resident - 1) / resident;
        const double cost = waves * (1.0 + rows / 32.0);
        if (cost < bestCost) { bestCost = cost; best = rows; }
    }
    const Variant v = variantFor(q.H, best);
    ensureDynamicSmem(reinterpret_cast<const void *>(v.kernel), v.smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>((q.B + best - 1) / best * v.ctas));
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = v.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(v.ctas);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    {
        KernelTimer timer__("recurrentBackward", st);
        RXMET_CUDA(cudaLaunchKernelEx(&cfg, v.kernel, args));
    }
    afterLaunch("recurrentBackwardUmma");
}

}  // namespace gru
}  // namespace rxmet
