// One step after another of a recurrence on byte-plane codes, the product W_hh h on tcgen05 kind::i8, a thread per hidden
// unit: layers of up to 128 units inside one CTA, wider ones (up to 256) over a cluster.
//
// The accumulator of gate g is a tile of its own with the units as lanes, so that a thread finds the sums of ALL gates of its
// unit in its own tensor-memory lane: linear stages and cell follow in the same registers, without the exchange through
// shared memory and the barrier that plane_recurrence_umma.cuh needs for its tiles of mixed gates.  A CTA of U < 128 units
// fills the 128 lanes with 128 / U copies of its weights; each copy serves other rows.  The weights stay in tensor memory for the whole
// sequence (A operand: lane = channel, column = four bytes along K), the hidden codes of the rows are the B operand in shared
// memory, plane p of row r in accumulator column r PLANES + p.  Per step:
//   product -> linear stages and cell (ROWS x U cells, one to four per thread) -> new codes into the operand
//   (one CTA) or, staged, as one bulk copy to every CTA of the cluster -> control warp starts the next product.
// The warps only ARRIVE at the barrier behind the codes: what a step stores leaves and what the next but one reads is asked for
// while the next product runs.  Lanes beyond the last unit or row repeat the last one - the same values to the same places -
// instead of branching.
// What it replaced (a quarter of K per lane on dp4a, or a cluster of two with mixed gate tiles), T = 100, H = 128, 16-bit LSTM inference: 1 row 74 -> 55 us,
// 128 rows 116 -> 56, 700 rows 180 -> 141; training with all checkpoints: 128 rows 248 -> 72, 300 rows 229 -> 132; 8-bit training,
// 256 rows 162 -> 95.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <type_traits>

#include "cluster_device.cuh"
#include "common.h"
#include "dependent_launch.cuh"
#include "plane_recurrence_umma.cuh"

namespace rxmet {
namespace unitrec {

using namespace umma;
using planerec::Problem;

template <int N>
__device__ __forceinline__ void tmemLoad(uint32_t addr, uint32_t *r) {
    if constexpr (N == 1) asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r[0]) : "r"(addr));
    else if constexpr (N == 2) asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];\n" : "=r"(r[0]), "=r"(r[1]) : "r"(addr));
    else {
        static_assert(N % 4 == 0, "one, two or a multiple of four columns");
#pragma unroll
        for (int i = 0; i < N; i += 4) planerec::tmemLoad4(addr + i, r + i);
    }
}

// A word of the initial codes at Problem::h0.
template <int PLANES>
__device__ __forceinline__ uint32_t planeWord(const Problem &p, int row, int plane, int kw) {
    return __ldg(p.h0 + (static_cast<size_t>(row) * PLANES + plane) * ((p.H + 15) / 16 * 4) + kw);
}

template <class Cell, int HP, int U, int ROWS, int PLANES>
struct Geometry {
    static_assert(HP % U == 0 && 128 % U == 0 && U % 32 == 0, "units of a CTA");
    static constexpr int kCtas = HP / U, kGates = Cell::kGates, kCopies = 128 / U;
    // Two CTAs of eight epilogue warps on an SM rather than one of sixteen: as fast where both have rows (LSTM training, H = 128, 592
    // rows: 149 against 153 us), faster where one has them (256 rows: 100 against 129 us), and another pass finds room beside it.
    static constexpr int kGroups = ROWS / kCopies < 1 ? 1 : ROWS / kCopies > 2 ? 2 : ROWS / kCopies;   // warps of a quarter
    static constexpr int kWarps = 4 * kGroups, kThreads = 32 * (kWarps + 1);                            // and the control warp
    static constexpr int kRows = ROWS <= kCopies * kGroups ? 1 : ROWS / (kCopies * kGroups);            // rows of a thread
    static_assert(kRows * kCopies * kGroups >= ROWS && (kRows == 1 || kRows * kCopies * kGroups == ROWS), "rows divide");
    static constexpr int kCols = (PLANES * ROWS + 15) / 16 * 16;          // accumulator columns of a gate
    static constexpr uint32_t kColsA = HP / 4;                             // tensor-memory columns of its weights
    static constexpr uint32_t kTmemCols = planerec::powerOfTwoFrom(kGates * (kCols + kColsA));
    static_assert(kTmemCols <= 512, "tensor memory has 512 columns");
    static constexpr int kResident = kTmemCols <= 256 ? 2 : 1;             // CTAs of an SM
    static constexpr uint32_t kGroupStride = kCols * 16 + 16;              // next 16 bytes along K; the odd 16 bytes part the banks of a warp's two groups
    static constexpr uint32_t kOperandBytes = HP / 16 * kGroupStride;
    static constexpr uint32_t kSlabBytes = U / 16 * kGroupStride;          // this CTA's units
    static constexpr size_t kSharedBytes = kCtas == 1 ? (kOperandBytes + 127) / 128 * 128 : (2 * kOperandBytes + 2 * kSlabBytes + 127) / 128 * 128;
};

// Cell contract (device functions unless marked; `at` = first row of the step in the [T][B] arrays, `shared` = address of the
// operator's part of shared memory):
//   kGates, kTwoRows, kSignedCodes                          accumulator tiles; whether a thread has registers for two rows; codes as signed bytes
//   size_t sharedBytes()                                    host: size of that part
//   uint32_t weightWord(gate, unit, kw)                     four weight bytes along K
//   uint32_t codeWord(Problem, row, plane, kw)              four bytes of the initial codes; [B][PLANES][kWords] words at Problem::h0 or its own
//   void init(uint8_t *, shared, tid, threads)              fills it
//   bool valid()                                            false: the inputs are not good, outputs become NaN
//   Unit unitOf(shared, unit)                               constants of a unit (all lanes of the warp call it); Unit::plain, uniform in the
//                                                           warp: the usual parameters, for which advance<.., true> has the short forms
//   void begin(State &, row, unit)                          state of a row from h0
//   void fetch(Fetch &, at, row, unit)                      operands of a step
//   uint32_t advance<PLANES, PLAIN>(Unit, State &, Fetch, acc[gates][PLANES], Out &)   one step: new code - grid minimum
//   void store(Unit, Out, at, row, unit, good)              outputs of the step; good = false: make them NaN
//   void finish(State, row, unit, good)                     after the last step
template <class Cell, int HP, int U, int ROWS, int PLANES>
__global__ void __launch_bounds__(Geometry<Cell, HP, U, ROWS, PLANES>::kThreads, Geometry<Cell, HP, U, ROWS, PLANES>::kResident)
unitRecurrence(const __grid_constant__ Problem p, const __grid_constant__ Cell c) {
    using G = Geometry<Cell, HP, U, ROWS, PLANES>;
    constexpr int NC = G::kCtas, kGates = G::kGates, kRows = G::kRows;
    extern __shared__ __align__(128) uint8_t smemU[];
    __shared__ __align__(8) uint64_t productBar, codeBar[2];
    __shared__ uint32_t tmemSlot;
    __shared__ volatile int failed;   // the control warp's wait gave up
    uint8_t *operand = smemU;                                   // [NC == 1 ? 1 : 2][HP / 16][kCols + 1][16]
    uint8_t *staging = NC == 1 ? operand : operand + 2 * G::kOperandBytes;   // [2][U / 16][kCols + 1][16]
    const uint32_t shared = smemAddr(smemU) + static_cast<uint32_t>(G::kSharedBytes);   // the operator's own part

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    const int quarter = warp & 3, group = warp >> 2;
    const uint32_t rank = NC == 1 ? 0u : cluster::rank();
    const int local = quarter % (U / 32) * 32 + lane, slot = static_cast<int>(rank) * U + local;   // place of the unit in the CTA and in K
    const int unit = min(slot, p.H - 1);
    const int b0 = static_cast<int>(blockIdx.x) / NC * ROWS;
    const int rowInCta = (group * G::kCopies + quarter / (U / 32)) * kRows;   // first row of the thread
    const bool live = warp < G::kWarps && slot - lane < p.H && rowInCta < ROWS;   // uniform in the warp

    if (tid == 0) {
        failed = 0;
        cluster::initBarrier(&productBar, 1);
        for (int i = 0; i < 2; ++i) cluster::initBarrier(&codeBar[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        if (NC > 1)
            for (int i = 0; i < 2; ++i) cluster::arriveExpect(smemAddr(&codeBar[i]), NC * G::kSlabBytes);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    c.init(smemU + G::kSharedBytes, shared, tid, G::kThreads);
    for (uint32_t i = tid; i < G::kSharedBytes / 16; i += G::kThreads) reinterpret_cast<uint4 *>(operand)[i] = make_uint4(0u, 0u, 0u, 0u);
    waitForPredecessor();   // what is above needs nothing from earlier kernels
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const int kWords = (p.H + 15) / 16 * 4;   // words of a plane row
    for (int i = tid; i < ROWS * PLANES * (kWords / 4); i += G::kThreads) {
        const int kg = i % (kWords / 4), n = i / (kWords / 4), row = min(b0 + n / PLANES, p.B - 1);
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = c.codeWord(p, row, n % PLANES, 4 * kg + e);
        *reinterpret_cast<uint4 *>(operand + kg * G::kGroupStride + n * 16) = make_uint4(w[0], w[1], w[2], w[3]);
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0), tmemWeights = tmem + kGates * G::kCols;
    const uint32_t quarterBase = static_cast<uint32_t>(32 * quarter) << 16;
    if (warp < G::kWarps)   // the warps of a quarter share its weights
#pragma unroll 4
        for (int i = group; i < kGates * (HP / 16); i += G::kGroups) {
            const int g = i / (HP / 16), kw = i % (HP / 16) * 4;
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = kw + e < kWords ? c.weightWord(g, unit, kw + e) : 0u;
            planerec::tmemStore4(tmemWeights + quarterBase + g * G::kColsA + kw, w[0], w[1], w[2], w[3]);
        }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    if constexpr (NC > 1) cluster::barrierAll();   // every CTA's barriers are armed before anyone sends
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    bool alive = true;   // false once one of this warp's waits gave up
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (alive) alive = __all_sync(0xffffffffu, waitPhase(bar, parity));
    };
    // The barrier behind the codes of a step.  A warp whose wait gave up must not run ahead of the others: it waits here.
    auto codesWritten = [&] {
        if (alive) asm volatile("bar.arrive 1, %0;" ::"n"(G::kThreads) : "memory");
        else asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");
    };
    if (warp == G::kWarps) {
        // ---- control warp: products and copies; lane d sends to CTA d
        constexpr uint32_t kIdesc = planeproj::instructionDescriptor(G::kCols) | (Cell::kSignedCodes ? 1u << 10 : 0u);   // B format signed 8-bit
        const uint64_t descB0 = operandDescriptor(smemAddr(operand), G::kGroupStride, kCore);
        const uint32_t peer = static_cast<uint32_t>(lane) % NC;
        const uint32_t sendTo = NC == 1 ? 0u : cluster::remote(smemAddr(operand), peer) + rank * G::kSlabBytes;
        const uint32_t sendBar = NC == 1 ? 0u : cluster::remote(smemAddr(&codeBar[0]), peer);
#pragma unroll 1
        for (int t = 0; t < p.T; ++t) {
            const uint32_t bar = smemAddr(&codeBar[0]) + (t & 1) * 8;
            if (NC > 1 && t > 0) {
                wait(bar, ((t - 1) >> 1) & 1);
                if (!alive) failed = 1;
            }
            if (electOne()) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t descB = NC == 1 ? descB0 : descB0 + static_cast<uint64_t>((t & 1) * (G::kOperandBytes >> 4));
#pragma unroll
                for (int g = 0; g < kGates; ++g)
#pragma unroll
                    for (int ks = 0; ks < HP / 32; ++ks)
                        planerec::mmaI8TmemA(tmem + g * G::kCols, tmemWeights + g * G::kColsA + ks * 8,
                                             descB + static_cast<uint64_t>(ks * ((2 * G::kGroupStride) >> 4)), kIdesc, ks > 0 ? 1u : 0u);
                commitTo(smemAddr(&productBar));
                if (NC > 1 && t > 0) cluster::arriveExpect(bar, NC * G::kSlabBytes);   // for step t + 2
            }
            __syncwarp();
            asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");   // the codes of step t are written
            if (NC > 1 && t + 1 < p.T && lane < NC)
                cluster::copyTo(sendTo + ((t + 1) & 1) * G::kOperandBytes, smemAddr(staging) + (t & 1) * G::kSlabBytes, G::kSlabBytes,
                                sendBar + ((t + 1) & 1) * 8);
        }
    } else if (!live) {
        for (int t = 0; t < p.T; ++t) asm volatile("bar.sync 1, %0;" ::"n"(G::kThreads) : "memory");
    } else {
        const bool valid = c.valid();
        const typename Cell::Unit mine = c.unitOf(shared, unit);
        int row[kRows];
        typename Cell::State state[kRows];
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            row[r] = min(b0 + rowInCta + r, p.B - 1);
            c.begin(state[r], row[r], unit);
        }
        const uint32_t column = tmem + quarterBase + rowInCta * PLANES;
        uint8_t *codes = staging + local / 16 * G::kGroupStride + rowInCta * (PLANES * 16) + (local & 15);
        auto run = [&](auto plainTag) {
            constexpr bool kPlain = decltype(plainTag)::value;
            struct Operands {
                typename Cell::Fetch of[kRows];
            };
            auto fetch = [&](int t, Operands &to) {
                const size_t at = static_cast<size_t>(min(t, p.T - 1)) * p.B;
#pragma unroll
                for (int r = 0; r < kRows; ++r) c.fetch(to.of[r], at, row[r], unit);
            };
            auto step = [&](int t, Operands &now) {
                wait(smemAddr(&productBar), t & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t acc[kGates][kRows * PLANES];
#pragma unroll
                for (int g = 0; g < kGates; ++g) tmemLoad<kRows * PLANES>(column + g * G::kCols, acc[g]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                typename Cell::Out out[kRows];
#pragma unroll
                for (int r = 0; r < kRows; ++r) {
                    uint32_t sums[kGates][PLANES];
#pragma unroll
                    for (int g = 0; g < kGates; ++g)
#pragma unroll
                        for (int pl = 0; pl < PLANES; ++pl) sums[g][pl] = acc[g][r * PLANES + pl];
                    const uint32_t u = c.template advance<PLANES, kPlain>(mine, state[r], now.of[r], sums, out[r]);
                    uint8_t *to = codes + (NC == 1 ? 0u : (t & 1) * G::kSlabBytes) + r * (PLANES * 16);
                    if (PLANES == 2) to[0] = static_cast<uint8_t>(u >> 8);
                    to[(PLANES - 1) * 16] = static_cast<uint8_t>(u);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                codesWritten();
                // under the next product
                const size_t at = static_cast<size_t>(t) * p.B;
                const bool good = valid && alive && (NC == 1 || !failed);
#pragma unroll
                for (int r = 0; r < kRows; ++r) c.store(mine, out[r], at, row[r], unit, good);
                fetch(t + 2, now);
            };
            Operands even, odd;
            fetch(0, even);
            fetch(1, odd);
            int t = 0;
#pragma unroll 1
            for (; t + 1 < p.T; t += 2) {
                step(t, even);
                step(t + 1, odd);
            }
            if (t < p.T) step(t, even);
        };
        if (mine.plain) run(std::true_type{});
        else run(std::false_type{});
#pragma unroll
        for (int r = 0; r < kRows; ++r) c.finish(state[r], row[r], unit, valid && alive && (NC == 1 || !failed));
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols) : "memory");
    if constexpr (NC > 1) cluster::barrierAll();   // nobody leaves while a peer may still copy into its shared memory
}

template <class Cell, int HP, int U, int ROWS, int PLANES>
size_t sharedBytes(const Cell &cell) {
    using G = Geometry<Cell, HP, U, ROWS, PLANES>;
    // CTAs by themselves need not keep clusters out, only one CTA too many of their own kind, which would wait there for another's whole sequence
    const size_t least = G::kCtas > 1 ? cluster::leastShared(G::kTmemCols) : static_cast<size_t>(currentDevice().smemMax) / (512 / G::kTmemCols + 1) + 1024;
    return std::max(G::kSharedBytes + cell.sharedBytes(), least);
}

// CTAs without a cluster that an SM holds: as many as its tensor memory, unless the operator's tables are large (16-bit LSTM layers whose
// activations need 32 inputs a line have 120 kB of them; an SM has 228 kB, of which a CTA takes 1 kB by itself and less than 512 bytes statically).
template <class Cell, int HP, int U, int ROWS, int PLANES>
int residentCtas(const Cell &cell) {
    const size_t each = sharedBytes<Cell, HP, U, ROWS, PLANES>(cell) + 1024 + 512, all = static_cast<size_t>(currentDevice().smemMax) + 1024;
    return std::max(1, std::min(Geometry<Cell, HP, U, ROWS, PLANES>::kResident, static_cast<int>(all / each)));
}

// SMs that the most CTAs launchRows() takes for `rows` rows need beside a kernel that holds the others: clusters lie within one of about eight groups of
// SMs, each of which may have up to a cluster less one too many.  Launched beside a projection that leaves them no more than their number, clusters of
// three came to lie two on an SM: 16-bit GRU, T = 98, B = 64, H = 160 141 us, behind the projection's end 113; T = 98, B = 40,
// H = 256 142 and 121.
inline int smsFor(int rows, int H) {
    const int ctas = (H + 63) / 64;
    return H <= 128 ? rows : (rows + 3) / 4 * ctas + 8 * (ctas - 1);
}

// `early`: before the kernel in front of it has ended (its prologue runs beside that one's end).
template <class Cell, int HP, int U, int ROWS, int PLANES>
void launch(const char *name, const Problem &p, const Cell &cell, bool early, cudaStream_t st) {
    using G = Geometry<Cell, HP, U, ROWS, PLANES>;
    const auto kernel = unitRecurrence<Cell, HP, U, ROWS, PLANES>;
    const size_t smem = sharedBytes<Cell, HP, U, ROWS, PLANES>(cell);
    ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>((p.B + ROWS - 1) / ROWS * G::kCtas));
    cfg.blockDim = dim3(G::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attrs[2] = {};
    attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[0].val.programmaticStreamSerializationAllowed = early ? 1 : 0;
    attrs[1].id = cudaLaunchAttributeClusterDimension;
    attrs[1].val.clusterDim.x = G::kCtas;
    attrs[1].val.clusterDim.y = attrs[1].val.clusterDim.z = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = G::kCtas > 1 ? 2 : 1;
    {
        KernelTimer timer__(name, st);
        RXMET_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, cell));
    }
    afterLaunch(name);
}

// Rows of a CTA (up to 128 units) or of a cluster: as few as let all of them run at the same time, two of them on an SM.  A step of few
// rows is a chain of about 0.5 us (one CTA) or 1.1 us (a cluster), one of many is bound by issue, and two CTAs of an SM share it
// better than one of twice the rows (W8 / A16 LSTM inference, T = 100, H = 128: one row a CTA 56 us at 128 rows, two 66 at 256 and 94 at 592, where
// four take 99; four 144 at 1184, where two take 182 in two waves).
template <class Cell, int HP, int PLANES>
void launchRows(const char *name, const Problem &p, const Cell &cell, bool early, cudaStream_t st) {
    constexpr int U = HP <= 128 ? HP : 64, kLeast = HP > 128 ? 4 : 128 / U;
    auto fits = [&](auto rows) {
        constexpr int R = decltype(rows)::value;
        using G = Geometry<Cell, HP, U, R, PLANES>;
        const int groups = (p.B + R - 1) / R;
        if (HP == U) return groups <= (U == 128 && R == 1 ? 1 : residentCtas<Cell, HP, U, R, PLANES>(cell)) * smsPerPass();
        // the query counts one CTA of a cluster per SM (33 clusters of four); 36 clusters of eight rows run at the same time all the same
        return groups <= G::kResident * residentClusters(reinterpret_cast<const void *>(unitRecurrence<Cell, HP, U, R, PLANES>), G::kCtas,
                                                         G::kThreads, sharedBytes<Cell, HP, U, R, PLANES>(cell)) / concurrentPasses();
    };
    auto with = [&](auto rows) { unitrec::launch<Cell, HP, U, decltype(rows)::value, PLANES>(name, p, cell, early, st); };
    if (fits(std::integral_constant<int, kLeast>{})) return with(std::integral_constant<int, kLeast>{});
    constexpr int kNext = 2 * kLeast, kMost = HP > 128 ? kNext : 2 * kNext;
    if constexpr (kNext < kMost && Cell::kTwoRows) {
        if (!fits(std::integral_constant<int, kNext>{})) return with(std::integral_constant<int, kMost>{});
    }
    with(std::integral_constant<int, kNext>{});
}

}  // namespace unitrec
}  // namespace rxmet
