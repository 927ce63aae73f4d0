// One step after another of a recurrence on byte-plane codes (QuantLSTM W4 / W8 beyond 128 units, 16-bit activations) over a
// thread-block cluster, the product W_hh h on tcgen05 kind::i8.
//
// The H / U CTAs of a cluster advance ROWS batch rows together; a CTA owns U hidden units.  Their gate channels are the
// accumulator lanes - tiles of 128 lanes = 4 quarters (gates) x 32 units - and their
// weights stay in tensor memory for the whole sequence as the A operand (lane = channel, column = four bytes along K).
// The rows of a CTA fall into one to three groups that run on their own (operands, barriers, eight epilogue warps and a control warp
// each), so that the tensor pipe and the copies of one work under the epilogue of the others; only the weights and the operator's tables are
// shared.  The hidden codes of a group's rows, split into unsigned byte planes, are the B operand: plane p of row r is accumulator column
// p rows + r, so the weights are read once for both planes.  Per step and group:
//   product -> phase A (warp = quarter, lane = unit: the operator's linear stage and, where it likes, its gate) -> exchange
//   through shared memory inside the four warps of a tile -> phase B (lane = unit, a quarter of the rows per warp: the
//   cell) -> the new codes of the CTA's units, staged in operand layout, travel as one bulk copy to every CTA.
//
// Bound: the chain of one step where rows are few - about 0.3 k cycles of tcgen05, 0.4 k of copy latency, 0.2 k of
// barriers and the operator's epilogue at H = 256 -, issue and the table look-ups where they are many.  The operand in shared memory
// instead of tensor memory or an MMA issue loop that is not warp-uniform double the first part.  Row groups that shared product and
// barriers took turns with them, T = 100, H = 512: 256 rows, inference 377 -> 301 us, training 580 -> 500; 2048 rows 2045 -> 1390 us.
//
// Synchronisation: operand and staging buffers by step parity; a CTA sends the codes of step t only after it has those of
// step t - 1 of every peer, and a peer sends those only after its product of step t - 1 is complete: the operand
// buffer of step t (= t - 2) and the staging buffer it came from are free by then.  The epilogue warps only arrive at the barrier behind
// the codes.  Every wait is bounded; a warp whose wait gave up waits no more and reports it to the operator, which turns its outputs into NaN.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "cluster_device.cuh"
#include "common.h"
#include "plane_proj_umma.cuh"

namespace rxmet {
namespace planerec {

using namespace umma;

// D += A B with A (signed bytes) in tensor memory
__device__ __forceinline__ void mmaI8TmemA(uint32_t tmemD, uint32_t tmemA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n"
        :
        : "r"(tmemD), "r"(tmemA), "l"(descB), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}
__device__ __forceinline__ void tmemStore4(uint32_t addr, uint32_t v0, uint32_t v1, uint32_t v2, uint32_t v3) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v0), "r"(v1), "r"(v2), "r"(v3) : "memory");
}
__device__ __forceinline__ void tmemLoad4(uint32_t addr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

constexpr uint32_t powerOfTwoFrom(uint32_t n) {
    uint32_t p = 32;
    while (p < n) p *= 2;
    return p;
}

template <int HP, int U, int ROWS, int PLANES>
struct Geometry {
    static constexpr int kCtas = HP / U, kTiles = U / 32;
    // Epilogue warps of all row groups; each group has a control warp beside them.  Three row groups where they divide the rows.
    static constexpr int kWarps = ROWS * kTiles < 16 ? 8 : kTiles == 2 && ROWS % 12 == 0 ? 24 : 16;
    static constexpr int kRowGroups = kWarps / (4 * kTiles);
    static constexpr int kThreads = 32 * (kWarps + kRowGroups), kGroupThreads = 32 * (4 * kTiles + 1);
    static constexpr int kRowsA = ROWS / kRowGroups;            // rows of a group = of a lane in phase A
    static constexpr int kRowsB = kRowsA / 4;                   // cells of a lane in phase B
    static_assert(kRowsA % 4 == 0 && kRowsA * kRowGroups == ROWS, "rows divide into quads");
    static constexpr int kPadK = (HP + 31) / 32 * 32;
    static constexpr int kCols = (PLANES * kRowsA + 15) / 16 * 16;        // accumulator columns of a tile and row group
    static constexpr uint32_t kColsA = kPadK / 4;                          // tensor-memory columns of its weights
    static constexpr uint32_t kTmemCols = powerOfTwoFrom(kTiles * (kRowGroups * kCols + kColsA));
    static_assert(kTmemCols <= 512, "tensor memory has 512 columns");
    static constexpr uint32_t kGroupStride = kCols * 16 + 16;              // next 16 bytes along K; the odd 16 bytes part the banks of a warp's two groups
    static constexpr uint32_t kOperandBytes = kPadK / 16 * kGroupStride;
    static constexpr uint32_t kSlabBytes = U / 16 * kGroupStride;          // this CTA's units
    static constexpr uint32_t kBufferBytes = 2 * kOperandBytes + 2 * kSlabBytes;   // of a row group
    static constexpr uint32_t kExchangeBytes = kTiles * 4 * ROWS * 32 * 4;
    static constexpr size_t kSharedBytes = kRowGroups * kBufferBytes + kExchangeBytes;
};

struct Problem {
    int T, B, H;
    const uint32_t *h0;   // [B][PLANES][H padded to 16, / 4] words of four code bytes: the initial state
};

// Cell contract (device functions unless marked; `at` = first row of the step in the [T][B] arrays, `shared` = address of the
// operator's part of shared memory):
//   kGates, kSaves, kFull, kChunk                           quarters in use; whether storeLinear has anything to store; whether H is HP;
//                                                           most rows of phase A at a time
//   size_t sharedBytes()                                    host: size of that part
//   uint32_t weightWord(gate, unit, kw)                     four weight bytes along K, 0 for an empty quarter
//   void init(uint8_t *, tid, threads)                      fills it
//   bool valid()                                            false: the inputs are not good, outputs become NaN
//   Lane lane(shared, gate, unit, real)                     constants of phase A (all lanes of the warp call it)
//   void begin(shared, State &, row, unit)                  state of one cell of phase B from h0
//   void fetch(Fetch &, at, row, gate, unit), fetchB(FetchB &, at, row, unit)     operands of a step, asked for before the product is awaited
//   uint32_t linear<STRIDE>(shared, Lane, Fetch, acc, Saved &)    phase A; plane p of the sum at acc[p STRIDE]
//   kTotalFrom                                              rows of a cluster from which a step leaves no row out: the linear stage comes in two
//                                                           halves then, totals<STRIDE, ROWS>(Lane, acc) and linearOfTotal, with fetchRow for fetch,
//                                                           and has to be safe with any operand, also with what lies up to 64 rows behind the last row.
//                                                           Rows and units that do not exist are computed like the others - without a branch per row
//                                                           the rows of a thread interleave - and only their stores are left out, by
//                                                           storeRows(State[], FetchB[], at, row, unit, good, count) and storeLinearRows(Lane, Saved[],
//                                                           at, row, gate, unit, count): the first `count` rows of the array
//   uint32_t cell(shared, State &, FetchB, v[4])            phase B: new code - grid minimum
//   void store<LANES>(State, FetchB, at, row, unit, good, part)   outputs of the step; good = false: make them NaN
//   void storeLinear(Lane, Saved, at, row, gate, unit)      what phase A saves
//   void finish(State, row, unit, good)                     after the last step
template <class Cell, int HP, int U, int ROWS, int PLANES>
__global__ void __launch_bounds__(Geometry<HP, U, ROWS, PLANES>::kThreads, 1)
planeRecurrence(const __grid_constant__ Problem p, const __grid_constant__ Cell c) {
    using G = Geometry<HP, U, ROWS, PLANES>;
    constexpr int MT = G::kTiles, NC = G::kCtas, kFirstGroupBarrier = 1 + G::kWarps / 4;   // named barriers: one per tile and row group, one per group
    extern __shared__ __align__(128) uint8_t smemR[];
    __shared__ __align__(8) uint64_t productBars[G::kRowGroups], codeBars[G::kRowGroups][2];
    __shared__ uint32_t tmemSlot;
    __shared__ volatile int failed[G::kRowGroups];   // the wait of a group's control warp gave up
    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    const bool control = warp >= G::kWarps;
    const int quarter = warp & 3, tile = (warp >> 2) % MT, rowGroup = control ? warp - G::kWarps : (warp >> 2) / MT;
    uint8_t *operand = smemR + rowGroup * G::kBufferBytes;                   // [2][K / 16][kCols + 1][16]
    uint8_t *staging = operand + 2 * G::kOperandBytes;                       // [2][U / 16][kCols + 1][16]
    uint32_t *exchange = reinterpret_cast<uint32_t *>(smemR + G::kRowGroups * G::kBufferBytes);   // [tile][row group][4 gates][rowsA][32 units]
    const uint32_t shared = smemAddr(smemR) + static_cast<uint32_t>(G::kSharedBytes);                    // the operator's own part
    uint64_t &productBar = productBars[rowGroup], (&codeBar)[2] = codeBars[rowGroup];

    const uint32_t rank = cluster::rank();
    const int unit = static_cast<int>(rank) * U + tile * 32 + lane;
    const int b0 = static_cast<int>(blockIdx.x) / NC * ROWS;
    const int rowA = b0 + rowGroup * G::kRowsA, rowB = rowA + quarter * G::kRowsB;   // first rows of the two phases

    if (tid == 0) {
        for (int g = 0; g < G::kRowGroups; ++g) {
            failed[g] = 0;
            cluster::initBarrier(&productBars[g], 1);
            for (int i = 0; i < 2; ++i) cluster::initBarrier(&codeBars[g][i], 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        for (int g = 0; g < G::kRowGroups; ++g)
            for (int i = 0; i < 2; ++i) cluster::arriveExpect(smemAddr(&codeBars[g][i]), NC * G::kSlabBytes);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(G::kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    c.init(smemR + G::kSharedBytes, tid, G::kThreads);
    for (uint32_t i = tid; i < G::kRowGroups * G::kBufferBytes / 16; i += G::kThreads) reinterpret_cast<uint4 *>(smemR)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    const int H = p.H, kWords = (H + 15) / 16 * 4;   // words of a plane row
    for (int i = tid; i < ROWS * PLANES * (kWords / 4); i += G::kThreads) {
        const int kg = i % (kWords / 4), n = i / (kWords / 4), pl = n / ROWS, r = n - pl * ROWS, g = r / G::kRowsA;
        if (b0 + r < p.B)
            *reinterpret_cast<uint4 *>(smemR + g * G::kBufferBytes + kg * G::kGroupStride + (pl * G::kRowsA + r - g * G::kRowsA) * 16) =
                *reinterpret_cast<const uint4 *>(p.h0 + (static_cast<size_t>(b0 + r) * PLANES + pl) * kWords + 4 * kg);
    }
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0), tmemWeights = tmem + MT * G::kRowGroups * G::kCols;
    const uint32_t quarterBase = static_cast<uint32_t>(32 * quarter) << 16;
    if (rowGroup == 0 && !control)
        for (int kw = 0; kw < G::kPadK / 4; kw += 4) {
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = (kw + e < kWords && unit < H) ? c.weightWord(quarter, unit, kw + e) : 0u;
            tmemStore4(tmemWeights + quarterBase + tile * G::kColsA + kw, w[0], w[1], w[2], w[3]);
        }
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
    cluster::barrierAll();   // every CTA's barriers are armed before anyone sends
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    constexpr uint32_t kIdesc = planeproj::instructionDescriptor(G::kCols);
    bool alive = true;   // false once a wait of this warp gave up
    auto wait = [&](uint32_t bar, uint32_t parity) {
        if (alive) alive = __all_sync(0xffffffffu, G::kWarps > 8 ? waitSuspended(bar, parity) : waitPhase(bar, parity));   // polling wakes 2 % of a step earlier
    };
    const uint32_t tmemGroup = tmem + rowGroup * G::kCols;   // accumulators of this row group, MT tiles of kRowGroups kCols
    if (control) {
        // ---- control warp of a row group: products and copies; lane d sends to CTA d
        const uint32_t peer = static_cast<uint32_t>(lane) % NC;
        const uint32_t sendTo = cluster::remote(smemAddr(operand), peer) + rank * G::kSlabBytes;
        const uint32_t sendBar = cluster::remote(smemAddr(&codeBar[0]), peer);
        const uint64_t descB0 = operandDescriptor(smemAddr(operand), G::kGroupStride, kCore);
#pragma unroll 1
        for (int t = 0; t < p.T; ++t) {
            const uint32_t bar = smemAddr(&codeBar[0]) + (t & 1) * 8;
            if (t > 0) wait(bar, ((t - 1) >> 1) & 1);
            if (!alive) failed[rowGroup] = 1;
            if (electOne()) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t descB = descB0 + static_cast<uint64_t>((t & 1) * (G::kOperandBytes >> 4));
#pragma unroll
                for (int m = 0; m < MT; ++m)
#pragma unroll
                    for (int ks = 0; ks < G::kPadK / 32; ++ks)
                        mmaI8TmemA(tmemGroup + m * (G::kRowGroups * G::kCols), tmemWeights + m * G::kColsA + ks * 8,
                                   descB + static_cast<uint64_t>(ks * ((2 * G::kGroupStride) >> 4)), kIdesc, ks > 0 ? 1u : 0u);
                commitTo(smemAddr(&productBar));
                if (t > 0) cluster::arriveExpect(bar, NC * G::kSlabBytes);   // for step t + 2
            }
            __syncwarp();
            asm volatile("bar.sync %0, %1;" ::"r"(kFirstGroupBarrier + rowGroup), "n"(G::kGroupThreads) : "memory");   // the codes of step t are staged
            if (t + 1 < p.T && lane < NC)
                cluster::copyTo(sendTo + ((t + 1) & 1) * G::kOperandBytes, smemAddr(staging) + (t & 1) * G::kSlabBytes, G::kSlabBytes,
                                sendBar + ((t + 1) & 1) * 8);
        }
    } else {
        // Units beyond the layer's width compute on zero weights and store nothing.  Where a step leaves no row out (kAll) their codes
        // reach the operand all the same; they meet zero weights there too, those of every k >= H.
        const bool real = Cell::kFull || unit < H;
        const bool valid = c.valid();
        // rows of phase A in one go: as many as the operator allows and the rows divide into
        constexpr int kChunk = G::kRowsA <= Cell::kChunk ? G::kRowsA : (G::kRowsA % Cell::kChunk == 0 ? Cell::kChunk : 4);
        constexpr bool kDefer = G::kRowsA == 4;   // more rows keep the epilogue busy by themselves; held back they would spill
        constexpr bool kAll = ROWS >= Cell::kTotalFrom;
        const typename Cell::Lane mine = c.lane(shared, quarter, unit, real);
        typename Cell::State state[G::kRowsB] = {};
#pragma unroll
        for (int i = 0; i < G::kRowsB; ++i)
            if (real && rowB + i < p.B) c.begin(shared, state[i], rowB + i, unit);
        const uint32_t column = tmemGroup + quarterBase + tile * (G::kRowGroups * G::kCols);
        uint32_t *exchangeTile = exchange + (tile * G::kRowGroups + rowGroup) * (4 * G::kRowsA * 32) + lane;
        uint8_t *stageMine = staging + (tile * 2 + (lane >> 4)) * G::kGroupStride + (rowB - rowA) * 16 + (lane & 15);
#pragma unroll 1
        for (int t = 0; t < p.T; ++t) {
            const size_t at = static_cast<size_t>(t) * p.B;   // first row of the step in the [T][B] arrays
            // Phase A walks its rows kChunk at a time.  With kAll the operands of all of them are asked for before the product is
            // awaited (a chunk is too short to hide a load: a training step of 24 rows took 7.2 us with a chunk's lead); else the loop
            // is rolled and the operands of the next chunk are asked for before the current ones are used.
            constexpr int kFetched = kAll ? G::kRowsA : kChunk, kUnroll = kAll ? G::kRowsA / kChunk : 1;
            typename Cell::Fetch in[kFetched];
            typename Cell::FetchB inB[G::kRowsB];
            if constexpr (kAll)
                for (int i = 0; i < G::kRowsB; ++i) inB[i] = {};
            auto fetchA = [&](auto &to, int first, int count) {
#pragma unroll
                for (int r = 0; r < count; ++r)
                    if constexpr (kAll) c.fetchRow(to[r], at, rowA + first + r, quarter, unit);
                    else if (real && rowA + first + r < p.B) c.fetch(to[r], at, rowA + first + r, quarter, unit);
            };
            fetchA(in, 0, kFetched);
#pragma unroll
            for (int i = 0; i < G::kRowsB; ++i)
                if (real && rowB + i < p.B) c.fetchB(inB[i], at, rowB + i, unit);
            wait(smemAddr(&productBar), t & 1);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            typename Cell::Saved saved[kChunk];
#pragma unroll kUnroll
            for (int first = 0; first < G::kRowsA; first += kChunk) {
                uint32_t acc[PLANES * kChunk];
#pragma unroll
                for (int pl = 0; pl < PLANES; ++pl)
#pragma unroll
                    for (int r = 0; r < kChunk; r += 4) tmemLoad4(column + pl * G::kRowsA + first + r, acc + pl * kChunk + r);
                typename Cell::Fetch later[kChunk];
                if (!kAll && first + kChunk < G::kRowsA) fetchA(later, first + kChunk, kChunk);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (quarter < Cell::kGates) {
                    if constexpr (kAll) {
                        c.template totals<kChunk, kChunk>(mine, acc);
#pragma unroll
                        for (int r = 0; r < kChunk; ++r)
                            exchangeTile[(quarter * G::kRowsA + first + r) * 32] = c.linearOfTotal(shared, mine, in[first + r], acc[r], saved[r]);
                    } else
#pragma unroll
                    for (int r = 0; r < kChunk; ++r)
                        if (rowA + first + r < p.B)
                            exchangeTile[(quarter * G::kRowsA + first + r) * 32] = c.template linear<kChunk>(shared, mine, in[r], acc + r, saved[r]);
                    if constexpr (Cell::kSaves && !kDefer && kAll) {
                        c.storeLinearRows(mine, saved, at, rowA + first, quarter, unit, real ? p.B - rowA - first : 0);
                    } else if (Cell::kSaves && !kDefer) {
#pragma unroll
                        for (int r = 0; r < kChunk; ++r)
                            if (real && rowA + first + r < p.B) c.storeLinear(mine, saved[r], at, rowA + first + r, quarter, unit);
                    }
                }
                if (!kAll && G::kRowsA > kChunk) {
#pragma unroll
                    for (int r = 0; r < kChunk; ++r) in[r] = later[r];
                }
            }
            asm volatile("bar.sync %0, 128;" ::"r"(1 + (warp >> 2)) : "memory");   // the four quarters of this tile and row group
#pragma unroll
            for (int i = 0; i < G::kRowsB; ++i) {
                const bool exists = real && rowB + i < p.B;
                if (!kAll && !exists) continue;
                uint32_t v[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) v[g] = g < Cell::kGates ? exchangeTile[(g * G::kRowsA + quarter * G::kRowsB + i) * 32] : 0u;
                const uint32_t u = c.cell(shared, state[i], inB[i], v);
                uint8_t *dst = stageMine + (t & 1) * G::kSlabBytes + i * 16;
                if (PLANES == 2) {
                    dst[0] = static_cast<uint8_t>(u >> 8);
                    dst[G::kRowsA * 16] = static_cast<uint8_t>(u);
                } else {
                    dst[0] = static_cast<uint8_t>(u);
                }
                if (!kDefer && !kAll && exists) c.store(state[i], inB[i], at, rowB + i, unit, valid && alive && !failed[rowGroup]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            // the control warp sends the codes; a warp whose wait gave up must not run ahead of the others and waits here
            if (alive) asm volatile("bar.arrive %0, %1;" ::"r"(kFirstGroupBarrier + rowGroup), "n"(G::kGroupThreads) : "memory");
            else asm volatile("bar.sync %0, %1;" ::"r"(kFirstGroupBarrier + rowGroup), "n"(G::kGroupThreads) : "memory");
            if constexpr (!kDefer && kAll) c.storeRows(state, inB, at, rowB, unit, valid && alive && !failed[rowGroup], real ? p.B - rowB : 0);
            if constexpr (kDefer && kAll) {   // what nobody waits for leaves while the codes travel and the next product runs
                c.storeRows(state, inB, at, rowB, unit, valid && alive && !failed[rowGroup], real ? p.B - rowB : 0);
                if constexpr (Cell::kSaves) {
                    if (quarter < Cell::kGates) c.storeLinearRows(mine, saved, at, rowA, quarter, unit, real ? p.B - rowA : 0);
                }
            } else if (kDefer) {
#pragma unroll
                for (int i = 0; i < G::kRowsB; ++i)
                    if (real && rowB + i < p.B) c.store(state[i], inB[i], at, rowB + i, unit, valid && alive && !failed[rowGroup]);
                if (Cell::kSaves && quarter < Cell::kGates) {
#pragma unroll
                    for (int r = 0; r < kChunk; ++r)
                        if (real && rowA + r < p.B) c.storeLinear(mine, saved[r], at, rowA + r, quarter, unit);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < G::kRowsB; ++i)
            if (real && rowB + i < p.B) c.finish(state[i], rowB + i, unit, valid && alive && !failed[rowGroup]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(G::kTmemCols) : "memory");
    cluster::barrierAll();   // nobody leaves while a peer may still copy into its shared memory
}

template <class Cell, int HP, int U, int ROWS, int PLANES>
size_t sharedBytes(const Cell &cell) {
    using G = Geometry<HP, U, ROWS, PLANES>;
    return std::max(G::kSharedBytes + cell.sharedBytes(), cluster::leastShared(G::kTmemCols));
}

// Launches a variant with its clusters.
template <class Cell, int HP, int U, int ROWS, int PLANES>
void launch(const char *name, const Problem &p, const Cell &cell, cudaStream_t st) {
    using G = Geometry<HP, U, ROWS, PLANES>;
    const auto kernel = planeRecurrence<Cell, HP, U, ROWS, PLANES>;
    const size_t smem = sharedBytes<Cell, HP, U, ROWS, PLANES>(cell);
    ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>((p.B + ROWS - 1) / ROWS * G::kCtas));
    cfg.blockDim = dim3(G::kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = G::kCtas;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    {
        KernelTimer timer__(name, st);
        RXMET_CUDA(cudaLaunchKernelEx(&cfg, kernel, p, cell));
    }
    afterLaunch(name);
}

// Rows of a cluster among ROWS...: the number of waves times the cost of a step, which is about 1 + rows / PER of the
// chain of a short one - as few rows as let all clusters run at the same time, or many where they cannot.  Four rows only
// where they leave half of the GPU free: the other direction of a layer may run beside this pass.
template <class Cell, int HP, int U, int PLANES, int PER, int... ROWS>
void launchBest(const char *name, const Problem &p, const Cell &cell, cudaStream_t st) {
    double bestCost = 1e30;
    int best = 0;
    (
        [&] {
            using G = Geometry<HP, U, ROWS, PLANES>;
            // a single wave of it would not beat what is found already: do not even load the variant
            if (1.0 + ROWS / static_cast<double>(PER) >= bestCost || sharedBytes<Cell, HP, U, ROWS, PLANES>(cell) > static_cast<size_t>(currentDevice().smemMax)) return;
            const int resident = std::max(1, residentClusters(reinterpret_cast<const void *>(planeRecurrence<Cell, HP, U, ROWS, PLANES>), G::kCtas,
                                                              G::kThreads, sharedBytes<Cell, HP, U, ROWS, PLANES>(cell)) / concurrentPasses());
            const int clusters = (p.B + ROWS - 1) / ROWS, waves = (clusters + resident - 1) / resident;
            if (ROWS == 4 && G::kTmemCols > 256 && 2 * clusters > resident) return;
            const double cost = waves * (1.0 + ROWS / static_cast<double>(PER));
            if (cost < bestCost) { bestCost = cost; best = ROWS; }
        }(),
        ...);
    (
        [&] {
            if (best == ROWS) launch<Cell, HP, U, ROWS, PLANES>(name, p, cell, st);
        }(),
        ...);
}

}  // namespace planerec
}  // namespace rxmet
