// Input projection of the byte-plane paths (16-bit or 8-bit activation codes as one or two unsigned byte
// planes, signed 8-bit weight codes) as a tcgen05.mma kind::i8 GEMM with exact 32-bit integer accumulators in
// tensor memory, shared by the QuantGRU W8 / A16 forward and the wide QuantLSTM forward:
//
//   acc_p[row][c] = sum_k plane_p[row][k] * w[k][c]        (p = high, low byte plane)
//   out[row][c]   = epilogue(c, acc_high, acc_low)         (the caller's functor: exact combine, rescale,
//                                                           clamp, masks - whatever its operator defines)
//
// The product is computed transposed, D[channel][row], so that a lane of tensor memory is a channel: the
// per-channel constants of the epilogue live in registers and, for one row, the lanes of a warp store
// neighbouring channels.
//
// A work item is a tile of NR rows and a tile of 128 channels; a CTA takes the channel tiles of one share of a row tile one after
// another.  Few row tiles are cut into shares of fewer channel tiles, so that a short call fills the GPU as well.  Warps by role:
//   weights   one lane copies weight tiles, packed beforehand in the canonical K-major A layout, in slices of at most 256 k-bytes
//             into a ring (bulk copies)
//   rows      places the planes of a row tile into one of two B buffers, 16 bytes at a time
//   products  one thread issues PLANES x K/32 MMAs per item into one of two accumulator buffers
//   epilogue  sixteen warps: tensor-memory quarter x four groups of rows
// so that copies, products and the epilogue of different items run at the same time.  Every mbarrier wait is bounded; one
// that gives up ends all further waiting of its warp, sets the status word, and the CTA still frees its tensor memory.
//
// Bound: the stores of the results and the issue of the epilogue.  I = 256, C = 2048, 4.1 M rows (33.5 GB of 32-bit results) 15.0 -> 7.2 ms;
// I = 512, C = 768, 12,800 rows on half of the SMs 81 -> 44 us; I = 80, C = 512, 25,600 rows 25 -> 20 us, I = 40 30 -> 26 us with checkpoints; 1000 rows, C = 2048
// 79 -> 16 us, where eight CTAs had been at work.  The form before it fetched every weight tile through registers between two barriers of
// all warps; two warps that placed the planes 16 bytes at a time took 3 us a row tile, which shares of a row tile made the bound.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "dependent_launch.cuh"
#include "tensor_map.cuh"
#include "umma_device.cuh"

namespace rxmet {
namespace planeproj {

using namespace umma;

constexpr int kChannelTile = 128;
constexpr int kEpilogueWarps = 16, kProductWarp = 16, kRowWarp = 17, kWeightWarp = 18;
constexpr int kThreads = 32 * (kWeightWarp + 1);
constexpr int kSlice = 256;   // k-bytes of a slice of a weight tile

// kind::i8 with a signed A (weights) and an unsigned B (byte planes): 32-bit integer accumulator (bits [4,6)
// = 2), A format signed 8-bit (bits [7,10) = 1), B format unsigned 8-bit (bits [10,13) = 0), both K-major,
// N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t instructionDescriptor(int n) {
    return (2u << 4) | (1u << 7) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
}

__device__ __forceinline__ void mmaI8(uint32_t tmemD, uint64_t descA, uint64_t descB, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, {%5, %5, %5, %5}, p;\n\t"
        "}\n"
        :
        : "r"(tmemD), "l"(descA), "l"(descB), "r"(idesc), "r"(accumulate), "r"(0u)
        : "memory");
}

struct Problem {
    const uint32_t *planes = nullptr;   // [rows][PLANES][kWords] words of four unsigned bytes, kWords a multiple of 4
    int rows = 0, kWords = 0;
    const uint4 *tiles = nullptr;       // packed weight tiles (tilePlace), 128 * kPad bytes each
    int C = 0;                          // channels beyond C in the last tile are computed and dropped
    int ring = 0, shares = 0;           // slices of weight tiles in shared memory, shares of a row tile's channel tiles (launch())
    int *status = nullptr;              // device word, set to 1 when a bounded wait of the kernel gave up
    bool early = false;                 // a dependent kernel starts beside this one (launch())
};

__host__ __device__ inline int paddedK(int kWords) { return (kWords * 4 + 31) / 32 * 32; }
__host__ __device__ inline int paddedC(int C) { return (C + kChannelTile - 1) / kChannelTile * kChannelTile; }
// Where the 16 bytes from k-group kg of channel c lie among the packed tiles, in units of 16 bytes: tiles of 128 channels, slices of kSlice
// k-bytes, eight channels, k-groups, channels.
__host__ __device__ inline size_t tilePlace(int c, int kg, int kPad) {
    const int slice = kg / (kSlice / 16), groups = min(kPad / 16 - slice * (kSlice / 16), kSlice / 16);
    return static_cast<size_t>(c / kChannelTile) * (kChannelTile * (kPad / 16)) + slice * (kChannelTile * (kSlice / 16)) +
           (c % kChannelTile / 8) * (groups * 8) + kg % (kSlice / 16) * 8 + c % 8;
}
// Rows of a tile, and slices of weight tiles that fit beside the planes of two row tiles.
__host__ __device__ constexpr int rowsPerTile(int kPad) { return kPad <= 256 ? 128 : 64; }
inline int ringSlices(int kPad, int planes) {
    const int sliceBytes = kChannelTile * (kPad < kSlice ? kPad : kSlice), rows = 2 * planes * rowsPerTile(kPad) * kPad;
    return std::min(4, (225 * 1024 - rows) / sliceBytes);
}
// Whether the operands fit one SM.
inline bool fits(int kPad, int planes) { return kPad <= 512 && ringSlices(kPad, planes) >= 2 && encodeTiled() != nullptr; }
inline size_t sharedBytes(int kPad, int planes) {
    return static_cast<size_t>(ringSlices(kPad, planes)) * kChannelTile * std::min(kPad, kSlice) + 2 * static_cast<size_t>(planes) * rowsPerTile(kPad) * kPad;
}

// Epilogue functor contract:
//   struct Loaded; __device__ Loaded load(int c) const;    what a channel reads from memory, asked for one item ahead
//   struct Channel;                                        per-channel constants; Channel::small, uniform in the warp: storeRows takes it
//   __device__ Channel channel(const Loaded &, int c) const;
//   __device__ void store(const Channel &, size_t row, int c, const int32_t (&acc)[PLANES]) const;
//   __device__ void storeRows<N>(const Channel &, size_t row, int c, const uint32_t (&acc)[PLANES][N], int count) const;
//                                                          the first `count` of N rows from `row` on
// f(j) for the first `count` of N rows; whole groups without a test per row.
template <int N, class F>
__device__ __forceinline__ void eachRow(int count, F f) {
    if (count >= N) {
#pragma unroll
        for (int j = 0; j < N; ++j) f(j);
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j)
            if (j < count) f(j);
    }
}
// One column of an array, walked row by row.  The pointer is hidden from the compiler after every step: unrolled, it computes a 64-bit
// product per row instead of an addition, and keeps sixteen of them.
template <class T>
struct Column {
    T *at;
    uint32_t rowBytes;
    __device__ __forceinline__ Column(T *array, size_t row, uint32_t c, uint32_t C) : at(array + row * C + c), rowBytes(C * sizeof(T)) {}
    __device__ __forceinline__ void put(T value) {
        *at = value;
        at = reinterpret_cast<T *>(reinterpret_cast<char *>(at) + rowBytes);
        asm volatile("" : "+l"(at));
    }
};

template <class Epilogue, int PLANES, int NR>
__global__ void __launch_bounds__(kThreads, 1) planeProjUmma(const __grid_constant__ Problem p, const __grid_constant__ Epilogue epi, const __grid_constant__ CUtensorMap rowsMap) {
    constexpr uint32_t kBufCols = PLANES * NR;
    constexpr uint32_t kTmemCols = 2 * kBufCols;   // a power of two for the sizes instantiated (128 .. 512)
    constexpr uint32_t kIdesc = instructionDescriptor(NR);
    constexpr int kMaxSlices = 4;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t weightFull[kMaxSlices], weightFree[kMaxSlices], rowsFull[2], rowsFree[2], accFull[2], accFree[2];
    __shared__ uint32_t tmemSlot;
    __shared__ int failed;

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    const int C = p.C, kWords = p.kWords, kPad = paddedK(kWords), ring = p.ring;
    const uint32_t sliceBytes = static_cast<uint32_t>(kChannelTile) * min(kPad, kSlice);
    const uint32_t planeBytes = static_cast<uint32_t>(NR) * kPad;
    constexpr uint32_t kGroupBytes = NR * 16;   // rows: next 16 bytes along K
    uint8_t *weights = smem;                      // [ring][16 channel groups][slice / 16][8][16]
    uint8_t *rowPlanes = smem + ring * sliceBytes;   // [2][PLANES][kPad / 16][NR][16]

    if (tid == 0) {
        failed = 0;
        auto init = [](uint64_t *bar, uint32_t count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
        };
        for (int i = 0; i < kMaxSlices; ++i) { init(&weightFull[i], 1); init(&weightFree[i], 1); }
        for (int i = 0; i < 2; ++i) { init(&rowsFull[i], 1); init(&rowsFree[i], 1); init(&accFull[i], 1); init(&accFree[i], kEpilogueWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // the k padding of the planes is never written again
    for (uint32_t i = tid; i < 2 * PLANES * planeBytes / 16; i += kThreads) reinterpret_cast<uint4 *>(rowPlanes)[i] = make_uint4(0u, 0u, 0u, 0u);
    waitForPredecessor();   // what is above needs nothing from earlier kernels
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (p.early) letDependentsStart();   // every CTA that has come here has its tensor memory
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0);

    const int channelTiles = paddedC(C) / kChannelTile, slices = (kPad + kSlice - 1) / kSlice;
    const int shares = p.shares, units = (p.rows + NR - 1) / NR * shares;   // a unit: one share of the channel tiles of a row tile
    auto tilesFrom = [&](int share) { return share * channelTiles / shares; };

    bool alive = true;   // false once a wait of this warp gave up
    auto wait = [&](uint64_t *bar, uint32_t parity) {
        if (alive) alive = __all_sync(0xffffffffu, waitPhase(smemAddr(bar), parity));
    };
    auto arrive = [&](uint64_t *bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory"); };

    if (warp == kWeightWarp) {
        uint32_t n = 0;   // slices so far
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x)
            for (int ct = tilesFrom(unit % shares); ct < tilesFrom(unit % shares + 1); ++ct)
                for (int s = 0; s < slices; ++s, ++n) {
                    const uint32_t at = n % ring, round = n / ring;
                    if (round > 0) wait(&weightFree[at], (round - 1) & 1);
                    const uint32_t bytes = static_cast<uint32_t>(kChannelTile) * min(kPad - s * kSlice, kSlice);
                    if (electOne()) {
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(&weightFull[at])), "r"(bytes) : "memory");
                        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                         smemAddr(weights + at * sliceBytes)),
                                     "l"(p.tiles + (static_cast<size_t>(ct) * kChannelTile * kPad + static_cast<size_t>(s) * kChannelTile * kSlice) / 16),
                                     "r"(bytes), "r"(smemAddr(&weightFull[at]))
                                     : "memory");
                    }
                    __syncwarp();
                }
        // nothing is left in flight, whatever the other warps gave up on
        for (uint32_t i = n > static_cast<uint32_t>(ring) ? n - ring : 0; i < n; ++i)
            if (!waitPhase(smemAddr(&weightFull[i % ring]), (i / ring) & 1)) alive = false;
    } else if (warp == kRowWarp) {
        const int kGroups = kWords / 4;
        uint32_t n = 0;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++n) {
            const uint32_t buf = n & 1, bar = smemAddr(&rowsFull[buf]);
            if (n > 1) wait(&rowsFree[buf], ((n >> 1) - 1) & 1);
            if (lane == 0) asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(PLANES * kGroups * kGroupBytes) : "memory");
            __syncwarp();
            for (int i = lane; i < PLANES * kGroups; i += 32) {
                const int pl = i / kGroups, kg = i - pl * kGroups;
                copyBox(smemAddr(rowPlanes + (buf * PLANES + pl) * planeBytes + kg * kGroupBytes), &rowsMap, 4 * i, unit / shares * NR, bar);
            }
        }
        // nothing is left in flight, whatever the other warps gave up on
        for (uint32_t i = n > 2 ? n - 2 : 0; i < n; ++i)
            if (!waitPhase(smemAddr(&rowsFull[i & 1]), (i >> 1) & 1)) alive = false;
    } else if (warp == kProductWarp) {
        uint32_t n = 0, item = 0, unitIndex = 0;
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x, ++unitIndex) {
            const uint32_t rowBuf = unitIndex & 1;
            wait(&rowsFull[rowBuf], (unitIndex >> 1) & 1);
            for (int ct = tilesFrom(unit % shares); ct < tilesFrom(unit % shares + 1); ++ct, ++item) {
                const uint32_t buf = item & 1;
                if (item > 1) wait(&accFree[buf], ((item >> 1) - 1) & 1);
                for (int s = 0; s < slices; ++s, ++n) {
                    const uint32_t at = n % ring;
                    wait(&weightFull[at], (n / ring) & 1);
                    if (electOne()) {
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const int sliceK = min(kPad - s * kSlice, kSlice);
                        const uint64_t descA = operandDescriptor(smemAddr(weights + at * sliceBytes), kCore, static_cast<uint32_t>(sliceK / 16) * kCore);
                        constexpr uint64_t kStep = (2 * kCore) >> 4;   // the start-address field counts 16-byte units
#pragma unroll
                        for (int pl = 0; pl < PLANES; ++pl) {
                            const uint64_t descB = operandDescriptor(smemAddr(rowPlanes + (rowBuf * PLANES + pl) * planeBytes + s * (kSlice / 16) * kGroupBytes), kGroupBytes, kCore);
                            for (int ks = 0; ks < sliceK / 32; ++ks)
                                mmaI8(tmem + buf * kBufCols + pl * NR, descA + ks * kStep, descB + ks * ((2 * kGroupBytes) >> 4), kIdesc, s + ks > 0 ? 1u : 0u);
                        }
                        commitTo(smemAddr(&weightFree[at]));
                        if (s + 1 == slices) {
                            commitTo(smemAddr(&accFull[buf]));
                            if (ct + 1 == tilesFrom(unit % shares + 1)) commitTo(smemAddr(&rowsFree[rowBuf]));
                        }
                    }
                    __syncwarp();
                }
            }
        }
    } else {
        const int q = warp & 3, group = warp >> 2;   // tensor-memory lane quarter (32 channels) of this warp, row-chunk group
        uint32_t item = 0;
        auto channelOf = [&](int ct) { return min(ct * kChannelTile + 32 * q + lane, C - 1); };
        typename Epilogue::Loaded loaded = epi.load(channelOf(tilesFrom(blockIdx.x % shares)));
        for (int unit = blockIdx.x; unit < units; unit += gridDim.x) {
            const int tilesEnd = tilesFrom(unit % shares + 1);
            for (int ct = tilesFrom(unit % shares); ct < tilesEnd; ++ct, ++item) {
                const uint32_t buf = item & 1;
                const int c = ct * kChannelTile + 32 * q + lane;
                const bool real = c < C;
                const typename Epilogue::Channel ch = epi.channel(loaded, min(c, C - 1));
                loaded = epi.load(channelOf(ct + 1 < tilesEnd ? ct + 1 : tilesFrom((unit + gridDim.x) % shares)));
                wait(&accFull[buf], (item >> 1) & 1);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int chunk = group; chunk < NR / 16; chunk += kEpilogueWarps / 4) {
                    uint32_t acc[PLANES][16];
#pragma unroll
                    for (int pl = 0; pl < PLANES; ++pl) {
                        asm volatile(
                            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                            "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                            : "=r"(acc[pl][0]), "=r"(acc[pl][1]), "=r"(acc[pl][2]), "=r"(acc[pl][3]), "=r"(acc[pl][4]), "=r"(acc[pl][5]),
                              "=r"(acc[pl][6]), "=r"(acc[pl][7]), "=r"(acc[pl][8]), "=r"(acc[pl][9]), "=r"(acc[pl][10]), "=r"(acc[pl][11]),
                              "=r"(acc[pl][12]), "=r"(acc[pl][13]), "=r"(acc[pl][14]), "=r"(acc[pl][15])
                            : "r"(tmem + (static_cast<uint32_t>(32 * q) << 16) + static_cast<uint32_t>(buf * kBufCols + pl * NR + 16 * chunk)));
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (chunk + kEpilogueWarps / 4 >= NR / 16) {   // the products of the item after next may overwrite this buffer
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) arrive(&accFree[buf]);
                    }
                    const int row0 = unit / shares * NR + 16 * chunk;
                    if (ch.small) {
                        epi.template storeRows<16>(ch, static_cast<size_t>(row0), c, acc, real ? p.rows - row0 : 0);
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        if (row0 + j >= p.rows) break;
                        int32_t a[PLANES];
#pragma unroll
                        for (int pl = 0; pl < PLANES; ++pl) a[pl] = static_cast<int32_t>(acc[pl][j]);
                        if (real) epi.store(ch, static_cast<size_t>(row0 + j), c, a);
                    }
                }
            }
        }
    }
    if (!alive && lane == 0) atomicExch(&failed, 1);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    if (tid == 0 && failed && p.status) atomicExch(p.status, 1);
}

// Launches the projection on at most `sms` SMs.  `dependents`: SMs that the recurrence behind it needs (unitrec::smsFor), which starts with the first CTAs of the
// projection where both find SMs of their own, and prepares itself beside them, else when the last of them has gone (16-bit GRU inference, 1 row: T = 1, H = 128
// 27 -> 21 us, T = 40, H = 100 45 -> 41 us; before it had to wait for the projection's end to be launched at all).
template <int PLANES, class Epilogue>
void launch(const char *name, Problem p, const Epilogue &epi, int sms, int dependents, cudaStream_t st) {
    const int kPad = paddedK(p.kWords), rows = rowsPerTile(kPad), rowTiles = (p.rows + rows - 1) / rows, channelTiles = paddedC(p.C) / kChannelTile;
    p.ring = ringSlices(kPad, PLANES);
    // Shares of a row tile that leave the SMs least to wait for: 200 row tiles of 25,600 rows are two rounds of 148 CTAs, 400 halves are three
    // of half the length.  A share reads the planes of its rows again, so fewer where it makes no difference.
    p.shares = 1;
    double least = 1e30;
    for (int shares = 1; shares <= channelTiles; ++shares) {
        const double time = static_cast<double>((static_cast<long long>(rowTiles) * shares + sms - 1) / sms) * ((channelTiles + shares - 1) / shares + 0.25);
        if (time < least * 0.99) { least = time; p.shares = shares; }
    }
    const size_t smem = sharedBytes(kPad, PLANES);
    const int grid = std::max(1, std::min(rowTiles * p.shares, sms));
    p.early = grid + dependents <= sms;
    const CUtensorMap map = boxMap(p.planes, p.rows, PLANES * p.kWords, CU_TENSOR_MAP_SWIZZLE_NONE, 4, rows);
    auto run = [&](auto kernel) {
        ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
        {
            KernelTimer timer__(name, st);
            launchDependent(kernel, grid, kThreads, smem, st, p, epi, map);
        }
        afterLaunch(name);
    };
    if (rows == 128) run(planeProjUmma<Epilogue, PLANES, 128>);
    else run(planeProjUmma<Epilogue, PLANES, 64>);
}

}  // namespace planeproj
}  // namespace rxmet
