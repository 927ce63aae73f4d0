// Weight gradients on tcgen05.mma, the gradients as A operand in tensor memory.
//
//   partial[s][m][n] = sum over the rows k of split s of code[k][m] * B[k][n]      (m < M)
//   partial[s][M][n] = sum over the same rows of B[k][n]                            (bias gradient)
//
// Codes are small integers (activation codes minus their zero point), exact in bf16 as one term, or as 256 floor(a / 256) and a mod 256 on
// grids of more than 8 bits.  B (fp32 gradients) is split into three bf16 terms that together carry all 24 bits, so that every product is exact
// and only the accumulation rounds.
//
// The product is computed transposed: a lane of tensor memory is a gate channel n, an accumulator column an element m.  A CTA owns 128
// channels, up to 256 elements of one of the two problems of a layer, and a range of rows.  A chunk of 32 rows is two MMA k-steps.  Warps by role:
//   copies      fetches the raw rows of a chunk as TMA boxes of 32 rows x 128 bytes into a ring
//   gradients   sixteen warps, two groups that take chunks in turn: thread = channel and sixteen rows; reads its column (neighbouring lanes,
//               neighbouring words), adds it to the bias gradient, stores the three terms to its own tensor-memory lane
//   codes       eight warps: raw codes -> bf16 in the canonical MN-major B layout in shared memory, 8 x 16-byte rows of a core matrix at a time
//   products    one thread issues the MMAs of a chunk (k-steps, code terms, gradient terms, in this order)
// Accumulators leave without a turn: neighbouring lanes are neighbouring channels of a row of `partial`.
//
// The tensor core truncates each addition to an accumulator.  Up to 128 elements the first terms, which carry the sum's size, have accumulators
// of their own, one for each k-step of a chunk, that are added to the others' at the end: a sixth of the additions that truncate at that size.
//
// Bound: codes of one term hand-overs and reading (102,400 more rows of 40 + 128 elements and 384 channels 92 us = 4.2 TB/s; DRAM 47 %, issue 48 %, tensor pipe
// 18 %), of two terms the tensor pipe (77 %; 51,200 more rows, 256 + 256 elements, 1024 channels 209 us = 1.54 PFLOP/s).  With both operands in shared
// memory (the form before) the MMAs alone took 3/4 of its bandwidth beside the copies and the conversion.  256,000 rows, 256 + 512 elements,
// 2048 channels, two terms 4.25 -> 3.13 ms; 12,800 rows, 512 + 256, 768 channels 94 -> 61 us; 25,600 rows, 40 + 128, one term, 512 channels 41.7 -> 39.4 us.  384
// channels by itself 28.5 (another kernel, of 192 channels a CTA) -> 30.5 us, in a step from the end of the input gradient on 28.4 -> 27.1, because it prepares
// itself under that one's tail: one kernel for all widths, with a sixth of the other's error.
// A last tile of 64 channels (192, 576) is half empty; passes of 25,600 rows, I 40, against that form all the same: 64 units 162 -> 157 us (16-bit codes 201 -> 186),
// 192 units 422 -> 372 (485 -> 413).
// Error against 64 bits, 2-norm, normal gradients: 25,600 rows, one term 1.0e-6 -> 1.7e-7 (512 channels), 1.9e-6 -> 1.5e-7 (384); 12,800 rows, two terms 8.0e-6, as before.
//
// Every mbarrier wait is bounded; one that gives up ends all further waiting of the CTA and sets the status word (the reduction that follows turns
// its outputs into NaN); copies and products in flight are awaited and tensor memory is freed all the same.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "backward_cluster_device.cuh"
#include "common.h"
#include "dependent_launch.cuh"
#include "tensor_map.cuh"
#include "umma_device.cuh"
#include "weight_grad_mma.h"

namespace rxmet {
namespace wgrad {
namespace {

using namespace umma;

constexpr int kRows = kBoxRows;                       // of a chunk
constexpr int kGradientWarps = 16, kCodeWarps = 8, kConvWarps = kGradientWarps + kCodeWarps;
constexpr int kCopyWarp = kConvWarps, kProductWarp = kConvWarps + 1, kThreads = 32 * (kProductWarp + 1);
constexpr int kMaxElements = 256, kMaxBoxes = kMaxElements / kBoxCols;   // of a CTA
constexpr int kMaxRing = 4, kMaxStages = 4;
constexpr uint32_t kStageCols = 3 * kRows / 2;        // tensor-memory columns of a chunk: three terms, two rows a column
constexpr uint32_t kTmemCols = 512;
constexpr int kMaxTiles = 16;                          // element tiles of both problems

// An element tile of a problem, all splits and channel tiles of it.
struct Tile {
    int problem, m0, elements;      // elements: of this tile
    int NP, boxes;                  // elements padded to 16, boxes of 32
    int accs, stages, ring;
    int firstBlock, splits, chunks;   // chunks of a split
};
struct Pair {
    Problem of[2];
    CUtensorMap gradients[2], codes[2], first[2];
    Tile tile[kMaxTiles];
    int tiles, channelTiles, N;
    int firstChunks[2], totalChunks[2];   // chunks that Problem::aFirst gives the codes of; all chunks
};

// Codes of one term: two groups of warps take chunks in turn, which hides their hand-overs (T = 100, B = 256, H = 128, four gates 42.4 -> 38.9 us); of two
// terms: all take every chunk (a layer of 512 inputs, 256 units, 12,800 rows 62 -> 59 us).
template <int TERMS>   // of a code
__global__ void __launch_bounds__(kThreads, 1) weightGradUmma(const __grid_constant__ Pair set) {
    constexpr int kCodeGroups = TERMS == 1 ? 2 : 1, kChunkWarps = kGradientWarps / 2 + kCodeWarps / kCodeGroups;   // of a chunk
    extern __shared__ __align__(1024) uint8_t smemRaw[];
    __shared__ __align__(8) uint64_t rawFull[2 * kMaxRing], rawFree[kMaxRing], termsFull[kMaxStages], termsFree[kMaxStages], accFull;
    __shared__ uint32_t tmemSlot;
    __shared__ volatile int failed;
    __shared__ float biasParts[4][kTileM];

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    int t = 0;
    while (t + 1 < set.tiles && static_cast<int>(blockIdx.x) >= set.tile[t + 1].firstBlock) ++t;
    const Tile &tile = set.tile[t];
    const Problem &p = set.of[tile.problem];
    const int local = static_cast<int>(blockIdx.x) - tile.firstBlock, split = local / set.channelTiles, n0 = (local - split * set.channelTiles) * kTileM, N = set.N;
    const int chunkBegin = split * tile.chunks, chunks = min(tile.chunks, set.totalChunks[tile.problem] - chunkBegin);
    const int NP = tile.NP, boxes = tile.boxes, gradientBoxes = min(kTileM / kBoxCols, (N - n0 + kBoxCols - 1) / kBoxCols);
    const uint32_t slotBytes = static_cast<uint32_t>(kTileM / kBoxCols + boxes) * kBoxBytes;
    const uint32_t kStride = static_cast<uint32_t>(boxes) * (kBoxCols / 8) * kCore;   // codes: next eight rows
    const uint32_t termBytes = (kRows / 8) * kStride, stageBytes = TERMS * termBytes;
    uint8_t *raw = smemRaw + ((1024u - (smemAddr(smemRaw) & 1023u)) & 1023u);   // swizzled boxes start on 1024 bytes
    uint8_t *stages = raw + tile.ring * slotBytes;

    if (tid == 0) {
        failed = 0;
        auto init = [](uint64_t *bar, uint32_t count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
        };
        for (int i = 0; i < 2 * kMaxRing; ++i) init(&rawFull[i], 1);
        for (int i = 0; i < kMaxRing; ++i) init(&rawFree[i], kChunkWarps);
        for (int i = 0; i < kMaxStages; ++i) { init(&termsFull[i], kChunkWarps); init(&termsFree[i], 1); }
        init(&accFull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    waitForPredecessor();   // what is above needs nothing from earlier kernels
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0), stageBase = tmem + tile.accs * NP;

    auto wait = [&](uint64_t *bar, uint32_t parity) {   // one that gives up ends all further waiting of the CTA
        if (testPhase(smemAddr(bar), parity)) return;
        if (!failed && !waitSuspended(smemAddr(bar), parity)) failed = 1;
    };
    auto arrive = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory");
    };
    // Rows of a chunk: those of Problem::aFirst come first, in chunks of their own, then the others.
    const int firstChunks = set.firstChunks[tile.problem];
    auto rowOf = [&](int chunk) { return chunk < firstChunks ? chunk * kRows : p.firstRows + (chunk - firstChunks) * kRows; };
    // ... of which the first this many are the chunk's own; rows beyond the last one are read as zeros
    auto validOf = [&](int chunk) { return chunk < firstChunks ? min(kRows, p.firstRows - chunk * kRows) : kRows; };

    if (warp < kGradientWarps) {
        const int quarter = warp & 3, half = (warp >> 2) & 1, group = warp >> 3;
        const uint32_t lanes = static_cast<uint32_t>(32 * quarter) << 16;
        const bool real = quarter < gradientBoxes;   // lanes of absent channels keep what they held
        RingTurn slot(tile.ring, group);
        Turn stage;
        stage.step(tile.stages, group);
        float bias = 0.0f;
        for (int c = group; c < chunks; c += 2, slot.step(2), stage.step(tile.stages, 2)) {
            const int valid = validOf(chunkBegin + c) - 16 * half, place = slot.place();
            wait(&rawFull[slot.full.at], slot.full.parity);
            const float *column = reinterpret_cast<const float *>(raw + place * slotBytes + quarter * kBoxBytes) + 16 * half * kBoxCols + lane;
            float v[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) v[i] = column[i * kBoxCols];
            if (valid < 16) {
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = i < valid ? v[i] : 0.0f;
            }
            arrive(&rawFree[place]);
            float sum[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) sum[i] = v[i] + v[i + 8];
#pragma unroll
            for (int n = 4; n > 0; n /= 2)
#pragma unroll
                for (int i = 0; i < n; ++i) sum[i] += sum[i + n];
            bias += sum[0];
            if (stage.again) wait(&termsFree[stage.at], stage.parity ^ 1u);
            __syncwarp();
            if (real) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t to = stageBase + lanes + stage.at * kStageCols + 8 * half;
#pragma unroll
                for (int term = 0; term < 3; ++term) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        w[i] = packBf16(v[2 * i], v[2 * i + 1]);
                        v[2 * i] -= bf16Lo(w[i]);
                        v[2 * i + 1] -= bf16Hi(w[i]);
                    }
                    bwdcluster::tmemStore8(to + term * (kRows / 2), w);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            arrive(&termsFull[stage.at]);
        }
        biasParts[2 * group + half][32 * quarter + lane] = bias;
        asm volatile("bar.sync 1, %0;" ::"n"(32 * kGradientWarps) : "memory");
        const int at = 32 * quarter + lane;
        if (warp < 4 && tile.m0 == 0 && n0 + at < N)
            p.partial[(static_cast<size_t>(split) * (p.M + 1) + p.M) * N + n0 + at] = (biasParts[0][at] + biasParts[1][at]) + (biasParts[2][at] + biasParts[3][at]);
    } else if (warp < kConvWarps) {
        // warp -> eight rows of every other chunk, or of every chunk and every other box; lane -> row and eight elements of a box
        const int second = (warp - kGradientWarps) >> 2, turn = kCodeGroups == 2 ? second : 0, firstBox = kCodeGroups == 2 ? 0 : second, group = warp & 3, row8 = lane & 7, eighth = lane >> 3, row = 8 * group + row8;
        // 1.5 * 2^23 rounds to integers, which sit in the low bits, 1.5 * 2^31 to multiples of 256
        constexpr float kMagic = 12582912.0f, kMagic256 = 3221225472.0f;
        const float inverse = p.aInvScale, offset = kMagic + (p.aCodes ? static_cast<float>(p.aZero) : p.aFloatZero);   // exact: below 2^24
        auto run = [&](auto integersTag) {
            constexpr bool kIntegers = decltype(integersTag)::value;
            RingTurn slot(tile.ring, turn);
            Turn stage;
            stage.step(tile.stages, turn);
            for (int c = turn; c < chunks; c += kCodeGroups, slot.step(kCodeGroups), stage.step(tile.stages, kCodeGroups)) {
                const bool mine = row < validOf(chunkBegin + c);
                const int place = slot.place();
                wait(&rawFull[slot.full.at], slot.full.parity);
                if (stage.again) wait(&termsFree[stage.at], stage.parity ^ 1u);
                const uint8_t *from = raw + place * slotBytes + kTileM / kBoxCols * kBoxBytes + row * 128;
                uint8_t *to = stages + stage.at * stageBytes + group * kStride + eighth * kCore + row8 * 16;
#pragma unroll 2
                for (int box = firstBox; box < boxes; box += 3 - kCodeGroups) {
                    const uint4 a = *reinterpret_cast<const uint4 *>(from + box * kBoxBytes + (((2 * eighth) ^ row8) << 4));
                    const uint4 b = *reinterpret_cast<const uint4 *>(from + box * kBoxBytes + (((2 * eighth + 1) ^ row8) << 4));
                    const uint32_t q[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
                    float x[8];
                    // boxes beyond the last element decode to some finite value that only reaches accumulator columns nobody reads
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        x[i] = __fadd_rn(kIntegers ? __uint_as_float(0x4b400000u + q[i]) : __fmaf_rn(__uint_as_float(q[i]), inverse, kMagic), -offset);
                    uint32_t word[4];
                    uint8_t *at = to + box * (kBoxCols / 8) * kCore;
                    if (TERMS == 2) {   // 256 floor(x / 256): x - 127.5 is no tie
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float u = __fadd_rn(__fadd_rn(x[2 * i] - 127.5f, kMagic256), -kMagic256), v = __fadd_rn(__fadd_rn(x[2 * i + 1] - 127.5f, kMagic256), -kMagic256);
                            word[i] = mine ? packBf16(u, v) : 0u;
                            x[2 * i] -= u;
                            x[2 * i + 1] -= v;
                        }
                        *reinterpret_cast<uint4 *>(at) = make_uint4(word[0], word[1], word[2], word[3]);
                        at += termBytes;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i) word[i] = mine ? packBf16(x[2 * i], x[2 * i + 1]) : 0u;
                    *reinterpret_cast<uint4 *>(at) = make_uint4(word[0], word[1], word[2], word[3]);
                }
                arrive(&rawFree[place]);
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                arrive(&termsFull[stage.at]);
            }
        };
        if (p.aCodes) run(std::true_type{});
        else run(std::false_type{});
    } else if (warp == kCopyWarp) {
        // a box per lane: a lone lane takes 90 cycles a box, longer than 128 elements take to multiply
        const CUtensorMap *gradients = &set.gradients[tile.problem], *codes = &set.codes[tile.problem], *first = &set.first[tile.problem];
        fillRing(chunks, tile.ring, rawFull, rawFree, failed, wait, [&](int c, int place, uint64_t *full) {
            const int chunk = chunkBegin + c, row = rowOf(chunk);
            const uint32_t bar = smemAddr(full), to = smemAddr(raw + place * slotBytes);
            if (lane == 0)
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"((gradientBoxes + boxes) * kBoxBytes) : "memory");
            __syncwarp();
            if (lane < gradientBoxes) {
                copyBox(to + lane * kBoxBytes, gradients, n0 + lane * kBoxCols, row, bar);
            } else if (lane >= kTileM / kBoxCols && lane < kTileM / kBoxCols + boxes) {
                const int b = lane - kTileM / kBoxCols;
                copyBox(to + lane * kBoxBytes, chunk < firstChunks ? first : codes, tile.m0 + b * kBoxCols, chunk < firstChunks ? row : row - p.firstRows, bar);
            }
        });
    } else if (electOne()) {
        // A: K-major in tensor memory, B: MN-major in shared memory
        const uint32_t idesc = instructionDescriptor(NP, true), others = tmem + (tile.accs - 1) * NP;
        const uint64_t descB0 = operandDescriptor(smemAddr(stages), kStride, kCore);
        const bool parted = tile.accs == 3;
        Turn stage;
        for (int c = 0; c < chunks; ++c, stage.step(tile.stages)) {
            wait(&termsFull[stage.at], stage.parity);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t terms = stageBase + stage.at * kStageCols;
            const uint64_t descB = descB0 + static_cast<uint64_t>((stage.at * stageBytes) >> 4);
#pragma unroll
            for (int ks = 0; ks < kRows / 16; ++ks)
#pragma unroll
                for (int a = 0; a < TERMS; ++a)
#pragma unroll
                    for (int term = 0; term < 3; ++term)
                        bwdcluster::mmaBf16TmemA(term > 0 ? others : parted ? tmem + ks * NP : tmem, terms + term * (kRows / 2) + 8 * ks,
                                                 descB + static_cast<uint64_t>((a * termBytes + 2 * ks * kStride) >> 4), idesc,
                                                 (c > 0 || a > 0 || (parted ? term > 1 || (term == 1 && ks > 0) : ks > 0 || term > 0)) ? 1u : 0u);
            commitTo(smemAddr(&termsFree[stage.at]));
            if (c + 1 == chunks) commitTo(smemAddr(&accFull));
        }
        letDependentsStart();   // the reduction is launched under the last products and the epilogue
    }
    __syncwarp();

    // accumulators -> partial: lane = channel
    if (chunks > 0) {
        if (warp == kProductWarp && lane == 0) waitPhase(smemAddr(&accFull), 0);   // nothing is left in flight, whatever was given up
        if (warp < kGradientWarps) {
            wait(&accFull, 0);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int quarter = warp & 3, n = n0 + 32 * quarter + lane;
            float *out = p.partial + (static_cast<size_t>(split) * (p.M + 1) + tile.m0) * N + n;
            const uint32_t from = tmem + (static_cast<uint32_t>(32 * quarter) << 16);
            for (int m = 16 * (warp >> 2); m < tile.elements; m += 16 * (kGradientWarps / 4)) {
                uint32_t r[3][16];
#pragma unroll
                for (int acc = 0; acc < 3; ++acc) {
                    if (acc > 0 && tile.accs == 1) break;
                    bwdcluster::tmemLoad<8>(from + acc * NP + m, *reinterpret_cast<uint32_t (*)[8]>(r[acc]));
                    bwdcluster::tmemLoad<8>(from + acc * NP + m + 8, *reinterpret_cast<uint32_t (*)[8]>(r[acc] + 8));
                }
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    float v = __uint_as_float(r[0][i]);
                    if (tile.accs == 3) v = (v + __uint_as_float(r[1][i])) + __uint_as_float(r[2][i]);
                    if (m + i < tile.elements && n < N) out[static_cast<size_t>(m + i) * N] = v;
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
    if (tid == 0 && failed && p.status) atomicExch(p.status, 1);
}

int elementTiles(int M) { return (M + kMaxElements - 1) / kMaxElements; }
int channelTiles(int N) { return (N + kTileM - 1) / kTileM; }
int paddedTile(int M) { return ((M + elementTiles(M) - 1) / elementTiles(M) + 15) / 16 * 16; }   // elements of a tile
int chunksOf(int K, int firstRows) { return (firstRows + kRows - 1) / kRows + (K - firstRows + kRows - 1) / kRows; }

size_t slotBytes(const Tile &t) { return static_cast<size_t>(kTileM / kBoxCols + t.boxes) * kBoxBytes; }
size_t stageBytes(const Tile &t, int terms) { return static_cast<size_t>(terms) * kRows * t.boxes * kBoxCols * 2; }

}  // namespace

bool tensorMemoryPath(int Ma, int Mb, int N) {
    static const bool disabled = std::getenv("RXMET_WGRAD_MMA_SYNC") != nullptr;
    return !disabled && Ma >= 4 && Mb >= 4 && Ma % 4 == 0 && Mb % 4 == 0 && (N % 128 == 0 || N % 192 == 0) && elementTiles(Ma) + elementTiles(Mb) <= kMaxTiles &&
           encodeTiled() != nullptr;
}

int tileSplitBound(int M, int N) { return std::max(1, kMaxSms / (elementTiles(M) * channelTiles(N))); }

// A chunk costs a CTA what it has to read or, with two terms a code, its products; the SMs are shared out so that both problems end together.
PairPlan planPair(const Problem &a, const Problem &b, int K, int N, bool wide, int sms) {
    const Problem *of[2] = {&a, &b};
    int tiles[2], chunks[2];
    double cost[2];
    for (int i = 0; i < 2; ++i) {
        const int NP = paddedTile(of[i]->M);
        tiles[i] = elementTiles(of[i]->M) * channelTiles(N);
        chunks[i] = chunksOf(K, of[i]->firstRows);
        cost[i] = std::max((wide ? 6.0 : 3.0) * NP, 500.0 + 4.0 * NP);
    }
    sms = std::min(sms, kMaxSms);
    int best[2] = {1, 1};
    double least = 1e30;
    for (int s = 1; s == 1 || (s <= chunks[0] && s * tiles[0] + tiles[1] <= sms); ++s) {
        const int other = std::max(1, std::min(chunks[1], (sms - s * tiles[0]) / tiles[1]));
        const double time = std::max(cost[0] * ((chunks[0] + s - 1) / s), cost[1] * ((chunks[1] + other - 1) / other));
        if (time < least) { least = time; best[0] = s; best[1] = other; }
    }
    PairPlan plan;
    for (int i = 0; i < 2; ++i) {
        const int each = (chunks[i] + best[i] - 1) / best[i];
        plan.chunks[i] = each;
        plan.splits[i] = (chunks[i] + each - 1) / each;
    }
    return plan;
}

PairPlan chainPlan(int K) {
    PairPlan plan;
    for (int i = 0; i < 2; ++i) {
        plan.chunks[i] = kChainRows / kRows;
        plan.splits[i] = chainChunks(K);
    }
    return plan;
}

PairPlan finePlan(const Problem &a, const Problem &b, int K, int N, int sms) {
    const Problem *of[2] = {&a, &b};
    const int room = std::min(tileSplitBound(a.M, N), tileSplitBound(b.M, N)), tiles = (elementTiles(a.M) + elementTiles(b.M)) * channelTiles(N);
    int chunks[2], least = 1;
    for (int i = 0; i < 2; ++i) {
        chunks[i] = chunksOf(K, of[i]->firstRows);
        least = std::max(least, (chunks[i] * kRows + kChainRows - 1) / kChainRows);
    }
    PairPlan plan{};
    if (least > room) return plan;
    const int waves = (least * tiles + sms - 1) / sms, splits = std::min(room, std::max(least, waves * sms / tiles));
    for (int i = 0; i < 2; ++i) {
        plan.chunks[i] = (chunks[i] + splits - 1) / splits;
        plan.splits[i] = (chunks[i] + plan.chunks[i] - 1) / plan.chunks[i];
    }
    return plan;
}

int planRows(const PairPlan &plan) { return std::max(plan.chunks[0], plan.chunks[1]) * kRows; }

void launchPair(const Problem &a, const Problem &b, int K, int N, const PairPlan &plan, bool wide, cudaStream_t st) {
    Pair set;
    set.of[0] = a;
    set.of[1] = b;
    set.tiles = 0;
    set.channelTiles = channelTiles(N);
    set.N = N;
    const int terms = wide ? 2 : 1;
    size_t smem = 0;
    int blocks = 0;
    RXMET_REQUIRE(elementTiles(a.M) + elementTiles(b.M) <= kMaxTiles, "weight gradient: %d and %d elements", a.M, b.M);
    for (int i : {a.M >= b.M ? 0 : 1, a.M >= b.M ? 1 : 0}) {   // the larger problem's CTAs first
        const Problem &p = set.of[i];
        RXMET_REQUIRE(alignedTo(p.B, 16) && alignedTo(p.aCodes, 16) && alignedTo(p.aFloat, 16) && alignedTo(p.aFirst, 16) && p.M % 4 == 0 && N % 4 == 0,
                      "weight gradient: misaligned operands");
        const void *codes = p.aCodes ? static_cast<const void *>(p.aCodes) : static_cast<const void *>(p.aFloat);
        set.gradients[i] = boxMap(p.B, K, N, CU_TENSOR_MAP_SWIZZLE_NONE);
        // a sequence of one step has no rows but the first ones
        set.codes[i] = boxMap(K > p.firstRows ? codes : p.aFirst, std::max(1, K > p.firstRows ? K - p.firstRows : p.firstRows), p.M, CU_TENSOR_MAP_SWIZZLE_128B);
        set.first[i] = p.firstRows > 0 ? boxMap(p.aFirst, p.firstRows, p.M, CU_TENSOR_MAP_SWIZZLE_128B) : set.codes[i];
        set.firstChunks[i] = (p.firstRows + kRows - 1) / kRows;
        set.totalChunks[i] = chunksOf(K, p.firstRows);
        const int each = paddedTile(p.M);
        for (int m0 = 0; m0 < p.M; m0 += each) {
            Tile &t = set.tile[set.tiles++];
            t.problem = i;
            t.m0 = m0;
            t.elements = std::min(each, p.M - m0);
            t.NP = each;
            t.boxes = (each + kBoxCols - 1) / kBoxCols;
            t.accs = each <= 128 ? 3 : 1;
            t.stages = std::min<int>(kMaxStages, (kTmemCols - t.accs * each) / kStageCols);
            t.ring = kMaxRing;
            const size_t most = 222 * 1024;
            while (t.stages > 2 && 2 * slotBytes(t) + t.stages * stageBytes(t, terms) > most) --t.stages;
            while (t.ring > 2 && t.ring * slotBytes(t) + t.stages * stageBytes(t, terms) > most) --t.ring;
            while (t.stages > 2 && t.ring == 2 && 3 * slotBytes(t) + (t.stages - 1) * stageBytes(t, terms) <= most) { --t.stages; t.ring = 3; }
            smem = std::max(smem, 1024 + t.ring * slotBytes(t) + t.stages * stageBytes(t, terms));
            t.firstBlock = blocks;
            t.splits = plan.splits[i];
            t.chunks = plan.chunks[i];
            blocks += t.splits * set.channelTiles;
        }
    }
    auto run = [&](auto kernel) {
        ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
        KernelTimer timer__("weightGradUmma", st);
        launchDependent(kernel, static_cast<unsigned>(blocks), kThreads, smem, st, set);
    };
    if (wide) run(weightGradUmma<2>);
    else run(weightGradUmma<1>);
}

namespace {

// blockIdx.y: which of the two.  Bound by memory, 16 bytes a load: the counts are multiples of four (N is).
__global__ void foldPartials(float4 *a, size_t countA, float4 *b, size_t countB, int partials, bool first) {
    float4 *sums = blockIdx.y == 0 ? a : b;
    const size_t count = blockIdx.y == 0 ? countA : countB;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < count; i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float4 s = sums[count + i];
#pragma unroll 4
        for (int p = 2; p <= partials; ++p) {
            const float4 v = sums[p * count + i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        if (!first) {
            const float4 v = sums[i];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        sums[i] = s;
    }
}

}  // namespace

void addPartials(float *a, size_t countA, float *b, size_t countB, int partials, bool first, cudaStream_t st) {
    const size_t most = std::max(countA, countB) / 4;
    {
        KernelTimer timer__("foldPartials", st);
        foldPartials<<<dim3(static_cast<unsigned>(std::min<size_t>((most + 255) / 256, 148 * 8)), 2), 256, 0, st>>>(
            reinterpret_cast<float4 *>(a), countA / 4, reinterpret_cast<float4 *>(b), countB / 4, partials, first);
    }
    afterLaunch("foldPartials");
}

}  // namespace wgrad

namespace {

__device__ __forceinline__ void initProbeBarrier(uint64_t &bar) { asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(umma::smemAddr(&bar)) : "memory"); }
__device__ __forceinline__ void arriveOnProbe(uint64_t *bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(umma::smemAddr(bar)) : "memory"); }

// One warp polls a barrier that nothing completes, with the poll loop of the tcgen05 kernels, then fills a ring whose places nothing frees, with
// the loop of their copy warps.  status: 1 where both gave up, the lanes of the second after the same chunk; 2 otherwise.
__global__ void boundedWaitProbe(int *status, unsigned int *polls) {
    constexpr int kRing = 2;
    __shared__ __align__(8) uint64_t bar, full[2 * kRing], freed[kRing];
    __shared__ volatile int failed;
    if (threadIdx.x == 0) {
        failed = 0;
        initProbeBarrier(bar);
        for (uint64_t &b : full) initProbeBarrier(b);
        for (uint64_t &b : freed) initProbeBarrier(b);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    uint32_t made = 0;
    const bool completed = umma::waitPhase(umma::smemAddr(&bar), 0, &made);
    const int issued = umma::fillRing(
        8, kRing, full, freed, failed,
        [&](uint64_t *b, uint32_t parity) {
            if (threadIdx.x == 5 && !umma::waitPhase(umma::smemAddr(b), parity)) failed = 1;   // one lane finds out
        },
        [&](int, int, uint64_t *b) {
            if (threadIdx.x == 0) arriveOnProbe(b);
        });
    const bool together = __all_sync(0xffffffffu, issued == kRing);
    if (threadIdx.x == 0) {
        *polls = made;
        atomicExch(status, !completed && failed && together ? 1 : 2);
    }
}

// Two warps that take the chunks of a ring of an odd number of places in turn, as the warps of the gradient kernels do; the first chunk lands
// long after those behind it.  status: 3 where a warp was let through to a chunk that had not been asked for, or a wait gave up.
__global__ void ringTurnProbe(int *status) {
    constexpr int kRing = 3, kChunks = 24;
    __shared__ __align__(8) uint64_t full[2 * kRing], freed[kRing];
    __shared__ volatile int failed, asked;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        failed = asked = 0;
        for (uint64_t &b : full) initProbeBarrier(b);
        for (uint64_t &b : freed) initProbeBarrier(b);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto wait = [&](uint64_t *b, uint32_t parity) {
        if (!failed && !umma::waitPhase(umma::smemAddr(b), parity)) failed = 1;
    };
    if (warp == 0) {
        umma::fillRing(kChunks, kRing, full, freed, failed, wait, [&](int i, int, uint64_t *b) {
            if (lane == 0) {
                asked = i + 1;
                if (i > 0) arriveOnProbe(b);
            }
            __syncwarp();
        });
    } else if (warp == 1) {   // the first chunk
        for (int i = 0; i < 1000; ++i) __nanosleep(100);
        if (lane == 0) arriveOnProbe(&full[0]);
    } else {
        umma::RingTurn turn(kRing, warp - 2);
        for (int c = warp - 2; c < kChunks && !__any_sync(0xffffffffu, failed); c += 2, turn.step(2)) {
            wait(&full[turn.full.at], turn.full.parity);
            if (c >= asked) failed = 1;   // let through too early
            if (__any_sync(0xffffffffu, failed)) break;
            if (lane == 0) arriveOnProbe(&freed[turn.place()]);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && failed) atomicExch(status, 3);
}

}  // namespace
}  // namespace rxmet

extern "C" int rxmet_selftest_bounded_wait(int *status_dev, unsigned int *polls_out, void *stream) {
    using namespace rxmet;
    return guarded([&] {
        RXMET_REQUIRE(status_dev != nullptr, "status_dev must not be null");
        cudaStream_t st = static_cast<cudaStream_t>(stream);
        unsigned int *pollsDev = reinterpret_cast<unsigned int *>(status_dev + 1);
        RXMET_CUDA(cudaMemsetAsync(status_dev, 0, 2 * sizeof(int), st));
        boundedWaitProbe<<<1, 32, 0, st>>>(status_dev, pollsDev);
        afterLaunch("boundedWaitProbe");
        ringTurnProbe<<<1, 128, 0, st>>>(status_dev);
        afterLaunch("ringTurnProbe");
        int status = 0;
        unsigned int polls = 0;
        RXMET_CUDA(cudaMemcpyAsync(&status, status_dev, sizeof(int), cudaMemcpyDeviceToHost, st));
        RXMET_CUDA(cudaMemcpyAsync(&polls, pollsDev, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
        RXMET_CUDA(cudaStreamSynchronize(st));
        if (polls_out) *polls_out = polls;
        if (status != 1) fail(RXMET_ERR_CUDA, "a bounded device-side wait did not give up as it should (%d)", status);
        fail(RXMET_ERR_DEVICE_TIMEOUT, "a bounded device-side wait ran out after %u polls", polls);
    });
}
