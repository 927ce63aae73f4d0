// dx = (G * kScale) code on tcgen05.mma, the gradients as A operand in tensor memory.
//
// A CTA walks a contiguous range of rows in tiles of 128 rows (= the lanes of tensor memory) and, with more than 256 columns, one slab
// of columns.  The accumulator D[128][NP] of a tile sums over K in chunks of 32 channels.  Warps by role:
//   gradients   copies a chunk's rows as TMA boxes of 32 rows x 128 bytes (128-byte swizzle), one a lane, into a ring
//   converters  sixteen warps, two groups that take chunks in turn: thread = row and sixteen channels; reads its pieces, scales them,
//               splits them into three bf16 terms that carry all 24 bits and stores these to its own tensor-memory lane
//   weights     up to 64 columns the codes, exact in bf16, are converted once per CTA and stay in shared memory; beyond, packWeights lays
//               them out before and one lane copies them chunk by chunk (bulk copies)
//   products    one thread issues the six MMAs of a chunk (2 k-steps x 3 terms, in this order) into one of two accumulators (one beyond 128 columns)
//   epilogue    eight warps: accumulator rows through shared memory, so that a store covers 128 bytes of a row, masked
// so that a tile leaves under the products of the next one.  Every mbarrier wait is bounded; one that gives up ends all further waiting of
// the CTA, turns the outputs that follow into NaN and sets the status word; copies and products in flight are awaited and
// tensor memory is freed all the same.
//
// Bound: the hand-overs and the conversion of a chunk (0.50 us a chunk and SM up to 128 columns; issue 39 %, DRAM 40 %, tensor pipe 11 %); beyond 128
// columns the products of a tile wait for the read-out of the one accumulator (256 columns: 30.7 us a tile of 32 chunks, 47.4 of 64, that is 0.52 a chunk, of
// which the MMAs take 0.41, and 14 for the read-out; tensor pipe 40 %).  The forms before it wrote the terms to shared memory, where the MMAs read them again: half of its bandwidth beside copies and conversion; they walked
// whole tiles (two rounds where a CTA has 173 rows) and left the epilogue outside.  In a step, with what surrounds the kernel: 25,600 rows x 384 -> 40
// columns 26.8 -> 23.7 us, 25,600 x 512 -> 40 31.7 -> 26.1, 12,800 x 768 -> 40 41.4 -> 24.7, 256,000 x 2048 -> 256 943 -> 664; by itself, back to back, 17, 21, 18 us
// and 12,800 x 768 -> 512 59 -> 40.
#include <algorithm>
#include <cstdlib>

#include "backward_cluster_device.cuh"
#include "common.h"
#include "dependent_launch.cuh"
#include "input_grad_umma.h"
#include "tensor_map.cuh"
#include "umma_device.cuh"

namespace rxmet {
namespace igrad {
namespace {

using namespace umma;

constexpr int kChunk = kBoxCols;                               // channels: two k-steps
constexpr int kConvWarps = 16, kEpilogueWarps = 8, kFillWarps = kConvWarps + kEpilogueWarps;
constexpr int kGradientWarp = kFillWarps, kWeightWarp = kFillWarps + 1, kProductWarp = kFillWarps + 2;
constexpr int kThreads = 32 * (kProductWarp + 1);
constexpr int kMaxRing = 6, kMaxStages = 8, kWeightRing = 4;
constexpr uint32_t kRawBytes = kTileM / kBoxRows * kBoxBytes;   // 16 KB
constexpr uint32_t kStageCols = 3 * kChunk / 2;               // tensor-memory columns of a chunk: three terms, two channels a column
constexpr uint32_t kGroupStride = kChunk / 8 * kCore;          // weights: next eight columns
constexpr uint32_t kTmemCols = 512;
constexpr int kResidentColumns = 64, kMaxColumns = 256;        // of a CTA
constexpr int kMaxK = 8192;

struct Shape {
    int NP, slabs;        // padded columns of a slab
    int accs, stages;     // accumulators and operand stages in tensor memory
    int ring;             // chunks of gradients in shared memory
    int rowsPerCta;       // a multiple of kBoxRows
};

// codes -> bf16: packed[slab][chunk][n / 8][k-group][n % 8][8 k]; one thread per 16-byte row.
struct WeightRow {
    float c[8];
    __device__ __forceinline__ void load(const Problem &p, int n, int k0) {
        if (n >= p.N) {
#pragma unroll
            for (int j = 0; j < 8; ++j) c[j] = 0.0f;
        } else if (p.codesNK) {   // K is a multiple of 32
            const int32_t *at = p.codesNK + static_cast<size_t>(n) * p.K + k0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                int4 q;
                if ((reinterpret_cast<uintptr_t>(at) & 15) == 0) q = __ldg(reinterpret_cast<const int4 *>(at) + h);
                else q = make_int4(__ldg(at + 4 * h), __ldg(at + 4 * h + 1), __ldg(at + 4 * h + 2), __ldg(at + 4 * h + 3));
                c[4 * h] = static_cast<float>(q.x); c[4 * h + 1] = static_cast<float>(q.y); c[4 * h + 2] = static_cast<float>(q.z); c[4 * h + 3] = static_cast<float>(q.w);
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; ++j) c[j] = __ldg(p.codesKN + static_cast<size_t>(k0 + j) * p.N + n);
        }
    }
    __device__ __forceinline__ uint4 packed() const {
        return make_uint4(packBf16(c[0], c[1]), packBf16(c[2], c[3]), packBf16(c[4], c[5]), packBf16(c[6], c[7]));
    }
};
__device__ __forceinline__ int rowPlace(int n, int k8, int NP) {   // in units of 16 bytes
    return (k8 / 4 * (NP / 8) + n / 8) * 32 + k8 % 4 * 8 + n % 8;
}
__global__ void packWeights(const Problem p, int NP, int slabs, uint4 *packed) {
    letDependentsStart();
    const int groups = p.K / 8, item = blockIdx.x * blockDim.x + threadIdx.x;
    if (item >= groups * NP * slabs) return;
    const int k8 = item % groups, n = item / groups, slab = n / NP;
    WeightRow row;
    row.load(p, n, 8 * k8);
    packed[static_cast<size_t>(slab) * groups * NP + rowPlace(n - slab * NP, k8, NP)] = row.packed();
}

template <bool STREAM>   // weights chunk by chunk
__global__ void __launch_bounds__(kThreads, 1)
inputGradUmma(const __grid_constant__ Problem p, const __grid_constant__ Shape s, const __grid_constant__ CUtensorMap gradients) {
    extern __shared__ __align__(1024) uint8_t smemRaw[];
    __shared__ __align__(8) uint64_t rawFull[2 * kMaxRing], rawFree[kMaxRing], termsFull[kMaxStages], termsFree[kMaxStages], weightsFull[kWeightRing],
        weightsFree[kWeightRing], accFull[2], accFree[2];
    __shared__ uint32_t tmemSlot;
    __shared__ volatile int failed;

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    const int K = p.K, NP = s.NP, chunks = K / kChunk, n0 = static_cast<int>(blockIdx.y) * NP, columns = min(p.N - n0, NP);
    const int rowBegin = min(p.rows, static_cast<int>(blockIdx.x) * s.rowsPerCta), rowEnd = min(p.rows, rowBegin + s.rowsPerCta);
    const int tiles = (rowEnd - rowBegin + kTileM - 1) / kTileM, total = tiles * chunks;
    const uint32_t weightBytes = static_cast<uint32_t>(NP) * kChunk * 2;   // of a chunk
    uint8_t *raw = smemRaw + ((1024u - (smemAddr(smemRaw) & 1023u)) & 1023u);   // swizzled boxes start on 1024 bytes
    uint8_t *turn = raw + s.ring * kRawBytes;                                    // [8 warps][32 rows][128 bytes]
    uint8_t *weights = turn + kEpilogueWarps * 4096;
    float *scale = reinterpret_cast<float *>(weights + (STREAM ? kWeightRing : chunks) * weightBytes);

    if (tid == 0) {
        failed = 0;
        auto init = [](uint64_t *bar, uint32_t count) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smemAddr(bar)), "r"(count) : "memory");
        };
        for (int i = 0; i < 2 * kMaxRing; ++i) init(&rawFull[i], 1);
        for (int i = 0; i < kMaxRing; ++i) init(&rawFree[i], kConvWarps / 2);
        for (int i = 0; i < kMaxStages; ++i) { init(&termsFull[i], kConvWarps / 2); init(&termsFree[i], 1); }
        for (int i = 0; i < kWeightRing; ++i) { init(&weightsFull[i], STREAM ? 1 : kFillWarps); init(&weightsFree[i], 1); }
        for (int i = 0; i < 2; ++i) { init(&accFull[i], 1); init(&accFree[i], kEpilogueWarps); }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "n"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    waitForPredecessor();   // what is above needs nothing from earlier kernels
    if (tid == 0 && blockIdx.x == 0 && blockIdx.y == 0 && p.clear) *p.clear = 0;
    for (int k = tid; k < K; k += kThreads) scale[k] = p.kScale ? __ldg(p.kScale + k) : 1.0f;
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = __shfl_sync(0xffffffffu, tmemSlot, 0), stageBase = tmem + s.accs * NP;

    auto wait = [&](uint64_t *bar, uint32_t parity) {   // one that gives up ends all further waiting of the CTA
        if (testPhase(smemAddr(bar), parity)) return;
        if (!failed && !waitSuspended(smemAddr(bar), parity)) failed = 1;
    };
    auto arrive = [&](uint64_t *bar) {
        __syncwarp();
        if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smemAddr(bar)) : "memory");
    };
    auto expect = [](uint64_t *bar, uint32_t bytes) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smemAddr(bar)), "r"(bytes) : "memory");
    };
    auto boxesOf = [&](int tile) { return min(kTileM / kBoxRows, (rowEnd - rowBegin - tile * kTileM + kBoxRows - 1) / kBoxRows); };
    if (!STREAM && warp < kFillWarps) {
        // consecutive threads walk whichever index of the codes is contiguous; three rows are asked for before the first is used
        constexpr int kAhead = 3, kFill = 32 * kFillWarps;
        const int inner = p.codesNK ? K / 8 : NP, items = NP * (K / 8);
        for (int first = tid; first < items; first += kAhead * kFill) {
            WeightRow rows[kAhead];
            int place[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) {
                const int item = min(first + i * kFill, items - 1), outer = item / inner, in = item - outer * inner;
                const int n = p.codesNK ? outer : in, k8 = p.codesNK ? in : outer;
                place[i] = rowPlace(n, k8, NP);
                rows[i].load(p, n, 8 * k8);
            }
#pragma unroll
            for (int i = 0; i < kAhead; ++i) reinterpret_cast<uint4 *>(weights)[place[i]] = rows[i].packed();
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        arrive(&weightsFull[0]);
    }

    if (warp < kConvWarps) {
        const int quarter = warp & 3, part = (warp >> 2) & 1, group = warp >> 3, sw = lane & 7;
        const uint32_t lanes = static_cast<uint32_t>(32 * quarter) << 16;
        RingTurn slot(s.ring, group);
        Turn stage;
        stage.step(s.stages, group);
        int tile = 0, c = group;
        while (c >= chunks) { c -= chunks; ++tile; }
        bool real = quarter < boxesOf(tile);   // lanes of absent rows keep what they held
        for (int g = group; g < total; g += 2) {
            const int place = slot.place();
            wait(&rawFull[slot.full.at], slot.full.parity);
            const uint8_t *row = raw + place * kRawBytes + quarter * kBoxBytes + lane * 128;
            float v[16];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 x = *reinterpret_cast<const float4 *>(row + (((4 * part + i) ^ sw) << 4));
                v[4 * i] = x.x; v[4 * i + 1] = x.y; v[4 * i + 2] = x.z; v[4 * i + 3] = x.w;
            }
            arrive(&rawFree[place]);
            if (stage.again) wait(&termsFree[stage.at], stage.parity ^ 1u);
            __syncwarp();
            if (real) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 f = *reinterpret_cast<const float4 *>(scale + c * kChunk + 16 * part + 4 * i);
                    v[4 * i] *= f.x; v[4 * i + 1] *= f.y; v[4 * i + 2] *= f.z; v[4 * i + 3] *= f.w;
                }
                const uint32_t to = stageBase + lanes + stage.at * kStageCols + 8 * part;
#pragma unroll
                for (int term = 0; term < 3; ++term) {
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        w[i] = packBf16(v[2 * i], v[2 * i + 1]);
                        v[2 * i] -= bf16Lo(w[i]);
                        v[2 * i + 1] -= bf16Hi(w[i]);
                    }
                    bwdcluster::tmemStore8(to + term * (kChunk / 2), w);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
            arrive(&termsFull[stage.at]);
            slot.step(2);
            stage.step(s.stages, 2);
            for (c += 2; c >= chunks; c -= chunks) real = quarter < boxesOf(++tile);
        }
    } else if (warp < kFillWarps) {
        // the two warps of a quarter take blocks of 32 columns in turn
        const int quarter = warp & 3, half = (warp - kConvWarps) >> 2;
        float4 *mine = reinterpret_cast<float4 *>(turn + (warp - kConvWarps) * 4096);
        const bool vectors = p.N % 4 == 0 && (reinterpret_cast<uintptr_t>(p.out) & 15) == 0 && (reinterpret_cast<uintptr_t>(p.mask) & 3) == 0;
        Turn acc;
        for (int tile = 0; tile < tiles; ++tile, acc.step(s.accs)) {
            wait(&accFull[acc.at], acc.parity);
            __syncwarp();
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int first = rowBegin + tile * kTileM + 32 * quarter, count = min(32, rowEnd - first);
            const uint32_t from = tmem + (static_cast<uint32_t>(32 * quarter) << 16) + acc.at * NP;
            const bool poison = failed != 0;
            for (int c0 = 32 * half; c0 < NP && count > 0; c0 += 64) {
                uint32_t r[32];
                if (c0 + 32 <= NP) {
                    tmemLoad32(from + c0, r);
                } else {
#pragma unroll
                    for (int i = 0; i < 2; ++i) bwdcluster::tmemLoad<8>(from + c0 + 8 * i, *reinterpret_cast<uint32_t (*)[8]>(r + 8 * i));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int i = 16; i < 32; ++i) r[i] = 0u;
                }
                // lane = row here: turn the 32 x 32 block so that eight lanes hold 128 bytes of a row
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    mine[lane * 8 + (i ^ (lane & 7))] =
                        make_float4(__uint_as_float(r[4 * i]), __uint_as_float(r[4 * i + 1]), __uint_as_float(r[4 * i + 2]), __uint_as_float(r[4 * i + 3]));
                __syncwarp();
                const int i = lane & 7, col = c0 + 4 * i, left = columns - col, at = lane >> 3;
                const size_t o = static_cast<size_t>(first + at) * p.N + n0 + col;
                if (left > 0) {
                    float *to = p.out + o;
                    const uint8_t *m = p.mask + o;
                    const size_t step = 4 * static_cast<size_t>(p.N);
                    uint32_t drop[8];   // a byte is 0xff where the mask drops the value
#pragma unroll
                    for (int pass = 0; pass < 8; ++pass) {
                        uint32_t word = p.maskKeeps ? 0x01010101u : 0u;
                        if (p.mask && 4 * pass + at < count) {
                            if (vectors) word = __ldg(reinterpret_cast<const uint32_t *>(m));
                            else
                                for (int e = 0; e < 4; ++e)
                                    if (e < left) word = (word & ~(0xffu << (8 * e))) | static_cast<uint32_t>(__ldg(m + e)) << (8 * e);
                        }
                        drop[pass] = p.maskKeeps ? __vcmpeq4(word, 0u) : __vcmpne4(word, 0u);
                        m += step;
                    }
                    float4 x[8];
#pragma unroll
                    for (int pass = 0; pass < 8; ++pass) x[pass] = mine[(4 * pass + at) * 8 + (i ^ ((4 * pass + at) & 7))];
#pragma unroll
                    for (int pass = 0; pass < 8; ++pass, to += step) {
                        if (drop[pass] != 0u) {   // rare; a product with 0 keeps NaN and signs
                            auto times = [&](float v, int e) { return drop[pass] >> (8 * e) & 1u ? v * 0.0f : v; };
                            x[pass] = make_float4(times(x[pass].x, 0), times(x[pass].y, 1), times(x[pass].z, 2), times(x[pass].w, 3));
                        }
                        if (poison) x[pass] = make_float4(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000), __int_as_float(0x7fc00000), __int_as_float(0x7fc00000));
                        if (4 * pass + at >= count) continue;
                        if (vectors) {
                            *reinterpret_cast<float4 *>(to) = x[pass];
                        } else {
                            const float v[4] = {x[pass].x, x[pass].y, x[pass].z, x[pass].w};
#pragma unroll
                            for (int e = 0; e < 4; ++e)
                                if (e < left) to[e] = v[e];
                        }
                    }
                }
                __syncwarp();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            arrive(&accFree[acc.at]);   // the products of a later tile may overwrite the accumulator
        }
    } else if (warp == kGradientWarp) {
        int tile = 0, c = 0;   // of the next chunk
        fillRing(total, s.ring, rawFull, rawFree, failed, wait, [&](int, int place, uint64_t *bar) {
            const int boxes = boxesOf(tile), row = rowBegin + tile * kTileM + lane * kBoxRows;
            if (lane == 0) expect(bar, boxes * kBoxBytes);
            __syncwarp();
            if (lane < boxes) copyBox(smemAddr(raw + place * kRawBytes + lane * kBoxBytes), &gradients, c * kChunk, row, smemAddr(bar));
            if (++c == chunks) {
                c = 0;
                ++tile;
            }
        });
    } else if (warp == kWeightWarp) {
        if (STREAM && electOne()) {
            Turn slot;
            int issued = 0;
            const uint8_t *first = static_cast<const uint8_t *>(p.packed) + static_cast<size_t>(blockIdx.y) * chunks * weightBytes;
            for (int tile = 0; tile < tiles && !failed; ++tile) {
                const uint8_t *src = first;
                for (int c = 0; c < chunks && !failed; ++c, src += weightBytes) {
                    if (slot.again) wait(&weightsFree[slot.at], slot.parity ^ 1u);
                    if (failed) break;
                    expect(&weightsFull[slot.at], weightBytes);
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                                     smemAddr(weights + slot.at * weightBytes)),
                                 "l"(src), "r"(weightBytes), "r"(smemAddr(&weightsFull[slot.at]))
                                 : "memory");
                    ++issued;
                    slot.step(kWeightRing);
                }
            }
            for (int g = max(0, issued - kWeightRing); g < issued; ++g) waitPhase(smemAddr(&weightsFull[g % kWeightRing]), (g / kWeightRing) & 1);
        }
    } else if (electOne()) {
        const uint32_t idesc = instructionDescriptor(NP, false);
        if (!STREAM) wait(&weightsFull[0], 0);
        Turn stage, slot, acc;
        for (int tile = 0; tile < tiles; ++tile, acc.step(s.accs)) {
            if (acc.again) wait(&accFree[acc.at], acc.parity ^ 1u);
            for (int c = 0; c < chunks; ++c) {
                wait(&termsFull[stage.at], stage.parity);
                if (STREAM) wait(&weightsFull[slot.at], slot.parity);
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t descB = operandDescriptor(smemAddr(weights + (STREAM ? slot.at : c) * weightBytes), kCore, kGroupStride);
                const uint32_t terms = stageBase + stage.at * kStageCols;
#pragma unroll
                for (int ks = 0; ks < kChunk / 16; ++ks)
#pragma unroll
                    for (int term = 0; term < 3; ++term)
                        bwdcluster::mmaBf16TmemA(tmem + acc.at * NP, terms + term * (kChunk / 2) + 8 * ks, descB + static_cast<uint64_t>(ks * ((2 * kCore) >> 4)), idesc,
                                                 (c > 0 || ks > 0 || term > 0) ? 1u : 0u);
                commitTo(smemAddr(&termsFree[stage.at]));
                if (STREAM) commitTo(smemAddr(&weightsFree[slot.at]));
                if (c + 1 == chunks) commitTo(smemAddr(&accFull[acc.at]));
                stage.step(s.stages);
                if (STREAM) slot.step(kWeightRing);
            }
        }
        letDependentsStart();   // the kernel behind this one is launched under the last products and the epilogue
        // nothing is left in flight when tensor memory is given back
        if (tiles > 0) waitPhase(smemAddr(&accFull[(tiles - 1) % s.accs]), ((tiles - 1) / s.accs) & 1);
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTmemCols) : "memory");
    if (tid == 0 && failed && p.status) atomicExch(p.status, 1);
}

// Columns of a CTA: all of them up to 256, else even slabs.
Shape shapeFor(int N) {
    Shape s{};
    s.slabs = (N + kMaxColumns - 1) / kMaxColumns;
    s.NP = ((N + s.slabs - 1) / s.slabs + 15) / 16 * 16;
    s.accs = s.NP <= 128 ? 2 : 1;
    s.stages = std::min<int>(kMaxStages, (kTmemCols - s.accs * s.NP) / kStageCols);
    return s;
}
size_t sharedBytes(const Shape &s, int K, bool stream, int ring) {
    return 1024 + ring * static_cast<size_t>(kRawBytes) + kEpilogueWarps * 4096 + static_cast<size_t>(stream ? kWeightRing : K / kChunk) * s.NP * kChunk * 2 +
           sizeof(float) * static_cast<size_t>(K);
}
// Weights stay in shared memory up to 64 columns where they leave room for a ring of four chunks.
bool resident(int K, int N) { return N <= kResidentColumns && sharedBytes(shapeFor(N), K, false, 4) <= 225 * 1024; }

}  // namespace

size_t packedBytes(int K, int N) {
    if (N < 1 || K < kChunk || K % kChunk != 0 || K > kMaxK || resident(K, N)) return 0;
    const Shape s = shapeFor(N);
    return static_cast<size_t>(s.slabs) * s.NP * K * 2;
}

bool eligible(int K, int N) {
    static const bool disabled = std::getenv("RXMET_IGRAD_SIMT") != nullptr;
    return !disabled && N >= 1 && K >= kChunk && K % kChunk == 0 && K <= kMaxK && encodeTiled() != nullptr;
}

void launch(const Problem &p, int sms, cudaStream_t st) {
    const bool stream = !resident(p.K, p.N);
    RXMET_REQUIRE(p.rows >= 1 && p.K % kChunk == 0 && p.K <= kMaxK && alignedTo(p.G, 16) && (!stream || (p.packed != nullptr && alignedTo(p.packed, 16))),
                  "input gradient: %d channels, %d columns", p.K, p.N);
    Shape s = shapeFor(p.N);
    const size_t most = std::min<size_t>(225 * 1024, currentDevice().smemMax);
    s.ring = kMaxRing;
    while (s.ring > 2 && sharedBytes(s, p.K, stream, s.ring) > most) --s.ring;
    const size_t smem = sharedBytes(s, p.K, stream, s.ring);
    const int boxes = (p.rows + kBoxRows - 1) / kBoxRows, most1 = std::max(1, sms / s.slabs);
    s.rowsPerCta = (boxes + most1 - 1) / most1 * kBoxRows;
    const CUtensorMap map = boxMap(p.G, p.rows, p.K, CU_TENSOR_MAP_SWIZZLE_128B);
    const dim3 grid(static_cast<unsigned>((p.rows + s.rowsPerCta - 1) / s.rowsPerCta), static_cast<unsigned>(s.slabs));
    KernelTimer timer__("inputGradUmma", st);
    if (stream) {
        const int items = p.K / 8 * s.NP * s.slabs;
        packWeights<<<(items + 255) / 256, 256, 0, st>>>(p, s.NP, s.slabs, static_cast<uint4 *>(p.packed));
        ensureDynamicSmem(reinterpret_cast<const void *>(inputGradUmma<true>), smem);
        launchDependent(inputGradUmma<true>, grid, kThreads, smem, st, p, s, map);
    } else {
        ensureDynamicSmem(reinterpret_cast<const void *>(inputGradUmma<false>), smem);
        launchDependent(inputGradUmma<false>, grid, kThreads, smem, st, p, s, map);
    }
}

}  // namespace igrad
}  // namespace rxmet
