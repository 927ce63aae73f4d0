// Input projection of the 8-bit QuantGRU path on the 5th-generation tensor cores:
//   ih[row][c] = epilogue( sum_k x_q[row][k] * W_q[k][c] )        for all T*B rows at once
// as tcgen05.mma kind::i8 (signed 8-bit codes, exact 32-bit integer accumulators in tensor memory)
// with the whole rescale / zero-point / clamp / keep-flag / gate-grid epilogue fused behind it
// (the reference runs a GEMM and a separate bias-and-rescale pass per call:
// operators/quant-gru/src/gru_forward_gpu_quant.cu:109-180, gru_forward_gpu_quant_fp.cu:1129).
//
// The product is computed TRANSPOSED, D[channel][row] = W_q^T x_q^T: the 128 lanes of tensor memory are
// 128 output channels, the columns are rows of the batch.  That puts one channel into one thread of the
// epilogue, so the per-channel constants (multiplier, shift, offset, gate rescale) live in registers, and
// for a given row the 32 lanes of a warp store 32 neighbouring channels: 64 contiguous bytes of codes.
//
// A CTA keeps one tile of 128 channels and walks a contiguous range of rows, 64 at a time.  Once: its channels' weight codes as the K-major
// A operand in the un-swizzled canonical layout (core matrix = 8 channels x 16 k-bytes) and the constants of the
// epilogue.  Per item: the code rows (contiguous in HBM) come into the canonical K-major B layout as 4-byte asynchronous copies (a row
// is I bytes, not a multiple of 16, so no bulk copy fits), asked for two items ahead; one thread issues K/32 MMAs into one of two
// accumulator buffers and commits them to that buffer's mbarrier; the epilogue of the previous item runs meanwhile: tcgen05.ld (lane =
// channel, 16 rows per load), integer rescale with round-half-even, clamp, optional second rescale onto the gate-input grid.
// Bound: issue of the epilogue.  25,600 rows, I = 40, 384 channels 24.0 -> 21.4 us against CTAs that walked items of all channel tiles,
// fetched each item's constants and waited for its rows.
// Every mbarrier wait is bounded; a wait that gives up sets the status word (the recurrent kernel that
// consumes the codes turns its outputs into NaN then) and the CTA still frees its tensor memory.
#include <algorithm>
#include <cstdlib>
#include <type_traits>

#include "common.h"
#include "dependent_launch.cuh"
#include "gru_device.cuh"
#include "input_proj_umma.h"
#include "plane_proj_umma.cuh"
#include "umma_device.cuh"

namespace rxmet {
namespace iproj {
namespace {

using namespace umma;
using gru::Rescale;

constexpr int kThreads = 512;

// kind::i8: 32-bit integer accumulator (bits [4,6) = 2), signed 8-bit A and B (bits [7,10) = [10,13) = 1),
// both K-major (bits 15, 16 clear), N >> 3 in [17,23), M >> 4 in [24,29).
__host__ __device__ constexpr uint32_t instructionDescriptorI8(int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kTileM >> 4) << 24);
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

// Rows of the batch per item = accumulator columns.  A CTA keeps one tile of 128 channels, whose constants stay in its threads' registers,
// and walks a contiguous range of rows, cut at multiples of 16.
constexpr int kRows = 64, kRowStep = 16;

__host__ __device__ inline int paddedC(int C) { return (C + kTileM - 1) / kTileM * kTileM; }
size_t sharedBytes(int kPad) { return static_cast<size_t>(kTileM + 2 * kRows) * kPad; }

__global__ void __launch_bounds__(kThreads, 2) inputProjUmma(const Problem p, int rowsPerCta) {
    constexpr uint32_t kTmemCols = 2 * kRows;
    constexpr uint32_t kIdesc = instructionDescriptorI8(kRows);
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[2];  // one per accumulator buffer
    __shared__ uint32_t tmemSlot;
    __shared__ int failed;

    const int tid = threadIdx.x, lane = tid & 31, warp = warpIndex();
    const int C = p.C, kWords = p.kWords, kPad = p.kPad, channelTiles = paddedC(C) / kTileM;
    const int ct = static_cast<int>(blockIdx.x) % channelTiles, rowBegin = static_cast<int>(blockIdx.x) / channelTiles * rowsPerCta;
    const int rowEnd = min(p.rows, rowBegin + rowsPerCta), items = (rowEnd - rowBegin + kRows - 1) / kRows;
    const uint32_t groupStride = static_cast<uint32_t>(kPad / 16) * kCore;  // next 8 channels / 8 rows
    uint8_t *weights = smem;                                               // [kTileM / 8][kPad / 16][8][16]
    uint8_t *rowStages = smem + static_cast<size_t>(kTileM) * kPad;             // 2 x [kRows / 8][kPad / 16][8][16]
    const size_t stageBytes = static_cast<size_t>(kRows) * kPad;

    if (tid == 0) {
        failed = 0;
        for (int i = 0; i < 2; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smemAddr(&bars[i])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smemAddr(&tmemSlot)), "r"(kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    // operands start as zeros: the k padding of both and the channels beyond C are never written again
    for (size_t i = tid; i < (static_cast<size_t>(kTileM) * kPad + 2 * stageBytes) / 16; i += kThreads)
        reinterpret_cast<uint4 *>(smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    waitForPredecessor();
    if (!p.late) letDependentsStart();
    // weight word (kw, c) = codes k = 4 kw .. 4 kw + 3 of channel c -> four consecutive bytes of row c
    for (int i = tid; i < kWords * kTileM; i += kThreads) {
        const int kw = i / kTileM, local = i % kTileM, c = ct * kTileM + local;
        if (c < C)
            *reinterpret_cast<int32_t *>(weights + (local >> 3) * groupStride + (kw >> 2) * kCore + (local & 7) * 16 + (kw & 3) * 4) = p.w[static_cast<size_t>(kw) * C + c];
    }

    // the code words of an item's rows are one contiguous run; rows beyond the range become zeros
    auto loadRows = [&](int item, int stage) {
        const size_t first = static_cast<size_t>(rowBegin + item * kRows) * kWords;
        const size_t limit = static_cast<size_t>(rowEnd) * kWords;
        uint8_t *dst = rowStages + stage * stageBytes;
        for (int i = tid; i < kRows * kWords; i += kThreads) {
            const int r = i / kWords, kw = i - r * kWords;
            const bool real = first + i < limit;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smemAddr(dst + (r >> 3) * groupStride + (kw >> 2) * kCore + (r & 7) * 16 + (kw & 3) * 4)),
                         "l"(p.x + (real ? first + i : 0)), "r"(real ? 4u : 0u)
                         : "memory");
        }
    };

    for (int n = 0; n < min(2, items); ++n) loadRows(n, n);

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmemSlot;

    const int32_t zpOut = p.zpOut, lo = p.lo, hi = p.hi;
    const int q = warp & 3, group = warp >> 2;  // tensor-memory lane quarter (32 channels) of this warp, row-chunk group
    // second rescale: |code| and |zero point| below 2^20 keep the product inside 32-bit pieces
    const bool gridsSmall = lo >= -(1 << 20) && hi <= (1 << 20) && zpOut >= -(1 << 20) && zpOut <= (1 << 20);

    const bool real = ct * kTileM + 32 * q + lane < C;
    const int c = min(ct * kTileM + 32 * q + lane, C - 1);  // this thread's channel
    // per-channel constants in registers.  Narrow channels (|offset| < 2^30, a multiplier that shrinks,
    // shift in [1, 31]) round with 32-bit pieces of the product; the others take the 64-bit form.
    const Rescale rs = p.rescale[c];
    const int64_t offset = p.biasAcc[c] - p.comp[c];
    const bool narrow = rs.shift >= 1 && rs.shift <= 31 && rs.mult > 0 && static_cast<int64_t>(rs.mult) <= (1ll << rs.shift) &&
                        offset > -(1ll << 30) && offset < (1ll << 30);
    const Rescale gateRs = p.pre.enabled ? p.pre.toGate[c / p.pre.hidden] : Rescale{1, 0};
    const bool gateNarrow = gridsSmall && gateRs.shift >= 1 && gateRs.shift <= 31 && gateRs.mult > 0 &&
                            static_cast<int64_t>(gateRs.mult) <= (1ll << min(gateRs.shift + 9, 31));
    const bool warpNarrow = __all_sync(0xffffffffu, narrow && (!p.pre.enabled || gateNarrow));
    // Narrow: half a unit rides in the addend, the floor is right then except for an exact tie, where it is the upper neighbour and an
    // odd one must step down.
    const int64_t plus = offset * rs.mult + (narrow ? int64_t{1} << (rs.shift - 1) : 0);
    const int64_t gatePlus = -static_cast<int64_t>(zpOut) * gateRs.mult + (gateNarrow ? int64_t{1} << (gateRs.shift - 1) : 0);
    const uint32_t tie = (1u << (rs.shift & 31)) - 1u, gateTie = (1u << (gateRs.shift & 31)) - 1u;
    auto rounded = [](int64_t sum, int shift, uint32_t mask) {
        const uint32_t low = static_cast<uint32_t>(sum);
        const int32_t q = static_cast<int32_t>(__funnelshift_r(low, static_cast<uint32_t>(static_cast<uint64_t>(sum) >> 32), shift));
        return (low & mask) == 0 ? q & ~1 : q;
    };

    auto epilogue = [&](int item) {
        const int buf = item & 1;
        if (!waitPhase(smemAddr(&bars[buf]), (item >> 1) & 1)) failed = 1;
        // the products have read this stage: the rows of the item after next come in under the epilogue
        if (item + 2 < items) loadRows(item + 2, buf);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int chunk = group; chunk < kRows / 16; chunk += kThreads / 128) {
            uint32_t acc[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                : "=r"(acc[0]), "=r"(acc[1]), "=r"(acc[2]), "=r"(acc[3]), "=r"(acc[4]), "=r"(acc[5]), "=r"(acc[6]), "=r"(acc[7]),
                  "=r"(acc[8]), "=r"(acc[9]), "=r"(acc[10]), "=r"(acc[11]), "=r"(acc[12]), "=r"(acc[13]), "=r"(acc[14]), "=r"(acc[15])
                : "r"(tmem + (static_cast<uint32_t>(32 * q) << 16) + static_cast<uint32_t>(buf * kRows + 16 * chunk)));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            const int row0 = rowBegin + item * kRows + 16 * chunk, count = real ? rowEnd - row0 : 0;
            planeproj::Column<int16_t> to(p.out, row0, c, C);
            planeproj::Column<uint8_t> toMask(p.mask, row0, c, C);
            if (warpNarrow) {
                auto rows = [&](auto preTag, auto maskTag) {
                    planeproj::eachRow<16>(count, [&](int j) {
                        const int32_t code = rounded(static_cast<int64_t>(static_cast<int32_t>(acc[j])) * rs.mult + plus, rs.shift, tie) + zpOut;
                        const int32_t inside = max(lo, min(code, hi));
                        if (decltype(maskTag)::value) toMask.put(static_cast<uint8_t>(inside == code ? 1 : 0));
                        to.put(static_cast<int16_t>(decltype(preTag)::value ? rounded(static_cast<int64_t>(inside) * gateRs.mult + gatePlus, gateRs.shift, gateTie)
                                                                            : inside));
                    });
                };
                if (p.pre.enabled && p.mask) rows(std::true_type{}, std::true_type{});
                else if (p.pre.enabled) rows(std::true_type{}, std::false_type{});
                else if (p.mask) rows(std::false_type{}, std::true_type{});
                else rows(std::false_type{}, std::false_type{});
                continue;
            }
            const int64_t mulAdd = offset * rs.mult, gateAdd = -static_cast<int64_t>(zpOut) * gateRs.mult;
#pragma unroll 1
            for (int j = 0; j < min(count, 16); ++j) {
                uint8_t keep;
                int32_t sum = 0;
#pragma unroll
                for (int e = 0; e < 16; ++e) sum = e == j ? static_cast<int32_t>(acc[e]) : sum;
                int32_t code = gru::clampCode(gru::rshiftRoundCalled(static_cast<int64_t>(sum) * rs.mult + mulAdd, rs.shift) + zpOut, lo, hi, keep);
                if (p.pre.enabled) code = gru::rshiftRoundCalled(static_cast<int64_t>(code) * gateRs.mult + gateAdd, gateRs.shift);
                to.put(static_cast<int16_t>(code));
                if (p.mask) toMask.put(keep);
            }
        }
        // the MMAs of the item after next overwrite this buffer: order them behind these loads
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    };

    for (int item = 0; item < items; ++item) {
        const int stage = item & 1;
        asm volatile("cp.async.wait_all;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (warp == 0 && electOne()) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t descA = operandDescriptor(smemAddr(weights), kCore, groupStride), descB = operandDescriptor(smemAddr(rowStages + stage * stageBytes), kCore, groupStride);
            constexpr uint64_t kStep = (2 * kCore) >> 4;   // the start-address field counts 16-byte units
            for (int ks = 0; ks < kPad / 32; ++ks)
                mmaI8(tmem + stage * kRows, descA + ks * kStep, descB + ks * kStep, kIdesc, ks > 0 ? 1u : 0u);
            commitTo(smemAddr(&bars[stage]));
        }
        if (item > 0) epilogue(item - 1);
    }
    if (items > 0) epilogue(items - 1);

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (p.late) letDependentsStart();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    if (tid == 0 && failed && p.status) atomicExch(p.status, 1);
}

}  // namespace

int paddedK(int kWords) { return (kWords * 4 + 31) / 32 * 32; }

bool eligible(int C, int kWords, const void *x) {
    static const bool disabled = std::getenv("RXMET_IPROJ_SIMT") != nullptr;
    if (disabled || kWords < 1 || !alignedTo(x, 4)) return false;
    return static_cast<size_t>(paddedC(C) + 2 * kRows) * paddedK(kWords) <= 200 * 1024;
}

void launch(const Problem &problem, int sms, cudaStream_t st) {
    Problem prob = problem;
    prob.kPad = paddedK(prob.kWords);
    const size_t smem = sharedBytes(prob.kPad);
    ensureDynamicSmem(reinterpret_cast<const void *>(inputProjUmma), smem);
    const int channelTiles = paddedC(prob.C) / kTileM, most = std::max(1, 2 * sms / channelTiles);   // ranges of rows
    // Up to two CTAs an SM a range is one item: cut finer, the projection of a few thousand rows sits on all SMs, and a recurrence that is launched
    // beside it finds room for its CTAs on some of them only (T 100, B 32, I 100, H 64: 3200 rows on 200 CTAs 60 us, on 100 43; a QAT step 142 and 119).
    const bool whole = (prob.rows + kRows - 1) / kRows * channelTiles <= 2 * sms;
    const int rowsPerCta = whole ? kRows : ((prob.rows + most - 1) / most + kRowStep - 1) / kRowStep * kRowStep;
    const int grid = (prob.rows + rowsPerCta - 1) / rowsPerCta * channelTiles;
    prob.late = prob.dependents > 0 && grid + prob.dependents > sms;
    KernelTimer timer__("inputLinear", st);
    launchDependent(inputProjUmma, grid, kThreads, smem, st, prob, rowsPerCta);
}

}  // namespace iproj
}  // namespace rxmet
