// Preparation of a quantized LSTM call on byte planes: codes of x, h0 and c0, packed weights with their addends, tensor-core tiles.
//
// Blocks by job: channels of weight_ih and weight_hh, then rows of h0, c0 and x.  One launch in the place of five and up to three memsets,
// between which the device waited 2 to 4 us each: 8-bit training, T = 100, B = 256, I = 40, H = 128 347 -> 326 us, two directions of 16-bit
// inference, T = 200, B = 128, H = 128 198 -> 180 us.  The pass over the inputs of a large call is bound by issue, then by memory: T = 1000, B = 4096,
// I = 256 (4.2 GB in, 2.1 GB out) 2.59 -> 1.40 ms, where a division in double and a 64-bit one per word took the rest.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "common.h"
#include "dependent_launch.cuh"
#include "lstm_device.cuh"
#include "lstm_prepare.h"
#include "plane_proj_umma.cuh"
#include "row_words.cuh"

namespace rxmet {
namespace lstm {
namespace {

using dev::CodeGrid;
using dev::rescaleF;

constexpr int kThreads = 256, kCount = 4;   // words a thread asks for at a time

// How a job is shared out, decided on the host.
struct Shares {
    int group[2];        // lanes of a channel: weight_ih, weight_hh
    int blocks[5];       // weight_ih, weight_hh, h0, c0, x
    bool vectors[5];     // the same order: 16-byte loads and stores of four columns, 4-byte stores of their flags
};

// Four values of a row from column k on; zeros beyond the last one.
__device__ __forceinline__ void loadFour(const PrepareRows &t, bool vectors, const RowWord &at, float (&v)[4]) {
    const int k = 4 * at.word;
    const float *from = t.src + at.row * t.cols + k;
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = 0.0f;
    if (!t.src || !at.real) return;
    if (vectors) {
        if (k >= t.cols) return;
        const float4 four = __ldcs(reinterpret_cast<const float4 *>(from));
        v[0] = four.x; v[1] = four.y; v[2] = four.z; v[3] = four.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (k + e < t.cols) v[e] = from[e];
    }
}
template <int PLANES>
__device__ __forceinline__ void storePlanes(const PrepareRows &t, const RowWord &at, uint32_t high, uint32_t low) {
    uint32_t *to = t.planes + at.row * (PLANES * t.words) + at.word;
    to[0] = PLANES == 2 ? high : low;
    if (PLANES == 2) to[t.words] = low;
}
// A word as the reference states it: any scale and any value.
template <int PLANES>
__device__ __forceinline__ void quantizeWord(const PrepareRows &t, bool vectors, const RowWord &at) {
    if (!at.real) return;
    float v[4];
    loadFour(t, vectors, at, v);
    uint32_t low = 0, high = 0;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int k = 4 * at.word + e;
        if (k >= t.cols) continue;
        const size_t o = at.row * t.cols + k;
        uint8_t clamped = 0;
        const int32_t q = t.src ? dev::quantizeCode(v[e], t.scale, t.zp, t.lo, t.hi, clamped) : min(max(t.zp, t.lo), t.hi);
        const uint32_t u = static_cast<uint32_t>(q - t.lo);
        low |= (u & 0xffu) << (8 * e);
        high |= (u >> 8 & 0xffu) << (8 * e);
        if (t.carrier) t.carrier[o] = static_cast<float>(q);
        if (t.clamped) t.clamped[o] = clamped;
        if (t.centred) t.centred[o] = static_cast<float>(q - t.zp);
    }
    if (t.planes) storePlanes<PLANES>(t, at, high, low);
}
// SAVES: something beside the planes is asked for.
template <int PLANES, bool SAVES>
__device__ __forceinline__ void quantizePlainRows(const CodeGrid &grid, const PrepareRows &t, bool vectors, int block, int blocks) {
    const float toBits = 8388608.0f - grid.lo;   // code + toBits = 2^23 + (code - lo)
    eachRowWord<kCount>(t.rows, t.words, block, blocks, [&](const RowWord (&at)[kCount]) {
        float v[kCount][4];
#pragma unroll
        for (int n = 0; n < kCount; ++n) loadFour(t, vectors, at[n], v[n]);
        uint32_t far = 0;
#pragma unroll
        for (int n = 0; n < kCount; ++n) {
            float x[4];
            if (!grid.codes(v[n], x)) far |= 1u << n;
            uint32_t bits[4], flags = 0;
            const int k = 4 * at[n].word;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float inside = fminf(fmaxf(x[e], grid.lo), grid.hi);
                if (SAVES) flags |= inside != x[e] ? 1u << (8 * e) : 0u;
                x[e] = inside;
                bits[e] = __float_as_uint(__fadd_rn(inside, toBits));
            }
            if (!at[n].real) continue;
            if (t.planes) {
                uint32_t low = __byte_perm(__byte_perm(bits[0], bits[1], 0x0040), __byte_perm(bits[2], bits[3], 0x0040), 0x5410);
                uint32_t high = __byte_perm(__byte_perm(bits[0], bits[1], 0x0051), __byte_perm(bits[2], bits[3], 0x0051), 0x5410);
                const int beyond = k + 4 - t.cols;   // columns of the padding
                if (beyond > 0) {
                    const uint32_t keep = beyond >= 4 ? 0u : 0xffffffffu >> (8 * beyond);
                    low &= keep;
                    high &= keep;
                }
                storePlanes<PLANES>(t, at[n], high, low);
            }
            if constexpr (SAVES) {
                const size_t o = at[n].row * t.cols + k;
                if (vectors) {
                    if (k >= t.cols) continue;
                    if (t.carrier) *reinterpret_cast<float4 *>(t.carrier + o) = make_float4(x[0], x[1], x[2], x[3]);
                    if (t.clamped) *reinterpret_cast<uint32_t *>(t.clamped + o) = flags;
                    if (t.centred) *reinterpret_cast<float4 *>(t.centred + o) = make_float4(x[0] - grid.zp, x[1] - grid.zp, x[2] - grid.zp, x[3] - grid.zp);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if (k + e >= t.cols) continue;
                        if (t.carrier) t.carrier[o + e] = x[e];
                        if (t.clamped) t.clamped[o + e] = static_cast<uint8_t>(flags >> (8 * e));
                        if (t.centred) t.centred[o + e] = x[e] - grid.zp;
                    }
                }
            }
        }
#pragma unroll 1
        for (int n = 0; far >> n; ++n)   // rare: written again
            if (far >> n & 1u) quantizeWord<PLANES>(t, vectors, n == 0 ? at[0] : n == 1 ? at[1] : n == 2 ? at[2] : at[3]);
    });
}
template <int PLANES>
__device__ __forceinline__ void quantizeRows(const PrepareRows &t, bool vectors, int block, int blocks) {
    static_assert(kCount == 4, "the words of a thread are named one by one");
    const CodeGrid grid(t.scale, t.zp, t.lo, t.hi);
    if (!grid.plain || !t.src) eachRowWord<1>(t.rows, t.words, block, blocks, [&](const RowWord (&at)[1]) { quantizeWord<PLANES>(t, vectors, at[0]); });
    else if (t.carrier || t.clamped || t.centred) quantizePlainRows<PLANES, true>(grid, t, vectors, block, blocks);
    else quantizePlainRows<PLANES, false>(grid, t, vectors, block, blocks);
}

// `group` neighbouring lanes a channel; they quantize consecutive words of its row and add up the codes.
template <bool IH>
__device__ __forceinline__ void quantizeWeights(const PrepareCall &a, const PrepareWeights &side, bool vectors, int group, int block) {
    const int C = 4 * a.H, lane = threadIdx.x % group, c = static_cast<int>((block * kThreads + threadIdx.x) / group);
    const bool real = c < C;
    const int allWords = IH && a.ihTiles ? planeproj::paddedK(side.words) / 4 : side.words;
    const int ch = min(c, C - 1), gate = ch / a.H, j = ch - gate * a.H;
    auto field = [&](int f) { return __ldg(a.channel + static_cast<size_t>(f) * C + ch); };
    const CodeGrid grid(field(side.scaleField), 0, a.wLo, a.wHi);
    const float *row = side.w + static_cast<size_t>(ch) * side.K;
    int32_t sum = 0;
    for (int kw = lane; kw < allWords; kw += group) {
        const int k = 4 * kw;
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (real && vectors) {
            if (k < side.K) {
                const float4 four = __ldg(reinterpret_cast<const float4 *>(row + k));
                v[0] = four.x; v[1] = four.y; v[2] = four.z; v[3] = four.w;
            }
        } else if (real) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (k + e < side.K) v[e] = __ldg(row + k + e);
        }
        uint32_t word = 0, flags = 0;
        int32_t codes[4];
        float x[4];
        if (grid.plain && grid.codes(v, x)) {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float inside = fminf(fmaxf(x[e], grid.lo), grid.hi);
                flags |= inside != x[e] ? 1u << e : 0u;
                codes[e] = static_cast<int32_t>(inside);
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                uint8_t clamped;
                codes[e] = dev::quantizeCode(v[e], grid.scale, 0, a.wLo, a.wHi, clamped);
                flags |= static_cast<uint32_t>(clamped) << e;
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if (!real || k + e >= side.K) continue;
            const int32_t q = codes[e];
            const size_t o = static_cast<size_t>(ch) * side.K + k + e;
            if (side.carrier) side.carrier[o] = static_cast<float>(q);
            if (side.clamped) side.clamped[o] = static_cast<uint8_t>(flags >> e & 1u);
            sum += q;
            word |= (static_cast<uint32_t>(q) & 0xffu) << (8 * e);
        }
        if constexpr (IH) {
            if (a.ihWords && real && kw < side.words) a.ihWords[static_cast<size_t>(kw) * C + c] = word;
            if (a.ihTiles && c < planeproj::paddedC(C)) a.ihTiles[4 * planeproj::tilePlace(c, kw / 4, 4 * allWords) + kw % 4] = word;
        } else if (real) {
            a.hhWords[((static_cast<size_t>(gate >> 1) * side.words + kw) * a.H + j) * 2 + (gate & 1)] = word;
        }
    }
    for (int o = group / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane != 0 || !real) return;
    int64_t addend = side.correction * static_cast<int64_t>(sum);
    if (side.b) {
        uint8_t clamped;
        const int32_t q = dev::quantizeCode(side.b[c], field(side.biasScaleField), 0, a.bLo, a.bHi, clamped);
        addend += static_cast<int64_t>(rescaleF(static_cast<float>(q), DevRescale{field(side.biasMultField), field(side.biasPow2Field)}));
        if (side.biasCarrier) side.biasCarrier[c] = static_cast<float>(q);
        if (side.biasClamped) side.biasClamped[c] = clamped;
    }
    side.addend[c] = addend;
}

template <int PLANES>
__global__ void __launch_bounds__(kThreads, 4) prepareCall(const __grid_constant__ PrepareCall a, const __grid_constant__ Shares s) {
    letDependentsStart();
    if (blockIdx.x == 0 && threadIdx.x == 0 && a.clear) *a.clear = 0;
    int block = static_cast<int>(blockIdx.x);
    if (block < s.blocks[0]) return quantizeWeights<true>(a, a.ih, s.vectors[0], s.group[0], block);
    block -= s.blocks[0];
    if (block < s.blocks[1]) return quantizeWeights<false>(a, a.hh, s.vectors[1], s.group[1], block);
    block -= s.blocks[1];
    if (block < s.blocks[2]) return quantizeRows<PLANES>(a.h0, s.vectors[2], block, s.blocks[2]);
    block -= s.blocks[2];
    if (block < s.blocks[3]) return quantizeRows<1>(a.c0, s.vectors[3], block, s.blocks[3]);
    quantizeRows<PLANES>(a.x, s.vectors[4], block - s.blocks[3], s.blocks[4]);
}

}  // namespace

void prepare(const PrepareCall &call, cudaStream_t st) {
    Shares s{};
    const int C = 4 * call.H, channels = call.ihTiles ? planeproj::paddedC(C) : C;
    auto weights = [&](int i, const PrepareWeights &w, int count) {
        s.group[i] = w.words <= 4 ? 4 : w.words <= 8 ? 8 : w.words <= 16 ? 16 : 32;
        s.blocks[i] = (count * s.group[i] + kThreads - 1) / kThreads;
        s.vectors[i] = w.K % 4 == 0 && alignedTo(w.w, 16);
    };
    weights(0, call.ih, channels);
    weights(1, call.hh, C);
    const int most = 8 * currentDevice().sms;
    auto rows = [&](int i, const PrepareRows &r) {
        s.blocks[i] = rowWordBlocks(r.rows, r.words, kCount, kThreads, most);
        s.vectors[i] = r.cols % 4 == 0 && alignedTo(r.src, 16) && alignedTo(r.carrier, 16) && alignedTo(r.centred, 16) && alignedTo(r.clamped, 4);
    };
    rows(2, call.h0);
    rows(3, call.c0);
    rows(4, call.x);
    const int grid = s.blocks[0] + s.blocks[1] + s.blocks[2] + s.blocks[3] + s.blocks[4];
    {
        KernelTimer timer__("lstmPrepare", st);
        if (call.planes == 2) prepareCall<2><<<grid, kThreads, 0, st>>>(call, s);
        else prepareCall<1><<<grid, kThreads, 0, st>>>(call, s);
    }
    afterLaunch("lstmPrepare");
}

}  // namespace lstm
}  // namespace rxmet
