// LSTM backward through time on real values, with the optional clamp masks of the QAT path.
//
// Launch plan (the reference runs T x (pointwise kernel + cuBLAS GEMM) and three cuBLAS GEMMs,
// operators/quant-lstm/src/lstm/backward_float_cuda.cu:50-104,189-330):
//   dequantWeights x2  : QAT only - q-carrier weight codes x per-channel scale -> real weights
//   recurrentBackward  : ONE launch for all T steps; a CTA owns BT batch rows, walks t = T-1..0,
//                        keeps dc in registers and dh in shared memory, writes the masked gate
//                        gradients of both linear branches, and propagates dh through weight_hh
//                        (rows resident in shared memory as far as they fit, the rest in registers)
//   gemmRowsTN + reduce: dW_ih = G_ih^T x, dW_hh = G_hh^T h_prev as split-K tile GEMMs over the T*B
//                        rows with fixed-order reduction (bit-reproducible), masks applied there
//   gemmNN             : dx = G_ih W_ih with the input clamp mask
//   columnSums + reduce: bias gradients
// Saved q-carrier tensors are dequantized while they are loaded: real = (value - zp) * scale.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "common.h"
#include "dependent_launch.cuh"
#include "input_grad_umma.h"
#include "lstm_backward_cluster.h"
#include "lstm_kernels.h"
#include "regroup.h"
#include "weight_grad_mma.h"

namespace rxmet {
namespace lstm {
namespace {

__device__ __forceinline__ void prefetchL2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ float keepOf(const uint8_t *mask, size_t i) { return (mask == nullptr || mask[i] == 0) ? 1.0f : 0.0f; }
__device__ __forceinline__ float realOf(float v, Dequant d) { return (v - d.zeroPoint) * d.scale; }

__global__ void dequantWeights(const float *__restrict__ codes, const float *__restrict__ channelScale, int rows, int cols,
                               float *__restrict__ out) {
    const size_t n = static_cast<size_t>(rows) * cols;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x)
        out[i] = codes[i] * channelScale[i / cols];
}

// One word of keep/drop flags per (t, b, j): bit 0 hidden, 1 tanh(cell), 2 cell, 3-6 gate outputs,
// 7-10 gate inputs, 11-14 ih linear, 15-18 hh linear (a set bit = clamped = no gradient).  Packing them
// once in a bandwidth-bound pass takes 19 byte loads per element off every step of the recurrence.
// `width` >= H: words per row of out, the ones beyond H keep everything.
__global__ void packStepMasks(const rxmet_lstm_backward_masks mk, size_t rows, int H, int width, uint32_t *__restrict__ out) {
    const size_t n = rows * width;
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t row = i / width, j = i - row * width, at = row * H + j, go = row * 4 * H + j;
        if (j >= static_cast<size_t>(H)) {
            out[i] = 0u;
            continue;
        }
        auto bit = [](const uint8_t *m, size_t idx) -> uint32_t { return (m != nullptr && m[idx] != 0) ? 1u : 0u; };
        uint32_t w = bit(mk.hidden_outputs, at) | (bit(mk.cell_tanh_outputs, at) << 1) | (bit(mk.cell_states, at) << 2);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const size_t o = go + static_cast<size_t>(g) * H;
            w |= (bit(mk.gate_outputs, o) << (3 + g)) | (bit(mk.gate_inputs, o) << (7 + g)) |
                 (bit(mk.weight_ih_linear, o) << (11 + g)) | (bit(mk.weight_hh_linear, o) << (15 + g));
        }
        out[i] = w;
    }
}

// The same packing, four hidden units per thread (H a multiple of 4, flag bytes 0 or 1, as every
// forward of this library writes them): 32-bit loads of four flag bytes, byte permutes spread them
// over the 16-bit lanes of two words and a multiply-add moves each pair into its bit position.
// Bits 0..14 are gathered in one pair of words, bits 15..18 in a second pair.
__global__ void packStepMasks4(const rxmet_lstm_backward_masks mk, size_t quads, int H, uint4 *__restrict__ out) {
    for (size_t q = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; q < quads;
         q += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t i = q * 4, row = i / H, j = i % H, go = row * 4 * H + j;
        uint32_t low01 = 0, low23 = 0, high01 = 0, high23 = 0;
        auto add = [](const void *m, size_t at, int pos, uint32_t &a01, uint32_t &a23) {
            const uint32_t w = m ? *reinterpret_cast<const uint32_t *>(static_cast<const uint8_t *>(m) + at) : 0u;
            a01 += __byte_perm(w, 0u, 0x4140) * (1u << pos);
            a23 += __byte_perm(w, 0u, 0x4342) * (1u << pos);
        };
        add(mk.hidden_outputs, i, 0, low01, low23);
        add(mk.cell_tanh_outputs, i, 1, low01, low23);
        add(mk.cell_states, i, 2, low01, low23);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const size_t o = go + static_cast<size_t>(g) * H;
            add(mk.gate_outputs, o, 3 + g, low01, low23);
            add(mk.gate_inputs, o, 7 + g, low01, low23);
            add(mk.weight_ih_linear, o, 11 + g, low01, low23);
            add(mk.weight_hh_linear, o, g, high01, high23);
        }
        out[q] = make_uint4((low01 & 0xffffu) | ((high01 & 0xffffu) << 15), (low01 >> 16) | ((high01 >> 16) << 15),
                            (low23 & 0xffffu) | ((high23 & 0xffffu) << 15), (low23 >> 16) | ((high23 >> 16) << 15));
    }
}

struct RecurrentArgs {
    int T, B, H, smemRows;  // smemRows: leading rows of each gate block held in shared memory
    int smemStride;         // floats between consecutive columns of the transposed copy (odd multiple of 4)
    const uint32_t *stepMasks;  // packed flags [T][B][H] or null
    const float *weightHh;  // real [4H][H]
    const float *c0;
    const float *gateOutputs, *cellStates, *cellTanh;
    const float *gradOutput, *gradFinalHidden, *gradFinalCell;
    Dequant dqC, dqGate[4], dqTanh;
    rxmet_lstm_backward_masks mk;
    float *gIh, *gHh;  // [T][B][4H]
    float *dh0, *dc0;  // [B][H] (masks applied)
};

// Rows of weight_hh that do not fit shared memory are kept in registers: thread (q, j) owns column j
// of the rows of gate q, the first smemRows of them in shared memory and up to kRegRows after that
// in registers, so that a step never goes to L2 for weights.
constexpr int kRegRows = 32;

template <int BT>
__global__ void __launch_bounds__(512) recurrentBackward(const __grid_constant__ RecurrentArgs a) {
    const int H = a.H, C = 4 * a.H, S = a.smemRows, R = H - S;
    extern __shared__ __align__(16) float smemF[];
    float *gS = smemF;               // [BT][C] gradient entering the hh branch
    float *partS = gS + BT * C;      // [4][BT][H] partial sums of dh
    float *wS = partS + 4 * BT * H;  // [4][S][H] leading rows of each gate block of weight_hh
    const int tid = threadIdx.x, nthreads = blockDim.x;
    const int b0 = blockIdx.x * BT, nb = min(BT, a.B - b0);
    // transposed per thread: the S leading rows of column j of gate block g are contiguous (stride SP),
    // so that phase A reads four of them with one 128-bit load
    const int SP = a.smemStride;
    for (int i = tid; i < 4 * S * H; i += nthreads) {
        const int g = i / (S * H), r = (i / H) % S, j = i % H;
        wS[(static_cast<size_t>(g) * H + j) * SP + r] = a.weightHh[(static_cast<size_t>(g) * H + r) * H + j];
    }
    for (int i = tid; i < 4 * BT * H; i += nthreads) partS[i] = 0.0f;
    for (int i = tid; i < BT * C; i += nthreads) gS[i] = 0.0f;

    const int elems = nb * H;
    const bool hasElem = tid < elems;
    const int eb = hasElem ? tid / H : 0, ej = hasElem ? tid % H : 0;
    const size_t stateIdx = static_cast<size_t>(b0 + eb) * H + ej;
    float dhCarry = hasElem ? a.gradFinalHidden[stateIdx] : 0.0f;
    float dc = hasElem ? a.gradFinalCell[stateIdx] : 0.0f;
    // phase A ownership: gate block q of the channels, hidden column j
    const bool hasColumn = tid < C;
    const int q = hasColumn ? tid / H : 0, cj = tid % H;
    float wr[kRegRows];
#pragma unroll
    for (int r = 0; r < kRegRows; ++r)
        wr[r] = (hasColumn && r < R) ? a.weightHh[(static_cast<size_t>(q) * H + S + r) * H + cj] : 0.0f;
    const bool vec = (H % 4 == 0) && (S % 4 == 0) && (SP % 4 == 0);
    __syncthreads();

    // inputs of one step for this thread's element, fetched one step ahead of their use
    struct StepIn {
        float gate[4], ct, cPrev, gradOut;
        uint32_t bits;
    };
    auto fetch = [&](int t, StepIn &in) {
        if (!hasElem) return;
        const size_t row = static_cast<size_t>(t) * a.B + b0 + eb, so = row * H + ej, go = row * C + ej;
#pragma unroll
        for (int g = 0; g < 4; ++g) in.gate[g] = a.gateOutputs[go + static_cast<size_t>(g) * H];
        in.ct = a.cellTanh[so];
        in.cPrev = t > 0 ? a.cellStates[so - static_cast<size_t>(a.B) * H] : (a.c0 ? a.c0[stateIdx] : a.dqC.zeroPoint);
        in.gradOut = a.gradOutput[so];
        in.bits = a.stepMasks ? a.stepMasks[so] : 0u;
    };
    StepIn cur{}, nxt{};
    fetch(a.T - 1, cur);

    for (int t = a.T - 1; t >= 0; --t) {
        const size_t rowBase = static_cast<size_t>(t) * a.B + b0;
        if (t > 0) fetch(t - 1, nxt);
        if (hasElem) {
            const size_t row = rowBase + eb, go = row * C + ej;
            auto keepBit = [&](int b) { return (cur.bits >> b) & 1u ? 0.0f : 1.0f; };
            const float ig = realOf(cur.gate[0], a.dqGate[0]), fg = realOf(cur.gate[1], a.dqGate[1]);
            const float cg = realOf(cur.gate[2], a.dqGate[2]), og = realOf(cur.gate[3], a.dqGate[3]);
            const float ct = realOf(cur.ct, a.dqTanh);
            const float cPrev = realOf(cur.cPrev, a.dqC);
            const float incoming = dhCarry + partS[(0 * BT + eb) * H + ej] + partS[(1 * BT + eb) * H + ej] +
                                   partS[(2 * BT + eb) * H + ej] + partS[(3 * BT + eb) * H + ej];
            const float dh = (incoming + cur.gradOut) * keepBit(0);
            const float gOut = dh * ct;
            const float gTanh = dh * og * keepBit(1);
            const float dcAll = dc + gTanh * (1.0f - ct * ct);
            const float mdc = dcAll * keepBit(2);
            const float go4[4] = {mdc * cg * keepBit(3), mdc * cPrev * keepBit(4), mdc * ig * keepBit(5), gOut * keepBit(6)};
            const float gi4[4] = {go4[0] * ig * (1.0f - ig), go4[1] * fg * (1.0f - fg), go4[2] * (1.0f - cg * cg),
                                  go4[3] * og * (1.0f - og)};
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const size_t o = go + static_cast<size_t>(g) * H;
                const float grad = gi4[g] * keepBit(7 + g);
                const float hh = grad * keepBit(15 + g);
                a.gIh[o] = grad * keepBit(11 + g);
                a.gHh[o] = hh;
                gS[eb * C + g * H + ej] = hh;
            }
            dc = mdc * fg;
            dhCarry = 0.0f;
        }
        cur = nxt;
        __syncthreads();
        if (hasColumn) {
            float acc[BT];
#pragma unroll
            for (int b = 0; b < BT; ++b) acc[b] = 0.0f;
            const float *wq = wS + (static_cast<size_t>(q) * H + cj) * SP;
            const float *gq = gS + q * H;
            if (vec) {
#pragma unroll 4
                for (int r = 0; r < S; r += 4) {
                    const float4 wv = *reinterpret_cast<const float4 *>(wq + r);
#pragma unroll
                    for (int b = 0; b < BT; ++b) {
                        const float4 gv = *reinterpret_cast<const float4 *>(gq + b * C + r);
                        acc[b] = fmaf(gv.x, wv.x, acc[b]);
                        acc[b] = fmaf(gv.y, wv.y, acc[b]);
                        acc[b] = fmaf(gv.z, wv.z, acc[b]);
                        acc[b] = fmaf(gv.w, wv.w, acc[b]);
                    }
                }
#pragma unroll
                for (int r = 0; r < kRegRows; r += 4) {
                    if (r < R) {
#pragma unroll
                        for (int b = 0; b < BT; ++b) {
                            const float4 gv = *reinterpret_cast<const float4 *>(gq + b * C + S + r);
                            acc[b] = fmaf(gv.x, wr[r], acc[b]);
                            acc[b] = fmaf(gv.y, wr[r + 1], acc[b]);
                            acc[b] = fmaf(gv.z, wr[r + 2], acc[b]);
                            acc[b] = fmaf(gv.w, wr[r + 3], acc[b]);
                        }
                    }
                }
            } else {
                for (int r = 0; r < S; ++r) {
                    const float w = wq[r];
#pragma unroll
                    for (int b = 0; b < BT; ++b) acc[b] = fmaf(gq[b * C + r], w, acc[b]);
                }
#pragma unroll
                for (int r = 0; r < kRegRows; ++r) {
                    if (r < R) {
#pragma unroll
                        for (int b = 0; b < BT; ++b) acc[b] = fmaf(gq[b * C + S + r], wr[r], acc[b]);
                    }
                }
            }
#pragma unroll
            for (int b = 0; b < BT; ++b) partS[(q * BT + b) * H + cj] = acc[b];
        }
        __syncthreads();
    }
    if (hasElem) {
        const float dh0 = dhCarry + partS[(0 * BT + eb) * H + ej] + partS[(1 * BT + eb) * H + ej] +
                          partS[(2 * BT + eb) * H + ej] + partS[(3 * BT + eb) * H + ej];
        a.dh0[stateIdx] = dh0 * keepOf(a.mk.initial_hidden, stateIdx);
        a.dc0[stateIdx] = dc * keepOf(a.mk.initial_cell, stateIdx);
    }
}

// ---- hidden sizes above 128 -------------------------------------------------------------------
//
// Thread (j, s) owns hidden unit j for RB batch rows of row group s: the pointwise derivative of its
// elements, then dh[b][j] = sum_c G_hh[b][c] * weight_hh[c][j] with column j of weight_hh streamed
// from L2 (coalesced over j) and the CTA's gate gradients read from shared memory as 16-byte
// broadcasts; dh and dc never leave the thread's registers.
template <int RB>
__global__ void __launch_bounds__(512, 1) recurrentBackwardWide(const __grid_constant__ RecurrentArgs a, const int HP) {
    const int H = a.H, C = 4 * a.H;
    extern __shared__ __align__(16) float smemF[];
    float *gS = smemF;  // [BT][C]
    const int tid = threadIdx.x, j = tid % HP, sg = tid / HP;
    const int BT = (blockDim.x / HP) * RB;
    const bool active = j < H;
    const int b0 = blockIdx.x * BT + sg * RB;
    for (int i = tid; i < BT * C; i += blockDim.x) gS[i] = 0.0f;
    float dhCarry[RB], dc[RB];
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        const bool valid = active && b0 + r < a.B;
        const size_t stateIdx = static_cast<size_t>(b0 + r) * H + j;
        dhCarry[r] = valid ? a.gradFinalHidden[stateIdx] : 0.0f;
        dc[r] = valid ? a.gradFinalCell[stateIdx] : 0.0f;
    }
    __syncthreads();
    for (int t = a.T - 1; t >= 0; --t) {
        if (active) {
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const int b = b0 + r;
                if (b >= a.B) continue;
                const size_t row = static_cast<size_t>(t) * a.B + b, so = row * H + j, go = row * C + j;
                const size_t stateIdx = static_cast<size_t>(b) * H + j;
                const uint32_t bits = a.stepMasks ? a.stepMasks[so] : 0u;
                auto keepBit = [&](int bit) { return (bits >> bit) & 1u ? 0.0f : 1.0f; };
                const float ig = realOf(a.gateOutputs[go], a.dqGate[0]);
                const float fg = realOf(a.gateOutputs[go + static_cast<size_t>(H)], a.dqGate[1]);
                const float cg = realOf(a.gateOutputs[go + 2 * static_cast<size_t>(H)], a.dqGate[2]);
                const float og = realOf(a.gateOutputs[go + 3 * static_cast<size_t>(H)], a.dqGate[3]);
                const float ct = realOf(a.cellTanh[so], a.dqTanh);
                const float cPrevCode = t > 0 ? a.cellStates[so - static_cast<size_t>(a.B) * H]
                                              : (a.c0 ? a.c0[stateIdx] : a.dqC.zeroPoint);
                const float cPrev = realOf(cPrevCode, a.dqC);
                const float dh = (dhCarry[r] + a.gradOutput[so]) * keepBit(0);
                const float gOut = dh * ct;
                const float gTanh = dh * og * keepBit(1);
                const float dcAll = dc[r] + gTanh * (1.0f - ct * ct);
                const float mdc = dcAll * keepBit(2);
                const float go4[4] = {mdc * cg * keepBit(3), mdc * cPrev * keepBit(4), mdc * ig * keepBit(5), gOut * keepBit(6)};
                const float gi4[4] = {go4[0] * ig * (1.0f - ig), go4[1] * fg * (1.0f - fg), go4[2] * (1.0f - cg * cg),
                                      go4[3] * og * (1.0f - og)};
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const size_t o = go + static_cast<size_t>(g) * H;
                    const float grad = gi4[g] * keepBit(7 + g);
                    const float hh = grad * keepBit(15 + g);
                    a.gIh[o] = grad * keepBit(11 + g);
                    a.gHh[o] = hh;
                    gS[(sg * RB + r) * C + g * H + j] = hh;
                }
                dc[r] = mdc * fg;
            }
        }
        __syncthreads();
        if (active) {
            float acc[RB];
#pragma unroll
            for (int r = 0; r < RB; ++r) acc[r] = 0.0f;
            const float *wp = a.weightHh + j;
            const float *gRows = gS + sg * RB * C;
            for (int c = 0; c < C; c += 4) {  // C = 4H is a multiple of 4
                float w[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i] = __ldg(wp + static_cast<size_t>(c + i) * H);
#pragma unroll
                for (int r = 0; r < RB; ++r) {
                    const float4 gv = *reinterpret_cast<const float4 *>(gRows + r * C + c);
                    acc[r] = fmaf(gv.x, w[0], acc[r]);
                    acc[r] = fmaf(gv.y, w[1], acc[r]);
                    acc[r] = fmaf(gv.z, w[2], acc[r]);
                    acc[r] = fmaf(gv.w, w[3], acc[r]);
                }
            }
#pragma unroll
            for (int r = 0; r < RB; ++r) dhCarry[r] = acc[r];
        }
        __syncthreads();
    }
    if (active) {
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            if (b0 + r >= a.B) continue;
            const size_t stateIdx = static_cast<size_t>(b0 + r) * H + j;
            a.dh0[stateIdx] = dhCarry[r] * keepOf(a.mk.initial_hidden, stateIdx);
            a.dc0[stateIdx] = dc[r] * keepOf(a.mk.initial_cell, stateIdx);
        }
    }
}

// Rows of a [rows, cols] operand that switches source after `split` rows (h_prev = [h0 ; hidden[0..T-2]]).
struct RowSource {
    const float *first;  // rows [0, split) ; null = zeros
    const float *rest;   // rows [split, ...) start here
    int split;
    Dequant dq;
    __device__ __forceinline__ float at(int row, int col, int cols) const {
        if (row < split) return first ? realOf(first[static_cast<size_t>(row) * cols + col], dq) : 0.0f;
        return realOf(rest[static_cast<size_t>(row - split) * cols + col], dq);
    }
};

constexpr int kTile = 64, kDepth = 16;

// partial[s][m][n] = sum over the s-th chunk of rows k of G[k][m] * X[k][n].
__global__ void __launch_bounds__(256) gemmRowsTN(const float *__restrict__ G, const RowSource X, int K, int M, int N,
                                                  int chunk, float *__restrict__ partial) {
    __shared__ float As[kDepth][kTile + 4];
    __shared__ float Bs[kDepth][kTile + 4];
    const int m0 = blockIdx.y * kTile, n0 = blockIdx.x * kTile;
    const int kBegin = blockIdx.z * chunk, kEnd = min(K, kBegin + chunk);
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4] = {};
    for (int k0 = kBegin; k0 < kEnd; k0 += kDepth) {
        for (int i = threadIdx.x; i < kDepth * kTile; i += 256) {
            const int kk = i / kTile, c = i % kTile, k = k0 + kk;
            As[kk][c] = (k < kEnd && m0 + c < M) ? G[static_cast<size_t>(k) * M + m0 + c] : 0.0f;
            Bs[kk][c] = (k < kEnd && n0 + c < N) ? X.at(k, n0 + c, N) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kDepth; ++kk) {
            float av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { av[i] = As[kk][ty * 4 + i]; bv[i] = Bs[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    float *out = partial + static_cast<size_t>(blockIdx.z) * M * N;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m < M && n < N) out[static_cast<size_t>(m) * N + n] = acc[i][j];
        }
}

// out[i] = keep[i] * sum_s partial[s][i], s ascending.
__global__ void reduceSplits(const float *__restrict__ partial, int splits, size_t n, const uint8_t *__restrict__ mask,
                             float *__restrict__ out) {
    for (size_t i = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float s = 0.0f;
        for (int p = 0; p < splits; ++p) s += partial[static_cast<size_t>(p) * n + i];
        out[i] = s * keepOf(mask, i);
    }
}

// out[m][n] = keep * sum_k A[m][k] * W[k][n]   (dx = G_ih W_ih: M = T*B, K = 4H, N = I).
__global__ void __launch_bounds__(256) gemmNN(const float *__restrict__ A, const float *__restrict__ W, int M, int N, int K,
                                              const uint8_t *__restrict__ mask, float *__restrict__ out) {
    __shared__ float As[kDepth][kTile + 1];
    __shared__ float Ws[kDepth][kTile + 4];
    const int m0 = blockIdx.x * kTile, n0 = blockIdx.y * kTile;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    float acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += kDepth) {
        for (int i = threadIdx.x; i < kTile * kDepth; i += 256) {
            const int r = i / kDepth, kk = i % kDepth;
            As[kk][r] = (m0 + r < M && k0 + kk < K) ? A[static_cast<size_t>(m0 + r) * K + k0 + kk] : 0.0f;
            const int wk = i / kTile, wc = i % kTile;
            Ws[wk][wc] = (k0 + wk < K && n0 + wc < N) ? W[static_cast<size_t>(k0 + wk) * N + n0 + wc] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kDepth; ++kk) {
            float av[4], bv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) { av[i] = As[kk][ty * 4 + i]; bv[i] = Ws[kk][tx * 4 + i]; }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int m = m0 + ty * 4 + i, n = n0 + tx * 4 + j;
            if (m < M && n < N) {
                const size_t o = static_cast<size_t>(m) * N + n;
                out[o] = acc[i][j] * keepOf(mask, o);
            }
        }
}

// weight[c][m] = scale * keep * sum_s partial[s][m][c] (m < M); bias[c] = keep * sum_s partial[s][M][c]:
// reduces the split-K partials of the tensor-core GEMM and writes the transposed [4H][M] layout.
// A CTA owns 32 channels x 8 rows; its four thread layers each sum every fourth split, and layer 0
// adds the four sums in layer order, so the result does not depend on the launch.
// A set status word (a bounded wait of the producing kernel gave up) turns the results into NaN.
// One launch reduces both problems of a step (blockIdx.z: 0 = weight_ih, 1 = weight_hh).
constexpr int kReduceLayers = 4, kReduceRows = 8;
struct ReduceJob {
    const float *partial;
    int splits, M;
    float scale;
    const uint8_t *weightMask, *biasMask;
    float *weight, *bias;
};
__global__ void __launch_bounds__(32 * kReduceRows * kReduceLayers)
reduceWeightGradT(const ReduceJob jobIh, const ReduceJob jobHh, int C, const int *__restrict__ status) {
    __shared__ float layer[kReduceLayers][kReduceRows][32];
    const ReduceJob &job = blockIdx.z == 0 ? jobIh : jobHh;
    const float *__restrict__ partial = job.partial;
    const int splits = job.splits, M = job.M;
    const float scale = job.scale;
    const uint8_t *__restrict__ weightMask = job.weightMask, *__restrict__ biasMask = job.biasMask;
    float *__restrict__ weight = job.weight, *__restrict__ bias = job.bias;
    waitForPredecessor();
    if (static_cast<int>(blockIdx.y) * kReduceRows > M) return;  // the other problem has more rows
    const size_t slab = static_cast<size_t>(M + 1) * C;
    const int c = blockIdx.x * 32 + threadIdx.x, m = blockIdx.y * kReduceRows + threadIdx.y;
    const bool inside = m <= M && c < C;
    float s = 0.0f;
    if (inside) {
        const float *src = partial + static_cast<size_t>(m) * C + c;
#pragma unroll 4
        for (int sp = threadIdx.z; sp < splits; sp += kReduceLayers) s += src[static_cast<size_t>(sp) * slab];
    }
    layer[threadIdx.z][threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.z != 0 || !inside) return;
    s = layer[0][threadIdx.y][threadIdx.x];
#pragma unroll
    for (int l = 1; l < kReduceLayers; ++l) s += layer[l][threadIdx.y][threadIdx.x];
    if (status && *status) s = __int_as_float(0x7fc00000);
    if (m < M) {
        const size_t o = static_cast<size_t>(c) * M + m;
        weight[o] = s * scale * keepOf(weightMask, o);
    } else if (bias) {
        bias[c] = s * keepOf(biasMask, c);
    }
}

// dx = G_ih W_ih for a narrow N (= input size <= 128): a CTA owns 64 rows, thread (row, quarter) keeps
// NO consecutive outputs in registers and walks K in chunks of 32 staged in shared memory (the G chunk
// transposed so that neighbouring rows read neighbouring banks, the W chunk read as warp-wide
// broadcasts).  The 64x64-tile kernel above wastes a third of its tile at N = 40.
constexpr int kDxRows = 64, kDxChunk = 32;
template <int NO>
__global__ void __launch_bounds__(256) inputGradNarrow(const float *__restrict__ G, const float *__restrict__ W, int M, int N,
                                                       int K, const uint8_t *__restrict__ mask, float *__restrict__ out) {
    __shared__ float Gs[kDxChunk][kDxRows + 1];
    __shared__ __align__(16) float Ws[kDxChunk][4 * NO];
    const int tid = threadIdx.x, r = tid % kDxRows, p = tid / kDxRows;
    const int row0 = blockIdx.x * kDxRows;
    float acc[NO];
#pragma unroll
    for (int i = 0; i < NO; ++i) acc[i] = 0.0f;
    for (int k0 = 0; k0 < K; k0 += kDxChunk) {
#pragma unroll
        for (int v = 0; v < 2; ++v) {
            const int lr = tid / 8 + v * 32, c4 = (tid % 8) * 4;
            float4 g = make_float4(0.f, 0.f, 0.f, 0.f);
            if (row0 + lr < M && k0 + c4 < K) g = *reinterpret_cast<const float4 *>(G + static_cast<size_t>(row0 + lr) * K + k0 + c4);
            Gs[c4][lr] = g.x; Gs[c4 + 1][lr] = g.y; Gs[c4 + 2][lr] = g.z; Gs[c4 + 3][lr] = g.w;
        }
        for (int i = tid; i < kDxChunk * 4 * NO; i += 256) {
            const int kk = i / (4 * NO), n = i % (4 * NO);
            Ws[kk][n] = (k0 + kk < K && n < N) ? W[static_cast<size_t>(k0 + kk) * N + n] : 0.0f;
        }
        __syncthreads();
#pragma unroll 8
        for (int kk = 0; kk < kDxChunk; ++kk) {
            const float g = Gs[kk][r];
#pragma unroll
            for (int i4 = 0; i4 < NO / 4; ++i4) {
                const float4 w = *reinterpret_cast<const float4 *>(&Ws[kk][p * NO + i4 * 4]);
                acc[i4 * 4 + 0] = fmaf(g, w.x, acc[i4 * 4 + 0]);
                acc[i4 * 4 + 1] = fmaf(g, w.y, acc[i4 * 4 + 1]);
                acc[i4 * 4 + 2] = fmaf(g, w.z, acc[i4 * 4 + 2]);
                acc[i4 * 4 + 3] = fmaf(g, w.w, acc[i4 * 4 + 3]);
            }
        }
        __syncthreads();
    }
    const int row = row0 + r;
    if (row >= M) return;
#pragma unroll
    for (int i = 0; i < NO; ++i) {
        const int n = p * NO + i;
        if (n < N) {
            const size_t o = static_cast<size_t>(row) * N + n;
            out[o] = acc[i] * keepOf(mask, o);
        }
    }
}

// partial[which][s][c] = sum over the s-th chunk of rows of g[n][c]; blockIdx.y selects G_ih or G_hh.
__global__ void columnSums(const float *__restrict__ gIh, const float *__restrict__ gHh, int rows, int C, int chunk,
                           float *__restrict__ partial) {
    const float *g = blockIdx.y == 0 ? gIh : gHh;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const int n0 = blockIdx.z * chunk, n1 = min(rows, n0 + chunk);
    float s = 0.0f;
    for (int n = n0; n < n1; ++n) s += g[static_cast<size_t>(n) * C + c];
    partial[(static_cast<size_t>(blockIdx.y) * gridDim.z + blockIdx.z) * C + c] = s;
}

int gridFor(size_t n, int block) { return static_cast<int>(std::min<size_t>((n + block - 1) / block, 148 * 8)); }

int splitsFor(int K, int tiles) {
    const int want = std::max(1, (2 * 148 + tiles - 1) / tiles);
    return std::max(1, std::min(want, (K + 255) / 256));
}
int tilesOf(int M, int N) { return ((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile); }

constexpr int kBiasSplits = 64;
constexpr int kMaxTensorSplits = 40;

}  // namespace

// Splits of the tensor-core weight-gradient partial arrays.
int tensorSplitBound(int rows, int I, int H, int M, int C, bool padded) {
    const int single = M <= 143 ? wgrad::splitBound(rows) : 1;
    return std::max({single, padded ? wgrad::chainPartials(rows) : 1, wgrad::tensorMemoryPath(I, H, C) ? wgrad::tileSplitBound(M, C) : 1});
}

namespace {

// Widths the tensor-core kernels tile: units in tiles of 32, inputs in groups of eight.
int tiledHidden(int H) { return (H + 31) / 32 * 32; }
int tiledInput(int I) { return I % 4 == 0 ? I : (I + 7) / 8 * 8; }

struct PaddedOperands {
    float *wIh, *wHh, *scales, *x, *h0, *c0, *gates, *cells, *tanhs, *hiddens, *gradOut, *gradHidden, *gradCell;
    float *dWIh, *dWHh, *dBIh, *dBHh, *dh0, *dc0;
    uint32_t *flags;
};
template <class W>
PaddedOperands layoutPadded(W &ws, int T, int B, int I, int H) {
    const size_t rows = static_cast<size_t>(T) * B, Hp = tiledHidden(H), Ip = tiledInput(I), C = 4 * Hp, state = static_cast<size_t>(B) * Hp;
    PaddedOperands o{};
    o.wIh = ws.template take<float>(C * I); o.wHh = ws.template take<float>(C * Hp); o.scales = ws.template take<float>(2 * C);
    o.x = ws.template take<float>(rows * Ip);
    o.h0 = ws.template take<float>(state); o.c0 = ws.template take<float>(state);
    o.gates = ws.template take<float>(rows * C); o.cells = ws.template take<float>(rows * Hp); o.tanhs = ws.template take<float>(rows * Hp);
    o.hiddens = ws.template take<float>(rows * Hp); o.gradOut = ws.template take<float>(rows * Hp);
    o.gradHidden = ws.template take<float>(state); o.gradCell = ws.template take<float>(state);
    o.dWIh = ws.template take<float>(C * Ip); o.dWHh = ws.template take<float>(C * Hp);
    o.dBIh = ws.template take<float>(C); o.dBHh = ws.template take<float>(C);
    o.dh0 = ws.template take<float>(state); o.dc0 = ws.template take<float>(state);
    o.flags = ws.template take<uint32_t>(rows * Hp);
    return o;
}
struct PaddedSizer {
    WorkspaceSizer ws;
    template <class T>
    T *take(size_t n) {
        ws.take<T>(n);
        return nullptr;
    }
};

// As backwardPadded of the GRU (gru_backward.cu): widths that no tile divides go through padded copies to the tensor-core
// kernels; the extra units have zero gradients.  T = 100, B = 100, I = 37, H = 150, 16 bits: the step 1893 -> 630 us.
bool paddedTakes(const BackwardCall &call) {
    static const bool disabled = std::getenv("RXMET_LSTM_BWD_SIMT") != nullptr || std::getenv("RXMET_LSTM_WGRAD_SIMT") != nullptr;
    if (disabled || !call.quantized || call.H > 512 || call.I > 512 || !call.weightCodesFitBf16 || !call.weightIhCodesFitBf16 ||
        !call.codesFitTwoTerms || call.h0 == nullptr || call.c0 == nullptr)
        return false;
    if (tiledHidden(call.H) == call.H && tiledInput(call.I) == call.I) return false;
    // dx and weight_ih have the caller's width: only the tensor-core kernel takes them beside operands of the padded one
    if (!igrad::eligible(4 * tiledHidden(call.H), call.I)) return false;
    return alignedTo(call.grads.input, 16) && (call.masks == nullptr || alignedTo(call.masks->input, 8));
}

void backwardPadded(const BackwardCall &call, void *workspace, size_t workspaceBytes, cudaStream_t st) {
    const int T = call.T, B = call.B, I = call.I, H = call.H, Hp = tiledHidden(H), Ip = tiledInput(I);
    const size_t rows = static_cast<size_t>(T) * B;
    const int steps = static_cast<int>(rows);
    const rxmet_lstm_backward_masks none{};
    const rxmet_lstm_backward_masks &mk = call.masks ? *call.masks : none;
    Workspace ws(workspace, workspaceBytes);
    const PaddedOperands o = layoutPadded(ws, T, B, I, H);
    auto copy = [](const void *src, void *dst, int rowGroups, int srcRows, int dstRows, int colGroups, int srcWidth, int dstWidth, float fill = 0.0f) {
        RegroupJob j;
        j.src = src; j.dst = dst; j.rowGroups = rowGroups; j.srcRows = srcRows; j.dstRows = dstRows;
        j.colGroups = colGroups; j.srcWidth = srcWidth; j.dstWidth = dstWidth;
        std::memcpy(&j.fill, &fill, sizeof(fill));
        return j;
    };
    BackwardCall inner = call;
    inner.H = Hp; inner.I = Ip; inner.dxColumns = I;
    inner.weightIh = o.wIh; inner.weightHh = o.wHh; inner.channelScales = o.scales; inner.x = o.x; inner.h0 = o.h0; inner.c0 = o.c0;
    inner.gateOutputs = o.gates; inner.cellStates = o.cells; inner.cellTanhOutputs = o.tanhs; inner.hiddenOutputs = o.hiddens;
    inner.gradOutput = o.gradOut; inner.gradFinalHidden = o.gradHidden; inner.gradFinalCell = o.gradCell;
    inner.grads.weight_ih = o.dWIh; inner.grads.weight_hh = o.dWHh; inner.grads.bias_ih = o.dBIh; inner.grads.bias_hh = o.dBHh;
    inner.grads.initial_hidden = o.dh0; inner.grads.initial_cell = o.dc0;
    const float zeroH = call.dqH.zeroPoint;   // codes of padded inputs and units: real zero
    const bool copyX = Ip != I || !alignedTo(call.x, 16);
    if (!copyX) inner.x = call.x;
    const RegroupJob in[] = {
        copy(call.gateOutputs, o.gates, 1, steps, steps, 4, H, Hp),
        copy(call.cellStates, o.cells, 1, steps, steps, 1, H, Hp),
        copy(call.cellTanhOutputs, o.tanhs, 1, steps, steps, 1, H, Hp),
        copy(call.hiddenOutputs, o.hiddens, 1, steps, steps, 1, H, Hp, zeroH),
        copy(call.gradOutput, o.gradOut, 1, steps, steps, 1, H, Hp),
        copy(call.x, copyX ? o.x : nullptr, 1, steps, steps, 1, I, Ip, call.dqX.zeroPoint),
        copy(call.gradFinalHidden, o.gradHidden, 1, B, B, 1, H, Hp),
        copy(call.gradFinalCell, o.gradCell, 1, B, B, 1, H, Hp),
        copy(call.h0, o.h0, 1, B, B, 1, H, Hp, zeroH),
        copy(call.c0, o.c0, 1, B, B, 1, H, Hp),
        copy(call.weightIh, o.wIh, 4, H, Hp, 1, I, I),
        copy(call.weightHh, o.wHh, 4, H, Hp, 1, H, Hp),
        copy(call.channelScales, o.scales, 1, 2, 2, 4, H, Hp),
    };
    regroup("lstmPadBackward", in, 13, st);
    rxmet_lstm_backward_masks innerMasks{};
    innerMasks.input = mk.input;
    inner.masks = &innerMasks;
    if (mk.hidden_outputs || mk.cell_tanh_outputs || mk.cell_states || mk.gate_outputs || mk.gate_inputs || mk.weight_ih_linear || mk.weight_hh_linear) {
        {
            KernelTimer timer__("lstmPackStepMasks", st);
            packStepMasks<<<gridFor(rows * Hp, 256), 256, 0, st>>>(mk, rows, H, Hp, o.flags);
        }
        afterLaunch("lstmPackStepMasks");
        inner.stepMasks = o.flags;
    }
    const size_t used = alignUp(ws.used(), 256);
    backward(inner, static_cast<char *>(workspace) + used, workspaceBytes - std::min(workspaceBytes, used), st);
    RegroupJob out[] = {
        copy(o.dWIh, call.grads.weight_ih, 4, Hp, H, 1, Ip, I), copy(o.dWHh, call.grads.weight_hh, 4, Hp, H, 1, Hp, H),
        copy(o.dBIh, call.grads.bias_ih, 1, 1, 1, 4, Hp, H), copy(o.dBHh, call.grads.bias_hh, 1, 1, 1, 4, Hp, H),
        copy(o.dh0, call.grads.initial_hidden, 1, B, B, 1, Hp, H), copy(o.dc0, call.grads.initial_cell, 1, B, B, 1, Hp, H),
    };
    const void *masks[] = {mk.weight_ih, mk.weight_hh, mk.bias_ih, mk.bias_hh, mk.initial_hidden, mk.initial_cell};
    for (int k = 0; k < 6; ++k) {
        out[k].mask = static_cast<const uint8_t *>(masks[k]);
        out[k].maskKeeps = 0;
    }
    regroup("lstmPadBackward", out, 6, st);
}

size_t tiledWorkspaceBytes(int T, int B, int I, int H, bool padded) {
    const size_t rows = static_cast<size_t>(T) * B, C = 4 * static_cast<size_t>(H);
    WorkspaceSizer ws;
    ws.take<float>(rows * C);  // G_ih
    ws.take<float>(rows * C);  // G_hh
    ws.take<float>(C * I);     // real weight_ih (QAT)
    ws.take<float>(C * H);     // real weight_hh (QAT)
    ws.take<float>(static_cast<size_t>(splitsFor(static_cast<int>(rows), tilesOf(static_cast<int>(C), I))) * C * I);
    ws.take<float>(static_cast<size_t>(splitsFor(static_cast<int>(rows), tilesOf(static_cast<int>(C), H))) * C * H);
    ws.take<float>(2 * kBiasSplits * C);
    ws.take<float>(rows * H);  // h_prev codes for the tensor-core weight gradient (QAT)
    ws.take<float>(static_cast<size_t>(tensorSplitBound(static_cast<int>(rows), I, H, I, static_cast<int>(C), padded)) * (I + 1) * C);
    ws.take<float>(static_cast<size_t>(tensorSplitBound(static_cast<int>(rows), I, H, H, static_cast<int>(C), padded)) * (H + 1) * C);
    ws.take<int>(1);              // status word of the tensor-memory weight-gradient kernel
    ws.take<uint32_t>(rows * H);  // packed per-step clamp flags
    ws.take<uint8_t>(igrad::packedBytes(static_cast<int>(C), I) + 256);   // weight operand of the input gradient
    return ws.used() + 1024;
}

// 0 where the widths are tiled already or beyond the padded route.
size_t paddedWorkspaceBytes(int T, int B, int I, int H) {
    if (H > 512 || I > 512 || (tiledHidden(H) == H && tiledInput(I) == I)) return 0;
    PaddedSizer sizer;
    layoutPadded(sizer, T, B, I, H);
    return sizer.ws.used() + 512 + tiledWorkspaceBytes(T, B, tiledInput(I), tiledHidden(H), true);
}

}  // namespace

size_t backwardWorkspaceBytes(int T, int B, int I, int H, bool padded) {
    return std::max(tiledWorkspaceBytes(T, B, I, H, false), padded ? paddedWorkspaceBytes(T, B, I, H) : 0);
}

void backward(const BackwardCall &call, void *workspace, size_t workspaceBytes, cudaStream_t st) {
    if (paddedTakes(call) && workspaceBytes >= paddedWorkspaceBytes(call.T, call.B, call.I, call.H)) return backwardPadded(call, workspace, workspaceBytes, st);
    const int T = call.T, B = call.B, I = call.I, H = call.H, C = 4 * H;
    if (H > 512) fail(RXMET_ERR_UNSUPPORTED, "hidden sizes up to 512 are built (got %d)", H);
    const bool wide = C > 512;
    const size_t rows = static_cast<size_t>(T) * B;
    Workspace ws(workspace, workspaceBytes);
    float *gIh = ws.take<float>(rows * C);
    float *gHh = ws.take<float>(rows * C);
    float *wIhReal = ws.take<float>(static_cast<size_t>(C) * I);
    float *wHhReal = ws.take<float>(static_cast<size_t>(C) * H);
    const int splitIh = splitsFor(static_cast<int>(rows), tilesOf(C, I));
    const int splitHh = splitsFor(static_cast<int>(rows), tilesOf(C, H));
    float *partIh = ws.take<float>(static_cast<size_t>(splitIh) * C * I);
    float *partHh = ws.take<float>(static_cast<size_t>(splitHh) * C * H);
    float *partBias = ws.take<float>(2 * kBiasSplits * static_cast<size_t>(C));
    const float *channelScales = call.channelScales;   // weight_ih, weight_hh
    const bool padded = call.dxColumns != 0;   // backwardPadded: as exact as the FP32 kernels that the caller's widths would take
    float *hPrev = ws.take<float>(rows * H);
    float *tensorIh = ws.take<float>(static_cast<size_t>(tensorSplitBound(static_cast<int>(rows), I, H, I, C, padded)) * (I + 1) * C);
    float *tensorHh = ws.take<float>(static_cast<size_t>(tensorSplitBound(static_cast<int>(rows), I, H, H, C, padded)) * (H + 1) * C);
    int *tensorStatus = ws.take<int>(1);
    uint32_t *stepMasks = ws.take<uint32_t>(rows * H);

    // Which kernels multiply by the saved integer weight codes directly (QAT on 8-bit grids); the
    // others read real-valued weights rebuilt here.
    const rxmet_lstm_backward_masks none{};
    const rxmet_lstm_backward_masks &mk = call.masks ? *call.masks : none;
    const bool anyStepMask = mk.hidden_outputs || mk.cell_tanh_outputs || mk.cell_states || mk.gate_outputs ||
                             mk.gate_inputs || mk.weight_ih_linear || mk.weight_hh_linear;
    const bool codes = call.quantized && call.weightCodesFitBf16 && std::getenv("RXMET_LSTM_BWD_SIMT") == nullptr;
    BackwardClusterArgs cl{};
    cl.T = T; cl.B = B; cl.H = H;
    cl.stepMasks = call.stepMasks ? call.stepMasks : anyStepMask ? stepMasks : nullptr;
    cl.weightCodes = call.weightHh; cl.channelScale = channelScales ? channelScales + C : nullptr; cl.c0 = call.c0;
    cl.gateOutputs = call.gateOutputs; cl.cellStates = call.cellStates; cl.cellTanh = call.cellTanhOutputs;
    cl.gradOutput = call.gradOutput; cl.gradFinalHidden = call.gradFinalHidden; cl.gradFinalCell = call.gradFinalCell;
    cl.dqC = call.dqC; cl.dqTanh = call.dqTanh;
    std::copy(call.dqGate, call.dqGate + 4, cl.dqGate);
    cl.maskH0 = static_cast<const uint8_t *>(mk.initial_hidden); cl.maskC0 = static_cast<const uint8_t *>(mk.initial_cell);
    cl.gIh = gIh; cl.gHh = gHh; cl.dh0 = call.grads.initial_hidden; cl.dc0 = call.grads.initial_cell;
    const bool clusterPath = codes && backwardClusterTakes(cl);
    // 16-byte copies of the caller's weight codes, float4 stores of dx and 8-byte loads of the input mask
    const bool tensorInputGrad = call.quantized && call.weightIhCodesFitBf16 && igrad::eligible(C, I) &&
                                 alignedTo(call.grads.input, 16) && alignedTo(call.weightIh, 16) &&
                                 (call.masks == nullptr || alignedTo(call.masks->input, 8));
    const float *wIh = call.weightIh, *wHh = call.weightHh;
    if (call.quantized) {
        RXMET_REQUIRE(channelScales, "per-channel weight scales missing");
        if (!tensorInputGrad) {
            KernelTimer timer__("lstmDequantWeights", st);
            dequantWeights<<<gridFor(static_cast<size_t>(C) * I, 256), 256, 0, st>>>(call.weightIh, channelScales, C, I, wIhReal);
            afterLaunch("lstmDequantWeights");
        }
        if (!clusterPath) {
            KernelTimer timer__("lstmDequantWeights", st);
            dequantWeights<<<gridFor(static_cast<size_t>(C) * H, 256), 256, 0, st>>>(call.weightHh, channelScales + C, C, H, wHhReal);
            afterLaunch("lstmDequantWeights");
        }
        wIh = wIhReal;
        wHh = wHhReal;
    }
    if (anyStepMask) {
        {
            KernelTimer timer__("lstmPackStepMasks", st);
            auto aligned4 = [](const void *ptr) { return (reinterpret_cast<uintptr_t>(ptr) & 3u) == 0; };
            if (H % 4 == 0 && aligned4(mk.hidden_outputs) && aligned4(mk.cell_tanh_outputs) && aligned4(mk.cell_states) &&
                aligned4(mk.gate_outputs) && aligned4(mk.gate_inputs) && aligned4(mk.weight_ih_linear) &&
                aligned4(mk.weight_hh_linear))
                packStepMasks4<<<gridFor(rows * H / 4, 256), 256, 0, st>>>(mk, rows * H / 4, H, reinterpret_cast<uint4 *>(stepMasks));
            else
                packStepMasks<<<gridFor(rows * H, 256), 256, 0, st>>>(mk, rows, H, H, stepMasks);
        }
        afterLaunch("lstmPackStepMasks");
    }
    {
        RecurrentArgs a{};
        a.T = T; a.B = B; a.H = H;
        a.stepMasks = cl.stepMasks;
        a.weightHh = wHh; a.c0 = call.c0;
        a.gateOutputs = call.gateOutputs; a.cellStates = call.cellStates; a.cellTanh = call.cellTanhOutputs;
        a.gradOutput = call.gradOutput; a.gradFinalHidden = call.gradFinalHidden; a.gradFinalCell = call.gradFinalCell;
        a.dqC = call.dqC; a.dqTanh = call.dqTanh;
        for (int g = 0; g < 4; ++g) a.dqGate[g] = call.dqGate[g];
        a.mk = mk; a.gIh = gIh; a.gHh = gHh; a.dh0 = call.grads.initial_hidden; a.dc0 = call.grads.initial_cell;
        const int smemMax = currentDevice().smemMax, sms = currentDevice().sms;
        const int bt = (B >= 4 * sms) ? 4 : ((B > sms) ? 2 : 1);
        const int block = (C + 31) / 32 * 32;
        if (clusterPath) backwardCluster(cl, st);
        else if (wide) {
            const int HP = (H + 31) / 32 * 32;
            const int groupsMax = std::max(1, 512 / HP);
            const int want = std::max(1, (B + smsPerPass() - 1) / smsPerPass());
            int rb = 1;
            while (rb < 8 && rb * groupsMax < want) rb *= 2;
            const int groups = std::max(1, std::min(groupsMax, (want + rb - 1) / rb));
            const int btWide = groups * rb;
            const size_t smem = sizeof(float) * static_cast<size_t>(btWide) * C;
            auto launchWide = [&](auto kernel) {
                ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
                KernelTimer timer__("lstmRecurrentBackwardWide", st);
                kernel<<<(B + btWide - 1) / btWide, groups * HP, smem, st>>>(a, HP);
            };
            if (rb == 1) launchWide(recurrentBackwardWide<1>);
            else if (rb == 2) launchWide(recurrentBackwardWide<2>);
            else if (rb == 4) launchWide(recurrentBackwardWide<4>);
            else launchWide(recurrentBackwardWide<8>);
            afterLaunch("lstmRecurrentBackwardWide");
        }
        auto launch = [&](auto kernel, int BT) {
            if (clusterPath || wide) return;
            const size_t base = sizeof(float) * (static_cast<size_t>(BT) * C + 4 * static_cast<size_t>(BT) * H);
            const size_t room = static_cast<size_t>(smemMax) > base + 1024 ? static_cast<size_t>(smemMax) - base - 1024 : 0;
            // rows per gate block in shared memory; the remaining rows of a block live in registers
            // column stride of the transposed copy: a multiple of 4 floats whose quarter is odd keeps the
            // 128-bit loads of eight neighbouring threads on distinct bank groups
            auto strideFor = [](int rows) {
                int sp = (rows + 3) / 4 * 4;
                if ((sp / 4) % 2 == 0) sp += 4;
                return sp;
            };
            int perGate = (H % 4 == 0) ? H : H / 4 * 4;
            while (perGate > 0 && sizeof(float) * 4 * static_cast<size_t>(H) * strideFor(perGate) > room) perGate -= 4;
            if (perGate < 0) perGate = 0;
            if (H - perGate > kRegRows)
                fail(RXMET_ERR_UNSUPPORTED, "hidden size %d leaves %d weight rows per gate outside shared memory and registers", H, H - perGate);
            a.smemRows = perGate;
            a.smemStride = strideFor(std::max(perGate, 1));
            const size_t smem = base + sizeof(float) * 4 * static_cast<size_t>(H) * a.smemStride;
            ensureDynamicSmem(reinterpret_cast<const void *>(kernel), smem);
            {
                KernelTimer timer__("lstmRecurrentBackward", st);
                kernel<<<(B + BT - 1) / BT, block, smem, st>>>(a);
            }
            afterLaunch("lstmRecurrentBackward");
        };
        if (bt == 4) launch(recurrentBackward<4>, 4);
        else if (bt == 2) launch(recurrentBackward<2>, 2);
        else launch(recurrentBackward<1>, 1);
    }
    if (call.quantized && !tensorInputGrad) RXMET_CUDA(cudaMemsetAsync(tensorStatus, 0, sizeof(int), st));   // the input gradient clears it itself
    if (tensorInputGrad) {
        // QAT: gradients times the integer weight codes on the tensor cores, scales folded into the gradients
        const int sms = currentDevice().sms;
        igrad::Problem pg{};
        pg.G = gIh; pg.kScale = channelScales; pg.codesKN = call.weightIh; pg.rows = static_cast<int>(rows); pg.K = C; pg.N = call.dxColumns ? call.dxColumns : I;
        pg.mask = static_cast<const uint8_t *>(mk.input); pg.maskKeeps = 0; pg.out = call.grads.input; pg.status = pg.clear = tensorStatus;
        if (const size_t bytes = igrad::packedBytes(C, pg.N)) pg.packed = ws.take<uint8_t>(bytes);
        igrad::launch(pg, sms, st);
        afterLaunch("inputGradUmma");
    } else if (I <= 128 && C % 4 == 0) {
        const int perThread = (I + 3) / 4;  // outputs per thread, four threads share a row
        const unsigned grid = static_cast<unsigned>((rows + kDxRows - 1) / kDxRows);
        const uint8_t *inputMask = static_cast<const uint8_t *>(mk.input);
        {
            KernelTimer timer__("lstmInputGradNarrow", st);
            if (perThread <= 4) inputGradNarrow<4><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
            else if (perThread <= 8) inputGradNarrow<8><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
            else if (perThread <= 12) inputGradNarrow<12><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
            else if (perThread <= 16) inputGradNarrow<16><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
            else if (perThread <= 24) inputGradNarrow<24><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
            else inputGradNarrow<32><<<grid, 256, 0, st>>>(gIh, wIh, static_cast<int>(rows), I, C, inputMask, call.grads.input);
        }
        afterLaunch("lstmInputGradNarrow");
    } else {
        {
            KernelTimer timer__("lstmGemmNN", st);
            gemmNN<<<dim3(static_cast<unsigned>((rows + kTile - 1) / kTile), (I + kTile - 1) / kTile), 256, 0, st>>>(
                gIh, wIh, static_cast<int>(rows), I, C, static_cast<const uint8_t *>(mk.input), call.grads.input);
        }
        afterLaunch("lstmGemmNN");
    }
    // QAT: x and h_prev are integer codes, which the tensor-core GEMM multiplies exactly; its ones row also yields the bias gradients.
    // A code is two exact bf16 terms when its grid is wider than 8 bits.
    const bool tensorMemory = wgrad::tensorMemoryPath(I, H, C);
    const bool aligned = call.quantized && I % 4 == 0 && H % 4 == 0 && alignedTo(call.x, 16);
    const bool oneTerm = aligned && call.codesFitTensorPath && I <= 140 && H <= 140 && (!padded || std::max(I, H) <= 128);   // chunks of rows: one kernel for both arrays
    const bool anyTerms = aligned && call.codesFitTwoTerms && (call.h0 || call.dqH.zeroPoint == 0.0f) && tensorMemory && std::getenv("RXMET_LSTM_WGRAD_SIMT") == nullptr;
    if (oneTerm || anyTerms) {
        // a missing h0 means real zeros, i.e. the zero-point code
        if (!call.h0 && call.dqH.zeroPoint != 0.0f) fail(RXMET_ERR_INVALID_ARGUMENT, "the QAT backward needs the quantized initial hidden state");
        const int K = static_cast<int>(rows);
        const bool wideCodes = !call.codesFitTensorPath;
        wgrad::Problem px{}, ph{};
        px.aFloat = call.x; px.aFloatZero = call.dqX.zeroPoint; px.M = I; px.B = gIh; px.partial = tensorIh;
        ph.aFloatZero = call.h0 ? call.dqH.zeroPoint : 0.0f; ph.M = H; ph.B = gHh; ph.partial = tensorHh;
        px.status = ph.status = tensorStatus;
        auto previous = [&] {   // hidden states of the step before as one array
            const size_t stateBytes = sizeof(float) * static_cast<size_t>(B) * H;
            if (call.h0) RXMET_CUDA(cudaMemcpyAsync(hPrev, call.h0, stateBytes, cudaMemcpyDeviceToDevice, st));
            else RXMET_CUDA(cudaMemsetAsync(hPrev, 0, stateBytes, st));
            if (T > 1)
                RXMET_CUDA(cudaMemcpyAsync(hPrev + static_cast<size_t>(B) * H, call.hiddenOutputs, stateBytes * (T - 1), cudaMemcpyDeviceToDevice, st));
            ph.aFloat = hPrev;
            ph.aFirst = nullptr;
            ph.firstRows = 0;
        };
        int splitsX, splitsH;
        if (tensorMemory) {
            if (call.h0 && alignedTo(call.h0, 16) && alignedTo(call.hiddenOutputs, 16)) {   // read where they are
                ph.aFirst = call.h0;   // a copy of all hidden states cost 12 us of a step of T = 100, B = 256, H = 128
                ph.firstRows = B;
                ph.aFloat = call.hiddenOutputs;
            } else {
                previous();
            }
            wgrad::PairPlan plan = wgrad::planPair(px, ph, K, C, wideCodes, currentDevice().sms);
            bool chain = padded && wgrad::planRows(plan) > wgrad::kChainRows;
            if (chain && wgrad::chainChunks(K) > wgrad::kChainGroup) {
                const wgrad::PairPlan fine = wgrad::finePlan(px, ph, K, C, currentDevice().sms);
                if (fine.splits[0] > 0) { plan = fine; chain = false; }
            }
            splitsX = plan.splits[0];
            splitsH = plan.splits[1];
            if (chain) {
                if (ph.aFirst) previous();
                splitsX = splitsH = wgrad::launchChained(px, ph, K, C, wideCodes, st);
            } else {
                wgrad::launchPair(px, ph, K, C, plan, wideCodes, st);
            }
        } else {
            previous();
            wgrad::Plan each = wgrad::plan(K, C, currentDevice().sms);
            if (each.splits > kMaxTensorSplits) {
                each.chunkK = ((K + kMaxTensorSplits - 1) / kMaxTensorSplits + 31) / 32 * 32;
                each.splits = (K + each.chunkK - 1) / each.chunkK;
            }
            splitsX = splitsH = each.splits;
            wgrad::launch(px, K, C, each, st);
            wgrad::launch(ph, K, C, each, st);
        }
        afterLaunch("weightGrad");
        {
            const ReduceJob jobIh{tensorIh, splitsX, I, call.dqX.scale, static_cast<const uint8_t *>(mk.weight_ih),
                                  static_cast<const uint8_t *>(mk.bias_ih), call.grads.weight_ih, call.grads.bias_ih};
            const ReduceJob jobHh{tensorHh, splitsH, H, call.dqH.scale, static_cast<const uint8_t *>(mk.weight_hh),
                                  static_cast<const uint8_t *>(mk.bias_hh), call.grads.weight_hh, call.grads.bias_hh};
            const int rowBlocks = (std::max(I, H) + 1 + kReduceRows - 1) / kReduceRows;
            KernelTimer timer__("lstmReduceWeightGradT", st);
            launchDependent(reduceWeightGradT, dim3((C + 31) / 32, rowBlocks, 2), dim3(32, kReduceRows, kReduceLayers), 0, st, jobIh, jobHh, C, tensorStatus);
        }
        afterLaunch("lstmReduceWeightGradT");
        return;
    }
    auto weightGrad = [&](const float *G, RowSource X, int N, int splits, float *partial, const uint8_t *mask, float *out) {
        const int chunk = ((static_cast<int>(rows) + splits - 1) / splits + kDepth - 1) / kDepth * kDepth;
        {
            KernelTimer timer__("lstmGemmRowsTN", st);
            gemmRowsTN<<<dim3((N + kTile - 1) / kTile, (C + kTile - 1) / kTile, splits), 256, 0, st>>>(
                G, X, static_cast<int>(rows), C, N, chunk, partial);
        }
        afterLaunch("lstmGemmRowsTN");
        {
            KernelTimer timer__("lstmReduceSplits", st);
            reduceSplits<<<gridFor(static_cast<size_t>(C) * N, 256), 256, 0, st>>>(partial, splits, static_cast<size_t>(C) * N, mask, out);
        }
        afterLaunch("lstmReduceSplits");
    };
    weightGrad(gIh, RowSource{call.x, call.x, 0, call.dqX}, I, splitIh, partIh, static_cast<const uint8_t *>(mk.weight_ih),
               call.grads.weight_ih);
    weightGrad(gHh, RowSource{call.h0, call.hiddenOutputs, B, call.dqH}, H, splitHh, partHh,
               static_cast<const uint8_t *>(mk.weight_hh), call.grads.weight_hh);
    if (call.grads.bias_ih || call.grads.bias_hh) {
        const int chunk = (static_cast<int>(rows) + kBiasSplits - 1) / kBiasSplits;
        {
            KernelTimer timer__("lstmColumnSums", st);
            columnSums<<<dim3((C + 127) / 128, 2, kBiasSplits), 128, 0, st>>>(gIh, gHh, static_cast<int>(rows), C, chunk, partBias);
        }
        afterLaunch("lstmColumnSums");
        float *dst[2] = {call.grads.bias_ih, call.grads.bias_hh};
        const uint8_t *msk[2] = {static_cast<const uint8_t *>(mk.bias_ih), static_cast<const uint8_t *>(mk.bias_hh)};
        for (int k = 0; k < 2; ++k) {
            if (!dst[k]) continue;
            {
                KernelTimer timer__("lstmReduceSplits", st);
                reduceSplits<<<gridFor(C, 128), 128, 0, st>>>(partBias + static_cast<size_t>(k) * kBiasSplits * C, kBiasSplits, C, msk[k], dst[k]);
            }
            afterLaunch("lstmReduceSplits");
        }
    }
}

}  // namespace lstm
}  // namespace rxmet
