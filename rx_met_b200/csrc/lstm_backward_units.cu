// Reverse recurrence of the LSTM QAT backward up to 128 units: the cell on top of unit_reverse_umma.cuh.  The arithmetic is that of
// lstm_backward_cluster.cuh, value for value.
#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"
#include "lstm_backward_cluster.h"
#include "unit_reverse_umma.cuh"

namespace rxmet {
namespace lstm {
namespace {

struct LstmReverseCell {
    static constexpr int kGates = 4, kWords = 8;
    BackwardClusterArgs a;
    bool vectors;   // the weight codes lie on a 16-byte boundary

    struct Unit {
        float scale[4];
    };
    struct State {
        float dh, dc;
    };
    // mdc = (dc + dh intoCell) keepCell, gate gradient g = f[g] mdc (f[3] dh), dc of the step before = mdc forget.  The flags 11..18
    // pick where a gate gradient goes.
    struct Factors {
        float f[4], intoCell, keepCell, forget, keepH, grad;
        uint32_t bits;
    };
    struct Out {
        float gate[4];
        uint32_t bits;
    };
    template <int H>
    __device__ __forceinline__ void tile(uint8_t *at, int lane, int m, int gate, int unit) const {   // eight lanes a channel of 32 output units
        const int first = min(m + lane % 8 * 4, H - 4);
        float v[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r) {   // channels 8 (r / 2) + 2 (lane / 8) + r % 2
            const float *src = a.weightCodes + (static_cast<size_t>(gate) * H + unit + r / 2 * 8 + lane / 8 * 2 + r % 2) * H + first;
            if (vectors) {
                const float4 x = __ldg(reinterpret_cast<const float4 *>(src));
                v[r][0] = x.x; v[r][1] = x.y; v[r][2] = x.z; v[r][3] = x.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[r][e] = __ldg(src + e);
            }
        }
#pragma unroll
        for (int r = 0; r < 8; r += 2)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                *reinterpret_cast<uint32_t *>(unitrev::tilePlace(at, lane % 8 * 4 + e, r / 2 * 8 + lane / 8 * 2)) = umma::packBf16(v[r][e], v[r + 1][e]);
    }
    __device__ __forceinline__ Unit unitOf(int unit) const {
        return Unit{{a.channelScale[unit], a.channelScale[a.H + unit], a.channelScale[2 * a.H + unit], a.channelScale[3 * a.H + unit]}};
    }
    __device__ __forceinline__ State begin(int row, int unit) const {
        const size_t o = static_cast<size_t>(row) * a.H + unit;
        return State{a.gradFinalHidden[o], a.gradFinalCell[o]};
    }
    template <uint32_t STRIDE>
    __device__ __forceinline__ void fetch(uint32_t dst, int t, int row, int unit) const {
        const size_t at = (static_cast<size_t>(t) * a.B + row) * a.H + unit;
        const float *gate = a.gateOutputs + (at - unit) * 4 + unit;
#pragma unroll
        for (int g = 0; g < 4; ++g) bwdcluster::copyAsync<4>(dst + g * STRIDE, gate + g * a.H);
        bwdcluster::copyAsync<4>(dst + 4 * STRIDE, a.cellTanh + at);
        bwdcluster::copyAsync<4>(dst + 5 * STRIDE, t > 0 ? a.cellStates + (at - static_cast<size_t>(a.B) * a.H) : a.c0 + at);
        bwdcluster::copyAsync<4>(dst + 6 * STRIDE, a.gradOutput + at);
        if (a.stepMasks) bwdcluster::copyAsync<4>(dst + 7 * STRIDE, a.stepMasks + at);
    }
    template <uint32_t STRIDE>
    __device__ __forceinline__ Factors factors(const uint8_t *from, int) const {
        auto operand = [&](int k) { return *reinterpret_cast<const float *>(from + k * STRIDE); };
        const uint32_t bits = a.stepMasks ? *reinterpret_cast<const uint32_t *>(from + 7 * STRIDE) : 0u;
        auto keep = [&](int pos) { return (bits >> pos) & 1u ? 0.0f : 1.0f; };
        auto real = [](float v, const Dequant &d) { return (v - d.zeroPoint) * d.scale; };
        const float ig = real(operand(0), a.dqGate[0]), fg = real(operand(1), a.dqGate[1]), cg = real(operand(2), a.dqGate[2]), og = real(operand(3), a.dqGate[3]);
        const float ct = real(operand(4), a.dqTanh), cPrev = real(operand(5), a.dqC);
        Factors r;
        r.f[0] = cg * ig * (1.0f - ig) * (keep(3) * keep(7));
        r.f[1] = cPrev * fg * (1.0f - fg) * (keep(4) * keep(8));
        r.f[2] = ig * (1.0f - cg * cg) * (keep(5) * keep(9));
        r.f[3] = ct * og * (1.0f - og) * (keep(6) * keep(10));
        r.intoCell = og * (1.0f - ct * ct) * keep(1);
        r.keepCell = keep(2);
        r.forget = fg;
        r.keepH = keep(0);
        r.grad = operand(6);
        r.bits = bits;
        return r;
    }
    __device__ __forceinline__ void advance(const Unit &u, const Factors &f, State &st, bool alive, float (&b)[4], Out &o) const {
        const float dh = alive ? (st.dh + f.grad) * f.keepH : __int_as_float(0x7fc00000);
        const float mdc = (st.dc + dh * f.intoCell) * f.keepCell;
#pragma unroll
        for (int g = 0; g < 3; ++g) o.gate[g] = f.f[g] * mdc;
        o.gate[3] = f.f[3] * dh;
        st.dc = mdc * f.forget;
        st.dh = 0.0f;
        o.bits = f.bits;
#pragma unroll
        for (int g = 0; g < 4; ++g) b[g] = (f.bits >> (15 + g)) & 1u ? 0.0f : o.gate[g] * u.scale[g];
    }
    __device__ __forceinline__ void store(const Out &o, int t, int row, int unit) const {
        const size_t at = (static_cast<size_t>(t) * a.B + row) * (4 * static_cast<size_t>(a.H)) + unit;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            a.gIh[at + g * a.H] = (o.bits >> (11 + g)) & 1u ? 0.0f : o.gate[g];
            a.gHh[at + g * a.H] = (o.bits >> (15 + g)) & 1u ? 0.0f : o.gate[g];
        }
    }
    __device__ __forceinline__ void finish(const State &st, int row, int unit, bool alive) const {
        const size_t o = static_cast<size_t>(row) * a.H + unit;
        auto keep = [&](const uint8_t *mask) { return mask == nullptr || mask[o] == 0 ? 1.0f : 0.0f; };
        const float bad = alive ? 0.0f : __int_as_float(0x7fc00000);
        a.dh0[o] = st.dh * keep(a.maskH0) + bad;
        a.dc0[o] = st.dc * keep(a.maskC0) + bad;
    }
};

}  // namespace

void backwardUnits(const BackwardClusterArgs &args, cudaStream_t st) {
    const LstmReverseCell cell{args, alignedTo(args.weightCodes, 16)};
    const unitrev::Problem p{args.T, args.B};
    const char *name = "lstmRecurrentBackwardCluster";
    switch (args.H) {
        case 32: return unitrev::launchRows<32>(name, p, cell, st);
        case 64: return unitrev::launchRows<64>(name, p, cell, st);
        case 96: return unitrev::launchRows<96>(name, p, cell, st);
        default: return unitrev::launchRows<128>(name, p, cell, st);
    }
}

}  // namespace lstm
}  // namespace rxmet
