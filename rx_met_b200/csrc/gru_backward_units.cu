// Reverse recurrence of the QuantGRU QAT backward up to 128 units: the cell on top of unit_reverse_umma.cuh.  The arithmetic is that
// of gru_backward_cluster.cu, value for value.
#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"
#include "gru_backward_cluster.h"
#include "unit_reverse_umma.cuh"

namespace rxmet {
namespace gru {
namespace {

struct GruReverseCell {
    static constexpr int kGates = 3, kWords = 7;
    BackwardQArgs a;
    const int32_t *Rq;   // [H][3H] codes

    struct Unit {
        float scale[3];
    };
    struct State {
        float dh;
    };
    // Every gradient of a step is linear in the incoming dh.  p: gate-input gradients of the input branch, q: of the recurrent branch.
    struct Factors {
        float p[3], q[3], z, keep, dh;
    };
    struct Out {
        float p[3], q[3];
    };
    template <int H>
    __device__ __forceinline__ void tile(uint8_t *at, int lane, int m, int gate, int unit) const {   // eight lanes a row of 32 codes
        int4 v[8];
#pragma unroll
        for (int r = 0; r < 8; ++r)
            v[r] = __ldg(reinterpret_cast<const int4 *>(Rq + static_cast<size_t>(min(m + 4 * r + lane / 8, H - 1)) * (3 * H) + gate * H + unit) + lane % 8);
#pragma unroll
        for (int r = 0; r < 8; ++r)
            *reinterpret_cast<uint2 *>(unitrev::tilePlace(at, 4 * r + lane / 8, lane % 8 * 4)) =
                make_uint2(umma::packBf16(static_cast<float>(v[r].x), static_cast<float>(v[r].y)), umma::packBf16(static_cast<float>(v[r].z), static_cast<float>(v[r].w)));
    }
    __device__ __forceinline__ Unit unitOf(int unit) const { return Unit{{a.scaleR[unit], a.scaleR[a.H + unit], a.scaleR[2 * a.H + unit]}}; }
    __device__ __forceinline__ State begin(int row, int unit) const { return State{a.dhIn ? a.dhIn[static_cast<size_t>(row) * a.H + unit] : 0.0f}; }
    template <uint32_t STRIDE>
    __device__ __forceinline__ void fetch(uint32_t dst, int t, int row, int unit) const {
        const size_t at = (static_cast<size_t>(t) * a.B + row) * a.H + unit;
        const float *v = a.v + (at - unit) * 4 + unit;
#pragma unroll
        for (int g = 0; g < 4; ++g) bwdcluster::copyAsync<4>(dst + g * STRIDE, v + g * a.H);
        bwdcluster::copyAsync<4>(dst + 4 * STRIDE, a.h + at);
        bwdcluster::copyAsync<4>(dst + 5 * STRIDE, a.dhNew + at + static_cast<size_t>(a.B) * a.H);
        if (a.stepBits) bwdcluster::copyAsync<4>(dst + 6 * STRIDE, a.stepBits + (at & ~static_cast<size_t>(1)));   // of a pair of units
    }
    template <uint32_t STRIDE>
    __device__ __forceinline__ Factors factors(const uint8_t *from, int unit) const {
        auto operand = [&](int k) { return *reinterpret_cast<const float *>(from + k * STRIDE); };
        const uint32_t pair = a.stepBits ? *reinterpret_cast<const uint32_t *>(from + 6 * STRIDE) : 0x1fff1fffu, bits = unit & 1 ? pair >> 16 : pair;
        auto keep = [&](int pos) { return static_cast<float>((bits >> pos) & 1u); };
        const float z = operand(0), r = operand(1), g = operand(2), qg = operand(3), hOld = operand(4);
        Factors f;
        f.z = z;
        f.keep = keep(12);
        f.dh = operand(5);
        const float fn = ((1.0f - g * g) * (1.0f - z)) * (keep(2) * keep(5));
        const float fr = ((r * (1.0f - r)) * (fn * qg)) * (keep(1) * keep(4));
        const float fz = ((z * (1.0f - z)) * (hOld - g)) * (keep(0) * keep(3));
        f.p[0] = fz * keep(9); f.p[1] = fr * keep(10); f.p[2] = fn * keep(11);
        f.q[0] = fz * keep(6); f.q[1] = fr * keep(7); f.q[2] = (fn * r) * keep(8);
        return f;
    }
    __device__ __forceinline__ void advance(const Unit &u, const Factors &f, State &st, bool alive, float (&b)[3], Out &o) const {
        const float dh = alive ? (f.dh + st.dh) * f.keep : __int_as_float(0x7fc00000);
        st.dh = f.z * dh;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            o.p[g] = f.p[g] * dh;
            o.q[g] = f.q[g] * dh;
            b[g] = o.q[g] * u.scale[g];
        }
    }
    __device__ __forceinline__ void store(const Out &o, int t, int row, int unit) const {
        const size_t at = (static_cast<size_t>(t) * a.B + row) * (3 * static_cast<size_t>(a.H)) + unit;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            a.dp[at + g * a.H] = o.p[g];
            a.dq[at + g * a.H] = o.q[g];
        }
    }
    __device__ __forceinline__ void finish(const State &st, int row, int unit, bool alive) const {
        const size_t o = static_cast<size_t>(row) * a.H + unit;
        const float keep = !a.carryOut && a.mH0 ? static_cast<float>(a.mH0[o]) : 1.0f;
        a.dh0[o] = st.dh * keep + (alive ? 0.0f : __int_as_float(0x7fc00000));
    }
};

}  // namespace

void backwardUnits(const BackwardQArgs &q, const int32_t *Rq, cudaStream_t st) {
    const GruReverseCell cell{q, Rq};
    const unitrev::Problem p{q.T, q.B};
    switch (q.H) {
        case 32: return unitrev::launchRows<32>("recurrentBackward", p, cell, st);
        case 64: return unitrev::launchRows<64>("recurrentBackward", p, cell, st);
        case 96: return unitrev::launchRows<96>("recurrentBackward", p, cell, st);
        default: return unitrev::launchRows<128>("recurrentBackward", p, cell, st);
    }
}

}  // namespace gru
}  // namespace rxmet
