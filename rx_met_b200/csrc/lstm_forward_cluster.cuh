// Wide QuantLSTM recurrence (weights <= 8 bits, activations of 9 to 16 bits, H <= 512) over thread-block clusters: the float
// q-carrier cell on top of plane_recurrence_umma.cuh.
//
// Every float rounding that decides a code is the reference's, value for value; what is cheaper than in the one-CTA kernels:
//  - activations come from the compact tables (a line per segment and a bit per input) in shared memory: two shared loads and
//    about fifteen instructions, where the full tables are gathers of one sector per lane from L2 - they bounded the large
//    batches and put two L2 round trips into the chain of every step;
//  - sums that provably fit 32 bits are combined in one multiply-add and converted once;
//  - rounding to an integer that is clamped to a grid below 2^22 adds and subtracts 1.5 * 2^23 (clamp first: the limits are
//    integers, so the order does not matter; a training forward clamps one step wider, which keeps the clamp flags).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

#include "common.h"
#include "lstm_device.cuh"
#include "lstm_kernels.h"
#include "plane_recurrence_umma.cuh"
#include "unit_recurrence_umma.cuh"

namespace rxmet {
namespace lstm {

constexpr float kRoundMagic = 12582912.0f;   // 1.5 * 2^23
__device__ __forceinline__ float roundSmall(float x) { return __fadd_rn(__fadd_rn(x, kRoundMagic), -kRoundMagic); }
__device__ __forceinline__ float clampF(float x, float lo, float hi) { return fminf(fmaxf(x, lo), hi); }

// Addresses and constants of one compact table, ready for lookup().
struct TableView {
    uint32_t segments, bits;   // shared addresses, moved by the exponent bits that an index carries
    float toIndex;             // x + toIndex = 2^23 + index
    float outLo, outHi;
};
__device__ __forceinline__ float lookup(const TableView &v, int segShift, float x, uint32_t &index) {
    index = __float_as_uint(__fadd_rn(x, v.toIndex));
    float slope, intercept;
    asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(slope), "=f"(intercept) : "r"(v.segments + ((index >> segShift) << 3)));
    uint32_t word;
    asm("ld.shared.u32 %0, [%1];" : "=r"(word) : "r"(v.bits + ((index >> 5) << 2)));
    // the bit of an input is bit 31 - (index & 31): shifted to the top it is added to the rounded value's last place, which is 1
    const uint32_t rounded = __float_as_uint(__fadd_rn(__fmaf_rn(slope, x, intercept), kRoundMagic)) + (__funnelshift_l(0u, word, index) >> 31);
    return clampF(__fadd_rn(__uint_as_float(rounded), -kRoundMagic), v.outLo, v.outHi);
}

// WIDTH: the hidden size where it is a compile-time constant, else 0.
template <bool TRAIN, int WIDTH = 0>
struct LstmPlaneCell {
    static constexpr int kGates = 4;
    static constexpr bool kSaves = TRAIN, kFull = WIDTH != 0;
    static constexpr int kChunk = TRAIN ? 4 : 16, kTotalFrom = 8;
    ScalarExec s;
    int width, kWords;
    __device__ __forceinline__ int hidden() const { return WIDTH ? WIDTH : width; }
    size_t B;
    int segShift, tableBytes;
    int segOffset[kTables], bitOffset[kTables], flagBelow[kTables], flagFrom[kTables];
    float inLo[kTables], outLo[kTables], outHi[kTables];
    const uint8_t *tables;
    const uint2 *words;        // [2 gate pairs][kWords][H]: (x, y) = gates (2 * pair, 2 * pair + 1)
    const int64_t *addend;     // [4H]
    const float *channel;
    const float *lhs;          // [T][B][4H]
    const float *c0;           // [B][H] centred cell codes
    float *output, *finalHidden, *finalCell;
    rxmet_lstm_trace ck;
    const int *poison;         // status word of the tensor-core projection: non-zero turns the outputs into NaN

    struct Lane {
        int64_t addend;
        float outScale, gateScale, giLo, giHi;   // multiplier times power of two: as exact as one after the other
        TableView table;
        float zpIn, zpOut;               // zero points and clamp limits that storeLinear needs
        int flagBelow, flagFrom;
        bool narrow;   // warp-uniform: the sum fits 32 bits
    };
    struct State {
        float cell, hidden, tanhC;
        uint32_t flags;   // clamped: bit 0 cell state, 1 tanh, 2 hidden
    };
    struct Fetch {
        float lhs;
    };
    struct FetchB {};
    struct Saved {
        float hh, gateIn, gateOut;
        uint32_t index;   // of the gate input in its table
        bool hhClamped, inClamped;
    };

    size_t sharedBytes() const { return static_cast<size_t>(tableBytes); }

    __device__ __forceinline__ uint32_t weightWord(int gate, int unit, int kw) const {
        const int H = hidden();
        const uint2 pair = __ldg(words + (static_cast<size_t>(gate >> 1) * kWords + kw) * H + unit);
        return (gate & 1) ? pair.y : pair.x;
    }
    __device__ __forceinline__ void init(uint8_t *shared, int tid, int threads) const {
        for (int i = tid; i < tableBytes / 16; i += threads)
            reinterpret_cast<uint4 *>(shared)[i] = __ldg(reinterpret_cast<const uint4 *>(tables) + i);
    }
    __device__ __forceinline__ TableView view(uint32_t shared, int t) const {
        constexpr uint32_t kExponent = 0x4B000000u;   // of 2^23
        return TableView{shared + segOffset[t] - ((kExponent >> segShift) << 3), shared + bitOffset[t] - ((kExponent >> 5) << 2),
                         8388608.0f - inLo[t], outLo[t], outHi[t]};
    }
    __device__ __forceinline__ Lane lane(uint32_t shared, int gate, int unit, bool real) const {
        const int H = hidden();
        Lane l;
        const int c = gate * H + unit, opIn = RXMET_LSTM_INPUT_GATE_INPUT + gate;
        const size_t C = 4 * static_cast<size_t>(H);
        l.addend = real ? addend[c] : 0;
        l.outScale = real ? __fmul_rn(channel[kHhOutMult * C + c], channel[kHhOutPow2 * C + c]) : 0.0f;
        l.gateScale = __fmul_rn(s.hhToGate[gate].mult, s.hhToGate[gate].pow2);
        l.giLo = static_cast<float>(s.lo[opIn] - s.zp[opIn]);
        l.giHi = static_cast<float>(s.hi[opIn] - s.zp[opIn]);
        l.table = view(shared, gate);
        l.zpIn = s.zpF[opIn];
        l.zpOut = s.zpF[RXMET_LSTM_INPUT_GATE_OUTPUT + gate];
        l.flagBelow = flagBelow[gate];
        l.flagFrom = flagFrom[gate];
        const int64_t wMax = max(-static_cast<int64_t>(s.lo[RXMET_LSTM_WEIGHT_HH]), static_cast<int64_t>(s.hi[RXMET_LSTM_WEIGHT_HH]));
        l.narrow = __all_sync(0xffffffffu, wMax * 65535 * H + llabs(l.addend) < (int64_t{1} << 31));
        return l;
    }
    // whether the projection before it went through; asked once, before the first step
    __device__ __forceinline__ bool valid() const { return poison == nullptr || *poison == 0; }
    __device__ __forceinline__ float scaleH(bool good) const { return good ? s.scale[RXMET_LSTM_OUTPUT] : __int_as_float(0x7fc00000); }
    // centred limits of an operator's grid
    __device__ __forceinline__ float lowOf(int op) const { return static_cast<float>(s.lo[op] - s.zp[op]); }
    __device__ __forceinline__ float highOf(int op) const { return static_cast<float>(s.hi[op] - s.zp[op]); }
    // clamp(rint(x)) on a grid of integers below 2^22 and, where it is saved, whether it clamped
    __device__ __forceinline__ float quantized(float x, float lo, float hi, bool &clamped) const {
        if (TRAIN) {
            const float r = roundSmall(clampF(x, lo - 1.0f, hi + 1.0f));
            clamped = r < lo || r > hi;
            return clampF(r, lo, hi);
        }
        clamped = false;
        return roundSmall(clampF(x, lo, hi));
    }

    __device__ __forceinline__ void begin(uint32_t, State &st, int row, int unit) const {
        const int H = hidden();
        st.cell = c0[static_cast<size_t>(row) * H + unit];
        st.hidden = st.tanhC = 0.0f;
        st.flags = 0;
    }
    __device__ __forceinline__ void fetch(Fetch &f, size_t at, uint32_t row, int gate, int unit) const {
        const int H = hidden();
        f.lhs = __ldg(lhs + at * (4 * static_cast<size_t>(H)) + (row * (4 * H) + gate * H + unit));
    }
    // the same for the rows of a thread: 64 bits all along, so that the rows are immediates of one address
    __device__ __forceinline__ void fetchRow(Fetch &f, size_t at, int row, int gate, int unit) const {
        const int H = hidden();
        f.lhs = __ldg(lhs + (at + static_cast<size_t>(row)) * (4 * static_cast<size_t>(H)) + (gate * H + unit));
    }
    __device__ __forceinline__ void fetchB(FetchB &, size_t, uint32_t, int) const {}
    // the sum of the planes as a float; NARROW: it fits 32 bits
    template <int PLANES, bool NARROW>
    __device__ __forceinline__ uint32_t total(const Lane &l, uint32_t high, uint32_t low) const {
        if (NARROW) return __float_as_uint(__int2float_rn(static_cast<int32_t>((PLANES == 2 ? high * 256u : 0u) + low + static_cast<uint32_t>(l.addend))));
        return __float_as_uint(__ll2float_rn((PLANES == 2 ? static_cast<int64_t>(static_cast<int32_t>(high)) << 8 : 0) + static_cast<int32_t>(low) + l.addend));
    }
    // the same for ROWS rows, in place of the plane sums; one branch for all of them
    template <int STRIDE, int ROWS>
    __device__ __forceinline__ void totals(const Lane &l, uint32_t *acc) const {
        if (l.narrow) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = total<2, true>(l, acc[r], acc[r + STRIDE]);
        } else {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = total<2, false>(l, acc[r], acc[r + STRIDE]);
        }
    }
    // gate output (centred code as a float)
    template <int STRIDE>
    __device__ __forceinline__ uint32_t linear(uint32_t shared, const Lane &l, const Fetch &in, const uint32_t *acc, Saved &saved) const {
        uint32_t sums[STRIDE + 1] = {acc[0]};
        sums[STRIDE] = acc[STRIDE];
        totals<STRIDE, 1>(l, sums);
        return linearOfTotal(shared, l, in, sums[0], saved);
    }
    __device__ __forceinline__ uint32_t linearOfTotal(uint32_t, const Lane &l, const Fetch &in, uint32_t sum32, Saved &saved) const {
        const float total = __uint_as_float(sum32);
        bool hhClamped;
        const float hh = quantized(__fmul_rn(total, l.outScale), lowOf(RXMET_LSTM_WEIGHT_HH_LINEAR),
                                   highOf(RXMET_LSTM_WEIGHT_HH_LINEAR), hhClamped);
        const float sum = __fadd_rn(in.lhs, roundSmall(__fmul_rn(hh, l.gateScale)));
        const float gateIn = clampF(sum, l.giLo, l.giHi);
        uint32_t index;
        const float gateOut = lookup(l.table, segShift, gateIn, index);
        if (TRAIN) saved = Saved{hh, gateIn, gateOut, index, hhClamped, sum < l.giLo || sum > l.giHi};
        return __float_as_uint(gateOut);
    }
    __device__ __forceinline__ uint32_t cell(uint32_t shared, State &st, const FetchB &, const uint32_t (&v)[4]) const {
        const float gI = __uint_as_float(v[0]), gF = __uint_as_float(v[1]), gG = __uint_as_float(v[2]), gO = __uint_as_float(v[3]);
        const float pf = __fmul_rn(gF, st.cell), pi = __fmul_rn(gI, gG);
        const float sf = dev::scaleCell(pf, s.forgetRatio, s.forgetMantissa, s.forgetExponent, s.forgetUsesFp);
        const float si = dev::scaleCell(pi, s.inputRatio, s.inputMantissa, s.inputExponent, s.inputUsesFp);
        bool cellClamped, hiddenClamped;
        st.cell = quantized(__fadd_rn(sf, si), lowOf(RXMET_LSTM_CELL_STATE), highOf(RXMET_LSTM_CELL_STATE), cellClamped);
        uint32_t index;
        st.tanhC = lookup(view(shared, 4), segShift, st.cell, index);
        st.hidden = quantized(__fmul_rn(__fmul_rn(gO, st.tanhC), __fmul_rn(s.productToOutput.mult, s.productToOutput.pow2)), lowOf(RXMET_LSTM_OUTPUT),
                              highOf(RXMET_LSTM_OUTPUT), hiddenClamped);
        if (TRAIN) st.flags = (cellClamped ? 1u : 0u) | (clampFlag(4, index) ? 2u : 0u) | (hiddenClamped ? 4u : 0u);
        return __float_as_uint(__fadd_rn(st.hidden, 8388608.0f + static_cast<float>(s.zp[RXMET_LSTM_OUTPUT] - s.lo[RXMET_LSTM_OUTPUT]))) & 0xffffu;
    }
    __device__ __forceinline__ bool clampFlag(int t, uint32_t index) const {
        const int i = static_cast<int>(index & 0x7fffffu);
        return i < flagBelow[t] || i >= flagFrom[t];
    }
    __device__ __forceinline__ void store(const State &st, const FetchB &, size_t at, uint32_t row, int unit, bool good) const {
        const int H = hidden();
        const size_t o = at * H + (row * H + unit);
        output[o] = __fmul_rn(st.hidden, scaleH(good));
        if (TRAIN) {
            if (ck.cell_states) ck.cell_states[o] = st.cell + s.zpF[RXMET_LSTM_CELL_STATE];
            if (ck.cell_states_clamped) ck.cell_states_clamped[o] = static_cast<uint8_t>(st.flags & 1u);
            if (ck.cell_tanh_outputs) ck.cell_tanh_outputs[o] = st.tanhC + s.zpF[RXMET_LSTM_CELL_TANH_OUTPUT];
            if (ck.cell_tanh_outputs_clamped) ck.cell_tanh_outputs_clamped[o] = static_cast<uint8_t>((st.flags >> 1) & 1u);
            if (ck.hidden_outputs) ck.hidden_outputs[o] = st.hidden + s.zpF[RXMET_LSTM_OUTPUT];
            if (ck.hidden_outputs_clamped) ck.hidden_outputs_clamped[o] = static_cast<uint8_t>((st.flags >> 2) & 1u);
        }
    }
    // The same for `count` of N consecutive rows: one address and one test per array.
    template <int N>
    __device__ __forceinline__ void storeRows(const State (&st)[N], const FetchB (&)[N], size_t at, int row, int unit, bool good, int count) const {
        const int H = hidden();
        const size_t o = (at + static_cast<size_t>(row)) * H + unit;
        auto put = [&](auto *to, auto value) {
            if (to == nullptr) return;
            to += o;
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i < count) to[static_cast<size_t>(i) * H] = value(st[i]);
        };
        const float scale = scaleH(good);
        put(output, [&](const State &v) { return __fmul_rn(v.hidden, scale); });
        if (!TRAIN) return;
        const float zpCell = s.zpF[RXMET_LSTM_CELL_STATE], zpTanh = s.zpF[RXMET_LSTM_CELL_TANH_OUTPUT], zpHidden = s.zpF[RXMET_LSTM_OUTPUT];
        put(ck.cell_states, [&](const State &v) { return v.cell + zpCell; });
        put(ck.cell_states_clamped, [&](const State &v) { return static_cast<uint8_t>(v.flags & 1u); });
        put(ck.cell_tanh_outputs, [&](const State &v) { return v.tanhC + zpTanh; });
        put(ck.cell_tanh_outputs_clamped, [&](const State &v) { return static_cast<uint8_t>((v.flags >> 1) & 1u); });
        put(ck.hidden_outputs, [&](const State &v) { return v.hidden + zpHidden; });
        put(ck.hidden_outputs_clamped, [&](const State &v) { return static_cast<uint8_t>((v.flags >> 2) & 1u); });
    }
    template <int N>
    __device__ __forceinline__ void storeLinearRows(const Lane &l, const Saved (&saved)[N], size_t at, int row, int gate, int unit, int count) const {
        const int H = hidden();
        const size_t o = (at + static_cast<size_t>(row)) * (4 * static_cast<size_t>(H)) + (gate * H + unit);
        auto put = [&](auto *to, auto value) {
            if (to == nullptr) return;
            to += o;
#pragma unroll
            for (int i = 0; i < N; ++i)
                if (i < count) to[static_cast<size_t>(i) * (4 * H)] = value(saved[i]);
        };
        const float zpLinear = s.zpF[RXMET_LSTM_WEIGHT_HH_LINEAR];
        put(ck.weight_hh_linear, [&](const Saved &v) { return v.hh + zpLinear; });
        put(ck.weight_hh_linear_clamped, [&](const Saved &v) { return static_cast<uint8_t>(v.hhClamped); });
        put(ck.gate_inputs, [&](const Saved &v) { return v.gateIn + l.zpIn; });
        put(ck.gate_inputs_clamped, [&](const Saved &v) { return static_cast<uint8_t>(v.inClamped); });
        put(ck.gate_outputs, [&](const Saved &v) { return v.gateOut + l.zpOut; });
        put(ck.gate_outputs_clamped, [&](const Saved &v) {
            const int index = static_cast<int>(v.index & 0x7fffffu);
            return static_cast<uint8_t>(index < l.flagBelow || index >= l.flagFrom);
        });
    }
    __device__ __forceinline__ void storeLinear(const Lane &l, const Saved &v, size_t at, uint32_t row, int gate, int unit) const {
        const int H = hidden();
        const size_t o = at * (4 * static_cast<size_t>(H)) + (row * (4 * H) + gate * H + unit);
        const int index = static_cast<int>(v.index & 0x7fffffu);
        if (ck.weight_hh_linear) ck.weight_hh_linear[o] = v.hh + s.zpF[RXMET_LSTM_WEIGHT_HH_LINEAR];
        if (ck.weight_hh_linear_clamped) ck.weight_hh_linear_clamped[o] = v.hhClamped;
        if (ck.gate_inputs) ck.gate_inputs[o] = v.gateIn + l.zpIn;
        if (ck.gate_inputs_clamped) ck.gate_inputs_clamped[o] = v.inClamped;
        if (ck.gate_outputs) ck.gate_outputs[o] = v.gateOut + l.zpOut;
        if (ck.gate_outputs_clamped) ck.gate_outputs_clamped[o] = index < l.flagBelow || index >= l.flagFrom;
    }
    __device__ __forceinline__ void finish(const State &st, int row, int unit, bool good) const {
        const int H = hidden();
        const size_t o = static_cast<size_t>(row) * H + unit;
        finalHidden[o] = __fmul_rn(st.hidden, scaleH(good));
        finalCell[o] = __fmul_rn(st.cell, good ? s.scale[RXMET_LSTM_CELL_STATE] : __int_as_float(0x7fc00000));
    }
};

// What a forward saves beside its outputs: nothing, some of the checkpoints, all of them.
enum class Saves { None, Some, All };

// The same cell with all gates of a unit in one thread (unit_recurrence_umma.cuh), one or two byte planes.  What is the same for all
// units is prepared on the host and read as constants: registers of a thread decide how many rows an SM has in flight.
struct LstmUnitConstants {
    struct Table {
        float toIndex, outLo, outHi;
        uint32_t segments, bits;          // offsets, moved by the exponent bits that an index carries
        uint32_t flagBelow, flagCount;    // clamped: index - flagBelow >= flagCount
    } table[kTables];
    float gateScale[4], giLo[4], giHi[4], zpIn[4], zpOut[4];
    float hhLo, hhHi, cLo, cHi, oLo, oHi, productScale, codePlus;
    int plain;                            // the cell's ratios are single factors
};
template <Saves SAVES, int PLANES, int WIDTH = 0>
struct LstmUnitCell : LstmPlaneCell<SAVES != Saves::None, WIDTH> {
    static constexpr bool kTrain = SAVES != Saves::None, kTwoRows = !kTrain, kSignedCodes = false;
    using Base = LstmPlaneCell<kTrain, WIDTH>;
    LstmUnitConstants k;
    struct Unit {
        int64_t addend[4];
        float outScale[4];
        bool narrow[4], plain;            // uniform in the warp: the sum fits 32 bits; all of them and k.plain
        uint32_t shared;
    };
    struct State {
        float cell, hidden;
    };
    struct Fetch {
        float lhs[4];
    };
    struct Out {
        float hh[4], sum[4], gate[4];   // hh before its clamp, gate input before its clamp, gate output
        uint32_t index[5];
        float cellRaw, cell, tanhC, hiddenRaw, hidden;   // Raw: before the clamp
    };
    // host: everything of k from the fields of the base
    void prepareConstants() {
        const auto &s = this->s;
        auto low = [&](int op) { return static_cast<float>(s.lo[op] - s.zp[op]); };
        auto high = [&](int op) { return static_cast<float>(s.hi[op] - s.zp[op]); };
        constexpr uint32_t kExponent = 0x4B000000u;   // of 2^23
        for (int t = 0; t < kTables; ++t)
            k.table[t] = {8388608.0f - this->inLo[t], this->outLo[t], this->outHi[t], static_cast<uint32_t>(this->segOffset[t]) - ((kExponent >> this->segShift) << 3),
                          static_cast<uint32_t>(this->bitOffset[t]) - ((kExponent >> 5) << 2), kExponent + static_cast<uint32_t>(this->flagBelow[t]),
                          static_cast<uint32_t>(this->flagFrom[t] - this->flagBelow[t])};
        for (int g = 0; g < 4; ++g) {
            const int in = RXMET_LSTM_INPUT_GATE_INPUT + g;
            k.gateScale[g] = s.hhToGate[g].mult * s.hhToGate[g].pow2;
            k.giLo[g] = low(in); k.giHi[g] = high(in);
            k.zpIn[g] = s.zpF[in]; k.zpOut[g] = s.zpF[RXMET_LSTM_INPUT_GATE_OUTPUT + g];
        }
        k.hhLo = low(RXMET_LSTM_WEIGHT_HH_LINEAR); k.hhHi = high(RXMET_LSTM_WEIGHT_HH_LINEAR);
        k.cLo = low(RXMET_LSTM_CELL_STATE); k.cHi = high(RXMET_LSTM_CELL_STATE);
        k.oLo = low(RXMET_LSTM_OUTPUT); k.oHi = high(RXMET_LSTM_OUTPUT);
        k.productScale = s.productToOutput.mult * s.productToOutput.pow2;
        k.codePlus = 8388608.0f + static_cast<float>(s.zp[RXMET_LSTM_OUTPUT] - s.lo[RXMET_LSTM_OUTPUT]);
        k.plain = !s.forgetUsesFp && !s.inputUsesFp;
    }
    __device__ __forceinline__ uint32_t codeWord(const planerec::Problem &p, int row, int plane, int kw) const { return unitrec::planeWord<PLANES>(p, row, plane, kw); }
    __device__ __forceinline__ void init(uint8_t *at, uint32_t, int tid, int threads) const { Base::init(at, tid, threads); }
    __device__ __forceinline__ Unit unitOf(uint32_t shared, int unit) const {
        Unit u;
        u.shared = shared;
        u.plain = k.plain;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const typename Base::Lane l = Base::lane(shared, g, unit, true);
            u.addend[g] = l.addend;
            u.outScale[g] = l.outScale;
            u.narrow[g] = l.narrow;
            u.plain = u.plain && l.narrow;
        }
        return u;
    }
    __device__ __forceinline__ void begin(State &st, int row, int unit) const {
        st.cell = this->c0[static_cast<size_t>(row) * this->hidden() + unit];
        st.hidden = 0.0f;
    }
    __device__ __forceinline__ void fetch(Fetch &f, size_t at, uint32_t row, int unit) const {
        const uint32_t H = this->hidden(), mine = row * (4 * H) + unit;
        const float *from = this->lhs + at * (4 * H);
#pragma unroll
        for (int g = 0; g < 4; ++g) f.lhs[g] = __ldg(from + g * H + mine);
    }
    // as Base::quantized, with the value before the clamp to the grid where flags are asked for
    __device__ __forceinline__ float rounded(float x, float lo, float hi) const {
        return kTrain ? roundSmall(clampF(x, lo - 1.0f, hi + 1.0f)) : roundSmall(clampF(x, lo, hi));
    }
    __device__ __forceinline__ float activation(const Unit &u, int t, float x, uint32_t &index) const {
        const LstmUnitConstants::Table &v = k.table[t];
        return lookup(TableView{u.shared + v.segments, u.shared + v.bits, v.toIndex, v.outLo, v.outHi}, this->segShift, x, index);
    }
    template <int, bool PLAIN>
    __device__ __forceinline__ uint32_t advance(const Unit &u, State &st, const Fetch &in, const uint32_t (&acc)[4][PLANES], Out &o) const {
        const auto &s = this->s;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            typename Base::Lane l;
            l.addend = u.addend[g];
            const uint32_t bits = PLAIN || u.narrow[g] ? Base::template total<PLANES, true>(l, acc[g][0], acc[g][PLANES - 1])
                                                       : Base::template total<PLANES, false>(l, acc[g][0], acc[g][PLANES - 1]);
            o.hh[g] = rounded(__fmul_rn(__uint_as_float(bits), u.outScale[g]), k.hhLo, k.hhHi);
            const float hh = kTrain ? clampF(o.hh[g], k.hhLo, k.hhHi) : o.hh[g];
            o.sum[g] = __fadd_rn(in.lhs[g], roundSmall(__fmul_rn(hh, k.gateScale[g])));
            o.gate[g] = activation(u, g, clampF(o.sum[g], k.giLo[g], k.giHi[g]), o.index[g]);
        }
        const float pf = __fmul_rn(o.gate[1], st.cell), pi = __fmul_rn(o.gate[0], o.gate[2]);
        const float sf = PLAIN ? __fmul_rn(pf, s.forgetRatio) : dev::scaleCell(pf, s.forgetRatio, s.forgetMantissa, s.forgetExponent, s.forgetUsesFp);
        const float si = PLAIN ? __fmul_rn(pi, s.inputRatio) : dev::scaleCell(pi, s.inputRatio, s.inputMantissa, s.inputExponent, s.inputUsesFp);
        o.cellRaw = rounded(__fadd_rn(sf, si), k.cLo, k.cHi);
        o.cell = st.cell = kTrain ? clampF(o.cellRaw, k.cLo, k.cHi) : o.cellRaw;
        o.tanhC = activation(u, 4, st.cell, o.index[4]);
        o.hiddenRaw = rounded(__fmul_rn(__fmul_rn(o.gate[3], o.tanhC), k.productScale), k.oLo, k.oHi);
        o.hidden = st.hidden = kTrain ? clampF(o.hiddenRaw, k.oLo, k.oHi) : o.hiddenRaw;
        return __float_as_uint(__fadd_rn(st.hidden, k.codePlus)) & 0xffffu;
    }
    __device__ __forceinline__ void store(const Unit &, const Out &v, size_t at, uint32_t row, int unit, bool good) const {
        const uint32_t H = this->hidden(), mine = row * H + unit, mine4 = row * (4 * H) + unit;
        const auto &s = this->s;
        const auto &ck = this->ck;
        (this->output + at * H)[mine] = __fmul_rn(v.hidden, Base::scaleH(good));
        if (!kTrain) return;
        auto put = [&](auto *to, auto value) {
            if (SAVES == Saves::All || to) (to + at * H)[mine] = value();
        };
        auto put4 = [&](auto *to, auto value) {
            if (SAVES != Saves::All && !to) return;
            auto *step = to + at * (4 * H);
#pragma unroll
            for (int g = 0; g < 4; ++g) (step + g * H)[mine4] = value(g);
        };
        auto flag = [](bool set) { return static_cast<uint8_t>(set ? 1 : 0); };
        auto clamped = [&](int t) { return flag(v.index[t] - k.table[t].flagBelow >= k.table[t].flagCount); };
        put4(ck.weight_hh_linear, [&](int g) { return clampF(v.hh[g], k.hhLo, k.hhHi) + s.zpF[RXMET_LSTM_WEIGHT_HH_LINEAR]; });
        put4(ck.weight_hh_linear_clamped, [&](int g) { return flag(v.hh[g] < k.hhLo || v.hh[g] > k.hhHi); });
        put4(ck.gate_inputs, [&](int g) { return clampF(v.sum[g], k.giLo[g], k.giHi[g]) + k.zpIn[g]; });
        put4(ck.gate_inputs_clamped, [&](int g) { return flag(v.sum[g] < k.giLo[g] || v.sum[g] > k.giHi[g]); });
        put4(ck.gate_outputs, [&](int g) { return v.gate[g] + k.zpOut[g]; });
        put4(ck.gate_outputs_clamped, [&](int g) { return clamped(g); });
        put(ck.cell_states, [&] { return v.cell + s.zpF[RXMET_LSTM_CELL_STATE]; });
        put(ck.cell_states_clamped, [&] { return flag(v.cellRaw < k.cLo || v.cellRaw > k.cHi); });
        put(ck.cell_tanh_outputs, [&] { return v.tanhC + s.zpF[RXMET_LSTM_CELL_TANH_OUTPUT]; });
        put(ck.cell_tanh_outputs_clamped, [&] { return clamped(4); });
        put(ck.hidden_outputs, [&] { return v.hidden + s.zpF[RXMET_LSTM_OUTPUT]; });
        put(ck.hidden_outputs_clamped, [&] { return flag(v.hiddenRaw < k.oLo || v.hiddenRaw > k.oHi); });
    }
    __device__ __forceinline__ void finish(const State &st, int row, int unit, bool good) const {
        const size_t o = static_cast<size_t>(row) * this->hidden() + unit;
        this->finalHidden[o] = __fmul_rn(st.hidden, Base::scaleH(good));
        this->finalCell[o] = __fmul_rn(st.cell, good ? this->s.scale[RXMET_LSTM_CELL_STATE] : __int_as_float(0x7fc00000));
    }
};

// Up to 128 units: inside one CTA, rows as few as let all CTAs run at the same time, up to four (64 units: eight).
template <Saves SAVES, int HP, int PLANES>
void launchLstmUnits(const char *name, const planerec::Problem &p, const LstmPlaneCell<SAVES != Saves::None> &cell, cudaStream_t st) {
    auto run = [&](auto width) {
        using Cell = LstmUnitCell<SAVES, PLANES, decltype(width)::value>;
        static_assert(sizeof(typename Cell::Base) == sizeof(cell), "the variants differ in the width only");
        Cell c;
        std::memcpy(static_cast<typename Cell::Base *>(&c), &cell, sizeof(cell));
        c.prepareConstants();
        unitrec::launchRows<Cell, HP, PLANES>(name, p, c, true, st);
    };
    if (p.H == HP) run(std::integral_constant<int, HP>{});
    else run(std::integral_constant<int, 0>{});
}
// Wider layers, over clusters.  Rows: a step of n rows costs about 1 + n / 5 of the chain of a one-row step.
template <bool TRAIN, int HP>
void launchLstmCluster(const planerec::Problem &p, const LstmPlaneCell<TRAIN> &cell, cudaStream_t st) {
    if (p.H == HP) {
        LstmPlaneCell<TRAIN, HP> full;
        static_assert(sizeof(full) == sizeof(cell), "the variants differ in the width only");
        std::memcpy(&full, &cell, sizeof(full));
        planerec::launchBest<LstmPlaneCell<TRAIN, HP>, HP, 64, 2, 5, 4, 8, 12, 16, 24, 32, 48>("lstmRecurrentWide", p, full, st);
    } else {
        planerec::launchBest<LstmPlaneCell<TRAIN>, HP, 64, 2, 5, 4, 8, 12, 16, 24, 32, 48>("lstmRecurrentWide", p, cell, st);
    }
}
// One padded width each, built in separate files (lstm_forward_cluster_*.cu, lstm_forward_units_*.cu).
template <bool TRAIN, int HP>
void lstmCluster(const planerec::Problem &p, const LstmPlaneCell<TRAIN> &cell, cudaStream_t st);
template <Saves SAVES, int HP, int PLANES>
void lstmUnits(const planerec::Problem &p, const LstmPlaneCell<SAVES != Saves::None> &cell, cudaStream_t st);

}  // namespace lstm
}  // namespace rxmet
