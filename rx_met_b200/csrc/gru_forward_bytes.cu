// 8-bit QuantGRU recurrence on small grids, H <= 256: the cell of recurrentLanesI8 (gru_forward_quant.cu) on top of
// unit_recurrence_umma.cuh, one plane of signed codes.
//
// The arithmetic is the integer carrier's, value for value: codes as differences to their zero points, activations from direct tables,
// input contributions rescaled by the projection, a rounding shift as an add of one half, a shift and, for the exact ties, a
// cleared lowest bit.  What is gained over the lanes is their product: 96 dp4a per thread and step at two rows of 128 units.
// Passes of T = 100, before -> now: inference, H = 128, 1 row 74 -> 63 us, 700 rows 303 -> 193; H = 256, 128 rows 221 -> 136 (on two planes before);
// training, H = 128, 128 rows 247 -> 213, H = 256 450 -> 351.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "common.h"
#include "gru_device.cuh"
#include "gru_forward_bytes.h"
#include "unit_recurrence_umma.cuh"

namespace rxmet {
namespace gru {
namespace {

// A rounding rescale of a 32-bit operand, shift in [0, 31]: half 0 and a mask that no remainder meets where the shift is 0.
struct SmallRescale {
    int32_t mult, shift, half;
    uint32_t mask;
};
__device__ __forceinline__ int32_t clearTie(int32_t q, uint32_t low, uint32_t mask) { return (low & mask) == 0 ? q & ~1 : q; }
__device__ __forceinline__ int32_t rescaleSmallTies(int32_t x, const SmallRescale &r) {   // |x * mult| + half < 2^31
    const int32_t v = x * r.mult + r.half;
    return clearTie(v >> r.shift, static_cast<uint32_t>(v), r.mask);
}
__device__ __forceinline__ int32_t roundWide(int64_t sum, int32_t shift, uint32_t mask) {   // half added already, quotient fits 32 bits, shift in [1, 31]
    const uint32_t low = static_cast<uint32_t>(sum), high = static_cast<uint32_t>(static_cast<uint64_t>(sum) >> 32);
    return clearTie(static_cast<int32_t>(__funnelshift_r(low, high, shift)), low, mask);
}
__device__ __forceinline__ int32_t clampTo(int32_t v, int32_t lo, int32_t hi) { return max(lo, min(v, hi)); }

struct ByteScalars {
    SmallRescale toUpdate, toReset, rhToNew, toH, newToH;
    int32_t loHh, hiHh, loH, hiH, last[3], toIndex[3], oneDiff;   // differences to the zero points; highest index of a table, zero point - grid minimum
    int32_t zpOut[3], zpHh, zpH, loOut[3], hiOut[3], loIn[3];
    float eff[3], effH, effHh;
    int plain;                      // both products of the cell round with 32-bit pieces
    Rescale rhGeneral, hGeneral;
};

enum class Saves { None, Packed, Bytes, Any };   // Bytes: all four flag tensors; Any: whatever of codes and flags is asked for

template <Saves SAVES, int WIDTH>
struct GruByteCell {
    static constexpr int kGates = 3;
    static constexpr bool kFlags = SAVES != Saves::None, kTwoRows = true, kSignedCodes = true;
    ByteScalars s;
    Lut luts[3];
    ByteRecurrence r;
    __device__ __forceinline__ int hidden() const { return WIDTH ? WIDTH : r.H; }
    __device__ __forceinline__ bool packs() const { return SAVES == Saves::Packed || (SAVES == Saves::Any && r.stepBits != nullptr); }

    // tables: the candidate's (entry, value on the h grid) pairs, then the other two gates'; an entry is the output's difference to its
    // zero point << 16 | inside the grid << gate
    size_t sharedBytes() const { return 8 * static_cast<size_t>(s.last[2] + 1) + 4 * static_cast<size_t>(s.last[0] + 1 + s.last[1] + 1); }
    struct Unit {
        int64_t plus[3];      // offset mult + 2^(shift - 1)
        int32_t mult[3], shift[3];
        uint32_t mask[3], table[3];   // shared addresses
        bool plain;
    };
    struct State {
        int32_t h;
    };
    struct Fetch {
        int32_t ih[3];
        uint32_t keepIh[3];
    };
    struct Out {
        int32_t gate[3], hh, h;
        uint32_t keep;   // bits 0..2 gate output z, r, n; 3..5 gate input; 6..8 hh linear; 9..11 ih linear; 12 hidden state
    };
    __device__ __forceinline__ uint32_t weightWord(int gate, int unit, int kw) const {
        const int H = hidden();
        return kw < r.kWords ? __ldg(r.words + static_cast<size_t>(kw) * 3 * H + gate * H + unit) : 0u;
    }
    __device__ __forceinline__ uint32_t codeWord(const planerec::Problem &, int row, int, int kw) const {
        if (kw >= r.kWords) return 0u;
        if (r.h0 == nullptr) return static_cast<uint32_t>(s.zpH & 0xff) * 0x01010101u;   // codes beyond the last unit meet zero weights
        return reinterpret_cast<const uint32_t *>(r.h0)[static_cast<size_t>(row) * r.kWords + kw];
    }
    __device__ __forceinline__ void init(uint8_t *at, uint32_t, int tid, int threads) const {
        auto entry = [&](int g, int i) {
            uint8_t keep;
            const int32_t code = clampCode(lutEval<true>(s.loIn[g] + i, luts[g]), s.loOut[g] + s.zpOut[g], s.hiOut[g] + s.zpOut[g], keep);
            return static_cast<int32_t>(static_cast<uint32_t>(code - s.zpOut[g]) << 16) | (keep << g);
        };
        int2 *tabN = reinterpret_cast<int2 *>(at);
        int32_t *tabZ = reinterpret_cast<int32_t *>(tabN + s.last[2] + 1), *tabR = tabZ + s.last[0] + 1;
        for (int i = tid; i <= s.last[0]; i += threads) tabZ[i] = entry(0, i);
        for (int i = tid; i <= s.last[1]; i += threads) tabR[i] = entry(1, i);
        for (int i = tid; i <= s.last[2]; i += threads) {
            const int32_t e = entry(2, i);
            tabN[i] = make_int2(e, rescaleSmallTies(e >> 16, s.newToH));
        }
    }
    __device__ __forceinline__ Unit unitOf(uint32_t shared, int unit) const {
        const int H = hidden();
        Unit u;
        bool narrow = s.plain;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const int c = g * H + unit;
            const Rescale rs = r.rescale[c];
            const int64_t offset = r.biasAcc[c] - r.comp[c];
            u.mult[g] = rs.mult;
            u.shift[g] = rs.shift;
            u.plus[g] = offset * rs.mult;
            u.mask[g] = (1u << (rs.shift & 31)) - 1u;
            narrow = narrow && rs.shift >= 1 && rs.shift <= 31 && rs.mult > 0 && static_cast<int64_t>(rs.mult) <= (1ll << rs.shift) &&
                     offset > -(1ll << 30) && offset < (1ll << 30);
        }
        u.plain = __all_sync(0xffffffffu, narrow);
        if (u.plain) {
#pragma unroll
            for (int g = 0; g < 3; ++g) u.plus[g] += int64_t{1} << (u.shift[g] - 1);
        }
        u.table[2] = shared;
        u.table[0] = shared + 8 * (s.last[2] + 1);
        u.table[1] = u.table[0] + 4 * (s.last[0] + 1);
        return u;
    }
    __device__ __forceinline__ bool valid() const { return r.poison == nullptr || *r.poison == 0; }
    __device__ __forceinline__ void begin(State &st, int row, int unit) const {
        const int H = hidden(), code = r.h0 ? r.h0[static_cast<size_t>(row) * (4 * r.kWords) + unit] : s.zpH;
        st.h = code - s.zpH;
        const size_t o = static_cast<size_t>(row) * H + unit;
        r.h[o] = static_cast<float>(st.h) * s.effH;
        if (SAVES == Saves::Any && r.hq) r.hq[o] = code;
    }
    __device__ __forceinline__ void fetch(Fetch &f, size_t at, uint32_t row, int unit) const {
        const uint32_t H = hidden(), mine = row * (3 * H) + unit;
        const int16_t *from = r.ih + at * (3 * H);
#pragma unroll
        for (int g = 0; g < 3; ++g) f.ih[g] = __ldg(from + mine + g * H);
        if (packs()) {
            const uint8_t *keep = r.maskIh + at * (3 * H);
#pragma unroll
            for (int g = 0; g < 3; ++g) f.keepIh[g] = __ldg(keep + mine + g * H);
        }
    }
    __device__ __forceinline__ int32_t index(int g, int32_t pre, uint32_t &keep) const {
        const int32_t i = clampTo(pre, 0, s.last[g]);
        if (kFlags && i == pre) keep += 8u << g;
        return i;
    }
    template <int PLANES, bool PLAIN>
    __device__ __forceinline__ uint32_t advance(const Unit &u, State &st, const Fetch &in, const uint32_t (&acc)[3][PLANES], Out &o) const {
        uint32_t keep = 0;
        int32_t hh[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const int64_t wide = static_cast<int64_t>(static_cast<int32_t>(acc[g][0])) * u.mult[g] + u.plus[g];
            const int32_t code = PLAIN ? roundWide(wide, u.shift[g], u.mask[g]) : rshiftRoundCalled(wide, u.shift[g]);
            hh[g] = clampTo(code, s.loHh, s.hiHh);
            if (kFlags && hh[g] == code) keep += 64u << g;
        }
        auto product = [&](int32_t x, const SmallRescale &r32, const Rescale &general) {
            if (PLAIN) return roundWide(static_cast<int64_t>(x) * r32.mult + r32.half, r32.shift, r32.mask);
            return rshiftRoundCalled(static_cast<int64_t>(x) * general.mult, general.shift);
        };
        int32_t z, rr, nEntry, fresh;
        asm("ld.shared.s32 %0, [%1];" : "=r"(z) : "r"(u.table[0] + 4 * index(0, in.ih[0] + rescaleSmallTies(hh[0], s.toUpdate) + s.toIndex[0], keep)));
        asm("ld.shared.s32 %0, [%1];" : "=r"(rr) : "r"(u.table[1] + 4 * index(1, in.ih[1] + rescaleSmallTies(hh[1], s.toReset) + s.toIndex[1], keep)));
        asm("ld.shared.v2.s32 {%0, %1}, [%2];"
            : "=r"(nEntry), "=r"(fresh)
            : "r"(u.table[2] + 8 * index(2, in.ih[2] + product((rr >> 16) * hh[2], s.rhToNew, s.rhGeneral) + s.toIndex[2], keep)));
        const int32_t zDiff = z >> 16;
        const int32_t code = product(zDiff * st.h + (s.oneDiff - zDiff) * fresh, s.toH, s.hGeneral);
        st.h = clampTo(code, s.loH, s.hiH);
        if (kFlags) {
            if (st.h == code) keep += 1u << 12;
            keep += static_cast<uint32_t>((z & 1) + (rr & 2) + (nEntry & 4));
            if (packs()) keep += (in.keepIh[0] << 9) + (in.keepIh[1] << 10) + (in.keepIh[2] << 11);
        }
        o = Out{{zDiff, rr >> 16, nEntry >> 16}, hh[2], st.h, keep};
        return static_cast<uint32_t>(st.h + s.zpH);
    }
    __device__ __forceinline__ void store(const Unit &, const Out &o, size_t at, uint32_t row, int unit, bool good) const {
        const uint32_t H = hidden(), mine = row * H + unit, mine3 = row * (3 * H) + unit, mine4 = row * (4 * H) + unit;
        (r.h + (at + r.B) * H)[mine] = static_cast<float>(o.h) * (good ? s.effH : __int_as_float(0x7fc00000));
        float *vStep = r.v + at * (4 * H);
#pragma unroll
        for (int g = 0; g < 3; ++g) (vStep + g * H)[mine4] = static_cast<float>(o.gate[g]) * (good ? s.eff[g] : __int_as_float(0x7fc00000));
        (vStep + 3 * H)[mine4] = static_cast<float>(o.hh) * (good ? s.effHh : __int_as_float(0x7fc00000));
        if (packs()) (r.stepBits + at * H)[mine] = static_cast<uint16_t>(o.keep);
        constexpr bool kAny = SAVES == Saves::Any;
        if (kAny && r.hq) (r.hq + (at + r.B) * H)[mine] = o.h + s.zpH;
        if (kAny && r.vq) {
            int32_t *to = r.vq + at * (4 * H);
#pragma unroll
            for (int g = 0; g < 3; ++g) (to + g * H)[mine4] = o.gate[g] + s.zpOut[g];
            (to + 3 * H)[mine4] = o.hh + s.zpHh;
        }
        if (SAVES == Saves::Bytes || (kAny && r.maskHh)) {
            uint8_t *to = r.maskHh + at * (3 * H);
#pragma unroll
            for (int g = 0; g < 3; ++g) (to + g * H)[mine3] = static_cast<uint8_t>((o.keep >> (6 + g)) & 1u);
        }
        if (SAVES == Saves::Bytes || (kAny && r.maskGateIn)) {
            uint8_t *toIn = r.maskGateIn + at * (3 * H), *toOut = r.maskGateOut + at * (3 * H);
#pragma unroll
            for (int g = 0; g < 3; ++g) {
                (toIn + g * H)[mine3] = static_cast<uint8_t>((o.keep >> (3 + g)) & 1u);
                (toOut + g * H)[mine3] = static_cast<uint8_t>((o.keep >> g) & 1u);
            }
            (r.maskH + at * H)[mine] = static_cast<uint8_t>((o.keep >> 12) & 1u);
        }
    }
    __device__ __forceinline__ void finish(const State &, int, int, bool) const {}
};

SmallRescale small(const Rescale &r) {
    const int n = r.shift & 31;
    return {r.mult, r.shift, n ? static_cast<int32_t>(1u << (n - 1)) : 0, n ? (1u << n) - 1u : 0xffffffffu};
}

template <int HP, Saves SAVES>
void launchFor(const ByteRecurrence &r, const ByteScalars &s, const GateExec &g, cudaStream_t st) {
    auto run = [&](auto width) {
        using Cell = GruByteCell<SAVES, decltype(width)::value>;
        Cell cell{};
        cell.s = s;
        cell.luts[0] = g.lut_update; cell.luts[1] = g.lut_reset; cell.luts[2] = g.lut_new;
        cell.r = r;
        unitrec::launchRows<Cell, HP, 1>("recurrentForward", planerec::Problem{r.T, r.B, r.H, nullptr}, cell, true, st);
    };
    if (r.H == HP) run(std::integral_constant<int, HP>{});
    else run(std::integral_constant<int, 0>{});
}
template <int HP>
void launchFor(const ByteRecurrence &r, const ByteScalars &s, const GateExec &g, cudaStream_t st) {
    if (r.hq || r.vq || (!r.maskHh != !r.maskGateIn) || (r.stepBits && r.maskHh)) launchFor<HP, Saves::Any>(r, s, g, st);
    else if (r.stepBits) launchFor<HP, Saves::Packed>(r, s, g, st);
    else if (r.maskHh) launchFor<HP, Saves::Bytes>(r, s, g, st);
    else launchFor<HP, Saves::None>(r, s, g, st);
}

}  // namespace

// Against the lanes: a step is shorter here, but there is more to prepare, and a layer of at most 64 units is padded to that.  Passes in us,
// lanes -> here:
//   inference beyond 64 units: H 65, 1 row T 40 27 -> 28, T 98 51 -> 47; 64 rows T 40 31 -> 33, T 64 40 -> 41, T 98 56 -> 55; H 128, 1 row T 8 17 -> 19, T 16
//     21 -> 21, T 40 36 -> 31; 128 rows T 16 23 -> 25, T 24 31 -> 31; 200 rows T 20, H 80 35 -> 27; 600 rows T 10, H 65 35 -> 33, H 128 47 -> 37
//   inference of 49 to 64 units: 300 rows T 10 19 -> 23, T 20 33 -> 29; 1200 rows T 40 89 -> 84
//   saving, beyond 64 units: H 65, 64 rows T 4 74 -> 79, T 12 86 -> 86, T 16 88 -> 86; H 128, 300 rows T 10 105 -> 96
//   saving, up to 64 units: 64, 64 rows T 40 84 -> 86, T 64 117 -> 105, 100 rows T 40 93 -> 87; 32, 128 rows T 40 103 -> 106, T 98 181 -> 161; 16, 300 rows
//     T 40 133 -> 123, 600 rows T 40 178 -> 169, 1200 rows 326 -> 334; 48, 1200 rows 369 -> 380; 64, 1200 rows 249 -> 232
bool forwardBytesTakes(int T, int B, int H, bool saves) {
    if (H > 256 || 4 * static_cast<uint64_t>(H) * B >= (uint64_t{1} << 32)) return false;
    if (H > 128) return true;
    const int sms = currentDevice().sms;
    const int64_t rows = static_cast<int64_t>(T) * B;
    if (saves) {
        if (H > 64) return T >= 16 || (H > 112 && B > 2 * sms);
        return static_cast<int64_t>(B) * H > 2048 && rows * H >= (B > 2 * sms ? 2 : 3) << 16 && (H == 64 || B <= 5 * sms);
    }
    if (H <= 64) return H > 48 && B > 2 * sms && (T >= 16 || B > 5 * sms);
    if (B > sms) return T >= 16 || B > 4 * sms;
    const bool crowded = (rows + 15) / 16 + B > sms;   // no SMs of their own beside the projection: nothing is prepared under it
    return T >= (H > 96 ? (crowded ? 24 : 16) : (crowded ? 64 : 48));
}

void forwardBytes(const ByteRecurrence &r, const GateExec &g, cudaStream_t st) {
    ByteScalars s{};
    const int inOp[3] = {RXMET_GRU_UPDATE_GATE_INPUT, RXMET_GRU_RESET_GATE_INPUT, RXMET_GRU_NEW_GATE_INPUT};
    const int outOp[3] = {RXMET_GRU_UPDATE_GATE_OUTPUT, RXMET_GRU_RESET_GATE_OUTPUT, RXMET_GRU_NEW_GATE_OUTPUT};
    s.toUpdate = small(g.hh_to_update); s.toReset = small(g.hh_to_reset); s.newToH = small(g.new_to_h);
    s.rhToNew = small(g.rh_to_new); s.toH = small(g.update_old_to_h);
    s.rhGeneral = g.rh_to_new; s.hGeneral = g.update_old_to_h;
    auto narrow = [](const Rescale &x) { return x.shift >= 1 && x.shift <= 31 && x.mult > 0 && static_cast<int64_t>(x.mult) <= (1ll << x.shift); };
    s.plain = narrow(g.rh_to_new) && narrow(g.update_old_to_h);
    for (int i = 0; i < 3; ++i) {
        s.last[i] = g.qhi[inOp[i]] - g.qlo[inOp[i]];
        s.toIndex[i] = g.zp[inOp[i]] - g.qlo[inOp[i]];
        s.loIn[i] = g.qlo[inOp[i]];
        s.zpOut[i] = g.zp[outOp[i]]; s.loOut[i] = g.qlo[outOp[i]] - s.zpOut[i]; s.hiOut[i] = g.qhi[outOp[i]] - s.zpOut[i];
        s.eff[i] = g.eff[outOp[i]];
    }
    s.zpHh = g.zp[RXMET_GRU_WEIGHT_HH_LINEAR]; s.zpH = g.zp[RXMET_GRU_H];
    s.loHh = g.qlo[RXMET_GRU_WEIGHT_HH_LINEAR] - s.zpHh; s.hiHh = g.qhi[RXMET_GRU_WEIGHT_HH_LINEAR] - s.zpHh;
    s.loH = g.qlo[RXMET_GRU_H] - s.zpH; s.hiH = g.qhi[RXMET_GRU_H] - s.zpH;
    s.effHh = g.eff[RXMET_GRU_WEIGHT_HH_LINEAR]; s.effH = g.eff[RXMET_GRU_H];
    s.oneDiff = g.quant_one - s.zpOut[0];
    if (r.H <= 64) launchFor<64>(r, s, g, st);
    else if (r.H <= 128) launchFor<128>(r, s, g, st);
    else if (r.H <= 192) launchFor<192>(r, s, g, st);
    else launchFor<256>(r, s, g, st);
}

}  // namespace gru
}  // namespace rxmet
