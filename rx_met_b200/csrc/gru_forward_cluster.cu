// W8 / A16 QuantGRU recurrence, H <= 256: the integer cell on top of unit_recurrence_umma.cuh.
//
// The arithmetic is the integer carrier's, value for value (gru_device.cuh): 64-bit rounding rescales and 16-segment tables.
// A step is bound by instructions and their chain, so an element executes as few as it can:
//   - every code is a difference to its zero point, zero points and halves are part of the constants;
//   - a rescale is one widening multiply-add, one funnel shift and, for the exact ties, a cleared lowest bit: shifts are known to lie
//     in [1, 31] where the operand is a grid difference;
//   - a table segment is found through a map of at most 257 buckets (the segment of the bucket's first code, and its only
//     threshold) instead of fifteen compare-and-selects.
// One direction, T = 100, before (clusters with mixed gate tiles, dp4a in lanes) -> now: H = 256, 128 rows, training 187 -> 119 us, 700 rows,
// inference 571 -> 341 us; H = 128, 300 rows, inference 162 -> 105, training 185 -> 134 us; H = 64, 300 rows 151 -> 65 us.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "common.h"
#include "gru_device.cuh"
#include "gru_forward_wide.h"
#include "unit_recurrence_umma.cuh"

namespace rxmet {
namespace gru {
namespace {

constexpr int kBuckets = 257;

// Table of one gate over d = gate-input code - zero point of the table.
struct FastLut {
    int4 segment[kSegments];          // slope; (term - output zero point) << 5 | shift; 2^(shift - 1); 0
    uint2 bucket[kBuckets + 3];       // the bucket's threshold; address of the segment before it, the one behind it follows
};
static_assert(sizeof(FastLut) % 16 == 0, "tables follow one another in shared memory");

// Rounding rescale of a 32-bit operand, shift in [1, 31], and of a product of two, shift in [1, 62].
struct ReadyRescale {
    int64_t plus;          // 2^(shift - 1), and whatever the operand is short of
    int32_t mult, shift;
    uint32_t mask;         // 2^shift - 1
};
struct ReadyWide {
    int64_t plus;          // 2^(shift - 1)
    int32_t mult, shift;
    uint32_t mask;         // 2^(shift % 32) - 1
};
// round_half_even(p / 2^n) for 1 <= n <= 31, low 32 bits, of sum = p + 2^(n-1): the floor is right except for an exact tie,
// where it is the upper neighbour and an odd one must step down.  n counts modulo 32, mask = 2^n - 1.
__device__ __forceinline__ int32_t roundShift31(int64_t sum, int n, uint32_t mask) {
    const uint32_t low = static_cast<uint32_t>(sum), high = static_cast<uint32_t>(static_cast<uint64_t>(sum) >> 32);
    const int32_t q = static_cast<int32_t>(__funnelshift_r(low, high, n));
    return (low & mask) == 0 ? q & ~1 : q;
}
__device__ __forceinline__ int32_t apply(int32_t x, const ReadyRescale &r) {
    return roundShift31(static_cast<int64_t>(x) * r.mult + r.plus, r.shift, r.mask);
}
__device__ __forceinline__ int32_t apply(int64_t x, const ReadyWide &r) {
    const int64_t sum = x * r.mult + r.plus;
    if (r.shift <= 31) return roundShift31(sum, r.shift, r.mask);
    const int32_t high = static_cast<int32_t>(sum >> 32), q = high >> (r.shift - 32);
    return (static_cast<uint32_t>(sum) | (static_cast<uint32_t>(high) & r.mask)) == 0 ? q & ~1 : q;
}
__device__ __forceinline__ int32_t clampTo(int32_t v, int32_t lo, int32_t hi) { return max(lo, min(v, hi)); }

// What the kernel needs of the parameters, prepared on the host.  Limits are differences to the zero point; those of a gate
// input, and `inPlus`, to the zero point of its table.
struct CellScalars {
    ReadyRescale ihTo[3], hhTo[2], newToH;
    ReadyWide rhToNew, oldToH;
    int32_t loHh, hiHh, inPlus[3], loIn[3], hiIn[3], loOut[3], hiOut[3], loH, hiH, oneDiff;
    int32_t zpHh, zpOut[3], zpH;
    int32_t bucketShift[3], firstBucket[3];
    float eff[3], effH, effHh;
};

// What a forward saves beside h and v: nothing, packed clamp flags, or whatever of codes and flags is asked for.
enum class Saves { None, Packed, Any };

// WIDTH: the hidden size where it is a compile-time constant (its multiples are address immediates then), else 0.
template <Saves SAVES, int WIDTH>
struct GruUnitCell {
    static constexpr int kGates = 3;
    static constexpr bool kFlags = SAVES != Saves::None, kTwoRows = true, kSignedCodes = false;
    CellScalars s;
    FastLut luts[3];
    int width;
    size_t B;
    __device__ __forceinline__ int hidden() const { return WIDTH ? WIDTH : width; }
    const uint32_t *words;    // [kWords][3H]
    const int64_t *addend;    // [3H]
    const Rescale *rescale;   // [3H]
    const int16_t *ih;        // [T][B][3H]
    const int16_t *h0;        // [B][hPad] codes
    int hPad;
    float *h, *v;             // [T+1][B][H], [T][B][4H] dequantized
    int32_t *hq, *vq;         // optional codes
    uint8_t *maskHh, *maskGateIn, *maskGateOut, *maskH;
    const uint8_t *maskIh;    // packed flags: those of the input projection, to be packed with the step's
    uint16_t *stepBits;
    const int *poison;        // status word of the tensor-core projection: non-zero turns the hidden outputs into NaN

    __device__ __forceinline__ bool packs() const { return SAVES == Saves::Packed || (SAVES == Saves::Any && stepBits != nullptr); }

    size_t sharedBytes() const { return sizeof(luts); }
    struct Unit {
        int64_t plus[3];      // (addend) mult + 2^(shift - 1)
        int32_t mult[3], shift[3];
        uint32_t mask[3], buckets[3];   // address of the bucket with number 0
        bool plain;           // the shifts of all lanes lie in [1, 31]
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
        return __ldg(words + static_cast<size_t>(kw) * 3 * H + gate * H + unit);
    }
    __device__ __forceinline__ uint32_t codeWord(const planerec::Problem &p, int row, int plane, int kw) const { return unitrec::planeWord<2>(p, row, plane, kw); }
    __device__ __forceinline__ void init(uint8_t *at, uint32_t shared, int tid, int threads) const {
        for (int i = tid; i < static_cast<int>(sizeof(luts) / 4); i += threads) {
            const int g = i / static_cast<int>(sizeof(FastLut) / 4), within = i % static_cast<int>(sizeof(FastLut) / 4);
            uint32_t word = reinterpret_cast<const uint32_t *>(luts)[i];
            if (within >= 4 * kSegments && (within & 1)) word += shared + g * static_cast<uint32_t>(sizeof(FastLut));   // a segment's address
            reinterpret_cast<uint32_t *>(at)[i] = word;
        }
    }
    __device__ __forceinline__ Unit unitOf(uint32_t shared, int unit) const {
        const int H = hidden();
        Unit u;
        bool narrow = true;
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const Rescale r = rescale[g * H + unit];
            narrow = narrow && r.shift >= 1 && r.shift <= 31;
            u.plus[g] = addend[g * H + unit];
            u.mult[g] = r.mult;
            u.shift[g] = r.shift;
            u.buckets[g] = shared + g * static_cast<uint32_t>(sizeof(FastLut)) + 16 * kSegments - 8u * static_cast<uint32_t>(s.firstBucket[g]);
        }
        u.plain = __all_sync(0xffffffffu, narrow);
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            u.mask[g] = (1u << (u.shift[g] & 31)) - 1u;
            if (u.plain) u.plus[g] = u.plus[g] * u.mult[g] + (int64_t{1} << (u.shift[g] - 1));
        }
        return u;
    }
    // whether the projection before it went through; asked once, before the first step
    __device__ __forceinline__ bool valid() const { return poison == nullptr || *poison == 0; }
    __device__ __forceinline__ void begin(State &st, int row, int unit) const {
        const int H = hidden(), code = h0[static_cast<size_t>(row) * hPad + unit];
        st.h = code - s.zpH;
        const size_t o = static_cast<size_t>(row) * H + unit;
        h[o] = static_cast<float>(st.h) * s.effH;
        if (SAVES == Saves::Any && hq) hq[o] = code;
    }
    __device__ __forceinline__ void fetch(Fetch &f, size_t at, uint32_t row, int unit) const {
        const uint32_t H = hidden(), mine = row * (3 * H) + unit;
        const int16_t *from = ih + at * (3 * H);
#pragma unroll
        for (int g = 0; g < 3; ++g) f.ih[g] = __ldg(from + mine + g * H);
        if (packs()) {
            const uint8_t *keep = maskIh + at * (3 * H);
#pragma unroll
            for (int g = 0; g < 3; ++g) f.keepIh[g] = __ldg(keep + mine + g * H);
        }
    }
    // rounded linear code; the sum of both planes fits 32 bits: |weights| <= 128, 256 units, codes up to 65535
    template <int PLANES, bool PLAIN>
    __device__ __forceinline__ int32_t linear(const Unit &u, int g, const uint32_t (&acc)[PLANES]) const {
        const int32_t sum = static_cast<int32_t>((PLANES == 2 ? acc[0] * 256u : 0u) + acc[PLANES - 1]);
        if (PLAIN) return roundShift31(static_cast<int64_t>(sum) * u.mult[g] + u.plus[g], u.shift[g], u.mask[g]);
        const int64_t prod = (sum + u.plus[g]) * u.mult[g];
        if (u.shift[g] < 1) return static_cast<int32_t>(prod << -u.shift[g]);
        return static_cast<int32_t>(rshiftRoundConst(prod, u.shift[g], (int64_t{1} << (u.shift[g] - 1)) - 1));
    }
    // gate output for a gate input
    __device__ __forceinline__ int32_t activation(const Unit &u, int g, int32_t sum, uint32_t &keep) const {
        const int32_t d = clampTo(sum, s.loIn[g], s.hiIn[g]);
        if (kFlags && d == sum) keep += 8u << g;
        int32_t threshold;
        uint32_t at;
        asm("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(threshold), "=r"(at) : "r"(u.buckets[g] + (static_cast<uint32_t>(d >> s.bucketShift[g]) << 3)));
        if (d >= threshold) at += 16;
        int32_t slope, term;
        uint32_t half, zero;
        asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(slope), "=r"(term), "=r"(half), "=r"(zero) : "r"(at));
        const int64_t product = static_cast<int64_t>(slope) * d + static_cast<int64_t>((static_cast<uint64_t>(zero) << 32) | half);
        const int32_t y = roundShift31(product, term, 2u * half - 1u) + (term >> 5);
        const int32_t out = clampTo(y, s.loOut[g], s.hiOut[g]);
        if (kFlags && out == y) keep += 1u << g;
        return out;
    }
    template <int PLANES, bool PLAIN>
    __device__ __forceinline__ uint32_t advance(const Unit &u, State &st, const Fetch &in, const uint32_t (&acc)[3][PLANES], Out &o) const {
        uint32_t keep = 0;
        int32_t hh[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            const int32_t code = linear<PLANES, PLAIN>(u, g, acc[g]);
            hh[g] = clampTo(code, s.loHh, s.hiHh);
            if (kFlags && hh[g] == code) keep += 64u << g;
        }
        const int32_t z = activation(u, 0, apply(in.ih[0], s.ihTo[0]) + apply(hh[0], s.hhTo[0]) + s.inPlus[0], keep);
        const int32_t r = activation(u, 1, apply(in.ih[1], s.ihTo[1]) + apply(hh[1], s.hhTo[1]) + s.inPlus[1], keep);
        const int32_t n = activation(u, 2, apply(in.ih[2], s.ihTo[2]) + apply(static_cast<int64_t>(r) * hh[2], s.rhToNew) + s.inPlus[2], keep);
        const int32_t fresh = apply(n, s.newToH);
        const int32_t code = apply(static_cast<int64_t>(z) * st.h + static_cast<int64_t>(s.oneDiff - z) * fresh, s.oldToH);
        st.h = clampTo(code, s.loH, s.hiH);
        if (kFlags && st.h == code) keep += 1u << 12;
        if (packs()) keep += (in.keepIh[0] << 9) + (in.keepIh[1] << 10) + (in.keepIh[2] << 11);
        o = Out{{z, r, n}, hh[2], st.h, keep};
        return static_cast<uint32_t>(st.h - s.loH);
    }
    __device__ __forceinline__ void store(const Unit &, const Out &o, size_t at, uint32_t row, int unit, bool good) const {
        const uint32_t H = hidden(), mine = row * H + unit, mine3 = row * (3 * H) + unit, mine4 = row * (4 * H) + unit;
        (h + (at + B) * H)[mine] = static_cast<float>(o.h) * (good ? s.effH : __int_as_float(0x7fc00000));
        float *vStep = v + at * (4 * H);
#pragma unroll
        for (int g = 0; g < 3; ++g) (vStep + g * H)[mine4] = static_cast<float>(o.gate[g]) * s.eff[g];
        (vStep + 3 * H)[mine4] = static_cast<float>(o.hh) * s.effHh;
        if (packs()) (stepBits + at * H)[mine] = static_cast<uint16_t>(o.keep);
        if (SAVES == Saves::Any) {
            if (hq) (hq + (at + B) * H)[mine] = o.h + s.zpH;
            if (vq) {
                int32_t *to = vq + at * (4 * H);
#pragma unroll
                for (int g = 0; g < 3; ++g) (to + g * H)[mine4] = o.gate[g] + s.zpOut[g];
                (to + 3 * H)[mine4] = o.hh + s.zpHh;
            }
            if (maskHh) {
                uint8_t *to = maskHh + at * (3 * H);
#pragma unroll
                for (int g = 0; g < 3; ++g) (to + g * H)[mine3] = static_cast<uint8_t>((o.keep >> (6 + g)) & 1u);
            }
            if (maskGateIn) {
                uint8_t *toIn = maskGateIn + at * (3 * H), *toOut = maskGateOut + at * (3 * H);
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    (toIn + g * H)[mine3] = static_cast<uint8_t>((o.keep >> (3 + g)) & 1u);
                    (toOut + g * H)[mine3] = static_cast<uint8_t>((o.keep >> g) & 1u);
                }
                (maskH + at * H)[mine] = static_cast<uint8_t>((o.keep >> 12) & 1u);
            }
        }
    }
    __device__ __forceinline__ void finish(const State &, int, int, bool) const {}
};

// `short31` is what the operand is short of: rescale(x + short31)
bool ready(const Rescale &r, ReadyRescale &out, int64_t short31 = 0) {
    if (r.shift < 1 || r.shift > 31) return false;
    out = ReadyRescale{short31 * r.mult + (int64_t{1} << (r.shift - 1)), r.mult, r.shift, (1u << r.shift) - 1u};
    return true;
}
bool ready(const Rescale &r, ReadyWide &out) {
    if (r.shift < 1 || r.shift > 62) return false;
    out = ReadyWide{int64_t{1} << (r.shift - 1), r.mult, r.shift, (1u << (r.shift & 31)) - 1u};
    return true;
}

// Bucket map of one table over the gate-input grid; false when a shift leaves [1, 31] or a bucket holds two thresholds.
bool ready(const Lut &lut, int32_t lo, int32_t hi, int32_t zpOut, FastLut &out, int32_t &bucketShift, int32_t &firstBucket) {
    const int64_t dLo = static_cast<int64_t>(lo) - lut.zp_x, dHi = static_cast<int64_t>(hi) - lut.zp_x;
    if (dHi < dLo || dHi - dLo > 65535 || std::max(-dLo, dHi) > (1 << 24)) return false;
    // the segments that codes of the grid use, in order; segment i is the first whose threshold exceeds the code, else the last
    int64_t from = dLo, behind[kSegments] = {};
    int used = 0;
    for (int i = 0; i < kSegments && from <= dHi; ++i) {
        const int64_t until = i == kSegments - 1 ? dHi + 1 : std::min<int64_t>(static_cast<int64_t>(lut.threshold[i]) - lut.zp_x, dHi + 1);
        if (until <= from) continue;
        const int64_t term = static_cast<int64_t>(lut.term_c[i]) - zpOut;
        if (lut.n_bx[i] < 1 || lut.n_bx[i] > 31 || std::abs(term) >= (int64_t{1} << 26)) return false;
        out.segment[used] = make_int4(lut.q_b[i], static_cast<int>(static_cast<uint32_t>(term) << 5 | static_cast<uint32_t>(lut.n_bx[i])),
                                      static_cast<int>(1u << (lut.n_bx[i] - 1)), 0);
        behind[used++] = from = until;
    }
    bucketShift = 0;
    while ((dHi >> bucketShift) - (dLo >> bucketShift) >= kBuckets) ++bucketShift;
    firstBucket = static_cast<int32_t>(dLo >> bucketShift);
    int segment = 0;
    for (int b = 0; b < kBuckets; ++b) {
        const int64_t first = std::max(dLo, static_cast<int64_t>(firstBucket + b) << bucketShift),
                      last = std::min(dHi, (static_cast<int64_t>(firstBucket + b + 1) << bucketShift) - 1);
        out.bucket[b] = make_uint2(static_cast<uint32_t>(INT32_MAX), 0u);
        if (first > last) continue;
        while (behind[segment] <= first) ++segment;
        out.bucket[b].y = 16u * static_cast<uint32_t>(segment);
        if (behind[segment] > last) continue;
        out.bucket[b].x = static_cast<uint32_t>(static_cast<int32_t>(behind[segment]));
        if (behind[segment + 1] <= last) return false;
    }
    return true;
}

// Everything of the cell that does not depend on the width or on what is saved.
struct Prepared {
    CellScalars s;
    FastLut luts[3];
};

template <int HP, Saves SAVES, int WIDTH>
void launchFor(const WideRecurrence &r, const Prepared &prepared, cudaStream_t st) {
    using Cell = GruUnitCell<SAVES, WIDTH>;
    Cell cell{};
    cell.s = prepared.s;
    std::copy(prepared.luts, prepared.luts + 3, cell.luts);
    cell.width = r.H;
    cell.B = static_cast<size_t>(r.B);
    cell.words = r.words; cell.addend = r.addend; cell.rescale = r.rescale; cell.ih = r.ih; cell.h0 = r.h0; cell.hPad = r.hPad;
    cell.h = r.h; cell.v = r.v; cell.hq = r.hq; cell.vq = r.vq;
    cell.maskHh = r.maskHh; cell.maskGateIn = r.maskGateIn; cell.maskGateOut = r.maskGateOut; cell.maskH = r.maskH;
    cell.maskIh = r.maskIh; cell.stepBits = r.stepBits;
    cell.poison = r.poison;
    unitrec::launchRows<Cell, HP, 2>("recurrentForward", planerec::Problem{r.T, r.B, r.H, r.h0Planes}, cell, true, st);
}
template <int HP>
void launchFor(const WideRecurrence &r, const Prepared &prepared, cudaStream_t st) {
    auto run = [&](auto width) {
        constexpr int kWidth = decltype(width)::value;
        if (r.hq || r.vq || r.maskHh || r.maskGateIn) launchFor<HP, Saves::Any, kWidth>(r, prepared, st);
        else if (r.stepBits) launchFor<HP, Saves::Packed, kWidth>(r, prepared, st);
        else launchFor<HP, Saves::None, kWidth>(r, prepared, st);
    };
    if (r.H == HP) run(std::integral_constant<int, HP>{});
    else run(std::integral_constant<int, 0>{});
}

bool prepare(const Exec &e, Prepared &cell) {
    const GateExec &g = e.gate;
    CellScalars &s = cell.s;
    const int inOp[3] = {RXMET_GRU_UPDATE_GATE_INPUT, RXMET_GRU_RESET_GATE_INPUT, RXMET_GRU_NEW_GATE_INPUT};
    const int outOp[3] = {RXMET_GRU_UPDATE_GATE_OUTPUT, RXMET_GRU_RESET_GATE_OUTPUT, RXMET_GRU_NEW_GATE_OUTPUT};
    const Lut *luts[3] = {&g.lut_update, &g.lut_reset, &g.lut_new};
    const Rescale ihTo[3] = {g.ih_to_update, g.ih_to_reset, g.ih_to_new}, hhTo[2] = {g.hh_to_update, g.hh_to_reset};
    const int32_t zpIh = g.zp[RXMET_GRU_WEIGHT_IH_LINEAR];
    bool ok = ready(g.rh_to_new, s.rhToNew) && ready(g.new_to_h, s.newToH) && ready(g.update_old_to_h, s.oldToH);
    for (int i = 0; i < 3 && ok; ++i) {
        const int32_t zpX = luts[i]->zp_x;
        ok = ready(ihTo[i], s.ihTo[i], -static_cast<int64_t>(zpIh)) && (i == 2 || ready(hhTo[i], s.hhTo[i])) &&
             ready(*luts[i], g.qlo[inOp[i]], g.qhi[inOp[i]], g.zp[outOp[i]], cell.luts[i], s.bucketShift[i], s.firstBucket[i]);
        s.inPlus[i] = g.zp[inOp[i]] - zpX; s.loIn[i] = g.qlo[inOp[i]] - zpX; s.hiIn[i] = g.qhi[inOp[i]] - zpX;
        s.zpOut[i] = g.zp[outOp[i]]; s.loOut[i] = g.qlo[outOp[i]] - s.zpOut[i]; s.hiOut[i] = g.qhi[outOp[i]] - s.zpOut[i];
        s.eff[i] = g.eff[outOp[i]];
    }
    if (!ok) return false;
    s.zpHh = g.zp[RXMET_GRU_WEIGHT_HH_LINEAR];
    s.loHh = g.qlo[RXMET_GRU_WEIGHT_HH_LINEAR] - s.zpHh; s.hiHh = g.qhi[RXMET_GRU_WEIGHT_HH_LINEAR] - s.zpHh;
    s.effHh = g.eff[RXMET_GRU_WEIGHT_HH_LINEAR];
    s.zpH = g.zp[RXMET_GRU_H]; s.loH = g.qlo[RXMET_GRU_H] - s.zpH; s.hiH = g.qhi[RXMET_GRU_H] - s.zpH; s.effH = g.eff[RXMET_GRU_H];
    s.oneDiff = g.quant_one - s.zpOut[0];
    return true;
}

}  // namespace

bool forwardWideClusterTakes(const Exec &e, int B, int H) {
    Prepared prepared;
    return H <= 256 && 4 * static_cast<uint64_t>(H) * B < (uint64_t{1} << 32) && prepare(e, prepared);   // offsets inside a step have 32 bits
}

void forwardWideCluster(const WideRecurrence &r, const Exec &e, cudaStream_t st) {
    Prepared prepared;
    prepare(e, prepared);
    if (r.H <= 32) launchFor<32>(r, prepared, st);
    else if (r.H <= 64) launchFor<64>(r, prepared, st);
    else if (r.H <= 128) launchFor<128>(r, prepared, st);
    else if (r.H <= 192) launchFor<192>(r, prepared, st);
    else launchFor<256>(r, prepared, st);
}

}  // namespace gru
}  // namespace rxmet
