// W8 / A16 QuantGRU recurrence over thread-block clusters: the integer cell on top of plane_recurrence_umma.cuh.
//
// The arithmetic is the integer carrier's, value for value (gru_device.cuh): 64-bit rounding rescales and 16-segment tables.
// What differs from the generic cell is how much of it an element executes: shifts are known to lie in [1, 31] where the
// operand is a grid difference, so a rescale is one widening multiply, one add and two funnel shifts; a table segment is found through a 256-bucket map (the segment of the
// bucket's first code and the one behind its only threshold) instead of fifteen compare-and-selects; the scalar
// constants come from the constant bank.
// T = 100, B = 128, H = 256, one direction of two at a time: 490 -> 190 us per pass (recurrentPlanes, dp4a).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "common.h"
#include "gru_device.cuh"
#include "gru_forward_wide.h"
#include "lane_recurrence.cuh"
#include "plane_recurrence_umma.cuh"

namespace rxmet {
namespace gru {
namespace {

constexpr int kBuckets = 256;

struct FastLut {
    int4 segment[kSegments];          // q_b, n_bx, term_c, 2^(n_bx - 1)
    uint2 bucket[kBuckets];           // the bucket's threshold; byte offset of the segment before it | of the one behind it << 16
};
static_assert(sizeof(int4) * kSegments == 256, "activation() addresses the buckets behind the segments");

// round_half_even(p / 2^n) for 1 <= n <= 31, low 32 bits, of sum = p + 2^(n-1): the floor is right except for an exact tie,
// where it is the upper neighbour and an odd one must step down.  mask = 2^n - 1.
__device__ __forceinline__ int32_t roundShift31(int64_t sum, int n, uint32_t mask) {
    const uint32_t low = static_cast<uint32_t>(sum), high = static_cast<uint32_t>(static_cast<uint64_t>(sum) >> 32);
    const int32_t q = static_cast<int32_t>(__funnelshift_r(low, high, n));
    return (low & mask) == 0 ? q & ~1 : q;
}

// Rounding rescale of a 32-bit operand, shift in [1, 31], and of a product of two, shift in [1, 62].
struct ReadyRescale {
    int32_t mult, shift;
    uint32_t half, mask;   // 2^(shift - 1), 2^shift - 1
};
struct ReadyWide {
    int32_t mult, shift;
    int64_t roundAdd;      // 2^(shift - 1) - 1
};
__device__ __forceinline__ int32_t apply(int32_t x, const ReadyRescale &r) {
    return roundShift31(static_cast<int64_t>(x) * r.mult + r.half, r.shift, r.mask);
}
__device__ __forceinline__ int32_t apply(int64_t x, const ReadyWide &r) {
    const int64_t p = x * r.mult;
    if (r.shift <= 31) return roundShift31(p + r.roundAdd + 1, r.shift, 2u * static_cast<uint32_t>(r.roundAdd) + 1u);
    return static_cast<int32_t>(rshiftRoundConst(p, r.shift, r.roundAdd));
}

// What the kernel needs of the tables, prepared on the host.
struct CellScalars {
    ReadyRescale ihTo[3], hhTo[2], newToH;
    ReadyWide rhToNew, oldToH;
    int32_t zpIh, zpHh, zpIn[3], loIn[3], hiIn[3], zpOut[3], loOut[3], hiOut[3], zpH, loH, hiH, loHh, hiHh, quantOne;
    int32_t zpX[3], bucketShift[3];
    float eff[3], effH, effHh;
};

// What a training forward saves of the clamp flags.
enum class Flags { None, Bytes, Packed };

// WIDTH: the hidden size where it is a compile-time constant (its multiples are address immediates then), else 0.
template <Flags FLAGS, int WIDTH>
struct GruPlaneCell {
    static constexpr int kGates = 3;
    static constexpr bool kSaves = false, kFull = WIDTH != 0;
    static constexpr int kChunk = 8, kTotalFrom = 16;   // a training step of eight rows is 10 % shorter with a branch per row
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

    size_t sharedBytes() const { return sizeof(luts); }
    struct Lane {
        int64_t addend, roundAdd;   // narrow: (sum + addend) mult + 2^(shift - 1) = sum mult + addend
        int32_t mult, shift;
        uint32_t mask;
        bool narrow;   // warp-uniform: the shifts of all lanes lie in [1, 31]
    };
    struct State {
        int32_t h, code[3], hhn;
        uint32_t keep;   // bits 0..2 gate output z, r, n; 3..5 gate input; 6..8 hh linear; 12 hidden state
    };
    struct Fetch {};
    struct Saved {};
    struct FetchB {
        int32_t ih[3];
        uint32_t keepIh[3];
    };

    __device__ __forceinline__ uint32_t weightWord(int gate, int unit, int kw) const {
        const int H = hidden();
        return gate < 3 ? __ldg(words + static_cast<size_t>(kw) * 3 * H + gate * H + unit) : 0u;
    }
    __device__ __forceinline__ void init(uint8_t *shared, int tid, int threads) const {
        for (int i = tid; i < static_cast<int>(sizeof(luts) / 4); i += threads)
            reinterpret_cast<uint32_t *>(shared)[i] = reinterpret_cast<const uint32_t *>(luts)[i];
    }
    __device__ __forceinline__ Lane lane(uint32_t, int gate, int unit, bool real) const {
        const int H = hidden();
        Lane l{0, 0, 0, 1, 1u, false};
        if (gate < 3 && real) {
            const Rescale r = rescale[gate * H + unit];
            l.addend = addend[gate * H + unit];
            l.mult = r.mult;
            l.shift = r.shift;
        }
        l.roundAdd = l.shift >= 1 ? (int64_t{1} << (l.shift - 1)) - 1 : 0;
        l.narrow = __all_sync(0xffffffffu, l.shift >= 1 && l.shift <= 31);
        if (l.narrow) {
            l.addend = l.addend * l.mult + (int64_t{1} << (l.shift - 1));
            l.mask = (1u << l.shift) - 1u;
        }
        return l;
    }
    // whether the projection before it went through; asked once, before the first step
    __device__ __forceinline__ bool valid() const { return poison == nullptr || *poison == 0; }
    __device__ __forceinline__ float scaleH(bool good) const { return good ? s.effH : __int_as_float(0x7fc00000); }
    __device__ __forceinline__ void begin(uint32_t, State &st, int row, int unit) const {
        const int H = hidden();
        st.h = h0[static_cast<size_t>(row) * hPad + unit];
        const size_t o = static_cast<size_t>(row) * H + unit;
        h[o] = static_cast<float>(st.h - s.zpH) * scaleH(true);
        if (hq) hq[o] = st.h;
    }
    __device__ __forceinline__ void fetch(Fetch &, size_t, uint32_t, int, int) const {}
    __device__ __forceinline__ void fetchRow(Fetch &, size_t, int, int, int) const {}
    __device__ __forceinline__ void fetchB(FetchB &f, size_t at, uint32_t row, int unit) const {
        const int H = hidden();
        const int16_t *from = ih + at * (3 * H) + (row * (3 * H) + unit);
#pragma unroll
        for (int g = 0; g < 3; ++g) f.ih[g] = __ldg(from + g * H);
        if (FLAGS == Flags::Packed) {
            const uint8_t *keep = maskIh + at * (3 * H) + (row * (3 * H) + unit);
#pragma unroll
            for (int g = 0; g < 3; ++g) f.keepIh[g] = __ldg(keep + g * H);
        }
    }
    // hh linear code, its keep flag in bit 0
    template <int STRIDE>
    __device__ __forceinline__ uint32_t linear(uint32_t, const Lane &l, const Fetch &, const uint32_t *acc, Saved &) const {
        const int64_t sum = (static_cast<int64_t>(static_cast<int32_t>(acc[0])) << 8) + static_cast<int32_t>(acc[STRIDE]);
        const int64_t prod = (sum + l.addend) * l.mult;
        int32_t res;
        if (l.narrow) res = roundShift31(sum * l.mult + l.addend, l.shift, l.mask);
        else res = l.shift >= 1 ? static_cast<int32_t>(rshiftRoundConst(prod, l.shift, l.roundAdd)) : static_cast<int32_t>(prod << -l.shift);
        uint8_t keep;
        const int32_t code = clampCode(res + s.zpHh, s.loHh, s.hiHh, keep);
        return static_cast<uint32_t>(code * 2 + keep);
    }
    // the same of ROWS rows in place of the plane sums, one branch for all of them (T = 100, H = 256, 1024 rows in clusters of 16:
    // 631 -> 572 us)
    template <int STRIDE, int ROWS>
    __device__ __forceinline__ void totals(const Lane &l, uint32_t *acc) const {
        auto sumOf = [&](int r) { return (static_cast<int64_t>(static_cast<int32_t>(acc[r])) << 8) + static_cast<int32_t>(acc[r + STRIDE]); };
        auto codeOf = [&](int32_t res) {
            uint8_t keep;
            const int32_t code = clampCode(res + s.zpHh, s.loHh, s.hiHh, keep);
            return static_cast<uint32_t>(code * 2 + keep);
        };
        if (l.narrow) {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) acc[r] = codeOf(roundShift31(sumOf(r) * l.mult + l.addend, l.shift, l.mask));
        } else {
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const int64_t prod = (sumOf(r) + l.addend) * l.mult;
                acc[r] = codeOf(l.shift >= 1 ? static_cast<int32_t>(rshiftRoundConst(prod, l.shift, l.roundAdd)) : static_cast<int32_t>(prod << -l.shift));
            }
        }
    }
    __device__ __forceinline__ uint32_t linearOfTotal(uint32_t, const Lane &, const Fetch &, uint32_t code, Saved &) const { return code; }
    __device__ __forceinline__ int32_t activation(uint32_t shared, int g, int32_t qx, uint32_t &keepOut) const {
        const uint32_t lut = shared + g * static_cast<uint32_t>(sizeof(FastLut));
        int32_t threshold;
        uint32_t segments;
        asm("ld.shared.v2.u32 {%0, %1}, [%2];"
            : "=r"(threshold), "=r"(segments)
            : "r"(lut + 256 + (static_cast<uint32_t>(qx - s.loIn[g]) >> s.bucketShift[g]) * 8));
        int4 e;
        asm("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
            : "=r"(e.x), "=r"(e.y), "=r"(e.z), "=r"(e.w)
            : "r"(lut + (qx < threshold ? segments & 0xffffu : segments >> 16)));
        const int64_t sum = static_cast<int64_t>(e.x) * (qx - s.zpX[g]) + static_cast<uint32_t>(e.w);
        const int32_t y = roundShift31(sum, e.y, 2u * static_cast<uint32_t>(e.w) - 1u) + e.z;
        uint8_t keep;
        const int32_t code = clampCode(y, s.loOut[g], s.hiOut[g], keep);
        keepOut |= static_cast<uint32_t>(keep) << g;
        return code;
    }
    __device__ __forceinline__ uint32_t cell(uint32_t shared, State &st, const FetchB &in, const uint32_t (&v)[4]) const {
        uint32_t keep = 0;
        int32_t hh[3];
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            hh[g] = static_cast<int32_t>(v[g]) >> 1;
            keep |= (v[g] & 1u) << (6 + g);
        }
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            uint8_t k;
            const int32_t pre = clampCode(apply(in.ih[g] - s.zpIh, s.ihTo[g]) + apply(hh[g] - s.zpHh, s.hhTo[g]) + s.zpIn[g], s.loIn[g], s.hiIn[g], k);
            keep |= static_cast<uint32_t>(k) << (3 + g);
            st.code[g] = activation(shared, g, pre, keep);
        }
        {
            uint8_t k;
            const int64_t prod = static_cast<int64_t>(st.code[1] - s.zpOut[1]) * (hh[2] - s.zpHh);
            const int32_t pre = clampCode(apply(in.ih[2] - s.zpIh, s.ihTo[2]) + apply(prod, s.rhToNew) + s.zpIn[2], s.loIn[2], s.hiIn[2], k);
            keep |= static_cast<uint32_t>(k) << 5;
            st.code[2] = activation(shared, 2, pre, keep);
        }
        {
            uint8_t k;
            const int32_t fresh = apply(st.code[2] - s.zpOut[2], s.newToH);
            const int64_t sum = static_cast<int64_t>(st.code[0] - s.zpOut[0]) * (st.h - s.zpH) + static_cast<int64_t>(s.quantOne - st.code[0]) * fresh;
            st.h = clampCode(apply(sum, s.oldToH) + s.zpH, s.loH, s.hiH, k);
            keep |= static_cast<uint32_t>(k) << 12;
        }
        st.hhn = hh[2];
        st.keep = keep;
        return static_cast<uint32_t>(st.h - s.loH);
    }
    // All lanes of a cell store all of it: picking a lane's share costs more than the stores (H = 64: 93 against 77 us).
    template <int LANES = 1>
    __device__ __forceinline__ void store(const State &st, const FetchB &in, size_t at, uint32_t row, int unit, bool good, int = 0) const {
        const int H = hidden();
        const uint32_t mine = row * H + unit, mine3 = row * (3 * H) + unit;
        h[(at + B) * H + mine] = static_cast<float>(st.h - s.zpH) * scaleH(good);
        float *vRow = v + at * (4 * H) + (row * (4 * H) + unit);
#pragma unroll
        for (int g = 0; g < 3; ++g) vRow[g * H] = static_cast<float>(st.code[g] - s.zpOut[g]) * s.eff[g];
        vRow[3 * H] = static_cast<float>(st.hhn - s.zpHh) * s.effHh;
        if (hq) hq[(at + B) * H + mine] = st.h;
        if (vq) {
            int32_t *to = vq + at * (4 * H) + (row * (4 * H) + unit);
#pragma unroll
            for (int g = 0; g < 3; ++g) to[g * H] = st.code[g];
            to[3 * H] = st.hhn;
        }
        if (FLAGS == Flags::Packed)
            stepBits[at * H + mine] = static_cast<uint16_t>(st.keep | (in.keepIh[0] << 9) | (in.keepIh[1] << 10) | (in.keepIh[2] << 11));
        if (FLAGS == Flags::Bytes) {
            if (maskHh) {
                uint8_t *to = maskHh + at * (3 * H) + mine3;
#pragma unroll
                for (int g = 0; g < 3; ++g) to[g * H] = static_cast<uint8_t>((st.keep >> (6 + g)) & 1u);
            }
            if (maskGateIn) {
                uint8_t *toIn = maskGateIn + at * (3 * H) + mine3, *toOut = maskGateOut + at * (3 * H) + mine3;
#pragma unroll
                for (int g = 0; g < 3; ++g) {
                    toIn[g * H] = static_cast<uint8_t>((st.keep >> (3 + g)) & 1u);
                    toOut[g * H] = static_cast<uint8_t>((st.keep >> g) & 1u);
                }
                maskH[at * H + mine] = static_cast<uint8_t>((st.keep >> 12) & 1u);
            }
        }
    }
    template <int N>
    __device__ __forceinline__ void storeRows(const State (&st)[N], const FetchB (&in)[N], size_t at, int row, int unit, bool good, int count) const {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i < count) store(st[i], in[i], at, row + i, unit, good);
    }
    __device__ __forceinline__ void storeLinear(const Lane &, const Saved &, size_t, uint32_t, int, int) const {}
    __device__ __forceinline__ void finish(const State &, int, int, bool) const {}
};

bool ready(const Rescale &r, ReadyRescale &out) {
    if (r.shift < 1 || r.shift > 31) return false;
    out = ReadyRescale{r.mult, r.shift, 1u << (r.shift - 1), (1u << r.shift) - 1u};
    return true;
}
bool ready(const Rescale &r, ReadyWide &out) {
    if (r.shift < 1 || r.shift > 62) return false;
    out = ReadyWide{r.mult, r.shift, (int64_t{1} << (r.shift - 1)) - 1};
    return true;
}

// Bucket map of one table over the gate-input grid; false when a shift leaves [1, 31] or a bucket holds two thresholds.
bool ready(const Lut &lut, int32_t lo, int32_t hi, FastLut &out, int32_t &bucketShift) {
    const int64_t span = static_cast<int64_t>(hi) - lo + 1;
    bucketShift = 0;
    while ((span - 1) >> bucketShift >= kBuckets) ++bucketShift;
    auto segmentOf = [&](int64_t q) {
        for (int i = 0; i < kSegments - 1; ++i)
            if (q < lut.threshold[i]) return i;
        return kSegments - 1;
    };
    for (int i = 0; i < kSegments; ++i) {
        if (lut.n_bx[i] < 1 || lut.n_bx[i] > 31) return false;
        out.segment[i] = make_int4(lut.q_b[i], lut.n_bx[i], lut.term_c[i], static_cast<int>(1u << (lut.n_bx[i] - 1)));
    }
    for (int b = 0; b < kBuckets; ++b) {
        const int64_t first = lo + (static_cast<int64_t>(b) << bucketShift), last = std::min<int64_t>(first + (int64_t{1} << bucketShift) - 1, hi);
        if (first > hi) {
            out.bucket[b] = make_uint2(0u, 0u);
            continue;
        }
        const int s0 = segmentOf(first), s1 = segmentOf(last);
        // only the threshold of s0 may lie in (first, last]
        if (s1 != s0 && segmentOf(lut.threshold[s0]) != s1) return false;
        const int32_t threshold = s0 == s1 ? INT32_MAX : lut.threshold[s0];
        out.bucket[b] = make_uint2(static_cast<uint32_t>(threshold), static_cast<uint32_t>(16 * s0) | (static_cast<uint32_t>(16 * s1) << 16));
    }
    return true;
}

// Everything of the cell that does not depend on the width or on what is saved.
struct Prepared {
    CellScalars s;
    FastLut luts[3];
};

template <int HP, Flags FLAGS, int WIDTH>
void launchFor(const WideRecurrence &r, const Prepared &prepared, cudaStream_t st) {
    using Cell = GruPlaneCell<FLAGS, WIDTH>;
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
    const planerec::Problem problem{r.T, r.B, r.H, r.h0Planes};
    if constexpr (HP == 64 || HP == 128)
        if (lanerec::launch<Cell, HP / 4, 2>("recurrentForward", problem, cell, st)) return;
    if constexpr (HP < 64) planerec::launchBest<Cell, HP, HP, 2, 32, 8, 16>("recurrentForward", problem, cell, st);
    else planerec::launchBest<Cell, HP, 64, 2, 32, 4, 8, 16>("recurrentForward", problem, cell, st);
}
template <int HP>
void launchFor(const WideRecurrence &r, const Prepared &prepared, cudaStream_t st) {
    auto run = [&](auto width) {
        constexpr int kWidth = decltype(width)::value;
        if (r.stepBits) launchFor<HP, Flags::Packed, kWidth>(r, prepared, st);
        else if (r.maskHh || r.maskGateIn) launchFor<HP, Flags::Bytes, kWidth>(r, prepared, st);
        else launchFor<HP, Flags::None, kWidth>(r, prepared, st);
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
    bool ok = ready(g.rh_to_new, s.rhToNew) && ready(g.new_to_h, s.newToH) && ready(g.update_old_to_h, s.oldToH);
    for (int i = 0; i < 3 && ok; ++i) {
        ok = ready(ihTo[i], s.ihTo[i]) && (i == 2 || ready(hhTo[i], s.hhTo[i])) &&
             ready(*luts[i], g.qlo[inOp[i]], g.qhi[inOp[i]], cell.luts[i], s.bucketShift[i]);
        s.zpIn[i] = g.zp[inOp[i]]; s.loIn[i] = g.qlo[inOp[i]]; s.hiIn[i] = g.qhi[inOp[i]];
        s.zpOut[i] = g.zp[outOp[i]]; s.loOut[i] = g.qlo[outOp[i]]; s.hiOut[i] = g.qhi[outOp[i]];
        s.zpX[i] = luts[i]->zp_x; s.eff[i] = g.eff[outOp[i]];
    }
    if (!ok) return false;
    s.zpIh = g.zp[RXMET_GRU_WEIGHT_IH_LINEAR];
    s.zpHh = g.zp[RXMET_GRU_WEIGHT_HH_LINEAR]; s.loHh = g.qlo[RXMET_GRU_WEIGHT_HH_LINEAR]; s.hiHh = g.qhi[RXMET_GRU_WEIGHT_HH_LINEAR];
    s.effHh = g.eff[RXMET_GRU_WEIGHT_HH_LINEAR];
    s.zpH = g.zp[RXMET_GRU_H]; s.loH = g.qlo[RXMET_GRU_H]; s.hiH = g.qhi[RXMET_GRU_H]; s.effH = g.eff[RXMET_GRU_H];
    s.quantOne = g.quant_one;
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
    if (r.H <= 32 && lanerec::rowsFor<16, 2>(r.B) == 0) launchFor<32>(r, prepared, st);
    else if (r.H <= 64) launchFor<64>(r, prepared, st);
    else if (r.H <= 128) launchFor<128>(r, prepared, st);
    else if (r.H <= 192) launchFor<192>(r, prepared, st);
    else launchFor<256>(r, prepared, st);
}

}  // namespace gru
}  // namespace rxmet
