// Device-side scalar arithmetic of the QuantLSTM q-carrier, shared by the forward kernels.
// Every function keeps the float roundings of the reference literally (no contraction, one rounding
// per reference operation), because those roundings decide integer codes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "lstm_params.h"

namespace rxmet {
namespace lstm {
namespace dev {

// rint((v * M) * 2^-shift) with the product rounded once in float
// (applyRescaleCore, operators/quant-lstm/include/quantization/float_carrier_ops.h:77-92).
__device__ __forceinline__ float rescaleF(float v, DevRescale r) {
    return rintf(__fmul_rn(__fmul_rn(v, r.mult), r.pow2));
}

// value -> clamp(rint(value / scale) + zp): division and rounding in double as the reference does
// (quantizeFp, float_carrier_ops.h:49-59).
__device__ __forceinline__ int32_t quantizeCode(float v, float scale, int32_t zp, int32_t lo, int32_t hi, uint8_t &clamped) {
    const double t = rint(static_cast<double>(v) / static_cast<double>(scale)) + static_cast<double>(zp);
    clamped = (t < static_cast<double>(lo)) || (t > static_cast<double>(hi));
    return t <= static_cast<double>(lo) ? lo : (t >= static_cast<double>(hi) ? hi : static_cast<int32_t>(t));
}

// The same codes and flags, four at a time, without a double-precision division per value.  n = v / scale rounded from the reciprocal is
// the nearest integer or, close to a tie, its neighbour; v - n scale is exact in one fused multiply-add and says which.  A quotient of two
// floats below 2^19 in magnitude that is no tie is at least 2^-45 of its size away from one, so that the reference's quotient in
// double rounds to the same integer.  Codes stay floats: integers below 2^24 throughout.
struct CodeGrid {
    float scale, inverse, half, zp, lo, hi;
    bool plain;   // the form above holds: not for scales near the ends of the float range or wide grids
    __device__ __forceinline__ CodeGrid(float s, int32_t z, int32_t l, int32_t h) {
        scale = s; half = 0.5f * s; zp = static_cast<float>(z); lo = static_cast<float>(l); hi = static_cast<float>(h);
        inverse = __frcp_rn(s);
        constexpr int kLimit = 1 << 21;
        plain = s > 0x1p-100f && s < 0x1p100f && abs(z) < kLimit && abs(l) < kLimit && abs(h) < kLimit;
    }
    // Codes before the clamp to [lo, hi]; false: a quotient beyond 2^19 or NaN is among them, take quantizeCode for all.
    __device__ __forceinline__ bool codes(const float (&v)[4], float (&x)[4]) const {
        float rest[4], shifted[4], size = 0.0f, off = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float t = __fmul_rn(v[e], inverse);
            size += fabsf(t);
            shifted[e] = __fadd_rn(t, 12582912.0f);   // 1.5 * 2^23: the integer in the low bits
            x[e] = __fadd_rn(shifted[e], -12582912.0f);
            rest[e] = __fmaf_rn(-x[e], scale, v[e]);
            off = fmaxf(off, fabsf(rest[e]));
        }
        if (off >= half) {   // ties and their neighbours
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float far = fabsf(rest[e]);
                if (far > half || (far == half && (__float_as_int(shifted[e]) & 1))) x[e] += copysignf(1.0f, rest[e]);
            }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] += zp;
        return size < 524288.0f;
    }
};

// accumulator (already a float) -> centred linear code (code - zero point) and its clamp flag
// (linearValue, operators/quant-lstm/src/lstm/forward_quantized_fp_cpu.cc:17-45).
__device__ __forceinline__ float linearCentredF(float total, DevRescale out, float cLo, float cHi, uint8_t &clamped) {
    const float r = rescaleF(total, out);
    clamped = (r < cLo) || (r > cHi);
    return fminf(fmaxf(r, cLo), cHi);
}

// Cell-update ratio (scaleCellProductFpCore, operators/quant-lstm/include/lstm/quantized_cell_fp.h:72-80).
// The double-precision form (ratios that do not fit Q31) sits behind a call, so that the common
// single multiply is not accompanied by a speculative evaluation of it.
static __device__ __noinline__ float scaleCellWide(float product, double mantissa, int exponent) {
    return static_cast<float>(ldexp(static_cast<double>(product) * mantissa, exponent));
}
__device__ __forceinline__ float scaleCell(float product, float ratio, double mantissa, int exponent, int usesFp) {
    if (usesFp) return scaleCellWide(product, mantissa, exponent);
    return __fmul_rn(product, ratio);
}

// Four signed bytes times four unsigned bytes, accumulated.
__device__ __forceinline__ int32_t dotSignedUnsigned(uint32_t signedBytes, uint32_t unsignedBytes, int32_t acc) {
    int32_t d;
    asm("dp4a.s32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(signedBytes), "r"(unsignedBytes), "r"(acc));
    return d;
}

}  // namespace dev
}  // namespace lstm
}  // namespace rxmet
