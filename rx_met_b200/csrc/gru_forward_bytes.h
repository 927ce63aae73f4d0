// The 8-bit QuantGRU recurrence on the kernel with a thread per unit (gru_forward_bytes.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gru_params.h"

namespace rxmet {
namespace gru {

// Operands of a recurrence on small 8-bit grids whose input contributions are rescaled to the gate inputs already (mode 2 of
// gru_forward_quant.cu).
struct ByteRecurrence {
    int T, B, H, kWords;
    const uint32_t *words;     // [kWords][3H]: four recurrent weight codes along K
    const int64_t *comp, *biasAcc;   // [3H] zero-point correction and bias on the accumulator grid
    const Rescale *rescale;    // [3H]
    const int16_t *ih;         // [T][B][3H]
    const int8_t *h0;          // [B][4 kWords] codes; null: the zero point
    float *h, *v;              // [T+1][B][H], [T][B][4H] dequantized
    int32_t *hq, *vq;          // optional codes
    uint8_t *maskHh, *maskGateIn, *maskGateOut, *maskH;   // optional keep flags
    const uint8_t *maskIh;     // with stepBits: the input projection's keep flags
    uint16_t *stepBits;        // optional [T][B][H]: the 13 flags of an element packed
    const int *poison;         // status word of the tensor-core projection: non-zero turns the hidden outputs into NaN
};
// Whether it takes the shape (offsets inside a step have to fit 32 bits) and is the faster kernel for it; saves: codes or flags are asked for.
bool forwardBytesTakes(int T, int B, int H, bool saves);
void forwardBytes(const ByteRecurrence &r, const GateExec &g, cudaStream_t stream);

}  // namespace gru
}  // namespace rxmet
