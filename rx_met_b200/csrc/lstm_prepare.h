// Everything a quantized LSTM call on byte planes needs before its input projection, in one launch (lstm_prepare.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "lstm_params.h"

namespace rxmet {
namespace lstm {

// A tensor [rows][cols] on one grid.
struct PrepareRows {
    const float *src;     // null: real zeros
    size_t rows;
    int cols, words;      // words of four codes of a row, padding included
    float scale;
    int32_t zp, lo, hi;
    uint32_t *planes;     // optional [rows][planes][words]: code - lo, the high bytes first where there are two planes
    float *centred;       // optional [rows][cols]: code - zp
    float *carrier;       // optional [rows][cols]: the code
    uint8_t *clamped;     // optional [rows][cols]
};
// The weights of one side, [4H][K].
struct PrepareWeights {
    const float *w, *b;            // b: optional
    int K, words;                  // words of four codes of a channel, padding included
    int scaleField, biasScaleField, biasMultField, biasPow2Field;
    int64_t correction;            // grid minimum - zero point of the codes they are multiplied with
    int64_t *addend;               // [4H] correction * row sum + rescaled bias
    float *carrier, *biasCarrier;  // optional
    uint8_t *clamped, *biasClamped;
};
struct PrepareCall {
    int H, planes;
    const float *channel;          // kChannelFields x 4H
    int32_t wLo, wHi, bLo, bHi;
    PrepareWeights ih, hh;
    uint32_t *ihWords;             // optional [words][4H]
    uint32_t *ihTiles;             // optional tensor-core tiles (plane_proj_umma.cuh), k padding and channels beyond 4H zero
    uint32_t *hhWords;             // [2 gate pairs][words][H][2]
    PrepareRows x, h0, c0;
    int *clear;                    // status word of a later kernel, set to 0
};
// Kernels launched behind it may start early (dependent_launch.cuh).
void prepare(const PrepareCall &call, cudaStream_t stream);

}  // namespace lstm
}  // namespace rxmet
