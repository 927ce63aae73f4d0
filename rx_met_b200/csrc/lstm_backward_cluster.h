#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "lstm_kernels.h"

namespace rxmet {
namespace lstm {

// What the reverse recurrence over thread-block clusters reads and writes (QAT: saved tensors are codes held in floats).
struct BackwardClusterArgs {
    int T, B, H;
    const uint32_t *stepMasks;    // packed clamp flags [T][B][H] (packStepMasks) or null
    const float *weightCodes;     // [4H][H] integer codes of at most 8 bits
    const float *channelScale;    // [4H]
    const float *c0;              // [B][H] codes
    const float *gateOutputs, *cellStates, *cellTanh;
    const float *gradOutput, *gradFinalHidden, *gradFinalCell;
    Dequant dqC, dqGate[4], dqTanh;
    const uint8_t *maskH0, *maskC0;   // optional, non-zero = clamped
    float *gIh, *gHh;             // [T][B][4H]
    float *dh0, *dc0;             // [B][H]
};

// True when the kernel takes the call: hidden units in tiles of 32, at most 512 of them, pointers aligned for its paired accesses.
bool backwardClusterTakes(const BackwardClusterArgs &args);
void backwardCluster(const BackwardClusterArgs &args, cudaStream_t stream);
// Its part up to 128 units, in steps of 32 (lstm_backward_units.cu).
void backwardUnits(const BackwardClusterArgs &args, cudaStream_t stream);

}  // namespace lstm
}  // namespace rxmet
