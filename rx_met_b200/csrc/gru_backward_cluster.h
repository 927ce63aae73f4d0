// Reverse-time recurrence of the GRU backward over thread-block clusters (QAT, 8-bit weight codes).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace rxmet {
namespace gru {

// What every kernel of the reverse recurrence reads and writes.
struct BackwardQArgs {
    int T, B, H;
    const uint32_t *RB;      // packed codes of the register kernel, see packRecurrentBf16
    const float *scaleR;     // [3H] effective scale per column
    const float *h, *v, *dhNew;
    float *dp, *dq, *dh0;
    const uint8_t *mIh, *mHh, *mGateIn, *mGateOut, *mH, *mH0;
    const uint16_t *stepBits;  // packed keep flags, see packStepMasks; null = nothing was clamped
    // a sequence cut into time chunks: the gradient that flows into the chunk's last step from the later chunk, and
    // whether dh0 receives this chunk's outgoing gradient as it is (1) or, at the start of the sequence, under
    // the h0 mask (0)
    const float *dhIn;
    int carryOut;
};

// True when the cluster kernel takes the call: hidden units in tiles of 32, at most 256 of them, pointers aligned for its
// paired accesses.  `Rq` = [H][3H] int32 codes of at most 8 bits.
bool backwardClusterTakes(const BackwardQArgs &q, const int32_t *Rq);
void backwardCluster(const BackwardQArgs &q, const int32_t *Rq, cudaStream_t stream);
// Its part up to 128 units, in steps of 32 (gru_backward_units.cu).
void backwardUnits(const BackwardQArgs &q, const int32_t *Rq, cudaStream_t stream);

}  // namespace gru
}  // namespace rxmet
