// W8 / A16 forward of the QuantGRU integer carrier on byte planes (gru_forward_wide.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"
#include "gru_params.h"

namespace rxmet {
namespace gru {

// Operands in the workspace, filled by prepareWide (gru_forward_quant.cu).
struct WideOperands {
    int kI, kH, tileWords, hPad;        // words of a row of x / h (K padded to 16 bytes), of a channel's row in a tile; codes of a row of h0
    uint32_t *xPlanes, *h0Planes;       // [T*B][2][kI], [B][2][kH] words of four bytes of code - grid minimum, high bytes first
    int16_t *h0Codes;                   // [B][hPad]
    uint32_t *wWords, *rWords;          // [kI][3H], [kH][3H]: four weight codes along K per word
    int64_t *addX, *addH;               // [3H]: (grid minimum - zero point) * sum of the weight codes + bias on the accumulator grid
    uint4 *wTiles;                      // input weights as tensor-core tiles (plane_proj_umma.cuh); null: the dp4a projection runs
    int *projStatus;
    int16_t *ihCodes;                   // [T*B][3H]
};
WideOperands wideOperands(Workspace &workspace, int T, int B, int I, int H);

struct WideCall {
    int T, B, I, H;
    WideOperands operands;
    const Rescale *gemmX, *gemmH;
    float *h, *v;
    int32_t *hq, *vq;                   // optional
    uint8_t *maskIh, *maskHh, *maskGateIn, *maskGateOut, *maskH;  // optional keep flags
    uint16_t *stepBits;                 // optional packed flags
};

// Weight grids of at most 8 bits, x / h grids of at most 16 bits, linear grids of at most 16 bits, H <= 512.
bool forwardWideTakes(const Exec &exec, int I, int H);
size_t forwardWideExtraBytes(int T, int B, int I, int H);
void forwardWide(const WideCall &call, const Exec &exec, cudaStream_t stream);

// Operands of the recurrence alone, after the input projection.
struct WideRecurrence {
    int T, B, H;
    const uint32_t *words;     // [kWords][3H]: four recurrent weight bytes along K
    const int64_t *addend;     // [3H]
    const Rescale *rescale;    // [3H]
    const int16_t *ih;         // [T][B][3H]
    const int16_t *h0;         // [B][hPad] codes
    int hPad;
    const uint32_t *h0Planes;  // [B][2][kWords]
    float *h, *v;              // [T+1][B][H], [T][B][4H] dequantized
    int32_t *hq, *vq;          // optional codes
    uint8_t *maskHh, *maskGateIn, *maskGateOut, *maskH;
    const uint8_t *maskIh;     // with stepBits: the input projection's keep flags
    uint16_t *stepBits;        // optional [T][B][H]: the 13 flags of an element packed (instead of the byte masks)
    const int *poison;         // status word of the tensor-core projection: non-zero turns the hidden outputs into NaN
};
// The recurrence over thread-block clusters (gru_forward_cluster.cu), and whether it takes the shape and the parameters.
bool forwardWideClusterTakes(const Exec &exec, int B, int H);
void forwardWideCluster(const WideRecurrence &r, const Exec &exec, cudaStream_t stream);

}  // namespace gru
}  // namespace rxmet
