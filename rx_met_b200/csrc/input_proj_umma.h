// Input projection of the 8-bit QuantGRU path as a tcgen05 kind::i8 GEMM with the fused integer
// epilogue (input_proj_umma.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "gru_device.cuh"

namespace rxmet {
namespace iproj {

struct Problem {
    const int32_t *x = nullptr;        // [rows][kWords] words of four signed 8-bit codes, rows back to back
    int rows = 0, kWords = 0, kPad = 0;  // kPad (bytes of k per row in shared memory) is filled in by launch()
    const int32_t *w = nullptr;        // [kWords][C] words of four signed 8-bit weight codes
    int C = 0;
    const int64_t *comp = nullptr;     // [C] zero-point compensation sum_k W * zp_x
    const int64_t *biasAcc = nullptr;  // [C] bias on the accumulator grid
    const gru::Rescale *rescale = nullptr;  // [C] accumulator -> output grid
    int32_t zpOut = 0, lo = 0, hi = 0;
    gru::PreRescale pre{};
    int16_t *out = nullptr;            // [rows][C]
    uint8_t *mask = nullptr;           // [rows][C] keep flags, optional
    int *status = nullptr;             // device word, set to 1 when a bounded wait of the kernel gave up
    // SMs that the recurrence behind the projection needs, one a CTA or as unitrec::smsFor counts them.  Where both find SMs of their own it starts with the projection's first CTAs and prepares
    // itself beside them; where they do not, with the last (late, filled in by launch()): CTAs that take the room left among those of a
    // projection lie unevenly on the SMs for the whole sequence (inference in lanes: 16 units, T 200, 200 rows 141 -> 75 us, T 98, 300 rows 88 -> 48; 64 units,
    // 80 inputs, T 200, 128 rows 122 -> 89).
    int dependents = 0;
    bool late = false;
};

// Codes of all channels and two items of rows within 200 kB, rows of x on a word boundary.  RXMET_IPROJ_SIMT in the environment turns the path off.
bool eligible(int C, int kWords, const void *x);
void launch(const Problem &problem, int sms, cudaStream_t stream);

}  // namespace iproj
}  // namespace rxmet
