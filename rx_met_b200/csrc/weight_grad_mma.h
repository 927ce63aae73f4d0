// Tensor-core weight-gradient GEMM shared by the GRU and LSTM backward passes.
//
// partial[s][m][n] = sum over the s-th chunk of the K rows of A[k][m] * B[k][n], for m < M, and
// partial[s][M][n] = the column sums of B over the same rows, i.e. the bias gradient.
// A holds small integers (activation codes minus their zero point), which bf16 represents exactly:
// magnitude at most 256 as one term, or - for 16-bit activation grids - below 2^16 as the two terms
// 256 * floor(a / 256) and a mod 256; B (fp32 gradients) is split into three bf16 terms that together
// carry all 24 significand bits, so every product is exact and only the fp32 accumulation rounds.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace rxmet {
namespace wgrad {

struct Problem {
    const int32_t *aCodes = nullptr;  // [K][M] integer codes, or
    const float *aFloat = nullptr;    // [K][M] floats: the integer is rint(value * aInvScale) - aFloatZero
    float aInvScale = 1.0f;
    float aFloatZero = 0.0f;
    int32_t aZero = 0;                // zero point of aCodes
    int M = 0;                        // real rows (multiple of 4; the mma.sync kernel: at most 143); row M is the ones row
    const float *B = nullptr;         // [K][N] gradients, N a multiple of 4
    float *partial = nullptr;         // [splits][M+1][N]
    int *status = nullptr;            // device word, set to 1 when a bounded wait of the kernel gave up
    // tcgen05 kernel only: the codes of the first rows, where they are an array of their own; the others' lie at aFloat then
    const float *aFirst = nullptr;    // [firstRows][M]
    int firstRows = 0;
};

// The mma.sync kernel: one problem cut into K splits of chunkK rows each (a multiple of its K tile).
struct Plan {
    int splits = 0;
    int chunkK = 0;
};
Plan plan(int K, int N, int sms);
void launch(const Problem &problem, int K, int N, const Plan &plan, cudaStream_t stream);
// Upper bound of plan(...).splits over every device, for sizing the partial buffers.
int splitBound(int K);

// The tcgen05 kernel (weight_grad_umma.cu): two problems over the same K rows and N columns (the input and the recurrent weights of a step) in
// one launch.  M a multiple of 4 up to sixteen tiles of 256, N a multiple of 128 or 192; operands 16-byte aligned.  RXMET_WGRAD_MMA_SYNC in the environment turns it off.
constexpr int kMaxSms = 160;
struct PairPlan {
    int splits[2], chunks[2];   // of a and b: K splits, chunks of 32 rows in a split
};
bool tensorMemoryPath(int Ma, int Mb, int N);
// wide: |code - zero point| may exceed 256 (two terms a code)
PairPlan planPair(const Problem &a, const Problem &b, int K, int N, bool wide, int sms);
int planRows(const PairPlan &plan);   // most rows of a split
void launchPair(const Problem &a, const Problem &b, int K, int N, const PairPlan &plan, bool wide, cudaStream_t stream);
// Upper bound of a problem's splits over every device, for sizing its partial sums.
int tileSplitBound(int M, int N);

// The tensor core truncates every addition to an accumulator.  Largest error of a sum of n terms of one sign: up to 128 elements (accumulators for the
// leading terms) 4e-7 with 8-bit codes up to 4096 rows, 6e-9 n with 16-bit codes (512 rows: 3.1e-6, 4096: 2.3e-5); beyond 128 elements (one accumulator)
// 2e-8 n with 8-bit codes (384 rows: 7.4e-6) and 3.5e-8 n with 16-bit codes (384 rows: 1.3e-5).  Calls that would otherwise take
// the FP32 kernels therefore cut the rows into chunks of kChainRows, however many there are: up to kChainGroup chunks (three
// waves of the widest layers) leave their partial sums to the reduction that follows, more go in several launches, after each of which
// addPartials folds the partial sums into one more array of them, so that the arrays do not grow with the rows.
constexpr int kChainRows = 512, kChainGroup = 32;
inline int chainChunks(int K) { return (K + kChainRows - 1) / kChainRows; }
// Arrays of (M + 1) x N partial sums that launchChained() writes.
inline int chainPartials(int K) { return chainChunks(K) <= kChainGroup ? chainChunks(K) : kChainGroup + 1; }
// sums of a and b (sum[i] = or += partial[0][i] + partial[1][i] + ...), `partial` behind the sums
void addPartials(float *a, size_t countA, float *b, size_t countB, int partials, bool first, cudaStream_t stream);
PairPlan chainPlan(int K);   // kChainRows a split
// More chunks than kChainGroup in one launch all the same, where the partial sums that tileSplitBound makes room for are enough: as many splits, of at
// most kChainRows rows, as fill whole waves of CTAs.  No splits: not enough room.  8-bit GRU training, T = 100, B = 256, I = 40, H = 16: two launches and two
// folds 194 us a pass, one launch 179; LSTM, T = 200, B = 200, H = 30 381 -> 331.
PairPlan finePlan(const Problem &a, const Problem &b, int K, int N, int sms);
// Both problems in chunks of kChainRows; returns the number of partial sums at a.partial and b.partial.
inline int launchChained(const Problem &a, const Problem &b, int K, int N, bool wide, cudaStream_t stream) {
    const int chunks = chainChunks(K);
    if (chunks <= kChainGroup) {
        launchPair(a, b, K, N, chainPlan(K), wide, stream);
        return chunks;
    }
    const size_t countA = static_cast<size_t>(a.M + 1) * N, countB = static_cast<size_t>(b.M + 1) * N;
    for (int first = 0; first < chunks; first += kChainGroup) {
        const size_t row = static_cast<size_t>(first) * kChainRows;
        const int rows = std::min(K - static_cast<int>(row), kChainGroup * kChainRows);
        auto part = [&](Problem p, size_t count) {
            if (p.aCodes) p.aCodes += row * p.M;
            if (p.aFloat) p.aFloat += row * p.M;
            p.B += row * N;
            p.partial += count;
            return p;
        };
        launchPair(part(a, countA), part(b, countB), rows, N, chainPlan(rows), wide, stream);
        addPartials(a.partial, countA, b.partial, countB, chainChunks(rows), first == 0, stream);
    }
    return 1;
}
}  // namespace wgrad
}  // namespace rxmet
