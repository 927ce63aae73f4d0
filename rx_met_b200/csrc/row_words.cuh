// Walking a [rows][words] array by the CTAs of a job: every thread is given COUNT (row, word) pairs at a time, so that it can ask
// for all their operands before it uses the first.  The row comes from one high product: a 64-bit division per word costs more
// instructions than quantizing its four values.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace rxmet {

struct RowWord {
    size_t row;
    int word;
    bool real;
};

// f(const RowWord (&)[COUNT]) for all words of the array; `words` at most 2^15 / COUNT, `block` of `blocks` CTAs.
template <int COUNT, class F>
__device__ __forceinline__ void eachRowWord(size_t rows, int words, int block, int blocks, F f) {
    const uint32_t per = COUNT * blockDim.x, rowsOf = max(1u, per / static_cast<uint32_t>(words)), wordsOf = rowsOf * words;   // of a chunk
    // i / words = high word of i (2^32 / words + 1) for every i < 2^32 / words
    const uint32_t magic = words == 1 ? 0u : 0xffffffffu / static_cast<uint32_t>(words) + 1u;
    const size_t chunks = (rows + rowsOf - 1) / rowsOf;
    for (size_t chunk = block; chunk < chunks; chunk += blocks) {
        const size_t first = chunk * rowsOf;
        const uint32_t end = static_cast<uint32_t>(min(static_cast<size_t>(rowsOf), rows - first)) * words;
        for (uint32_t base = threadIdx.x; base < wordsOf; base += per) {
            RowWord at[COUNT];
#pragma unroll
            for (int n = 0; n < COUNT; ++n) {
                const uint32_t i = base + n * blockDim.x, r = words == 1 ? i : __umulhi(i, magic);
                at[n] = RowWord{first + r, static_cast<int>(i - r * words), i < end};
            }
            f(at);
        }
    }
}
// CTAs of `threads` threads that such a walk can use, at most `most`.
inline int rowWordBlocks(size_t rows, int words, int count, int threads, int most) {
    const size_t rowsOf = static_cast<size_t>(count) * threads / words > 0 ? static_cast<size_t>(count) * threads / words : 1;
    const size_t chunks = (rows + rowsOf - 1) / rowsOf;
    return static_cast<int>(chunks < 1 ? 1 : chunks < static_cast<size_t>(most) ? chunks : static_cast<size_t>(most));
}

}  // namespace rxmet
