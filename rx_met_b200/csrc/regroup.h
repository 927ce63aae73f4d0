// Arrays of 32-bit elements between a layer's own widths and widths that the tensor-core kernels tile.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace rxmet {

// dst[g][r][c][j] = src[g][r][c][j] for g < rowGroups, c < colGroups; elements that src does not have take `fill`.
struct RegroupJob {
    const void *src = nullptr;
    void *dst = nullptr;
    int rowGroups = 1, srcRows = 0, dstRows = 0;    // rows of a group
    int colGroups = 1, srcWidth = 0, dstWidth = 0;  // elements of a column group
    uint32_t fill = 0;
    const uint8_t *mask = nullptr;                  // optional, in the layout of dst: elements are floats, dropped ones become 0
    int maskKeeps = 1;                              // 1: a nonzero byte keeps the element, 0: it drops it
};

constexpr int kMaxRegroupJobs = 16;
// One launch; false where no array has anything to copy and nothing was launched.  Kernels behind it may start early, once everything before it is complete.
bool regroup(const char *name, const RegroupJob *jobs, int count, cudaStream_t stream);

}  // namespace rxmet
