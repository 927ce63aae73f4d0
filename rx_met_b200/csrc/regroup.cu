// One warp per (row, column group); bound by memory: 4 bytes in, 4 bytes out per element, coalesced along j.
#include "regroup.h"

#include <algorithm>

#include "common.h"

namespace rxmet {
namespace {

struct Jobs {
    RegroupJob job[kMaxRegroupJobs];
};

constexpr int kThreads = 256;

__global__ void __launch_bounds__(kThreads) regroupArrays(const __grid_constant__ Jobs jobs) {
    const RegroupJob &p = jobs.job[blockIdx.y];
    const int lane = threadIdx.x & 31;
    const size_t items = static_cast<size_t>(p.rowGroups) * p.dstRows * p.colGroups;
    const uint32_t *src = static_cast<const uint32_t *>(p.src);
    uint32_t *dst = static_cast<uint32_t *>(p.dst);
    for (size_t item = blockIdx.x * static_cast<size_t>(kThreads / 32) + threadIdx.x / 32; item < items;
         item += static_cast<size_t>(gridDim.x) * (kThreads / 32)) {
        const size_t row = item / p.colGroups;
        const int c = static_cast<int>(item - row * p.colGroups);
        const int g = static_cast<int>(row / p.dstRows), r = static_cast<int>(row - static_cast<size_t>(g) * p.dstRows);
        const size_t from = ((static_cast<size_t>(g) * p.srcRows + r) * p.colGroups + c) * p.srcWidth, to = item * p.dstWidth;
        const int width = r < p.srcRows ? p.srcWidth : 0;
        for (int j = lane; j < p.dstWidth; j += 32) {
            uint32_t v = j < width ? src[from + j] : p.fill;
            if (p.mask != nullptr && (p.mask[to + j] != 0) != (p.maskKeeps != 0)) v = 0u;
            dst[to + j] = v;
        }
    }
}

}  // namespace

void regroup(const char *name, const RegroupJob *jobs, int count, cudaStream_t st) {
    RXMET_REQUIRE(count <= kMaxRegroupJobs, "too many arrays in one launch");
    Jobs all{};
    size_t most = 1;
    int n = 0;
    for (int i = 0; i < count; ++i) {
        if (jobs[i].dst == nullptr) continue;
        all.job[n++] = jobs[i];
        most = std::max(most, static_cast<size_t>(jobs[i].rowGroups) * jobs[i].dstRows * jobs[i].colGroups);
    }
    if (n == 0) return;
    const size_t blocks = std::min<size_t>((most + kThreads / 32 - 1) / (kThreads / 32), 148 * 8);
    {
        KernelTimer timer__(name, st);
        regroupArrays<<<dim3(static_cast<unsigned>(blocks), static_cast<unsigned>(n)), kThreads, 0, st>>>(all);
    }
    afterLaunch(name);
}

}  // namespace rxmet
