// A warp takes four (row, column group) items at a time; bound by memory: 4 bytes in, 4 bytes out per element, coalesced along j.
// Blocks by array, as many as it has work for: with the largest array's number for each of them, most had nothing to do (T = 61, B = 45, H = 100:
// 10.1 -> 9.4 us, with packStepMasks beside it 16.3 -> 11.2).
#include "regroup.h"

#include <algorithm>

#include "common.h"
#include "dependent_launch.cuh"

namespace rxmet {
namespace {

struct Jobs {
    RegroupJob job[kMaxRegroupJobs];
    int firstBlock[kMaxRegroupJobs + 1];
    int count;
};

constexpr int kThreads = 256, kWarps = kThreads / 32, kItems = 4;

// Index: wide enough for all items, 32 bits wherever they do (a 64-bit division takes longer than the copy).
template <class Index>
__device__ __forceinline__ void regroupItems(const RegroupJob &p, Index items, int block, int blocks) {
    const int lane = threadIdx.x & 31;
    const uint32_t *__restrict__ src = static_cast<const uint32_t *>(p.src);
    uint32_t *__restrict__ dst = static_cast<uint32_t *>(p.dst);
    const Index colGroups = static_cast<Index>(p.colGroups), dstRows = static_cast<Index>(p.dstRows);
    for (Index first = static_cast<Index>(block * kWarps + static_cast<int>(threadIdx.x) / 32) * kItems; first < items; first += static_cast<Index>(blocks) * kWarps * kItems) {
        size_t from[kItems];
        int width[kItems];
#pragma unroll
        for (int n = 0; n < kItems; ++n) {
            const Index item = min(first + n, items - 1), row = item / colGroups, c = item - row * colGroups, g = row / dstRows, r = row - g * dstRows;
            from[n] = ((static_cast<size_t>(g) * p.srcRows + r) * p.colGroups + c) * p.srcWidth;
            width[n] = first + n >= items ? -1 : r < static_cast<Index>(p.srcRows) ? p.srcWidth : 0;   // -1: no such item
        }
        for (int j = lane; j < p.dstWidth; j += 32) {
            uint32_t v[kItems];
#pragma unroll
            for (int n = 0; n < kItems; ++n) v[n] = j < width[n] ? src[from[n] + j] : p.fill;
#pragma unroll
            for (int n = 0; n < kItems; ++n) {
                if (width[n] < 0) continue;
                const size_t to = static_cast<size_t>(first + n) * p.dstWidth + j;
                if (p.mask != nullptr && (p.mask[to] != 0) != (p.maskKeeps != 0)) v[n] = 0u;
                dst[to] = v[n];
            }
        }
    }
}

__global__ void __launch_bounds__(kThreads) regroupArrays(const __grid_constant__ Jobs jobs) {
    waitForPredecessor();
    letDependentsStart();
    int i = 0;
    while (i + 1 < jobs.count && static_cast<int>(blockIdx.x) >= jobs.firstBlock[i + 1]) ++i;
    const RegroupJob &p = jobs.job[i];
    const size_t items = static_cast<size_t>(p.rowGroups) * p.dstRows * p.colGroups;
    const int block = static_cast<int>(blockIdx.x) - jobs.firstBlock[i], blocks = jobs.firstBlock[i + 1] - jobs.firstBlock[i];
    if (items < (size_t{1} << 30)) regroupItems<uint32_t>(p, static_cast<uint32_t>(items), block, blocks);
    else regroupItems<size_t>(p, items, block, blocks);
}

}  // namespace

bool regroup(const char *name, const RegroupJob *jobs, int count, cudaStream_t st) {
    RXMET_REQUIRE(count <= kMaxRegroupJobs, "too many arrays in one launch");
    Jobs all{};
    const size_t most = 8 * static_cast<size_t>(currentDevice().sms);
    for (int i = 0; i < count; ++i) {
        if (jobs[i].dst == nullptr) continue;
        const size_t items = static_cast<size_t>(jobs[i].rowGroups) * jobs[i].dstRows * jobs[i].colGroups;
        all.job[all.count] = jobs[i];
        all.firstBlock[all.count + 1] = all.firstBlock[all.count] + static_cast<int>(std::min<size_t>((items + kWarps * kItems - 1) / (kWarps * kItems), most));
        ++all.count;
    }
    const int blocks = all.firstBlock[all.count];
    if (blocks == 0) return false;
    {
        KernelTimer timer__(name, st);
        launchDependent(regroupArrays, static_cast<unsigned>(blocks), kThreads, 0, st, all);
    }
    afterLaunch(name);
    return true;
}

}  // namespace rxmet
