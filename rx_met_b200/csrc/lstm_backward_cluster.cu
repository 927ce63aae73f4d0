// Reverse recurrence of the LSTM QAT backward over thread-block clusters: variants up to 256 hidden units and the launch.
#include <cuda_runtime.h>

#include <algorithm>

#include "lstm_backward_cluster.cuh"

namespace rxmet {
namespace lstm {
namespace {

using reverse::Variant;

template <int H, int ROWS>
Variant variant() {
    return reverse::variant<H, H % 64 == 0 ? 64 : 32, ROWS>();
}
template <int ROWS>
Variant variantFor(int H) {
    switch (H) {
        case 160: return variant<160, ROWS>();
        case 192: return variant<192, ROWS>();
        case 224: return variant<224, ROWS>();
        default: return variant<256, ROWS>();
    }
}
Variant variantFor(int H, int rows) {
    if (H > 256) return reverse::wideVariant(H, rows);
    return rows == 4 ? variantFor<4>(H) : rows == 8 ? variantFor<8>(H) : variantFor<16>(H);
}
int resident(const Variant &v) { return residentClusters(reinterpret_cast<const void *>(v.kernel), v.ctas, v.threads, v.smem); }

// A step of clusters of `rows` rows.  Beyond 256 units in us, as measured at 288 and 512 units and on a line between (384: 1.17, 1.35, 1.87, 2.22).  By 1 + rows / 32,
// which holds for the narrower ones, twenty rows cost 1.08 times sixteen instead of 1.2: of the calls with more than 560 rows some took 1 to 2.5 % longer
// (T = 60, H = 512, 1000 rows 3350 -> 3269 us a training pass).
double stepCost(int H, int rows) {
    if (H <= 256) return 1.0 + rows / 32.0;
    const double between = (H - 288) / 224.0;
    switch (rows) {
        case 4: return 1.13 + 0.11 * between;
        case 8: return 1.29 + 0.12 * between;
        case 16: return 1.66 + 0.56 * between;
        default: return 2.00 + 0.69 * between;
    }
}

}  // namespace

bool backwardClusterTakes(const BackwardClusterArgs &a) {
    for (const void *p : {static_cast<const void *>(a.gateOutputs), static_cast<const void *>(a.cellStates), static_cast<const void *>(a.cellTanh),
                          static_cast<const void *>(a.gradOutput), static_cast<const void *>(a.gradFinalHidden),
                          static_cast<const void *>(a.gradFinalCell), static_cast<const void *>(a.c0), static_cast<const void *>(a.dh0),
                          static_cast<const void *>(a.dc0), static_cast<const void *>(a.gIh), static_cast<const void *>(a.gHh),
                          static_cast<const void *>(a.channelScale), static_cast<const void *>(a.stepMasks)})
        if (!alignedTo(p, 8)) return false;
    return a.H % 32 == 0 && a.H >= 32 && a.H <= 512 && a.c0 != nullptr && (a.H <= 256 || resident(variantFor(a.H, 4)) > 0);
}

void backwardCluster(const BackwardClusterArgs &args, cudaStream_t st) {
    if (args.H <= 128) return backwardUnits(args, st);   // inside one CTA
    // Rows of a cluster: as few as let all clusters of the pass run at the same time; a second wave costs the whole chain again.
    int best = 4;
    double bestCost = 1e30;
    for (int rows : {4, 8, 16, 20}) {
        if (rows > 16 && args.H <= 256) break;
        const double step = stepCost(args.H, rows);
        if (step >= bestCost) break;   // not even in a single wave: leave the variant unloaded
        const Variant v = variantFor(args.H, rows);
        if (rows > 4 && resident(v) == 0) continue;
        const int held = std::max(1, resident(v) / concurrentPasses());
        const int clusters = (args.B + rows - 1) / rows, waves = (clusters + held - 1) / held;
        if (waves * step < bestCost) { bestCost = waves * step; best = rows; }
    }
    const Variant v = variantFor(args.H, best);
    ensureDynamicSmem(reinterpret_cast<const void *>(v.kernel), v.smem);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>((args.B + best - 1) / best * v.ctas));
    cfg.blockDim = dim3(static_cast<unsigned>(v.threads));
    cfg.dynamicSmemBytes = v.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = static_cast<unsigned>(v.ctas);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    {
        KernelTimer timer__("lstmRecurrentBackwardCluster", st);
        RXMET_CUDA(cudaLaunchKernelEx(&cfg, v.kernel, args));
    }
    afterLaunch("lstmRecurrentBackwardCluster");
}

}  // namespace lstm
}  // namespace rxmet
