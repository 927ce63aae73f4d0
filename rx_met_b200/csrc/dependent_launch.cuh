// Programmatic dependent launch: a kernel launched with launchDependent() may be scheduled while its predecessor on the
// stream still runs, and calls waitForPredecessor() before it touches anything an earlier kernel wrote or reads.  A kernel
// calls letDependentsStart() once its own wait is over: all its CTAs are resident then, so that waiting CTAs of the
// dependent cannot keep any of them from an SM.  Saves the launch latency between short kernels (1.5 to 3 us each).
// The one exception: packStepMasks (gru_backward.cu) waits only at its end when it is launched right behind regroupArrays, which lets it start after its
// own wait and writes nothing that it reads; the launch there makes sure of that.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "common.h"

namespace rxmet {

__device__ __forceinline__ void waitForPredecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void letDependentsStart() { asm volatile("griddepcontrol.launch_dependents;"); }

template <class... Params, class... Args>
void launchDependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, Args &&...args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    RXMET_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
}

}  // namespace rxmet
