// step_chain.cuh -- launches of step kernels that follow one another directly on a stream.
//
// Between two ordinary launches the chip is idle for about 2 us: the last blocks drain, then the next
// grid starts and its first blocks read their metadata. A step kernel launched `after` another one comes
// resident while the other's last blocks run (programmatic dependent launch), reads what no step
// changes, and waits at step_wait() for the other to end with its stores visible. us per step, ordinary
// launches -> chained ones: 129x97x113 with 3 FP32 species (two launches a step) 23.9 -> 18.7; 27 k
// nodes of FP32 flow 8.2 -> 3.0, 482 k 22.5 -> 15.2; 256x128x128 FP32 flow 52.4 -> 51.3.
#pragma once

#include <cuda_runtime.h>

#include <utility>

namespace clb {

// Called by every thread of a step kernel, after its reads of what no step kernel writes (node metadata,
// velocities, parameters) and before any other access to memory. Let the next kernel's blocks in only
// after the wait: so when they start, everything before the kernel they follow is complete.
__device__ __forceinline__ void step_wait() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

// kern<<<grid, block, smem, stream>>>(args...); after: the stream's latest work is a kernel that calls
// step_wait(), launched since the last change of anything read ahead of it.
template <typename... P, typename... A>
inline void launch_step(bool after, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr = {};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = after ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, P(std::forward<A>(args))...);
}

}  // namespace clb
