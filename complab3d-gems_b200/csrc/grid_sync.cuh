// grid_sync.cuh -- a grid-wide barrier for kernels launched cooperatively (all blocks resident), with
// a bounded wait.
#pragma once

#include <cstdint>

namespace clb {

// Device words of one launch's barrier, zero when the launch starts.
struct GridSync {
    unsigned arrived;  // blocks that reached a barrier, over all barriers of the launch
    unsigned abort;    // nonzero: a wait gave up
};

// The `round`-th barrier of the launch (1, 2, ...), called by every thread of every block. What the
// blocks wrote before it is visible after it: each block's threads meet, one of them publishes with a
// fence and an increment, waits for the others, fences, and releases its block. False when a wait
// gave up, after `polls` looks; the caller then sets the handle's flag and returns.
__device__ __forceinline__ bool grid_barrier(GridSync* g, unsigned round, uint32_t polls) {
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned target = round * gridDim.x;
        __threadfence();
        atomicAdd(&g->arrived, 1u);
        int ok = 0;
        for (uint32_t it = 0; it < polls; ++it) {
            if (*(volatile unsigned*)&g->arrived >= target) {
                ok = 1;
                break;
            }
            if ((it & 255u) == 255u && *(volatile unsigned*)&g->abort) break;
        }
        if (!ok) atomicExch(&g->abort, 1u);
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

}  // namespace clb
