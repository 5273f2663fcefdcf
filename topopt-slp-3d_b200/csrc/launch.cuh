// Launches of the kernels that a CG iteration is made of.
//
// An iteration is 20 to 60 short kernels, each waiting for the one before:
// with ordinary launches a grid is set up only after the last block of its
// predecessor is done and its writes are flushed, about 1 us in which nothing
// runs.  launch_dep lets a grid start while its predecessor still runs
// (programmatic dependent launch, also inside captured graphs); every kernel
// launched with it calls dep_wait before it touches memory that other kernels
// write or read, which returns when all work before it is complete and
// visible.  The vectors that kernels hand on are not read as read-only data
// (no __restrict__, no __ldg): the grid may have begun before they were written.
// 64x32x32 FP64 W-cycle step 6.27 -> 5.90 ms, 96x48x48 MR 2 5.32 -> 5.15 ms.
// Solves that share the GPU (the serving loop) launch the same kernels
// ordinarily: grids that wait early keep their blocks' places from the other
// streams (eight 32x16x16 requests: 9.57 against 9.27 ms).
#pragma once

#include <cuda_runtime.h>

#include "tosp_internal.h"

namespace tosp {

// Lets the next grid start; first thing in a kernel launched with launch_dep.
__device__ __forceinline__ void dep_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// Waits for all earlier work of the stream.
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void dep_enter() {
    dep_start();
    dep_wait();
}

template <typename... P, typename... A>
void launch_dep(void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at = {};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = dependent_launches() ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...);
    count_launch();
}

}  // namespace tosp
