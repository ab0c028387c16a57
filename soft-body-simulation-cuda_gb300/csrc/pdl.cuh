// Programmatic dependent launch (sm_90 and later), shared by the step
// kernels.  A kernel launched with programmatic stream serialization may be
// scheduled before its predecessor on the stream has finished: once every
// CTA of the predecessor has executed pdl_trigger (or exited).  Until its
// own pdl_wait returns -- after the predecessor grid has completed and its
// writes are visible -- it may only read data that no earlier kernel of
// the chain writes (layouts, coefficients, factor blocks).  Every CTA of a
// kernel launched this way waits before it can exit, so each grid
// completes after its predecessor and the order holds along the chain.
//
// The step's kernels trigger after their own wait, so that one successor at a
// time is scheduled early.  Triggered at entry, a chain cascades: ten or more
// grids become resident, each holding its CTAs' slots and waiting for the one
// before it (two refined steps of 18 launches an iteration take 1718 us that
// way, 930 us this way; two of the 10^3 dense cube 220 and 194 us).  The
// factorisation's panels, a few long CTAs at a time, gain from it and trigger
// at entry (10^3 dense: 5.9 ms against 8.1 ms).
#pragma once
#include <cuda_runtime.h>

#include "engine.h"

namespace pdgb {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// An SM changes its split between L1 and shared memory only when it is idle, so
// a kernel that wants another split than its predecessor cannot start beside
// it: the kernels of a chain all ask for the largest shared memory.
template <typename... P> inline void prefer_shared(void (*kernel)(P...)) {
    PDGB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                       cudaSharedmemCarveoutMaxShared));
}

template <typename... P, typename... A>
inline void launch_pdl_carve(void (*kernel)(P...), bool most_shared, int grid, int block, size_t smem, cudaStream_t s,
                             A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = cudaSharedmemCarveoutMaxShared;
    cfg.attrs = attr;
    cfg.numAttrs = most_shared ? 2 : 1;
    PDGB_CUDA_TRY(cudaLaunchKernelEx(&cfg, kernel, args...));
}

template <typename... P, typename... A>
inline void launch_pdl(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
    launch_pdl_carve(kernel, false, grid, block, smem, s, args...);
}

}  // namespace pdgb
