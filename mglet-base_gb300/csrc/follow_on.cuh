// follow_on.cuh -- programmatic launches: kernels of a chain that overlap at their ends.
#pragma once

#include "internal.h"

namespace mg {

// Launches that follow one another overlap at their ends: a launch may start
// when every CTA of the one before has passed follow_on(), reads its tables, and waits in
// follow_on() until the one before is complete.  A kernel calls it before its first look
// at anything a launch has written.
__device__ __forceinline__ void follow_on() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ int flag_at(const int* p) {
    int v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// A launch of such a kernel; nc > 1: in clusters of nc CTAs.
template <class... P, class... A>
int launch_follow_on(void (*k)(P...), dim3 grid, int threads, size_t smem, cudaStream_t s, int nc, A... args) {
    cudaLaunchAttribute at[2] = {};
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = nc;
    at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = at;
    cfg.numAttrs = nc > 1 ? 2 : 1;
    MG_CUDA(cudaLaunchKernelEx(&cfg, k, P(args)...));
    return 0;
}

}  // namespace mg
