// Kernel launches with programmatic dependent launch (PDL).
//
// Every kernel of the hot path calls grid_dep_wait() (griddepcontrol.wait: returns once
// the preceding kernel in stream order has completed and its writes are visible) before
// it reads anything, and grid_dep_launch() (griddepcontrol.launch_dependents) once the
// next kernel's blocks may be scheduled: the short per-stage kernels trigger at their
// start, the long tile kernel only before its last pass, so waiting blocks of the next
// kernel do not sit beside it while it still works.  The ordering is that of a plain
// stream launch; inside a captured graph the dependency becomes a programmatic edge.
// FFB_PDL=0 in the environment launches without the attribute (the device instructions
// are then no-ops).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace ffb {

bool pdl_enabled();

__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Loads of what the preceding kernel may still be writing when this one starts: its outputs,
// read after grid_dep_wait().  Such memory changes during this kernel's lifetime, so neither
// __ldg, whose value the compiler may take at any time, nor the non-coherent path (.nc, to which
// a const __restrict__ parameter leads as well) may read it.  Plain loads do, since the wait is a
// barrier to them; these do too, and keep their order among each other where a loop
// fetches ahead.  Tables written once before any launch may use __ldg.
__device__ __forceinline__ uint32_t ld_waited(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float ld_waited(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_waited(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_waited(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                            Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

}  // namespace ffb
