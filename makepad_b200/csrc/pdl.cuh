// Loads in kernels that start beside the kernel in front of them (programmatic dependent launch), of what that kernel writes.
//
// Behind griddepcontrol.wait such data is visible to ordinary loads only: the read-only path (__ldg, or loads through a const __restrict__ pointer,
// which the compiler may send that way) is for memory that nobody writes while the kernel runs, and nothing keeps the compiler from moving
// such a load in front of the wait.  So these kernels read through plain pointers, or through the loads below, which stay where they are.
#pragma once
#include <cuda_runtime.h>

namespace mpq {

// evict-first: read once
__device__ __forceinline__ float load_once(const float* p)
{
    float v;
    asm volatile("ld.global.cs.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ float4 load_once(const float4* p)
{
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p) : "memory");
    return v;
}

}  // namespace mpq
