// pdl.cuh -- the two halves of a programmatic dependent launch (launch_dependent in common.h).  A kernel launched that way may start
// while its predecessor in the stream still runs.  pdl_release() lets the successor's CTAs be scheduled as soon as every CTA of this
// grid has called it (or exited); pdl_acquire() returns once the predecessor grid has completed and its writes are visible.
// Everything a kernel does before pdl_acquire() may only touch memory no earlier kernel of the stream writes (weights); both are
// no-ops in an ordinary launch.
//
// A kernel's lifetime thus begins before its predecessor's last write.  Read-only loads (__ldg, const __restrict__ pointers) promise data
// that stays as it is for that whole time, and neither they nor the cache-hint intrinsics (__ldcs) are ordered with pdl_acquire() for the
// compiler.  So only a model's weights and tables and what is written before the step's first launch are read that way; everything a
// predecessor may write, any operand of a public operation among it, comes by plain loads through unrestricted pointers, which the memory
// clobber of pdl_acquire() keeps behind it, or by ld_cs() below.
#pragma once
#include <cuda_runtime.h>

namespace spt {

__device__ __forceinline__ void pdl_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_acquire() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// streaming loads (evict first) that stay behind pdl_acquire(): volatile statements keep their order
__device__ __forceinline__ uint4 ld_cs(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.cs.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_cs(const float4* p) {
    float4 v;
    asm volatile("ld.global.cs.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

}  // namespace spt
