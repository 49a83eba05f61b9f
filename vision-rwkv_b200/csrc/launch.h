// Launches behind the kernel before them in the stream.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <cstdint>
#include <utility>

// A kernel launched by launch_behind does this first, in every thread and before any access to global memory, any allocation of tensor memory and
// any wait for another block: it may have been started while the kernel before it ran, and nothing that is in the stream before it may be
// assumed done until here.  Its inputs are no __restrict__ pointers.
#ifdef __CUDACC__
__device__ __forceinline__ void wait_for_launch_before() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Loads behind that wait that keep their order with it and may be moved across stores, which none of the kernels makes to what it reads (a
// read-only load, __ldg or a pointer marked so, needs no order with anything: what it reads must not change from the kernel's start on).
__device__ __forceinline__ uint4 read_behind(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float4 read_behind(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ uint2 read_behind(const uint2* p) {
    uint2 v;
    asm volatile("ld.global.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ float2 read_behind(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0,%1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ uint32_t read_behind(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(__cvta_generic_to_global(p)));
    return v;
}
#endif

// kernel<<<grid, block, smem, stream>>>(args...) without waiting for the launch before to be flushed: the kernel waits for it by itself.  Two
// such launches in a row follow one another 1.5 to 2 us sooner, one behind any other kernel about 1 (elementwise kernels of 3 to 30 us): a VRWKV6-B inference of
// 64 images at 224 pixels 9069 -> 8782 us, a WKV6 layer's training at 196 tokens 259 -> 249.  The blocks start when all those of the kernel before
// are gone or, behind Bi-WKV's strips (and kernels of libraries), have said that others may start: they are all resident by then and need
// nothing that the new ones could hold, which do nothing but wait until they are gone.
// An error of the launch stays until record_launches asks for it (cudaGetLastError), as that of <<<>>> does.
template <typename... P, typename... A>
inline void launch_behind(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}
