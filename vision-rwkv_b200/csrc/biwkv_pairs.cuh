// Device helpers of the Bi-WKV kernels that work on pairs of channels in f32x2 registers and hand sums over within a cluster.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "sm100_async.cuh"

namespace biwkv {
namespace pairs {

constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float rcp(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float2 f2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 shfl2(float2 a, int mask) {
    return f2(__shfl_xor_sync(0xffffffffu, a.x, mask), __shfl_xor_sync(0xffffffffu, a.y, mask));
}
__device__ __forceinline__ float2 sel2(bool c, float2 a, float2 b) { return c ? a : b; }

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_arrive_relaxed() { asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// address of the same shared-memory location in the CTA of rank `rank` of this cluster
__device__ __forceinline__ uint32_t peer_addr(const void* local, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(sm100::smem_u32(local)), "r"(rank));
    return r;
}
__device__ __forceinline__ float ld_peer(uint32_t addr) {
    float v;
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
    return v;
}
// Asynchronous stores into another CTA's shared memory; the receiving CTA's mbarrier counts the
// bytes, so data and notification travel together and the sender needs no fence.
__device__ __forceinline__ void st_async4(uint32_t addr, float4 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
                 "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async2(uint32_t addr, float2 v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(addr), "f"(v.x),
                 "f"(v.y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async1(uint32_t addr, float v, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(addr), "f"(v), "r"(bar)
                 : "memory");
}


// a thread's two channels: numerators (n) and denominators (d) of a state, each packed (ch 2p, ch 2p+1)
struct Pair2 {
    float2 n, d;
};
// x * (hi + lo) + y, both channels
__device__ __forceinline__ float2 mulc_add(float2 x, float2 hi, float2 lo, float2 y) { return fma2(x, hi, fma2(x, lo, y)); }

__device__ __forceinline__ float2 round2(float2 v) { return __bfloat1622float2(__float22bfloat162_rn(v)); }

// The kernels read w and u in pairs.  A vector that starts at an odd float (cut out of a parameter buffer) goes through a copy:
// single loads in the kernels cost every call, up to 7 % where a sequence is long.
inline const float* paired(const float* x, int C, float* copy, cudaStream_t stream) {
    if ((reinterpret_cast<uintptr_t>(x) & 7u) == 0) return x;
    cudaMemcpyAsync(copy, x, static_cast<size_t>(C) * sizeof(float), cudaMemcpyDeviceToDevice, stream);
    return copy;
}

}  // namespace pairs
}  // namespace biwkv
