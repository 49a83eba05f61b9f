// Pieces of the matrix products on the 5th-generation tensor cores (linear_tc.cu, linear_batch.cu): tiles of 128 rows, operands by TMA in
// swizzled rows, sums in tensor memory.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "linear_routes.h"
#include "sm100_async.cuh"

namespace lineartc {

using sm100::smem_u32;

constexpr uint32_t kWaitLimit = 1u << 20;
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
                 : "memory");
}
// the same box into L2 only
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src),
                 "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory"); }
// K-major operand in 128-byte rows, swizzled; eight rows are 1024 bytes
__device__ __forceinline__ uint64_t operand(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3FFF) | static_cast<uint64_t>(1) << 16 | static_cast<uint64_t>(1024 >> 4) << 32 | static_cast<uint64_t>(1) << 46 |
           static_cast<uint64_t>(2) << 61;
}
// bfloat16 operands, float32 sums, kM x n
__host__ __device__ constexpr uint32_t instr(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(kM >> 4) << 24); }
template <int n>
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b),
                 "r"(instr(n)), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void load16(uint32_t at, uint32_t* x) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]), "=r"(x[8]), "=r"(x[9]), "=r"(x[10]),
                   "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
                 : "r"(at)
                 : "memory");
}

// two sums as bfloat16
__device__ __forceinline__ uint32_t narrow2(uint32_t a, uint32_t b) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b));
    return *reinterpret_cast<const uint32_t*>(&r);
}
// relu(x)^2 of two sums, rounded to bfloat16 before (what the linear layer returns) and after
__device__ __forceinline__ uint32_t relu_square2(uint32_t a, uint32_t b) {
    const float2 x = __bfloat1622float2(__floats2bfloat162_rn(__uint_as_float(a), __uint_as_float(b)));
    // x < 0 ? 0 : x keeps NaN
    const float p = x.x < 0.f ? 0.f : x.x, q = x.y < 0.f ? 0.f : x.y;
    const __nv_bfloat162 r = __floats2bfloat162_rn(p * p, q * q);
    return *reinterpret_cast<const uint32_t*>(&r);
}

constexpr int kMostProducts = 4;
struct Products {
    CUtensorMap x[kMostProducts], w[kMostProducts], out[kMostProducts];
};

// SMs of the current device, 0 where the kernels cannot be had: linear_tc.cu's, linear_batch.cu's for layers or the key layer K deep
int tile_sms();
int slab_sms(bool square, int K);
// linear_tc.cu: several layers of one shape, without the squared ReLU
int batch_by_tiles(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream);
// linear_batch.cu: the key layer where a slab of W fits a CTA's shared memory beside what is on its way
int run_square_by_slabs(long long rows, int K, int N, const uint16_t* x, const uint16_t* w, uint16_t* out, void* stream);

}  // namespace lineartc
