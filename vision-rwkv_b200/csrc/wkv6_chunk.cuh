// Building blocks of the chunked WKV6 kernels (wkv6_chunk.cu): fragment layouts, split-precision matrix
// products, token scans.
//
// Layout.  A chunk is 64 tokens of one (batch, head), in four 16-token blocks; a warp works on the rows of one block
// at a time.  Within a block a thread (g = lane / 4, q = lane % 4) holds rows g and g + 8 and, for kk = 0..3, the four
// CONTIGUOUS channels 16 kk + 4 q + {0..3}.  The contraction index of a matrix product may be numbered in any
// order as long as both operands agree, so these registers are at once
//   the A fragment (m16 k16) of the block for k-step kk,
//   the two B fragments (k16 n8, n = token) of its two 8-token halves, and
//   - products are laid out the same way over their columns - the C fragments of every result with channel columns.
// Loads and stores of 16-bit (8-byte) and 32-bit (16-byte) rows are therefore whole-sector accesses straight
// between global memory and fragments, and scaling a result by a per-(token, channel) factor is register-local.
// Where a product contracts over tokens its operand is needed transposed; such operands pass through shared
// memory as rows of 64 "positions" (position 16 kk + 8 h + 2 q + e holds channel 16 kk + 4 q + 2 h + e) that
// ldmatrix.trans reads in the right order.
//
// Precision.  A value enters a product as a sum of NS bfloat16 numbers (1: rounded; 2: 16 bits), and the products of
// parts whose error would be kept are accumulated in float32.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>
#include "launch.h"

namespace wkv6c {

constexpr int N = 64;              // head size
constexpr int kChunk = 64;         // tokens per chunk
constexpr int kBlock = 16;         // tokens per block
constexpr int kBlocks = kChunk / kBlock;
constexpr int kTab = 80;           // floats per row of a float table: 64 channels + 16, so that neighbouring rows use other banks
constexpr int kRow = 72;           // bfloat16 per shared row: 64 positions + 8 so that 8 rows start in 8 different bank groups
constexpr int kPlane = kChunk * kRow;
constexpr int kStateWords = N * N / 2;      // 32-bit words (bfloat16 pairs) of one state, one part
constexpr float kLog2e = 1.4426950408889634f;

typedef float Block[2][4][4];      // [row g / g + 8][kk][channel 16 kk + 4 q + e]
typedef float Acc[8][4];           // C fragments of a 16 x 64 result: [2 kk + h][row g: e, e + 1; row g + 8: e, e + 1]

__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

// (a, b) as NS packed bfloat16 pairs whose sum is (a, b) to 8 NS bits
template <int NS>
__device__ __forceinline__ void split(float a, float b, uint32_t (&out)[NS]) {
#pragma unroll
    for (int s = 0; s < NS; ++s) {
        const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
        out[s] = *reinterpret_cast<const uint32_t*>(&h);
        if (s + 1 < NS) {
            a -= __uint_as_float(out[s] << 16);
            b -= __uint_as_float(out[s] & 0xffff0000u);
        }
    }
}
__device__ __forceinline__ float lo_f(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float hi_f(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ uint32_t movm_trans(uint32_t x) {
    uint32_t y;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(y) : "r"(x));
    return y;
}
// the part products (ia, ib) that are kept for NA-part times NB-part operands: all whose size is above the dropped error
template <int NA, int NB>
struct Keep {
    static constexpr int kMax = NA > NB ? NA : NB;
    static __device__ constexpr bool on(int ia, int ib) { return ia + ib < kMax; }
};

// ---- operands --------------------------------------------------------------------------------------------
// A fragments of a block, k = channels
template <int NS>
struct AFrag {
    uint32_t w[NS][4][4];      // [part][kk][a0..a3]
    __device__ __forceinline__ void set(int kk, const float (&x0)[4], const float (&x1)[4]) {
        uint32_t t[NS];
        split<NS>(x0[0], x0[1], t);
#pragma unroll
        for (int s = 0; s < NS; ++s) w[s][kk][0] = t[s];
        split<NS>(x1[0], x1[1], t);
#pragma unroll
        for (int s = 0; s < NS; ++s) w[s][kk][1] = t[s];
        split<NS>(x0[2], x0[3], t);
#pragma unroll
        for (int s = 0; s < NS; ++s) w[s][kk][2] = t[s];
        split<NS>(x1[2], x1[3], t);
#pragma unroll
        for (int s = 0; s < NS; ++s) w[s][kk][3] = t[s];
    }
    __device__ __forceinline__ void set(const Block& x) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) set(kk, x[0][kk], x[1][kk]);
    }
};

// ---- products --------------------------------------------------------------------------------------------
// lane's address offset (in bfloat16) for ldmatrix of a 16-token block: B fragments with n = token, k = position
__device__ __forceinline__ int off_tok(int lane) { return (((lane >> 4) << 3) + (lane & 7)) * kRow + ((lane >> 3) & 1) * 8; }
// ... k = token, n = position (trans); the same order serves an A fragment with m = position, k = token (see ldsm4t uses)
__device__ __forceinline__ int off_pos(int lane) { return ((((lane >> 3) & 1) << 3) + (lane & 7)) * kRow + (lane >> 4) * 8; }
// A fragment with m = token, k = position
__device__ __forceinline__ int off_a(int lane) { return ((((lane >> 3) & 1) << 3) + (lane & 7)) * kRow + (lane >> 4) * 8; }

// C[16 x 16] += A(block, channels) * X(block `b` of the planes, tokens as columns)
template <int NA, int NB>
__device__ __forceinline__ void prod_tokens(float (&c)[2][4], const AFrag<NA>& a, const __nv_bfloat16* planes, int b, int lane) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
#pragma unroll
        for (int ib = 0; ib < NB; ++ib) {
            uint32_t r[4];
            ldsm4(r, smem_addr(planes + ib * kPlane + b * kBlock * kRow + kk * 16 + off_tok(lane)));
#pragma unroll
            for (int ia = 0; ia < NA; ++ia)
                if (Keep<NA, NB>::on(ia, ib)) {
                    mma(c[0], a.w[ia][kk], r[0], r[1]);
                    mma(c[1], a.w[ia][kk], r[2], r[3]);
                }
        }
    }
}
// One k-step (positions 16 kk ..) of a slice of a state, from global memory: the B fragments of the two 8-column halves.
// kTrans: the stored state's rows and columns are exchanged.
template <int NB, bool kTrans>
__device__ __forceinline__ void state_frag(uint32_t (&f)[NB][4], const uint4* state, int cs, int kk, int lane) {
#pragma unroll
    for (int ib = 0; ib < NB; ++ib) {
        const uint4 v = read_behind(state + ib * (kStateWords / 4) + ((kTrans ? kk * 4 + cs : cs * 4 + kk) * 32) + lane);
        if (kTrans) {
            f[ib][0] = movm_trans(v.x); f[ib][1] = movm_trans(v.z); f[ib][2] = movm_trans(v.y); f[ib][3] = movm_trans(v.w);
        } else {
            f[ib][0] = v.x; f[ib][1] = v.y; f[ib][2] = v.z; f[ib][3] = v.w;
        }
    }
}
__device__ __forceinline__ void zero(Acc& c) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) c[i][j] = 0.f;
}
// element of a C-fragment result at (row half, kk, e) in Block numbering
__device__ __forceinline__ float& at(Acc& c, int half, int kk, int e) { return c[2 * kk + (e >> 1)][half * 2 + (e & 1)]; }

// ---- loads -------------------------------------------------------------------------------------------------
template <typename T>
struct Raw;      // a block as it lies in memory
template <>
struct Raw<float> {
    float4 v[2][4];
    __device__ __forceinline__ void load(const float* p, int C, int rows, int g, int q) {      // p: row 0 of the block, channel 0 of the head
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                v[half][kk] = g + 8 * half < rows ? read_behind(reinterpret_cast<const float4*>(p + static_cast<size_t>(g + 8 * half) * C + 16 * kk + 4 * q))
                                                  : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __device__ __forceinline__ void get(int half, int kk, float (&x)[4]) const {
        x[0] = v[half][kk].x; x[1] = v[half][kk].y; x[2] = v[half][kk].z; x[3] = v[half][kk].w;
    }
};
template <>
struct Raw<__nv_bfloat16> {
    uint2 v[2][4];
    __device__ __forceinline__ void load(const __nv_bfloat16* p, int C, int rows, int g, int q) {
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
                v[half][kk] = g + 8 * half < rows ? read_behind(reinterpret_cast<const uint2*>(p + static_cast<size_t>(g + 8 * half) * C + 16 * kk + 4 * q))
                                                  : make_uint2(0u, 0u);
    }
    __device__ __forceinline__ void get(int half, int kk, float (&x)[4]) const {
        x[0] = lo_f(v[half][kk].x); x[1] = hi_f(v[half][kk].x); x[2] = lo_f(v[half][kk].y); x[3] = hi_f(v[half][kk].y);
    }
};
__device__ __forceinline__ void load4(const float* p, float (&x)[4]) {
    const float4 v = read_behind(reinterpret_cast<const float4*>(p));
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, float (&x)[4]) {
    const uint2 v = read_behind(reinterpret_cast<const uint2*>(p));
    x[0] = lo_f(v.x); x[1] = hi_f(v.x); x[2] = lo_f(v.y); x[3] = hi_f(v.y);
}
// raw inputs of the half-precision kernels are rounded to bfloat16 where they arrive as float
template <bool kRound>
__device__ __forceinline__ void round4(float (&x)[4]) {
    if (kRound) {
#pragma unroll
        for (int e = 0; e < 4; e += 2) {      // two at a time: a single conversion goes through the exponential's unit, an eighth of a pair's rate
            uint32_t t[1];
            split<1>(x[e], x[e + 1], t);
            x[e] = lo_f(t[0]);
            x[e + 1] = hi_f(t[0]);
        }
    }
}
// store 4 contiguous channels (`scalar`: the tensor is not aligned for vector stores)
__device__ __forceinline__ void put4(bool scalar, float* p, float a, float b, float c, float d) {
    if (!scalar) {
        *reinterpret_cast<float4*>(p) = make_float4(a, b, c, d);
    } else {
        p[0] = a; p[1] = b; p[2] = c; p[3] = d;
    }
}
__device__ __forceinline__ void put4(bool scalar, __nv_bfloat16* p, float a, float b, float c, float d) {
    uint32_t x[1], y[1];
    split<1>(a, b, x);
    split<1>(c, d, y);
    if (!scalar) {
        *reinterpret_cast<uint2*>(p) = make_uint2(x[0], y[0]);
    } else {
        p[0] = __float2bfloat16(a); p[1] = __float2bfloat16(b); p[2] = __float2bfloat16(c); p[3] = __float2bfloat16(d);
    }
}

// ---- tables: 64 rows (tokens) of kTab floats -------------------------------------------------------------------
// this thread's channels 16 kk + 4 q .. of a row
__device__ __forceinline__ void row4(const float* row, int kk, int q, float (&x)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(row + 16 * kk + 4 * q);
    x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
}
__device__ __forceinline__ void put_row4(float* row, int kk, int q, float a, float b, float c, float d) {
    *reinterpret_cast<float4*>(row + 16 * kk + 4 * q) = make_float4(a, b, c, d);
}

// ---- column layout: lane = channels 2 lane, 2 lane + 1, one token after the other --------------------------------
// index (in 32-bit words) of the lane's pair in a row of positions
__device__ __forceinline__ int col_word(int lane) { return 8 * (lane >> 3) + 4 * (lane & 1) + ((lane >> 1) & 3); }
template <int NS>
__device__ __forceinline__ void col_store(__nv_bfloat16* planes, int row, int word, float a, float b) {
    uint32_t t[NS];
    split<NS>(a, b, t);
#pragma unroll
    for (int s = 0; s < NS; ++s) *reinterpret_cast<uint32_t*>(planes + s * kPlane + row * kRow + 2 * word) = t[s];
}
template <typename T>
struct Pair;        // a lane's two channels of one token, as they lie in memory
template <>
struct Pair<float> {
    float2 v;
    __device__ __forceinline__ void load(const float* p, bool on) { v = on ? read_behind(reinterpret_cast<const float2*>(p)) : make_float2(0.f, 0.f); }
    __device__ __forceinline__ void lds(const float* p) { v = *reinterpret_cast<const float2*>(p); }
    __device__ __forceinline__ float2 get() const { return v; }
    __device__ __forceinline__ uint32_t bits() const { return 0u; }
};
template <>
struct Pair<__nv_bfloat16> {
    uint32_t v;
    __device__ __forceinline__ void load(const __nv_bfloat16* p, bool on) { v = on ? read_behind(reinterpret_cast<const uint32_t*>(p)) : 0u; }
    __device__ __forceinline__ void lds(const __nv_bfloat16* p) { v = *reinterpret_cast<const uint32_t*>(p); }
    __device__ __forceinline__ float2 get() const { return make_float2(lo_f(v), hi_f(v)); }
    __device__ __forceinline__ uint32_t bits() const { return v; }      // the pair as it is
};
// raw inputs of the half-precision kernels are rounded to bfloat16 where they arrive as float
template <bool kRound>
__device__ __forceinline__ float2 round2(float2 x) {
    if (!kRound) return x;
    uint32_t t[1];
    split<1>(x.x, x.y, t);
    return make_float2(lo_f(t[0]), hi_f(t[0]));
}
// log2 of a token's decay, bounded at -128: 2^-128 is flushed to zero already, and so bounded a sum over a block keeps its
// smaller terms to 1e-4 (and stays finite) whatever a token's decay is.  The bound is taken on w, which leaves the product and
// its sum one instruction.  NaN stays NaN.  0 where the token is off the end: a selected operand, since with the bound inside
// a conditional the walk over the chunks branched for every token (B=2, T=2000, H=3: forward 81 for 60 us).
constexpr float kDead = 6.4712f;      // 2^kDead log2 e = 128
__device__ __forceinline__ float log2_decay(float w, bool on) {
    float t;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(t) : "f"(on ? w * kLog2e : -INFINITY), "f"(kDead));
    return -kLog2e * ex2(t);
}
// d log(decay) / d w_raw; 0 where the decay is (its gradient is, and the sums it multiplies are zero only up to rounding)
__device__ __forceinline__ float decay_slope(float w) {
    const float t = w * kLog2e;
    return t >= kDead ? 0.f : -ex2(t);
}

}  // namespace wkv6c
