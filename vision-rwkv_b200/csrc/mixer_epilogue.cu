// What a block computes between its matrix products, for inference: one pass each instead of torch's chains.
//
//   sigmoid_gate    sigmoid(r) * y                   classification/mmcls_custom/models/backbones/vrwkv.py:182-187, 253-257
//   relu_square     relu(x)^2                        vrwkv.py:250-251
//   norm_residual   x + gamma * LayerNorm(a), or x + gamma * a             vrwkv.py:297-318 (post- and pre-norm blocks);
//                   a may be given as r, y of sigmoid(r) * y, the gate that the channel mix ends with (vrwkv.py:253-257)
//   head_norm_gate  (GroupNorm per 64-channel head) * activation(gate)     vrwkv6.py:133, 205-212, bfloat16 result
//
//   add_rows        rows of a table, repeated, plus bfloat16 a, in float32  vrwkv.py:392 (positions), vrwkv6.py:200 (decay)
//   widen           bfloat16 as float32                                   what autocast puts in front of a LayerNorm
//   patch_rows      an image's patches as bfloat16 rows of a matrix         the operand of the patch embedding, vrwkv.py:357
//
// All are bound by HBM.  Bytes per element under bfloat16 autocast, the tensor-op chains against these: the gate 4 + 6 + 6
// (activation, cast of y, product) against 6; relu_square 24 (relu, cast, square in float32, the linear layer's cast)
// against 4, or 6 with the float32 result that a norm behind it takes; norm_residual 34 (cast, norm, scale, add) against
// 10; head_norm_gate 6 + 4 and the cast of its consumer, 6, against 8.  Every intermediate that a chain holds in bfloat16 is
// rounded to bfloat16 here too, and products and sums are rounded one by one, so only the order of LayerNorm's sums
// differs from torch's.
// Networks at 224 pixels under bfloat16 autocast, these kernels and bfloat16 outputs of the token shift together: the small
// model on 256 images 20.2 -> 8.0 ms, the matrix-state base model on 64 images 15.7 -> 11.6 ms.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <type_traits>
#include "launch.h"
#include "vrwkv_b200.h"
#include "vrwkv_internal.h"

namespace epilogue {

constexpr int kThreads = 256;
constexpr int kVec = 8;            // elements per thread and step of the elementwise kernels
constexpr int kMaxC = 1024;        // of norm_residual: a row fits a warp's registers

// N consecutive elements as floats
template <int N>
__device__ __forceinline__ void load(const float* p, float (&v)[N]) {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(p + i);
        v[i] = t.x; v[i + 1] = t.y; v[i + 2] = t.z; v[i + 3] = t.w;
    }
}
__device__ __forceinline__ void widen(uint32_t w, float& a, float& b) {
    a = __uint_as_float(w << 16);
    b = __uint_as_float(w & 0xffff0000u);
}
__device__ __forceinline__ uint32_t narrow(float a, float b) {
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&t);
}
template <int N>
__device__ __forceinline__ void load(const __nv_bfloat16* p, float (&v)[N]) {
    if (N == 8) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        widen(t.x, v[0], v[1]); widen(t.y, v[2], v[3]); widen(t.z, v[N - 4], v[N - 3]); widen(t.w, v[N - 2], v[N - 1]);
    } else {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        widen(t.x, v[0], v[1]); widen(t.y, v[2], v[3]);
    }
}
__device__ __forceinline__ void store(float* p, const float (&v)[kVec]) {
#pragma unroll
    for (int i = 0; i < kVec; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
}
__device__ __forceinline__ void store(__nv_bfloat16* p, const float (&v)[kVec]) {
    *reinterpret_cast<uint4*>(p) = make_uint4(narrow(v[0], v[1]), narrow(v[2], v[3]), narrow(v[4], v[5]), narrow(v[6], v[7]));
}
// (a, b) as R.  Two at a time: a single conversion to bfloat16 goes through the unit of the exponential, an eighth of a pair's rate.
template <typename R>
__device__ __forceinline__ void round_pair(float&, float&) {}
template <>
__device__ __forceinline__ void round_pair<__nv_bfloat16>(float& a, float& b) { widen(narrow(a, b), a, b); }

// sigmoid(r) before it is rounded to R.  The gates were bound by these instructions and not by HBM: 50176 x 384 in bfloat16 25.0 -> 17.3 us
// (115 MB: 6.7 TB/s), the gate with norm and residual 42.3 -> 34.7 (231 MB), 12544 x 768 widened 13.9 -> 10.9.  For bfloat16 r the approximate exponential and reciprocal (2^-22 each) round to what
// 1 / (1 + expf(-r)) rounds to, for all 65536 of them (checked one by one; the quarters keep results below 2^-126, which the reciprocal
// would flush), in 5 instructions for some 30.
template <typename R>
__device__ __forceinline__ float sigmoid(float r) { return 1.f / (1.f + expf(-r)); }
template <>
__device__ __forceinline__ float sigmoid<__nv_bfloat16>(float r) {
    float e, q;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(r * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(fmaf(e, 0.25f, 0.25f)));
    return q * 0.25f;
}
// sigmoid(r) * y of two elements, rounded to R as its factors are
template <typename R>
__device__ __forceinline__ void gate_pair(float (&r)[2], float y0, float y1) {
    r[0] = sigmoid<R>(r[0]);
    r[1] = sigmoid<R>(r[1]);
    round_pair<R>(r[0], r[1]);
    round_pair<R>(y0, y1);
    r[0] *= y0;
    r[1] *= y1;
    round_pair<R>(r[0], r[1]);
}
__device__ __forceinline__ float relu2(float x) {
    const float t = x < 0.f ? 0.f : x;      // NaN stays NaN
    return t * t;
}

// out = sigmoid(r) * y; the last n % kVec elements go to one thread
// O = float with R = bfloat16: the rounded result, widened for a LayerNorm that takes it in float32 (the copy that torch makes of it
// under autocast is a pass of 6 bytes per element, this one of 2 more: the matrix-state base model on 64 images 10.15 -> 9.90 ms).
template <typename R, typename Y, typename O>
__global__ void __launch_bounds__(kThreads) sigmoid_gate_kernel(long long n, const R* r, const Y* y, O* __restrict__ out) {
    wait_for_launch_before();
    const long long i = (static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x) * kVec;
    if (i + kVec <= n) {
        float a[kVec], b[kVec];
        load(r + i, a);
        load(y + i, b);
#pragma unroll
        for (int j = 0; j < kVec; j += 2) {
            float g[2] = {a[j], a[j + 1]};
            gate_pair<R>(g, b[j], b[j + 1]);
            a[j] = g[0]; a[j + 1] = g[1];
        }
        store(out + i, a);
    } else {
        for (long long j = i; j < n; ++j) {
            float g[2] = {static_cast<float>(r[j]), 0.f};
            gate_pair<R>(g, static_cast<float>(y[j]), 0.f);
            out[j] = static_cast<O>(g[0]);
        }
    }
}

template <typename R, typename O>
__global__ void __launch_bounds__(kThreads) relu_square_kernel(long long n, const R* x, O* __restrict__ out) {
    wait_for_launch_before();
    const long long i = (static_cast<long long>(blockIdx.x) * kThreads + threadIdx.x) * kVec;
    if (i + kVec <= n) {
        float a[kVec];
        load(x + i, a);
#pragma unroll
        for (int j = 0; j < kVec; ++j) a[j] = relu2(a[j]);
        store(out + i, a);
    } else {
        for (long long j = i; j < n; ++j) out[j] = static_cast<O>(relu2(static_cast<float>(x[j])));
    }
}

// out[i] = table[i mod period] + a[i], eight elements (one 8-element vector of the table) per thread
__global__ void __launch_bounds__(kThreads) add_rows_kernel(unsigned vectors, unsigned period, const float* table,
                                                            const __nv_bfloat16* a, float* __restrict__ out) {
    wait_for_launch_before();
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= vectors) return;
    float v[kVec], t[kVec];
    load(a + static_cast<size_t>(i) * kVec, v);
    load(table + static_cast<size_t>(i % period) * kVec, t);
#pragma unroll
    for (int j = 0; j < kVec; ++j) v[j] += t[j];
    store(out + static_cast<size_t>(i) * kVec, v);
}

// HBM-bound: 12544 x 768 take 11.4 us (5.1 TB/s), torch's cast 21; the matrix-state base model on 64 images 9.62 -> 9.49 ms.
__global__ void __launch_bounds__(kThreads) widen_kernel(unsigned vectors, const __nv_bfloat16* a, float* __restrict__ out) {
    wait_for_launch_before();
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= vectors) return;
    float v[kVec];
    load(a + static_cast<size_t>(i) * kVec, v);
    store(out + static_cast<size_t>(i) * kVec, v);
}

// Weights as bfloat16, several arrays in one launch.  Autocast casts each on its own: 2 to 3 us of GPU time and 2 more to the next launch, for 0.05
// to 2.4 million values.  VRWKV6-B's 144 casts, 410 us without the gaps, are 24 launches of 156 us (5.3 TB/s); VRWKV-S's 84, 205 us, are 24 of 80.
// Networks: 8782 -> 8354 us (64 images), 5540 -> 5410 (256 images).
constexpr int kMostNarrowed = 16, kNarrowedIters = 4;
struct Narrowed {
    const float* src[kMostNarrowed];
    __nv_bfloat16* dst[kMostNarrowed];
    long long n[kMostNarrowed];
    unsigned first[kMostNarrowed + 1];      // blocks of the arrays before
};
constexpr int kNarrowedBlock = kThreads * kVec * kNarrowedIters;      // values of a block
__global__ void __launch_bounds__(kThreads) narrow_kernel(const __grid_constant__ Narrowed a, int count) {
    wait_for_launch_before();
    int of = 0;
    while (of + 1 < count && blockIdx.x >= a.first[of + 1]) ++of;
    const float* const src = a.src[of];
    __nv_bfloat16* const dst = a.dst[of];
    const long long n = a.n[of], base = static_cast<long long>(blockIdx.x - a.first[of]) * kNarrowedBlock + threadIdx.x * kVec;
    if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0 && base + (kNarrowedIters - 1) * kThreads * kVec + kVec <= n) {
        float v[kNarrowedIters][kVec];
#pragma unroll
        for (int i = 0; i < kNarrowedIters; ++i) load(src + base + i * kThreads * kVec, v[i]);
#pragma unroll
        for (int i = 0; i < kNarrowedIters; ++i) store(dst + base + i * kThreads * kVec, v[i]);
        return;
    }
    for (int i = 0; i < kNarrowedIters; ++i)
        for (int e = 0; e < kVec; ++e) {
            const long long at = base + i * kThreads * kVec + e;
            if (at < n) dst[at] = __float2bfloat16_rn(src[at]);
        }
}

// Row (b, h, w) of `out` holds the patch at (h, w) of image b in the order channel, row, column, which is that of a
// convolution's weights: a patch embedding (kernel = stride) is then one matrix product.  A thread moves 8 pixels of an
// image row; reads are contiguous over the whole image, writes are whole 32-byte sectors.  With the library's
// convolution, 1.14 ms of it, the small model took 8.0 ms for 256 images of 224 pixels, this way 6.7.
__global__ void __launch_bounds__(kThreads) patch_rows_kernel(unsigned vectors, int channels, int H, int W, int rows, int cols, int patch,
                                                              const float* img, __nv_bfloat16* __restrict__ out) {
    wait_for_launch_before();
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= vectors) return;
    const unsigned per_row = static_cast<unsigned>(cols * patch) / kVec, lines = static_cast<unsigned>(rows * patch);
    const unsigned x = i % per_row * kVec, line = i / per_row;
    const unsigned y = line % lines, plane = line / lines, c = plane % channels, b = plane / channels;
    float v[kVec];
    load(img + (static_cast<size_t>(plane) * H + y) * W + x, v);
    const size_t token = (static_cast<size_t>(b) * rows + y / patch) * cols + x / patch;
    store(out + ((token * channels + c) * patch + y % patch) * patch + x % patch, v);
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) v += __shfl_xor_sync(0xffffffffu, v, m);
    return v;
}

// One warp per row, lane = 4 channels of each 128; kIters = ceil(C / 128).  Both inputs of a row are requested before the
// first sum, so 6 C bytes per warp are in flight.  kGate: a holds y and `gate` r of a gate, whose result is rounded as
// sigmoid_gate_kernel stores it: 12 bytes per element instead of 6 + 10 and a launch (the small
// model on 256 images 6.80 -> 6.70 ms).
template <typename A, int kIters, bool kGate>
__global__ void __launch_bounds__(kThreads) norm_residual_kernel(int rows, int C, float eps, const A* a, const A* gate,
                                                                 const float* weight,
                                                                 const float* bias, const float* gamma,
                                                                 const float* x, float* __restrict__ out) {
    wait_for_launch_before();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const size_t base = static_cast<size_t>(row) * C + 4 * lane;
    float v[kIters][4], res[kIters][4], r[kGate ? kIters : 1][4];
#pragma unroll
    for (int i = 0; i < kIters; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = res[i][j] = 0.f;
        if (128 * i + 4 * lane < C) {
            load(a + base + 128 * i, v[i]);
            load(x + base + 128 * i, res[i]);
            if (kGate) load(gate + base + 128 * i, r[i]);
        }
    }
    if (kGate) {
#pragma unroll
        for (int i = 0; i < kIters; ++i)
            if (128 * i + 4 * lane < C) {
#pragma unroll
                for (int j = 0; j < 4; j += 2) {
                    float g[2] = {r[i][j], r[i][j + 1]};
                    gate_pair<A>(g, v[i][j], v[i][j + 1]);
                    v[i][j] = g[0]; v[i][j + 1] = g[1];
                }
            }
    }
    if (weight != nullptr) {
        const float inv = 1.f / static_cast<float>(C);
        float s = 0.f, q = 0.f;
#pragma unroll
        for (int i = 0; i < kIters; ++i) s += (v[i][0] + v[i][1]) + (v[i][2] + v[i][3]);
        const float mean = warp_sum(s) * inv;
#pragma unroll
        for (int i = 0; i < kIters; ++i)
            if (128 * i + 4 * lane < C) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    v[i][j] -= mean;
                    q = fmaf(v[i][j], v[i][j], q);
                }
            }
        const float rstd = rsqrtf(warp_sum(q) * inv + eps);
#pragma unroll
        for (int i = 0; i < kIters; ++i)
            if (128 * i + 4 * lane < C) {
                float w[4], b[4];
                load(weight + 128 * i + 4 * lane, w);
                load(bias + 128 * i + 4 * lane, b);
#pragma unroll
                for (int j = 0; j < 4; ++j) v[i][j] = fmaf(v[i][j] * rstd, w[j], b[j]);
            }
    }
#pragma unroll
    for (int i = 0; i < kIters; ++i)
        if (128 * i + 4 * lane < C) {
            float g[4] = {1.f, 1.f, 1.f, 1.f};
            if (gamma != nullptr) load(gamma + 128 * i + 4 * lane, g);
            float4 o;
            o.x = __fadd_rn(res[i][0], __fmul_rn(g[0], v[i][0])); o.y = __fadd_rn(res[i][1], __fmul_rn(g[1], v[i][1]));
            o.z = __fadd_rn(res[i][2], __fmul_rn(g[2], v[i][2])); o.w = __fadd_rn(res[i][3], __fmul_rn(g[3], v[i][3]));
            *reinterpret_cast<float4*>(out + base + 128 * i) = o;
        }
}

// The norm alone, rows as above.  A mean from one sum is off by its rounding, which on rows whose mean is three times their spread put
// results 1.35e-7 from float64 (torch's layer 1.07e-7, C = 192 to 768); what rounding left in it is summed up beside the squares and
// taken off, 5.2e-8 for any mean.  us, torch's layer / the norm as a case of the kernel above / this: 50176 x 384 95 / 25.2 / 24.4,
// 50176 x 1024 149 / 69.3 / 63.2, 196 x 1024 3.7 / 3.9 / 3.1.  Weight and bias are asked for one piece of the row ahead, two in wide rows, since
// a load is not moved over a store by itself (1568 x 640 2.9 -> 2.6; everything asked for before the first store 12544 x 1024 19.3 -> 20.3).
template <int kIters>
__global__ void __launch_bounds__(kThreads) layer_norm_kernel(int rows, int C, float eps, const float* x, const float* weight,
                                                              const float* bias, float* __restrict__ out) {
    wait_for_launch_before();
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * (kThreads / 32) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const size_t base = static_cast<size_t>(row) * C + 4 * lane;
    const float inv = 1.f / static_cast<float>(C);
    float v[kIters][4], s = 0.f, d = 0.f, q = 0.f;
#pragma unroll
    for (int i = 0; i < kIters; ++i) {
#pragma unroll
        for (int j = 0; j < 4; ++j) v[i][j] = 0.f;
        if (128 * i + 4 * lane < C) load(x + base + 128 * i, v[i]);
    }
#pragma unroll
    for (int i = 0; i < kIters; ++i) s += (v[i][0] + v[i][1]) + (v[i][2] + v[i][3]);
    const float mean = warp_sum(s) * inv;
#pragma unroll
    for (int i = 0; i < kIters; ++i)
        if (128 * i + 4 * lane < C) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[i][j] -= mean;
                q = fmaf(v[i][j], v[i][j], q);
            }
            d += (v[i][0] + v[i][1]) + (v[i][2] + v[i][3]);
        }
    const float rest = warp_sum(d) * inv;
    const float rstd = rsqrtf(fmaxf(fmaf(-rest, rest, warp_sum(q) * inv), 0.f) + eps), shift = -rest * rstd;
    constexpr int kAhead = kIters > 6 ? 2 : 1;
    float w[kAhead + 1][4], b[kAhead + 1][4];      // asked for before the results in front of them leave
    const auto scale_at = [&](int i) {
        if (i < kIters && 128 * i + 4 * lane < C) {
            load(weight + 128 * i + 4 * lane, w[i % (kAhead + 1)]);
            load(bias + 128 * i + 4 * lane, b[i % (kAhead + 1)]);
        }
    };
#pragma unroll
    for (int i = 0; i < kAhead; ++i) scale_at(i);
#pragma unroll
    for (int i = 0; i < kIters; ++i)
        if (128 * i + 4 * lane < C) {
            scale_at(i + kAhead);
            const int at = i % (kAhead + 1);
            float4 o;
            o.x = fmaf(fmaf(v[i][0], rstd, shift), w[at][0], b[at][0]); o.y = fmaf(fmaf(v[i][1], rstd, shift), w[at][1], b[at][1]);
            o.z = fmaf(fmaf(v[i][2], rstd, shift), w[at][2], b[at][2]); o.w = fmaf(fmaf(v[i][3], rstd, shift), w[at][3], b[at][3]);
            *reinterpret_cast<float4*>(out + base + 128 * i) = o;
        }
}

// Per-head norm and gate, eight lanes per 64-channel head: lane q holds channels 4 q .. 4 q + 3 and 32 behind them, in 16-byte accesses.  The
// sums go pair by pair in the order of normgate_forward_kernel (a warp per head, one pair per lane), and so give the bits of its float32 result before it
// is rounded: there lane l, of channels 2 l and 2 l + 1, meets l + 16 first, then 8, 4, 2 and 1 lanes away; here lanes 2 q and 2 q + 1 of that
// order are one thread's, whose two sums meet last.  12544 x 768 with a bfloat16 gate (77 MB): 19.5 us with a half-warp per head, accesses of 8 and 4
// bytes and four heads requested together, 14.9 now (two heads together 16.2, four 21.7: fewer threads on an SM); 50176 x 384 42.9 -> 34.3.
constexpr int kLanes = 8;
__device__ __forceinline__ float eight_lane_sum(float even, float odd) {
#pragma unroll
    for (int m = kLanes / 2; m >= 1; m >>= 1) {
        even += __shfl_xor_sync(0xffffffffu, even, m);
        odd += __shfl_xor_sync(0xffffffffu, odd, m);
    }
    return even + odd;
}
__device__ __forceinline__ float activation(float x, int act) {
    if (act == 0) return x;
    const float s = 1.f / (1.f + __expf(-x));
    return act == 1 ? s : x * s;
}
template <typename G>
__global__ void __launch_bounds__(kThreads) head_norm_gate_kernel(long long heads, int per_row, float eps, const float* x,
                                                                  const G* gate, int act, const float* gamma,
                                                                  const float* beta, __nv_bfloat16* __restrict__ out) {
    wait_for_launch_before();
    const int q = threadIdx.x & (kLanes - 1);
    const long long mine = static_cast<long long>(blockIdx.x) * (kThreads / kLanes) + threadIdx.x / kLanes;
    const long long head = min(mine, heads - 1);      // a repeated head is computed and not stored
    float v[2][4], g[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        load(x + head * 64 + 4 * q + 32 * i, v[i]);
        load(gate + head * 64 + 4 * q + 32 * i, g[i]);
    }
    const float inv = 1.f / 64.f;
    const float mean = eight_lane_sum((v[0][0] + v[0][1]) + (v[1][0] + v[1][1]), (v[0][2] + v[0][3]) + (v[1][2] + v[1][3])) * inv;
    float part[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            float s = 0.f;
            const float dx = v[i][2 * p] - mean, dy = v[i][2 * p + 1] - mean;
            s += dx * dx + dy * dy;
            part[p][i] = s;
        }
    const float rstd = rsqrtf(eight_lane_sum(part[0][0] + part[0][1], part[1][0] + part[1][1]) * inv + eps);
    if (mine < heads) {
        const int c = static_cast<int>(head % per_row) * 64 + 4 * q;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float ga[4], be[4], o[4];
            load(gamma + c + 32 * i, ga);
            load(beta + c + 32 * i, be);
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = ((v[i][e] - mean) * rstd * ga[e] + be[e]) * activation(g[i][e], act);
            *reinterpret_cast<uint2*>(out + head * 64 + 4 * q + 32 * i) = make_uint2(narrow(o[0], o[1]), narrow(o[2], o[3]));
        }
    }
}

static bool misaligned(std::initializer_list<const void*> ps) {
    uintptr_t bits = 0;
    for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
    return (bits & 15u) != 0;
}
static long long blocks_of(long long n) { return (n + static_cast<long long>(kThreads) * kVec - 1) / (static_cast<long long>(kThreads) * kVec); }

template <typename A, int kIters = 1>
static void launch_norm_residual(int rows, int C, float eps, const A* a, const A* gate, const float* weight, const float* bias, const float* gamma,
                                 const float* x, float* out, cudaStream_t s) {
    if constexpr (kIters < kMaxC / 128) {
        if (C > 128 * kIters) return launch_norm_residual<A, kIters + 1>(rows, C, eps, a, gate, weight, bias, gamma, x, out, s);
    }
    const int per = kThreads / 32, grid = (rows + per - 1) / per;
    if constexpr (std::is_same<A, __nv_bfloat16>::value) {
        if (gate != nullptr) {
            launch_behind(norm_residual_kernel<A, kIters, true>, grid, kThreads, 0, s, rows, C, eps, a, gate, weight, bias, gamma, x, out);
            return;
        }
    }
    launch_behind(norm_residual_kernel<A, kIters, false>, grid, kThreads, 0, s, rows, C, eps, a, nullptr, weight, bias, gamma, x, out);
}
template <int kIters = 1>
static void launch_layer_norm(int rows, int C, float eps, const float* x, const float* weight, const float* bias, float* out, cudaStream_t s) {
    if constexpr (kIters < kMaxC / 128) {
        if (C > 128 * kIters) return launch_layer_norm<kIters + 1>(rows, C, eps, x, weight, bias, out, s);
    }
    constexpr int kPer = kThreads / 32;
    launch_behind(layer_norm_kernel<kIters>, rows / kPer + (rows % kPer != 0 ? 1 : 0), kThreads, 0, s, rows, C, eps, x, weight, bias, out);
}

}  // namespace epilogue

extern "C" int vrwkv_sigmoid_gate(long long n, const void* r, int r_is_bf16, const void* y, int y_is_bf16, void* out, void* stream) {
    using namespace epilogue;
    if (n <= 0 || blocks_of(n) > 0x7fffffffLL) return VRWKV_ERR_SHAPE;
    if (!r || !y || !out) return VRWKV_ERR_NULL;
    if (misaligned({r, y, out})) return VRWKV_ERR_ALIGNMENT;
    if (y_is_bf16 && !r_is_bf16) return VRWKV_ERR_UNSUPPORTED;
    const unsigned grid = static_cast<unsigned>(blocks_of(n));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    using H = __nv_bfloat16;
    if (y_is_bf16) launch_behind(sigmoid_gate_kernel<H, H, H>, grid, kThreads, 0, s, n, static_cast<const H*>(r), static_cast<const H*>(y), static_cast<H*>(out));
    else if (r_is_bf16) launch_behind(sigmoid_gate_kernel<H, float, H>, grid, kThreads, 0, s, n, static_cast<const H*>(r), static_cast<const float*>(y), static_cast<H*>(out));
    else launch_behind(sigmoid_gate_kernel<float, float, float>, grid, kThreads, 0, s, n, static_cast<const float*>(r), static_cast<const float*>(y), static_cast<float*>(out));
    return record_launches(1);
}

extern "C" int vrwkv_sigmoid_gate_f32out(long long n, const uint16_t* r, const uint16_t* y, float* out, void* stream) {
    using namespace epilogue;
    if (n <= 0 || blocks_of(n) > 0x7fffffffLL) return VRWKV_ERR_SHAPE;
    if (!r || !y || !out) return VRWKV_ERR_NULL;
    if (misaligned({r, y, out})) return VRWKV_ERR_ALIGNMENT;
    using H = __nv_bfloat16;
    launch_behind(sigmoid_gate_kernel<H, H, float>, static_cast<unsigned>(blocks_of(n)), kThreads, 0, static_cast<cudaStream_t>(stream),
                  n, reinterpret_cast<const H*>(r), reinterpret_cast<const H*>(y), out);
    return record_launches(1);
}

extern "C" int vrwkv_relu_square(long long n, const void* x, int is_bf16, void* out, void* stream) {
    using namespace epilogue;
    if (n <= 0 || blocks_of(n) > 0x7fffffffLL) return VRWKV_ERR_SHAPE;
    if (!x || !out) return VRWKV_ERR_NULL;
    if (misaligned({x, out})) return VRWKV_ERR_ALIGNMENT;
    const unsigned grid = static_cast<unsigned>(blocks_of(n));
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    using H = __nv_bfloat16;
    if (is_bf16) launch_behind(relu_square_kernel<H, H>, grid, kThreads, 0, s, n, static_cast<const H*>(x), static_cast<H*>(out));
    else launch_behind(relu_square_kernel<float, float>, grid, kThreads, 0, s, n, static_cast<const float*>(x), static_cast<float*>(out));
    return record_launches(1);
}

extern "C" int vrwkv_relu_square_f32out(long long n, const uint16_t* x, float* out, void* stream) {
    using namespace epilogue;
    if (n <= 0 || blocks_of(n) > 0x7fffffffLL) return VRWKV_ERR_SHAPE;
    if (!x || !out) return VRWKV_ERR_NULL;
    if (misaligned({x, out})) return VRWKV_ERR_ALIGNMENT;
    launch_behind(relu_square_kernel<__nv_bfloat16, float>, static_cast<unsigned>(blocks_of(n)), kThreads, 0, static_cast<cudaStream_t>(stream),
                  n, reinterpret_cast<const __nv_bfloat16*>(x), out);
    return record_launches(1);
}

extern "C" int vrwkv_add_rows(long long n, long long period, const float* table, const uint16_t* a, float* out, void* stream) {
    using namespace epilogue;
    if (n <= 0 || period <= 0 || n % period != 0) return VRWKV_ERR_SHAPE;
    if (!table || !a || !out) return VRWKV_ERR_NULL;
    if (period % kVec != 0 || n / kVec > 0x7fffffffLL - kThreads) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({table, a, out})) return VRWKV_ERR_ALIGNMENT;
    const unsigned vectors = static_cast<unsigned>(n / kVec);
    launch_behind(add_rows_kernel, (vectors + kThreads - 1) / kThreads, kThreads, 0, static_cast<cudaStream_t>(stream),
                  vectors, static_cast<unsigned>(period / kVec), table, reinterpret_cast<const __nv_bfloat16*>(a), out);
    return record_launches(1);
}

extern "C" int vrwkv_widen(long long n, const uint16_t* a, float* out, void* stream) {
    using namespace epilogue;
    if (n <= 0) return VRWKV_ERR_SHAPE;
    if (!a || !out) return VRWKV_ERR_NULL;
    if (n % kVec != 0 || n / kVec > 0x7fffffffLL - kThreads) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({a, out})) return VRWKV_ERR_ALIGNMENT;
    const unsigned vectors = static_cast<unsigned>(n / kVec);
    launch_behind(widen_kernel, (vectors + kThreads - 1) / kThreads, kThreads, 0, static_cast<cudaStream_t>(stream),
                  vectors, reinterpret_cast<const __nv_bfloat16*>(a), out);
    return record_launches(1);
}

extern "C" int vrwkv_narrow(int count, const float* const* src, const long long* n, uint16_t* const* out, void* stream) {
    using namespace epilogue;
    if (count <= 0 || count > kMostNarrowed) return VRWKV_ERR_SHAPE;
    if (!src || !n || !out) return VRWKV_ERR_NULL;
    Narrowed a{};
    long long blocks = 0;
    for (int i = 0; i < count; ++i) {
        if (n[i] <= 0) return VRWKV_ERR_SHAPE;
        if (!src[i] || !out[i]) return VRWKV_ERR_NULL;
        if ((reinterpret_cast<uintptr_t>(src[i]) & 3u) || (reinterpret_cast<uintptr_t>(out[i]) & 1u)) return VRWKV_ERR_ALIGNMENT;
        a.src[i] = src[i]; a.dst[i] = reinterpret_cast<__nv_bfloat16*>(out[i]); a.n[i] = n[i];
        a.first[i] = static_cast<unsigned>(blocks);
        blocks += n[i] / kNarrowedBlock + (n[i] % kNarrowedBlock != 0 ? 1 : 0);
        if (blocks > 0x7fffffffLL) return VRWKV_ERR_UNSUPPORTED;
    }
    launch_behind(narrow_kernel, static_cast<unsigned>(blocks), kThreads, 0, static_cast<cudaStream_t>(stream), a, count);
    return record_launches(0);
}

extern "C" int vrwkv_patch_rows(int B, int channels, int H, int W, int patch, const float* img, uint16_t* out, void* stream) {
    using namespace epilogue;
    if (B <= 0 || channels <= 0 || patch <= 0 || H < patch || W < patch) return VRWKV_ERR_SHAPE;
    if (!img || !out) return VRWKV_ERR_NULL;
    const int rows = H / patch, cols = W / patch;
    const long long vectors = static_cast<long long>(B) * channels * rows * patch * cols * patch / kVec;
    // image rows start on 16-byte boundaries, 8 pixels never span two patches
    if (patch % kVec != 0 || W % 4 != 0 || vectors > 0x7fffffffLL - kThreads) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({img, out})) return VRWKV_ERR_ALIGNMENT;
    launch_behind(patch_rows_kernel, static_cast<unsigned>((vectors + kThreads - 1) / kThreads), kThreads, 0, static_cast<cudaStream_t>(stream),
                  static_cast<unsigned>(vectors), channels, H, W, rows, cols, patch, img, reinterpret_cast<__nv_bfloat16*>(out));
    return record_launches(1);
}

extern "C" int vrwkv_norm_residual(int rows, int C, float eps, const void* a, int a_is_bf16, const float* weight, const float* bias,
                                   const float* gamma, const float* x, float* out, void* stream) {
    using namespace epilogue;
    if (rows <= 0 || C <= 0) return VRWKV_ERR_SHAPE;
    if (!a || !x || !out || (weight != nullptr) != (bias != nullptr)) return VRWKV_ERR_NULL;
    if (C % 4 != 0 || C > kMaxC) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({a, weight, bias, gamma, x, out})) return VRWKV_ERR_ALIGNMENT;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (a_is_bf16) launch_norm_residual<__nv_bfloat16>(rows, C, eps, static_cast<const __nv_bfloat16*>(a), nullptr, weight, bias, gamma, x, out, s);
    else launch_norm_residual<float>(rows, C, eps, static_cast<const float*>(a), nullptr, weight, bias, gamma, x, out, s);
    return record_launches(1);
}

extern "C" int vrwkv_layer_norm(int rows, int C, float eps, const float* x, const float* weight, const float* bias, float* out, void* stream) {
    using namespace epilogue;
    if (rows <= 0 || C <= 0) return VRWKV_ERR_SHAPE;
    if (!x || !weight || !bias || !out) return VRWKV_ERR_NULL;
    if (C % 4 != 0 || C > kMaxC) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({x, weight, bias, out})) return VRWKV_ERR_ALIGNMENT;
    launch_layer_norm(rows, C, eps, x, weight, bias, out, static_cast<cudaStream_t>(stream));
    return record_launches(1);
}

extern "C" int vrwkv_gated_norm_residual(int rows, int C, float eps, const uint16_t* r, const uint16_t* y, const float* weight, const float* bias,
                                         const float* gamma, const float* x, float* out, void* stream) {
    using namespace epilogue;
    if (rows <= 0 || C <= 0) return VRWKV_ERR_SHAPE;
    if (!r || !y || !x || !out || (weight != nullptr) != (bias != nullptr)) return VRWKV_ERR_NULL;
    if (C % 4 != 0 || C > kMaxC) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned({r, y, weight, bias, gamma, x, out})) return VRWKV_ERR_ALIGNMENT;
    launch_norm_residual<__nv_bfloat16>(rows, C, eps, reinterpret_cast<const __nv_bfloat16*>(y), reinterpret_cast<const __nv_bfloat16*>(r), weight, bias,
                                        gamma, x, out, static_cast<cudaStream_t>(stream));
    return record_launches(1);
}

extern "C" int vrwkv_head_norm_gate_bf16out(int rows, int C, float eps, const float* x, const void* gate, int gate_is_bf16, int gate_act,
                                            const float* gamma, const float* beta, uint16_t* out, void* stream) {
    using namespace epilogue;
    if (rows <= 0 || C <= 0 || C % 64 != 0 || gate_act < 0 || gate_act > 2) return VRWKV_ERR_SHAPE;
    if (!x || !gate || !gamma || !beta || !out) return VRWKV_ERR_NULL;
    if (misaligned({x, gate, gamma, beta, out})) return VRWKV_ERR_ALIGNMENT;
    const long long heads = static_cast<long long>(rows) * (C / 64), per = kThreads / kLanes, grid = (heads + per - 1) / per;
    if (grid > 0x7fffffffLL) return VRWKV_ERR_SHAPE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto* const o = reinterpret_cast<__nv_bfloat16*>(out);
    if (gate_is_bf16)
        launch_behind(head_norm_gate_kernel<__nv_bfloat16>, static_cast<unsigned>(grid), kThreads, 0, s, heads, C / 64, eps, x, static_cast<const __nv_bfloat16*>(gate), gate_act,
                                                                               gamma, beta, o);
    else
        launch_behind(head_norm_gate_kernel<float>, static_cast<unsigned>(grid), kThreads, 0, s, heads, C / 64, eps, x, static_cast<const float*>(gate), gate_act, gamma,
                                                                               beta, o);
    return record_launches(1);
}
