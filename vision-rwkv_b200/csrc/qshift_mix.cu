// Fused Q-Shift + token-mix interpolation, forward and backward.
//
// In the backbones every mixing block first builds a shifted copy xx of its input x
// (tokens laid out as an H x W grid, channel quarters moved by `s` pixels right / left /
// down / up with zero fill at the border, the remaining channels copied) and then forms
// n interpolations  out_m = x * mix_m + xx * (1 - mix_m)  (n = 3 in the spatial mix: k, v, r;
// n = 2 in the channel mix: k, r) that feed the linear layers
// (classification/mmcls_custom/models/backbones/vrwkv.py:68-79, 156-164, 247-250).  Done
// with tensor ops that is a transpose, a zero fill, five strided copies, a transpose back and
// 3 n elementwise passes.  Here: one pass that reads x once (the shifted read is a second,
// cache-resident read of a neighbouring token row) and writes the n outputs; the backward
// reads the n output gradients and x once, writes gx, and reduces the n mix gradients in a
// fixed order.  Pure bandwidth work: 4 (1 + n) bytes per element forward, 4 (n + 2) backward.
#include <cuda_runtime.h>
#include <cstdint>
#include "launch.h"
#include "qshift_lines.cuh"
#include "vrwkv_internal.h"

namespace qshift {

constexpr int kMaxOut = 3;
constexpr int kThreads = 128;
constexpr int kTokensPerBlock = 32;

struct Args {
    int B, H, W, C;
    int group;     // channels per shifted group = int(C * gamma), or head_dim / 4 for the per-head variant
    int period;    // 0: the four groups are channels [0, 4 * group); n: they repeat every n channels (n = head_dim)
    int shift;     // pixels
    int n_out;
    const float* x;
    const float* mix[kMaxOut];     // (C,)
    float* out[kMaxOut];           // forward outputs (B, T, C)
    bool out_bf16;                 // ... in bfloat16 (what an autocast linear layer behind them would round them to)
    const float* gout[kMaxOut];    // backward: output gradients
    float* gx;
    float* partial;                // backward: [blocks_y][n_out][C]
};

// Token that channel c of token (h, w) reads its shifted value from; -1 = zero fill.
__device__ __forceinline__ int source_token(const Args& a, int h, int w, int c) {
    const int g = (a.period ? c % a.period : c) / a.group;
    int hs = h, ws = w;
    if (g == 0) ws = w - a.shift;
    else if (g == 1) ws = w + a.shift;
    else if (g == 2) hs = h - a.shift;
    else if (g == 3) hs = h + a.shift;
    if (hs < 0 || hs >= a.H || ws < 0 || ws >= a.W) return -1;
    return hs * a.W + ws;
}
// Token whose shifted value is read *from* (h, w) for channel c (the transpose); -1 = none.
__device__ __forceinline__ int reader_token(const Args& a, int h, int w, int c) {
    const int g = (a.period ? c % a.period : c) / a.group;
    int hd = h, wd = w;
    if (g == 0) wd = w + a.shift;
    else if (g == 1) wd = w - a.shift;
    else if (g == 2) hd = h + a.shift;
    else if (g == 3) hd = h - a.shift;
    if (hd < 0 || hd >= a.H || wd < 0 || wd >= a.W) return -1;
    return hd * a.W + wd;
}

// ---- any shift, any alignment: token by token ----------------------------------------------------
// kVec: 4 channels per thread (needs C % 4 == 0, group % 4 == 0 and 16-byte aligned tensors)
template <int kVec, typename Out>
__global__ void __launch_bounds__(kThreads) qshift_mix_forward(const Args a) {
    const int cv = (blockIdx.x * kThreads + threadIdx.x) * kVec;
    if (cv >= a.C) return;
    const int T = a.H * a.W;
    float mixv[kMaxOut][kVec];
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m)
        if (m < a.n_out)
#pragma unroll
            for (int j = 0; j < kVec; ++j) mixv[m][j] = a.mix[m][cv + j];
    const long long tok0 = static_cast<long long>(blockIdx.y) * kTokensPerBlock;
    const long long ntok = static_cast<long long>(a.B) * T;
    for (int i = 0; i < kTokensPerBlock; ++i) {
        const long long tok = tok0 + i;
        if (tok >= ntok) break;
        const int b = static_cast<int>(tok / T), t = static_cast<int>(tok % T);
        const int h = t / a.W, w = t % a.W;
        const size_t base = static_cast<size_t>(tok) * a.C + cv;
        float xv[kVec], sv[kVec];
        const int src = source_token(a, h, w, cv);          // one group per vector (group % kVec == 0)
        if (kVec == 4) {
            const float4 x4 = *reinterpret_cast<const float4*>(a.x + base);
            xv[0] = x4.x; xv[1] = x4.y; xv[2] = x4.z; xv[3] = x4.w;
            float4 s4 = make_float4(0.f, 0.f, 0.f, 0.f);
            if (src >= 0) s4 = *reinterpret_cast<const float4*>(a.x + (static_cast<size_t>(b) * T + src) * a.C + cv);
            sv[0] = s4.x; sv[1] = s4.y; sv[2] = s4.z; sv[3] = s4.w;
        } else {
            xv[0] = a.x[base];
            sv[0] = src >= 0 ? a.x[(static_cast<size_t>(b) * T + src) * a.C + cv] : 0.f;
        }
#pragma unroll
        for (int m = 0; m < kMaxOut; ++m) {
            if (m < a.n_out) {
                float o[kVec];
#pragma unroll
                for (int j = 0; j < kVec; ++j) o[j] = fmaf(mixv[m][j], xv[j] - sv[j], sv[j]);
                Out* const to = reinterpret_cast<Out*>(a.out[m]) + base;
                if (kVec == 4) qlines::st4(to, make_float4(o[0], o[1], o[2], o[3]));
                else *to = static_cast<Out>(o[0]);
            }
        }
    }
}

template <int kVec>
__global__ void __launch_bounds__(kThreads) qshift_mix_backward(const Args a) {
    const int cv = (blockIdx.x * kThreads + threadIdx.x) * kVec;
    if (cv >= a.C) return;
    const int T = a.H * a.W;
    float mixv[kMaxOut][kVec], gmix[kMaxOut][kVec];
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m)
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
            mixv[m][j] = m < a.n_out ? a.mix[m][cv + j] : 0.f;
            gmix[m][j] = 0.f;
        }
    const long long tok0 = static_cast<long long>(blockIdx.y) * kTokensPerBlock;
    const long long ntok = static_cast<long long>(a.B) * T;
    for (int i = 0; i < kTokensPerBlock; ++i) {
        const long long tok = tok0 + i;
        if (tok >= ntok) break;
        const int b = static_cast<int>(tok / T), t = static_cast<int>(tok % T);
        const int h = t / a.W, w = t % a.W;
        const size_t base = static_cast<size_t>(tok) * a.C + cv;
        const int src = source_token(a, h, w, cv);
        const int rdr = reader_token(a, h, w, cv);
        const size_t sbase = (static_cast<size_t>(b) * T + (src >= 0 ? src : 0)) * a.C + cv;
        const size_t rbase = (static_cast<size_t>(b) * T + (rdr >= 0 ? rdr : 0)) * a.C + cv;
        float xv[kVec], sv[kVec], gxv[kVec];
#pragma unroll
        for (int j = 0; j < kVec; ++j) {
            xv[j] = a.x[base + j];
            sv[j] = src >= 0 ? a.x[sbase + j] : 0.f;
            gxv[j] = 0.f;
        }
#pragma unroll
        for (int m = 0; m < kMaxOut; ++m) {
            if (m < a.n_out) {
#pragma unroll
                for (int j = 0; j < kVec; ++j) {
                    const float g = a.gout[m][base + j];
                    gxv[j] = fmaf(g, mixv[m][j], gxv[j]);
                    gmix[m][j] = fmaf(g, xv[j] - sv[j], gmix[m][j]);
                    if (rdr >= 0) gxv[j] = fmaf(a.gout[m][rbase + j], 1.f - mixv[m][j], gxv[j]);
                }
            }
        }
#pragma unroll
        for (int j = 0; j < kVec; ++j) a.gx[base + j] = gxv[j];
    }
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m)
        if (m < a.n_out)
#pragma unroll
            for (int j = 0; j < kVec; ++j)
                a.partial[(static_cast<size_t>(blockIdx.y) * a.n_out + m) * a.C + cv + j] = gmix[m][j];
}

// ---- a shift of one pixel: walks along the lines of the grid (qshift_lines.cuh) ----------------------
template <typename Out>
__global__ void __launch_bounds__(qlines::kMaxThreads) qshift_lines_forward(const Args a, const qlines::Grid g) {
    wait_for_launch_before();
    using namespace qlines;
    const int cv = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    if (cv >= g.C) return;
    const int which = group_of(g, cv);
    const unsigned first = (blockIdx.x * blockDim.y + threadIdx.y) * static_cast<unsigned>(g.per_walker);
    float4 mix[kMaxOut];
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m) mix[m] = m < a.n_out ? ld4(a.mix[m] + cv) : zero4();
    for (unsigned line = first; line < min(first + g.per_walker, g.lines); ++line) {
        const Stretch s = stretch_at(g, line, which, cv);
        float4 x[kStretch], prev = zero4();
        if (s.before) prev = ld4(a.x + s.base - s.step);
#pragma unroll
        for (int j = 0; j < kStretch; ++j) x[j] = j < s.n ? ld4(a.x + s.base + j * s.step) : zero4();
#pragma unroll
        for (int j = 0; j < kStretch; ++j) {
            if (j < s.n) {
                const float4 from = which > 3 ? x[j] : prev;
                const float4 d = sub4(x[j], from);
#pragma unroll
                for (int m = 0; m < kMaxOut; ++m)
                    if (m < a.n_out) st4(reinterpret_cast<Out*>(a.out[m]) + s.base + j * s.step, fma4(mix[m], d, from));
            }
            prev = x[j];
        }
    }
}

__global__ void __launch_bounds__(qlines::kMaxThreads, 2) qshift_lines_backward(const Args a, const qlines::Grid g) {
    wait_for_launch_before();
    using namespace qlines;
    const int cv = (blockIdx.y * blockDim.x + threadIdx.x) * 4;
    if (cv >= g.C) return;
    const int which = group_of(g, cv);
    const unsigned walker = blockIdx.x * blockDim.y + threadIdx.y, first = walker * static_cast<unsigned>(g.per_walker);
    float4 gmix[kMaxOut];
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m) gmix[m] = zero4();
    for (unsigned line = first; line < min(first + g.per_walker, g.lines); ++line) {
        const Stretch s = stretch_at(g, line, which, cv);
        float4 d[kStretch], gx[kStretch];          // x minus its shifted value; gradient of x
        {
            float4 prev = zero4();
            if (s.before) prev = ld4(a.x + s.base - s.step);
#pragma unroll
            for (int j = 0; j < kStretch; ++j) {
                d[j] = j < s.n ? ld4(a.x + s.base + j * s.step) : zero4();
                gx[j] = zero4();
            }
#pragma unroll
            for (int j = 0; j < kStretch; ++j) {
                const float4 x = d[j];
                d[j] = sub4(x, which > 3 ? x : prev);
                prev = x;
            }
        }
#pragma unroll
        for (int m = 0; m < kMaxOut; ++m) {
            if (m < a.n_out) {
                // the token that reads token j through the shift is token j + 1 of the line
                float4 go[kStretch + 1];
#pragma unroll
                for (int j = 0; j <= kStretch; ++j)
                    go[j] = j < s.n || (j == s.n && s.after) ? ld4(a.gout[m] + s.base + j * s.step) : zero4();
                const float4 mix = ld4(a.mix[m] + cv), rest = make_float4(1.f - mix.x, 1.f - mix.y, 1.f - mix.z, 1.f - mix.w);
#pragma unroll
                for (int j = 0; j < kStretch; ++j)
                    if (j < s.n) {
                        gmix[m] = fma4(go[j], d[j], gmix[m]);
                        gx[j] = fma4(which > 3 ? go[j] : go[j + 1], rest, fma4(go[j], mix, gx[j]));
                    }
            }
        }
#pragma unroll
        for (int j = 0; j < kStretch; ++j)
            if (j < s.n) st4(a.gx + s.base + j * s.step, gx[j]);
    }
#pragma unroll
    for (int m = 0; m < kMaxOut; ++m)
        if (m < a.n_out) st4(a.partial + (static_cast<size_t>(walker) * a.n_out + m) * g.C + cv, gmix[m]);
}

// gmix[m][c] = sum over row blocks of partial[block][m][c], fixed order
__global__ void __launch_bounds__(1024) qshift_reduce(const float* partial, int blocks, int n_out, int C,
                                                      float* __restrict__ gmix0, float* __restrict__ gmix1,
                                                      float* __restrict__ gmix2) {
    wait_for_launch_before();
    __shared__ float red[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x, m = blockIdx.y;
    // kAhead rows asked for together and added up in order (1152 rows of 3 x 1024: 17.7 -> 6.2 us), fewer one by one
    constexpr int kAhead = 12;
    float acc = 0.f;
    if (c < C) {
        const float* p = partial + static_cast<size_t>(m) * C + c;
        const size_t pitch = static_cast<size_t>(n_out) * C;
        int r = threadIdx.y;
        for (; r + 32 * (kAhead - 1) < blocks; r += 32 * kAhead) {
            float v[kAhead];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) v[i] = p[(r + 32 * i) * pitch];
#pragma unroll
            for (int i = 0; i < kAhead; ++i) acc += v[i];
        }
        for (; r < blocks; r += 32) acc += p[r * pitch];
    }
    red[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && c < C) {
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) total += red[r][threadIdx.x];
        (m == 0 ? gmix0 : m == 1 ? gmix1 : gmix2)[c] = total;
    }
}

static bool vector_ok(const Args& a, bool bwd) {
    if (a.C % 4 || a.group % 4) return false;
    uintptr_t bits = reinterpret_cast<uintptr_t>(a.x);
    for (int m = 0; m < a.n_out; ++m) {
        bits |= reinterpret_cast<uintptr_t>(a.mix[m]);
        bits |= reinterpret_cast<uintptr_t>(bwd ? static_cast<const void*>(a.gout[m]) : static_cast<const void*>(a.out[m]));
    }
    if (bwd) bits |= reinterpret_cast<uintptr_t>(a.gx) | reinterpret_cast<uintptr_t>(a.partial);
    return (bits & 15u) == 0;
}
// the walks cover a shift of one pixel (the only one the models use) on whole 4-channel vectors
static bool walks(const Args& a, const qlines::Grid& g, bool bwd) { return a.shift == 1 && g.lines != 0 && vector_ok(a, bwd); }

static int row_blocks(const Args& a) {
    const long long ntok = static_cast<long long>(a.B) * a.H * a.W;
    return static_cast<int>((ntok + kTokensPerBlock - 1) / kTokensPerBlock);
}

size_t backward_workspace(int B, int H, int W, int C, int n_out) {
    Args a{};
    a.B = B; a.H = H; a.W = W;
    // rows of partial sums of the general kernels, or of the walks (neither depends on the shift's group)
    const long long walkers = qlines::make_shape(qlines::make_grid(B, H, W, C, 1, 0)).walkers;
    return static_cast<size_t>(std::max<long long>(row_blocks(a), walkers)) * n_out * C * sizeof(float);
}

// One stretch per walker: with four, as the backward's partial sums want them, the blocks were one and a half rounds of what the device holds
// (256 x 14 x 14 x 384, three bfloat16 outputs: 896 of 592), the last one half empty: 36.9 -> 31.4 us, two outputs 28.8 -> 25.7; float32, 64 x 24 x 24 x
// 1024 103 -> 93.8; over twenty sizes of 2 to 75 million elements 0 to 19 % less.  (VRWKV6's shift without offsets, one output, is slower
// so: 43.5 -> 48.0 at the last size.)
template <typename Out>
static void forward_as(const Args& a, cudaStream_t stream) {
    const qlines::Grid g = qlines::make_grid(a.B, a.H, a.W, a.C, a.group, a.period, qlines::kStretch, 1);
    const int by = row_blocks(a);
    if (walks(a, g, false)) {
        const qlines::Shape s = qlines::make_shape(g);
        launch_behind(qshift_lines_forward<Out>, s.grid, s.block, 0, stream, a, g);
    } else if (vector_ok(a, false)) {
        qshift_mix_forward<4, Out><<<dim3((a.C / 4 + kThreads - 1) / kThreads, by), kThreads, 0, stream>>>(a);
    } else {
        qshift_mix_forward<1, Out><<<dim3((a.C + kThreads - 1) / kThreads, by), kThreads, 0, stream>>>(a);
    }
}

int forward(const Args& a, cudaStream_t stream) {
    if (a.out_bf16) forward_as<__nv_bfloat16>(a, stream);
    else forward_as<float>(a, stream);
    return 1;
}

int backward(const Args& a, float* const gmix[kMaxOut], cudaStream_t stream) {
    const qlines::Grid g = qlines::make_grid(a.B, a.H, a.W, a.C, a.group, a.period);
    int rows = row_blocks(a);
    if (walks(a, g, true)) {
        const qlines::Shape s = qlines::make_shape(g);
        rows = static_cast<int>(s.walkers);
        launch_behind(qshift_lines_backward, s.grid, s.block, 0, stream, a, g);
    } else if (a.C % 4 == 0 && a.group % 4 == 0) {
        // the vector form of the general kernel only needs the group boundary rule (scalar loads inside)
        qshift_mix_backward<4><<<dim3((a.C / 4 + kThreads - 1) / kThreads, rows), kThreads, 0, stream>>>(a);
    } else {
        qshift_mix_backward<1><<<dim3((a.C + kThreads - 1) / kThreads, rows), kThreads, 0, stream>>>(a);
    }
    launch_behind(qshift_reduce, dim3((a.C + 31) / 32, a.n_out), dim3(32, 32), 0, stream, a.partial, rows, a.n_out, a.C, gmix[0],
                                                                              gmix[1], gmix[2]);
    return 2;
}

}  // namespace qshift

// ---- C ABI --------------------------------------------------------------------------------------
#include "vrwkv_b200.h"

static int qshift_check(int B, int H, int W, int C, int group, int shift, int n_out) {
    if (B <= 0 || H <= 0 || W <= 0 || C <= 0 || group <= 0 || shift < 0 || n_out < 1 || n_out > 3) return VRWKV_ERR_SHAPE;
    if (4LL * group > C + 0LL && group * 4 > C) return VRWKV_ERR_SHAPE;      // at most four shifted groups fit
    if ((static_cast<long long>(B) * H * W + 31) / 32 > 65535LL * 32768) return VRWKV_ERR_SHAPE;
    return VRWKV_OK;
}

static int qshift_forward_any(int B, int H, int W, int C, int group, int period, int shift, int n_out, const float* x,
                              const float* const* mix, void* const* out, bool out_bf16, void* stream) {
    if (int st = qshift_check(B, H, W, C, group, shift, n_out)) return st;
    if (!x || !mix || !out) return VRWKV_ERR_NULL;
    qshift::Args a{};
    a.B = B; a.H = H; a.W = W; a.C = C; a.group = group; a.period = period; a.shift = shift; a.n_out = n_out; a.x = x;
    for (int m = 0; m < n_out; ++m) {
        if (!mix[m] || !out[m]) return VRWKV_ERR_NULL;
        a.mix[m] = mix[m];
        a.out[m] = static_cast<float*>(out[m]);
    }
    a.out_bf16 = out_bf16;
    return record_launches(qshift::forward(a, static_cast<cudaStream_t>(stream)));
}

static int qshift_backward_any(int B, int H, int W, int C, int group, int period, int shift, int n_out, const float* x,
                               const float* const* mix, const float* const* gout, float* gx, float* const* gmix,
                               void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = qshift_check(B, H, W, C, group, shift, n_out)) return st;
    if (!x || !mix || !gout || !gx || !gmix || !workspace) return VRWKV_ERR_NULL;
    if (workspace_bytes < qshift::backward_workspace(B, H, W, C, n_out)) return VRWKV_ERR_WORKSPACE;
    qshift::Args a{};
    a.B = B; a.H = H; a.W = W; a.C = C; a.group = group; a.period = period; a.shift = shift; a.n_out = n_out; a.x = x;
    a.gx = gx;
    a.partial = static_cast<float*>(workspace);
    float* gm[qshift::kMaxOut] = {nullptr, nullptr, nullptr};
    for (int m = 0; m < n_out; ++m) {
        if (!mix[m] || !gout[m] || !gmix[m]) return VRWKV_ERR_NULL;
        a.mix[m] = mix[m];
        a.gout[m] = gout[m];
        gm[m] = gmix[m];
    }
    return record_launches(qshift::backward(a, gm, static_cast<cudaStream_t>(stream)));
}

// head_dim channels per head, a multiple of 4 that divides C; the groups are its quarters
static int multihead_check(int C, int head_dim) {
    return (head_dim < 4 || head_dim % 4 != 0 || C % head_dim != 0) ? VRWKV_ERR_SHAPE : VRWKV_OK;
}

extern "C" int vrwkv_qshift_mix_forward_f32(int B, int H, int W, int C, int group, int shift, int n_out,
                                            const float* x, const float* const* mix, float* const* out,
                                            void* stream) {
    return qshift_forward_any(B, H, W, C, group, 0, shift, n_out, x, mix, reinterpret_cast<void* const*>(out), false, stream);
}

extern "C" int vrwkv_qshift_multihead_mix_forward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out,
                                                      const float* x, const float* const* mix, float* const* out,
                                                      void* stream) {
    if (int st = multihead_check(C, head_dim)) return st;
    return qshift_forward_any(B, H, W, C, head_dim / 4, head_dim, shift, n_out, x, mix, reinterpret_cast<void* const*>(out), false, stream);
}

extern "C" int vrwkv_qshift_mix_forward_bf16out(int B, int H, int W, int C, int group, int head_dim, int shift, int n_out, const float* x,
                                                const float* const* mix, uint16_t* const* out, void* stream) {
    if (head_dim)
        if (int st = multihead_check(C, head_dim)) return st;
    return qshift_forward_any(B, H, W, C, head_dim ? head_dim / 4 : group, head_dim, shift, n_out, x, mix,
                              reinterpret_cast<void* const*>(out), true, stream);
}

extern "C" size_t vrwkv_qshift_mix_backward_workspace_bytes(int B, int H, int W, int C, int n_out) {
    if (B <= 0 || H <= 0 || W <= 0 || C <= 0 || n_out < 1 || n_out > 3) return 0;
    return qshift::backward_workspace(B, H, W, C, n_out);
}

extern "C" int vrwkv_qshift_mix_backward_f32(int B, int H, int W, int C, int group, int shift, int n_out,
                                             const float* x, const float* const* mix, const float* const* gout,
                                             float* gx, float* const* gmix, void* workspace, size_t workspace_bytes,
                                             void* stream) {
    return qshift_backward_any(B, H, W, C, group, 0, shift, n_out, x, mix, gout, gx, gmix, workspace, workspace_bytes, stream);
}

extern "C" int vrwkv_qshift_multihead_mix_backward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out,
                                                       const float* x, const float* const* mix,
                                                       const float* const* gout, float* gx, float* const* gmix,
                                                       void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = multihead_check(C, head_dim)) return st;
    return qshift_backward_any(B, H, W, C, head_dim / 4, head_dim, shift, n_out, x, mix, gout, gx, gmix, workspace,
                               workspace_bytes, stream);
}
