// Work split of the one-pixel token shift kernels (qshift_mix.cu, qshift_ddlerp.cu): walks along the shift.
//
// With a shift of one pixel every shifted channel takes its value from the token before it on a line of the grid: a
// row for the horizontal groups, a column for the vertical ones, walked in the direction of the shift.  A thread owns
// 4 consecutive channels (one group) and a stretch of up to kStretch tokens of such a line, so each value that a
// neighbour needs is already in a register: one halo load per stretch replaces a second load per token, and all loads of a
// stretch are issued together (9 independent 16-byte loads in flight per thread and tensor).  Channels of different
// groups walk different lines; a warp's accesses still cover whole 32-byte sectors.  Token-by-token code with
// one load and a 64-bit division per token in flight measured 0.56 of the HBM rate; this measures 0.87 (B=64, 24 x 24, C=1024,
// three outputs, forward + backward: 376 and 238 us).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>

namespace qlines {

constexpr int kStretch = 8;        // tokens a thread holds at a time (at most)
constexpr int kMaxThreads = 256;   // of a block: channel vectors x walkers

struct Grid {
    int B, H, W, C;
    int group;     // channels per shifted group
    int period;    // 0: the four groups are channels [0, 4 * group); n: they repeat every n channels
    int row_parts, row_len;    // a row in row_parts stretches of row_len tokens
    int col_parts, col_len;    // a column likewise
    unsigned lines;            // stretches per walk kind, the larger of the two, over the batch
    int per_walker;            // consecutive stretches of one walker
};

struct Shape {
    dim3 grid, block;
    long long walkers;
};

// (host) stretches as even as possible; enough of them per walker that partial sums stay small beside the tensors, few
// enough that the blocks fill the device; at most most_per_walker
inline Grid make_grid(int B, int H, int W, int C, int group, int period, int stretch = kStretch, int most_per_walker = 4) {
    Grid g{};
    g.B = B; g.H = H; g.W = W; g.C = C; g.group = group; g.period = period;
    g.row_parts = (W + stretch - 1) / stretch;
    g.row_len = (W + g.row_parts - 1) / g.row_parts;
    g.col_parts = (H + stretch - 1) / stretch;
    g.col_len = (H + g.col_parts - 1) / g.col_parts;
    const long long each = std::max(static_cast<long long>(H) * g.row_parts, static_cast<long long>(W) * g.col_parts);
    const long long lines = each * B;
    g.lines = lines < (1LL << 31) ? static_cast<unsigned>(lines) : 0u;      // 0: too many, the caller takes its general kernels
    const int vecs = C / 4, by = std::max(1, kMaxThreads / std::max(1, vecs));
    // 148 SMs with four blocks each
    g.per_walker = static_cast<int>(std::min<long long>(most_per_walker, std::max<long long>(1, lines / (592LL * by))));
    return g;
}
inline Shape make_shape(const Grid& g) {
    Shape s;
    const int vecs = g.C / 4;
    const int bx = std::min(vecs, kMaxThreads), by = std::max(1, kMaxThreads / std::max(1, vecs));
    const long long walkers = (static_cast<long long>(g.lines) + g.per_walker - 1) / g.per_walker;
    s.block = dim3(bx, by);
    s.grid = dim3(static_cast<unsigned>((walkers + by - 1) / by), (vecs + bx - 1) / bx);
    s.walkers = static_cast<long long>(s.grid.x) * by;
    return s;
}

// One stretch of one thread's channels: element offset of its first token, element step to the next (in walk order), tokens
struct Stretch {
    size_t base;
    long long step;
    int n;
    bool before, after;     // a token of the line precedes / follows the stretch
};
// group of the 4 channels from cv: 0 left, 1 right, 2 upper, 3 lower neighbour, above: unshifted
__device__ __forceinline__ int group_of(const Grid& g, int cv) { return (g.period ? cv % g.period : cv) / g.group; }

__device__ __forceinline__ Stretch stretch_at(const Grid& g, unsigned line, int which, int cv) {
    const bool row = which < 2 || which > 3;
    const int parts = row ? g.row_parts : g.col_parts, len = row ? g.row_len : g.col_len;
    const int across = row ? g.H : g.W, along = row ? g.W : g.H;
    const unsigned each = g.lines / static_cast<unsigned>(g.B);
    const int b = static_cast<int>(line / each), i = static_cast<int>(line % each);
    Stretch s;
    s.n = 0;
    s.before = s.after = false;
    s.base = 0;
    s.step = 0;
    if (i >= across * parts) return s;         // the other walk kind has more stretches
    // rows: a row's stretches are neighbours; columns: the columns of one band of rows are
    const int q = row ? i / parts : i % across, part = row ? i % parts : i / across;
    const int j0 = part * len;
    s.n = min(len, along - j0);
    if (s.n <= 0) { s.n = 0; return s; }
    s.before = j0 > 0;
    s.after = j0 + s.n < along;
    const bool back = which == 1 || which == 3;            // the source is the NEXT token of the raster: walk backwards
    const int at = back ? along - 1 - j0 : j0;
    const long long tok = static_cast<long long>(b) * g.H * g.W + (row ? static_cast<long long>(q) * g.W + at : static_cast<long long>(at) * g.W + q);
    s.base = static_cast<size_t>(tok) * g.C + cv;
    s.step = (row ? 1LL : static_cast<long long>(g.W)) * g.C * (back ? -1 : 1);
    return s;
}

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 zero4() { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float4 sub4(float4 a, float4 b) { return make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w); }
// a * b + c
__device__ __forceinline__ float4 fma4(float4 a, float4 b, float4 c) {
    return make_float4(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z), fmaf(a.w, b.w, c.w));
}
__device__ __forceinline__ void st4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void st4(__nv_bfloat16* p, float4 v) {
    uint2 raw;
    *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(v.x, v.y);
    *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = raw;
}

__device__ __forceinline__ void st8(float* p, float4 a, float4 b) { st4(p, a); st4(p + 4, b); }
__device__ __forceinline__ void st8(__nv_bfloat16* p, float4 a, float4 b) {
    uint4 raw;
    *reinterpret_cast<__nv_bfloat162*>(&raw.x) = __floats2bfloat162_rn(a.x, a.y);
    *reinterpret_cast<__nv_bfloat162*>(&raw.y) = __floats2bfloat162_rn(a.z, a.w);
    *reinterpret_cast<__nv_bfloat162*>(&raw.z) = __floats2bfloat162_rn(b.x, b.y);
    *reinterpret_cast<__nv_bfloat162*>(&raw.w) = __floats2bfloat162_rn(b.z, b.w);
    *reinterpret_cast<uint4*>(p) = raw;
}

}  // namespace qlines
