// WKV6 (head size 64, bidirectional), forward and backward, in 64-token chunks on the tensor cores.
//
// With l_m = log2 of the decays (log2 e * -exp(w_raw)) and D(t, s) = 2^(sum of l strictly between t and s), the operator is
//   y_t = sum_{s != t} (sum_i r_t[i] D(t,s)[i] k_s[i]) v_s + (sum_i r_t[i] u[i] k_t[i]) v_t
// and its gradients are sums over the same pairs.  Two kernels:
//
//   1. states: per (batch, head, direction) one CTA walks the chunks and leaves in global memory the 64 x 64 state
//      that ENTERS every chunk,  X <- 2^(sum l) X + sum_s (x_s 2^(decay to the chunk's edge)) z_s^T,
//      (x, z) = (k, v) for the forward; the backward needs (k, v) and the adjoint pair (r, gy).
//   2. outputs: one CTA per chunk, all chunks in parallel, both directions at once: read-out of the entering states,
//      the 64 x 64 pairs inside the chunk, and (backward) the decay gradient.
//
// What bounds it: memory in the first kernel, shared-memory accesses in the second (below).  Per element of a (B, T, C) tensor the bfloat16
// forward moves 20 bytes in the first kernel and 18 in the second (the states are 4 of each), the backward 44 and 40, 2.0 + 1.8 and 4.4 + 4.0 GB
// at B=32, T=4096, H=12, which take 0.30 + 0.61 and 0.74 + 1.99 ms; the products are about 0.8 and 3.6 kFLOP
// (0.26 and 1.0 of them in the first kernel).  The walk of the first kernel is serial over T / 64 chunks but holds only the state update; everything else
// is parallel over chunks, which a walk over the whole sequence per CTA (16 tokens at a time with the state in tensor
// memory: 1.47 + 7.8 ms at B=32, T=4096, H=12) was not.  64-wide heads make 16 x 64 x 64 products: mma.sync keeps their
// operands, scalings and masks in registers, where tcgen05 would stage each through shared memory and tensor memory for
// a product that takes 30 cycles.  The chunk length trades state traffic (1 / length) against pairs inside the chunk.
//
// Stability.  Exponents are sums of l over stretches of one 16-token block, most of them differences of its running sums; l
// is bounded below where 2^l is zero anyway (log2_decay), so those differences are good to 1e-4 even next to a token that
// forgets everything.  Between blocks no exponent is positive: block b's tokens are scaled towards the block's edges
// (2^(<= 0)), and a block further away takes the decay across the blocks in between as one more factor <= 1.  Inside a block
// a row is scaled by 2^(-the block's sum) relative to that, up to 2^kSafe; where a channel's sum over the block is below
// -kSafe, the block takes its pairs in four levels of halves (16, 8, 4, 2 tokens), with factors <= 1 only.
//
// Decay gradient.  With R> = r gr>, K> = k gk> (one-sided parts, elementwise) and the mirrored R<, K<, the gradient with
// respect to l_m counts the pairs that have m strictly between them.  Counted from the chunk's right edge,
//   g_m = edge + sum_{t > m} (R> + K< - K> - R<)_t - K>_m - R<_m,   edge[i] = sum_j (S> A> + A< S<)[i][j]
// where S>, A< have passed the edge rightward and A>, S< leftward.  Rounding errors stay within one chunk.
//
// Reference being replaced: classification/mmcls_custom/models/backbones/cuda_v6/wkv6_cuda.cu:6-346.
#include <algorithm>
#include <atomic>
#include <mutex>
#include <set>
#include <utility>
#include "launch.h"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"
#include "wkv6_chunk.cuh"

namespace wkv6c {

constexpr float kSafe = 64.f;       // largest |sum of l| over a block for which its own pairs may use factors above 1

typedef float Table[kChunk][kTab];

// ---- kernel 1: states entering every chunk ----------------------------------------------------------------
struct StateArgs {
    int T, H, n_chunks;
    uint4* out;              // [pair][direction][b h][chunk][part][kStateWords / 4]
    size_t plane;            // uint4 per (pair, direction)
    unsigned* status;        // the launch's status word and its host-visible copy
    unsigned* mirror;
    unsigned limit;          // polls of a wait
    unsigned extra;          // test only: bytes that a barrier waits for and no copy brings
};
// Polls before a wait for a tile gives up.  After that nothing is copied to where it would have been, and what is under way is waited for a
// little longer, so that a CTA leaves no copy behind.
constexpr uint32_t kWaitLimit = 1u << 20;

// Shared memory of a CTA, twice (the next chunk's tiles arrive during the whole of a step): the tiles of one chunk as the copy engine delivers
// them (w | x, z of every pair).  The operands take their place: a warp reads its tokens' rows and writes the same rows, 16-byte pieces
// exchanged by the row's number so that ldmatrix meets no bank twice; x's second part lies behind the first in a float row, else in
// the row of w, which its warp has read by then.
//
// What bounds the walk: HBM, since the two directions meet the inputs at different times and each reads them (forward 2 x 8 and backward 2 x 14 bytes an
// element, states 4 and 16).  B=32, H=12, T=4096, forward / backward us: 301 / 745 (2.0 and 4.4 GB: 6.6 and 5.9 TB/s), T=196 17.7 / 40.7.  Operand planes
// beside one set of tiles, fetched while the products ran, and each pair's factors computed by its own warps: 450 / 902, 19.6 / 43.2; the
// present form with one set of tiles, three CTAs instead of two on an SM: 479 / 1000; with sixteen warps of four tokens: 329 / 991 (one CTA on an SM).
template <typename XT, typename ZT0, typename ZT1, int kX, int kPairs>
struct StateSmem {
    static constexpr uint32_t kWPitch = N * 4, kXPitch = N * sizeof(XT), kZ0Pitch = N * sizeof(ZT0), kZ1Pitch = N * sizeof(ZT1);
    static constexpr uint32_t w = 0, x0 = kChunk * kWPitch, z0 = x0 + kChunk * kXPitch;
    static constexpr uint32_t x1 = z0 + kChunk * kZ0Pitch, z1 = x1 + (kPairs > 1 ? kChunk * kXPitch : 0);
    static constexpr uint32_t loaded = z1 + (kPairs > 1 ? kChunk * kZ1Pitch : 0);
    // sums of l over each warp's tokens, and the state's decay across the chunk: 32 floats to a row.  A float z of the second pair leaves the
    // second half of its rows free when its warp has read them (1.3 KB too much for two CTAs on an SM otherwise).
    static constexpr bool kInside = kPairs > 1 && sizeof(ZT1) == 4 && sizeof(XT) == 2;
    static constexpr uint32_t sums = kInside ? z1 + 128 : 2 * loaded, kSumPitch = kInside ? kZ1Pitch : 128;
    static constexpr uint32_t bar = 2 * loaded + (kInside ? 0 : (4 * kPairs + 1) * N * 4);
    static constexpr size_t bytes = bar + 16;
};
struct Rows { uint32_t at, pitch; };      // an operand: 64 rows (tokens) of 128 bytes
// 32-bit word `word` of a row
__device__ __forceinline__ uint32_t word_at(Rows p, int row, int word) { return p.at + row * p.pitch + (((word >> 2) ^ (row & 7)) << 4) + ((word & 3) << 2); }
__device__ __forceinline__ uint32_t chunk_at(Rows p, int row, int chunk) { return p.at + row * p.pitch + ((chunk ^ (row & 7)) << 4); }
__device__ __forceinline__ void put_word(uint32_t at, uint32_t v) { asm volatile("st.shared.b32 [%0], %1;" ::"r"(at), "r"(v) : "memory"); }
// a token's channel pair as one bfloat16 pair
__device__ __forceinline__ uint32_t half_pair(const __nv_bfloat16* row, int lane) { return *reinterpret_cast<const uint32_t*>(row + 2 * lane); }
__device__ __forceinline__ uint32_t half_pair(const float* row, int lane) {
    const float2 v = *reinterpret_cast<const float2*>(row + 2 * lane);
    uint32_t t[1];
    split<1>(v.x, v.y, t);
    return t[0];
}

// grid (b h, direction); direction 0 walks rightward (decay to the chunk's right edge), 1 leftward; four warps per pair of
// inputs.  kX parts of the scaled x; kRows: the state's rows are the channels of x (else its columns).  A warp scales kTokens tokens of all
// pairs, which share the factors: lane = two channels, one token after the other, so decays, their running sums and the scaling need no
// shuffles.
template <typename XT, typename ZT0, typename ZT1, int kX, bool kRows, int kPairs>
__global__ void __launch_bounds__(128 * kPairs, kPairs == 1 ? 3 : 2)
wkv6_state_kernel(const StateArgs a, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mx0,
                  const __grid_constant__ CUtensorMap mz0, const __grid_constant__ CUtensorMap mx1, const __grid_constant__ CUtensorMap mz1) {
    wait_for_launch_before();
    typedef StateSmem<XT, ZT0, ZT1, kX, kPairs> S;
    constexpr int kWarps = 4 * kPairs, kTokens = kChunk / kWarps, kZ = 1;
    extern __shared__ __align__(1024) unsigned char smem[];
    const int bh = blockIdx.x, dir = blockIdx.y, w8 = threadIdx.x >> 5, pair = w8 >> 2, warp = w8 & 3;
    const int b = bh / a.H, h = bh - b * a.H;
    const int lane = threadIdx.x & 31, g = lane >> 2;
    constexpr int kState = kX * kStateWords / 4;
    uint4* out = a.out + (static_cast<size_t>(pair) * 2 + dir) * a.plane + static_cast<size_t>(bh) * a.n_chunks * kState;
    // where channel `ch` of warp j's sum is, and (behind another's, or in its writer's third and fourth row) of the state's decay
    unsigned char* raw = smem;
    const auto total_at = [&](int j, int ch) {
        return reinterpret_cast<float*>((S::kInside ? raw : smem) + S::sums + ((S::kInside ? j * kTokens : 2 * j) + (ch >> 5)) * S::kSumPitch + (ch & 31) * 4);
    };
    const auto decay_at = [&](int ch) {
        return reinterpret_cast<float*>((S::kInside ? raw : smem) + S::sums + ((S::kInside ? (dir == 0 ? 2 : kChunk - kTokens + 2) : 2 * kWarps) + (ch >> 5)) * S::kSumPitch + (ch & 31) * 4);
    };
    uint64_t* bar = reinterpret_cast<uint64_t*>(smem + S::bar);
    const uint32_t base_at = smem_addr(smem);
    uint32_t at = base_at;
    const auto part_of = [&](int p, int part) {      // x's parts
        const uint32_t x = at + (p == 0 ? S::x0 : S::x1);
        if (part == 0) return Rows{x, S::kXPitch};
        return sizeof(XT) == 4 ? Rows{x + 128, S::kXPitch} : Rows{at + S::w + p * 128, S::kWPitch};
    };
    const auto chunk_of = [&](int step) { return dir == 0 ? step : a.n_chunks - 1 - step; };
    const auto fetch = [&](int step) {
        const int t0 = chunk_of(step) * kChunk;
        unsigned char* const to = smem + (step & 1) * S::loaded;
        uint64_t* const full = bar + (step & 1);
        sm100::mbar_expect_tx(full, S::loaded + a.extra);
        sm100::tma_load_3d(to + S::w, &mw, full, h * N, t0, b);
        sm100::tma_load_3d(to + S::x0, &mx0, full, h * N, t0, b);
        sm100::tma_load_3d(to + S::z0, &mz0, full, h * N, t0, b);
        if (kPairs > 1) {
            sm100::tma_load_3d(to + S::x1, &mx1, full, h * N, t0, b);
            sm100::tma_load_3d(to + S::z1, &mz1, full, h * N, t0, b);
        }
    };
    const int last = a.n_chunks - 1;        // steps that update the state
    if (threadIdx.x == 0) {
        sm100::mbar_init(bar, 1);
        sm100::mbar_init(bar + 1, 1);
        sm100::mbar_init_fence();
        fetch(0);
        if (last > 1) fetch(1);
    }
    __syncthreads();
    const int row0 = w8 * kTokens, word = col_word(lane);
    Acc c;
    zero(c);
    int gave_up = last;      // the step whose tiles did not come
    for (int step = 0; step < last; ++step) {
        const int valid = a.T - chunk_of(step) * kChunk;
        if (step < gave_up && !sm100::mbar_wait(bar + (step & 1), step >> 1 & 1, a.limit)) {
            gave_up = step;
            report_failure(a.status, a.mirror, 2u);
        }
        at = base_at + (step & 1) * S::loaded;
        raw = smem + (step & 1) * S::loaded;
        float2 sum[kTokens];
        float2 run = make_float2(0.f, 0.f);
        {
            const float* wt = reinterpret_cast<const float*>(raw + S::w) + row0 * N + 2 * lane;
#pragma unroll
            for (int t = 0; t < kTokens; ++t) {
                const float2 w = *reinterpret_cast<const float2*>(wt + t * N);
                run.x += log2_decay(w.x, row0 + t < valid);
                run.y += log2_decay(w.y, row0 + t < valid);
                sum[t] = run;
            }
        }
        uint32_t zi[kTokens];
        if (S::kInside) {
#pragma unroll
            for (int t = 0; t < kTokens; ++t) zi[t] = half_pair(reinterpret_cast<const ZT1*>(raw + S::z1) + (row0 + t) * N, lane);
            __syncwarp();
        }
        *reinterpret_cast<float2*>(total_at(w8, 2 * lane)) = run;
        __syncthreads();
        // a token's factor: the decay from it to the chunk's edge.  Small sums first: the way to the end of the warp's tokens, then
        // the rest of the chunk
        float2 edge;
        {
            float2 t[kWarps];
#pragma unroll
            for (int j = 0; j < kWarps; ++j) {
                t[j] = *reinterpret_cast<const float2*>(total_at(j, 2 * lane));
                if (dir == 0 ? j <= w8 : j >= w8) t[j] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int d = 1; d < kWarps; d *= 2)
#pragma unroll
                for (int j = 0; j < kWarps; j += 2 * d) { t[j].x += t[j + d].x; t[j].y += t[j + d].y; }
            edge = t[0];
        }
        if (w8 == (dir == 0 ? 0 : kWarps - 1)) *reinterpret_cast<float2*>(decay_at(2 * lane)) = make_float2(ex2(edge.x + run.x), ex2(edge.y + run.y));
        if (dir == 0) {
#pragma unroll
            for (int t = 0; t < kTokens; ++t) sum[t] = make_float2(ex2(edge.x + (run.x - sum[t].x)), ex2(edge.y + (run.y - sum[t].y)));
        } else {
#pragma unroll
            for (int t = kTokens - 1; t >= 0; --t)
                sum[t] = t > 0 ? make_float2(ex2(edge.x + sum[t - 1].x), ex2(edge.y + sum[t - 1].y)) : make_float2(ex2(edge.x), ex2(edge.y));
        }
#pragma unroll
        for (int p = 0; p < kPairs; ++p) {
            const XT* x = reinterpret_cast<const XT*>(raw + (p == 0 ? S::x0 : S::x1)) + row0 * N;
            float2 xv[kTokens];
            uint32_t zv[kTokens];
#pragma unroll
            for (int t = 0; t < kTokens; ++t) {
                const uint32_t r = half_pair(x + t * N, lane);      // raw inputs are rounded to bfloat16 where they arrive as float
                xv[t] = make_float2(lo_f(r) * sum[t].x, hi_f(r) * sum[t].y);
                zv[t] = p == 0        ? half_pair(reinterpret_cast<const ZT0*>(raw + S::z0) + (row0 + t) * N, lane)
                        : S::kInside ? zi[t]
                                     : half_pair(reinterpret_cast<const ZT1*>(raw + S::z1) + (row0 + t) * N, lane);
            }
            __syncwarp();      // the rows have been read
            const Rows z = p == 0 ? Rows{at + S::z0, S::kZ0Pitch} : Rows{at + S::z1, S::kZ1Pitch};
#pragma unroll
            for (int t = 0; t < kTokens; ++t) {
                uint32_t parts[kX];
                split<kX>(xv[t].x, xv[t].y, parts);
#pragma unroll
                for (int i = 0; i < kX; ++i) put_word(word_at(part_of(p, i), row0 + t, word), parts[i]);
                put_word(word_at(z, row0 + t, word), zv[t]);
            }
        }
        __syncthreads();
        // decay of the state across the chunk
        if (kRows) {
            const int ch = 16 * warp + 4 * (g >> 1) + (g & 1);
            const float s0 = *decay_at(ch), s1 = *decay_at(ch + 2);
#pragma unroll
            for (int i = 0; i < 8; ++i) { c[i][0] *= s0; c[i][1] *= s0; c[i][2] *= s1; c[i][3] *= s1; }
        } else {
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float s[4];
                row4(decay_at(16 * kk + 4 * (lane & 3)), 0, 0, s);
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int e = 0; e < 4; ++e) c[2 * kk + (e >> 1)][half * 2 + (e & 1)] *= s[e];
            }
        }
        const Rows z = pair == 0 ? Rows{at + S::z0, S::kZ0Pitch} : Rows{at + S::z1, S::kZ1Pitch};
        constexpr int kM = kRows ? kX : kZ, kN = kRows ? kZ : kX;
#pragma unroll
        for (int s = 0; s < kBlocks; ++s) {
            uint32_t am[kM][4];
            const int rm = s * kBlock + ((lane >> 4) << 3) + (lane & 7), rn = s * kBlock + (((lane >> 3) & 1) << 3) + (lane & 7);
#pragma unroll
            for (int i = 0; i < kM; ++i) ldsm4t(am[i], chunk_at(kRows ? part_of(pair, i) : z, rm, 2 * warp + ((lane >> 3) & 1)));
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int ib = 0; ib < kN; ++ib) {
                    uint32_t r[4];
                    ldsm4t(r, chunk_at(kRows ? z : part_of(pair, ib), rn, 2 * kk + (lane >> 4)));
#pragma unroll
                    for (int ia = 0; ia < kM; ++ia)
                        if (Keep<kM, kN>::on(ia, ib)) {
                            mma(c[2 * kk], am[ia], r[0], r[1]);
                            mma(c[2 * kk + 1], am[ia], r[2], r[3]);
                        }
                }
        }
        sm100::fence_proxy_async_smem();      // the copy engine writes where the operands were
        __syncthreads();
        if (threadIdx.x == 0 && step + 2 < last && gave_up == last) fetch(step + 2);
        uint4* o = out + static_cast<size_t>(chunk_of(step + 1)) * kState;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            uint32_t w0[kX], w1[kX], w2[kX], w3[kX];
            split<kX>(c[2 * kk][0], c[2 * kk][1], w0);
            split<kX>(c[2 * kk + 1][0], c[2 * kk + 1][1], w1);
            split<kX>(c[2 * kk][2], c[2 * kk][3], w2);
            split<kX>(c[2 * kk + 1][2], c[2 * kk + 1][3], w3);
#pragma unroll
            for (int s = 0; s < kX; ++s)
                o[s * (kStateWords / 4) + (warp * 4 + kk) * 32 + lane] = make_uint4(w0[s], w1[s], w2[s], w3[s]);
        }
    }
    if (threadIdx.x == 0)
        for (int s = gave_up; s < last && s < gave_up + 2; ++s) sm100::mbar_wait(bar + (s & 1), s >> 1 & 1, a.limit / 64);
}

// ---- pieces of kernel 2 ----------------------------------------------------------------------------------------
// Eight warps.  Token-by-token matrices (pairs inside the chunk) are formed by warp (block, dir): the block's rows against
// itself and everything earlier (dir 0) or later (dir 1).  Results with channel columns are formed by warp (slice, half):
// 16 channels, 32 tokens, both directions, so that a warp reads only its slice of the states and planes.
// Table tab holds the inclusive sums of l over each block (row = token).

// x (16 x 64, A layout) of a row range of a tensor
template <typename T, bool kRound>
__device__ __forceinline__ void load_block(Block& x, const T* p, int C, int rows, int g, int q) {
    Raw<T> raw;
    raw.load(p, C, rows, g, q);
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
            float t[4];
            raw.get(half, kk, t);
            round4<kRound>(t);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[half][kk][e] = t[e];
        }
}
// Exponent of a row's factor towards the partners' side: dir 0: sum before the row (to the block's left edge), dir 1:
// sum after it (right edge); minus the block's whole sum when `inner` (the operand then meets the block's own partners,
// whose planes are scaled to the far edge).
__device__ __forceinline__ void row_exponents(const Table& tab, int blk, int row, int dir, bool inner, int kk, int q, float (&x)[4]) {
    float total[4] = {0.f, 0.f, 0.f, 0.f};
    if ((dir == 0) == inner) row4(tab[blk * kBlock + kBlock - 1], kk, q, total);
    if (dir == 0) {
        if (row == 0) {
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] = 0.f - total[e];
        } else {
            row4(tab[blk * kBlock + row - 1], kk, q, x);
#pragma unroll
            for (int e = 0; e < 4; ++e) x[e] -= total[e];
        }
    } else {
        row4(tab[blk * kBlock + row], kk, q, x);
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = total[e] - x[e];
    }
}
// columns times 2^(sum over block j)
__device__ __forceinline__ void cross_block(Block& x, const Table& tab, int j, int q) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        float f[4];
        row4(tab[j * kBlock + kBlock - 1], kk, q, f);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float d = ex2(f[e]);
            x[0][kk][e] *= d;
            x[1][kk][e] *= d;
        }
    }
}
__device__ __forceinline__ bool block_is_safe(const Table& tab, int blk, int lane) {
    const float2 t = *reinterpret_cast<const float2*>(&tab[blk * kBlock + kBlock - 1][2 * lane]);
    return !__any_sync(0xffffffffu, !(t.x > -kSafe && t.y > -kSafe));
}

// row and column of C-fragment element (nt, i) inside the block
__device__ __forceinline__ int frag_row(int i, int g) { return g + 8 * (i >> 1); }
__device__ __forceinline__ int frag_col(int nt, int i, int q) { return 8 * nt + 2 * q + (i & 1); }

// Levels of halves for a block whose decay is too strong for factors above 1: at half size hs a token is scaled towards
// the boundary between the two halves of its 2 hs tokens, the same factor whichever role it plays.
__device__ __forceinline__ void level_factors(const Table& tab, int blk, int hs, int row, int kk, int q, float (&f)[4]) {
    const int mid = (row & ~(2 * hs - 1)) + hs;          // first row behind the boundary
    float b[4], x[4];
    row4(tab[blk * kBlock + mid - 1], kk, q, b);
    const bool later = row >= mid;
    row4(tab[blk * kBlock + (later ? row - 1 : row)], kk, q, x);
#pragma unroll
    for (int e = 0; e < 4; ++e) f[e] = ex2(later ? x[e] - b[e] : b[e] - x[e]);
}
__device__ __forceinline__ bool on_level(int t, int s, int hs) { return (t / (2 * hs)) == (s / (2 * hs)) && ((t & hs) != (s & hs)); }
template <int NS>
__device__ __forceinline__ void level_frag(AFrag<NS>& o, const Block& x, const Table& tab, int blk, int hs, int g, int q) {
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        float f0[4], f1[4];
        level_factors(tab, blk, hs, g, kk, q, f0);
        level_factors(tab, blk, hs, g + 8, kk, q, f1);
#pragma unroll
        for (int e = 0; e < 4; ++e) { f0[e] *= x[0][kk][e]; f1[e] *= x[1][kk][e]; }
        o.set(kk, f0, f1);
    }
}
// p[row][col] = sum_i a_row[i] b_col[i] D(row, col)[i] for all pairs of the block (both directions)
template <int NS>
__device__ __noinline__ void strong_pairs(float (&p)[2][4], const Block& a, const Block& b, const Table& tab, int blk, int g, int q) {
#pragma unroll 1
    for (int hs = 8; hs >= 1; hs >>= 1) {
        AFrag<NS> A, Bf;
        level_frag<NS>(A, a, tab, blk, hs, g, q);
        level_frag<NS>(Bf, b, tab, blk, hs, g, q);
        float c[2][4] = {};
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int ib = 0; ib < NS; ++ib)
#pragma unroll
                for (int ia = 0; ia < NS; ++ia)
                    if (Keep<NS, NS>::on(ia, ib)) {      // a block's B fragments are its A fragments, half by half
                        mma(c[0], A.w[ia][kk], Bf.w[ib][kk][0], Bf.w[ib][kk][2]);
                        mma(c[1], A.w[ia][kk], Bf.w[ib][kk][1], Bf.w[ib][kk][3]);
                    }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (on_level(frag_row(i, g), frag_col(nt, i, q), hs)) p[nt][i] = c[nt][i];
    }
}
// out[row half][e] += sum_s m[t][s] D(t, s) (x) x_s over the pairs of block blk on one side (dir 0: s earlier), for the 16
// channels of slice cs; m: the whole matrix (planes of NS parts, transposed if kTransM), x: the block's rows of the partner
template <typename T, int NS, bool kTransM, bool kRound>
__device__ __noinline__ void strong_gradients(float (&out)[2][4], const __nv_bfloat16* m, const T* x, int C, int rows, const Table& tab,
                                              int blk, int cs, int dir, int lane) {
    const int g = lane >> 2, q = lane & 3;
    uint32_t a[NS][4];
#pragma unroll
    for (int ia = 0; ia < NS; ++ia) {
        if (kTransM) ldsm4t(a[ia], smem_addr(m + ia * kPlane + blk * kBlock * kRow + blk * kBlock + off_tok(lane)));
        else ldsm4(a[ia], smem_addr(m + ia * kPlane + blk * kBlock * kRow + blk * kBlock + off_a(lane)));
    }
    float xv[2][4];
#pragma unroll
    for (int half = 0; half < 2; ++half) {
#pragma unroll
        for (int e = 0; e < 4; ++e) xv[half][e] = 0.f;
        if (g + 8 * half < rows) load4(x + static_cast<size_t>(g + 8 * half) * C + 16 * cs + 4 * q, xv[half]);
        round4<kRound>(xv[half]);
    }
#pragma unroll 1
    for (int hs = 8; hs >= 1; hs >>= 1) {
        float f[2][4], c[2][4] = {};
        level_factors(tab, blk, hs, g, cs, q, f[0]);
        level_factors(tab, blk, hs, g + 8, cs, q, f[1]);
        // fragment words of m: word i holds row g (+ 8 for odd i), columns 2 q, 2 q + 1 (+ 8 for i >= 2)
        uint32_t am[NS][4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = g + 8 * (i & 1), col = 2 * q + 8 * (i >> 1);
            uint32_t keep = 0u;
            if (on_level(row, col, hs) && (dir == 0 ? col < row : col > row)) keep |= 0x0000ffffu;
            if (on_level(row, col + 1, hs) && (dir == 0 ? col + 1 < row : col + 1 > row)) keep |= 0xffff0000u;
#pragma unroll
            for (int ia = 0; ia < NS; ++ia) am[ia][i] = a[ia][i] & keep;
        }
        uint32_t w0[NS], w1[NS], w2[NS], w3[NS];
        split<NS>(xv[0][0] * f[0][0], xv[0][1] * f[0][1], w0);
        split<NS>(xv[1][0] * f[1][0], xv[1][1] * f[1][1], w1);
        split<NS>(xv[0][2] * f[0][2], xv[0][3] * f[0][3], w2);
        split<NS>(xv[1][2] * f[1][2], xv[1][3] * f[1][3], w3);
#pragma unroll
        for (int ib = 0; ib < NS; ++ib) {
            const uint32_t b0 = movm_trans(w0[ib]), b1 = movm_trans(w1[ib]), b2 = movm_trans(w2[ib]), b3 = movm_trans(w3[ib]);
#pragma unroll
            for (int ia = 0; ia < NS; ++ia)
                if (Keep<NS, NS>::on(ia, ib)) {
                    mma(c[0], am[ia], b0, b1);
                    mma(c[1], am[ia], b2, b3);
                }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int e = 0; e < 4; ++e) out[half][e] = fmaf(f[half][e], c[e >> 1][half * 2 + (e & 1)], out[half][e]);
    }
}
__device__ __forceinline__ void copy(Block& to, const Block& from) {
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int e = 0; e < 4; ++e) to[half][kk][e] = from[half][kk][e];
}

// sum over this thread's quad of x . u . y per row
__device__ __forceinline__ void bonus_terms(const Block& x, const Block& y, const float* u, int q, float (&out)[2]) {
    out[0] = out[1] = 0.f;
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
        float uu[4];
        row4(u, kk, q, uu);
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int e = 0; e < 4; ++e) out[half] += x[half][kk][e] * uu[e] * y[half][kk][e];
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        out[half] += __shfl_xor_sync(0xffffffffu, out[half], 1);
        out[half] += __shfl_xor_sync(0xffffffffu, out[half], 2);
    }
}
// sums of l over a block's tokens into the table (a warp per block, lane = two channels)
__device__ __forceinline__ void scan_block(Table& tab, const float* w, int C, int rows, int blk, int lane) {
    Pair<float> wr[kBlock];
#pragma unroll
    for (int t = 0; t < kBlock; ++t) wr[t].load(w + static_cast<size_t>(t) * C + 2 * lane, t < rows);
    float2 run = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        run.x += log2_decay(wr[t].v.x, t < rows);
        run.y += log2_decay(wr[t].v.y, t < rows);
        *reinterpret_cast<float2*>(&tab[blk * kBlock + t][2 * lane]) = run;
    }
}
// a block's rows as they are, into planes
template <typename T, int NS, bool kRound>
__device__ __forceinline__ void stage_rows(__nv_bfloat16* planes, const T* p, int C, int rows, int blk, int lane) {
    Pair<T> x[kBlock];
#pragma unroll
    for (int t = 0; t < kBlock; ++t) x[t].load(p + static_cast<size_t>(t) * C + 2 * lane, t < rows);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        const float2 v = round2<kRound>(x[t].get());
        col_store<NS>(planes, blk * kBlock + t, col_word(lane), v.x, v.y);
    }
}
template <typename T>
__device__ __forceinline__ void load_rows(Pair<T> (&x)[kBlock], const T* p, int C, int rows, int lane) {
#pragma unroll
    for (int t = 0; t < kBlock; ++t) x[t].load(p + static_cast<size_t>(t) * C + 2 * lane, t < rows);
}
// a block's rows scaled to its right edge (for partners later than it: dir 0) or left edge (dir 1), into planes
template <typename T, int NS, bool kRound>
__device__ __forceinline__ void stage_scaled(__nv_bfloat16* planes, const Pair<T> (&x)[kBlock], const Table& tab, int blk, int dir, int lane) {
    const float2 total = *reinterpret_cast<const float2*>(&tab[blk * kBlock + kBlock - 1][2 * lane]);
    float2 prev = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        const float2 v = round2<kRound>(x[t].get());
        const float2 s = *reinterpret_cast<const float2*>(&tab[blk * kBlock + t][2 * lane]);
        const float ex = dir == 0 ? total.x - s.x : prev.x, ey = dir == 0 ? total.y - s.y : prev.y;
        col_store<NS>(planes, blk * kBlock + t, col_word(lane), v.x * ex2(ex), v.y * ex2(ey));
        prev = s;
    }
}
// a 16 x 16 tile (C fragments) into planes of 64 x 64 token-by-token parts
template <int NS>
__device__ __forceinline__ void store_tile(__nv_bfloat16* planes, const float (&m)[2][4], int mrow, int mcol, int g, int q) {
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            uint32_t t[NS];
            split<NS>(m[nt][2 * half], m[nt][2 * half + 1], t);
#pragma unroll
            for (int s = 0; s < NS; ++s)
                *reinterpret_cast<uint32_t*>(planes + s * kPlane + (mrow * kBlock + g + 8 * half) * kRow + mcol * kBlock + 8 * nt + 2 * q) = t[s];
        }
}

// ---- inputs kept in shared memory: 64 rows of 128 bytes (64 bfloat16), 16-byte pieces exchanged by the row's number as the copy engine's
// 128-byte swizzle has them.  A row's four channels 4 q .. of 16 kk: rows g of a warp's eight meet each bank twice, the least for 256 bytes.
__device__ __forceinline__ uint2 raw4(const unsigned char* tile, int row, int kk, int q) {
    return *reinterpret_cast<const uint2*>(tile + row * 128 + (((2 * kk + (q >> 1)) ^ (row & 7)) << 4) + (q & 1) * 8);
}
__device__ __forceinline__ void load4(const unsigned char* tile, int row, int kk, int q, float (&x)[4]) {
    const uint2 v = raw4(tile, row, kk, q);
    x[0] = lo_f(v.x); x[1] = hi_f(v.x); x[2] = lo_f(v.y); x[3] = hi_f(v.y);
}
__device__ __forceinline__ uint32_t raw_word(int row, int lane) { return row * 128 + (((lane >> 2) ^ (row & 7)) << 4) + ((lane & 3) << 2); }
__device__ __forceinline__ void load_block(Block& x, const unsigned char* tile, int blk, int g, int q) {
#pragma unroll
    for (int half = 0; half < 2; ++half)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) load4(tile, blk * kBlock + g + 8 * half, kk, q, x[half][kk]);
}
// a block's rows scaled to its right edge (for partners later than it: dir 0) or left edge (dir 1), into planes
template <int NS>
__device__ __forceinline__ void stage_scaled(__nv_bfloat16* planes, const unsigned char* tile, const Table& tab, int blk, int dir, int lane) {
    const float2 total = *reinterpret_cast<const float2*>(&tab[blk * kBlock + kBlock - 1][2 * lane]);
    float2 prev = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        const uint32_t v = *reinterpret_cast<const uint32_t*>(tile + raw_word(blk * kBlock + t, lane));
        const float2 s = *reinterpret_cast<const float2*>(&tab[blk * kBlock + t][2 * lane]);
        const float ex = dir == 0 ? total.x - s.x : prev.x, ey = dir == 0 ? total.y - s.y : prev.y;
        col_store<NS>(planes, blk * kBlock + t, col_word(lane), lo_f(v) * ex2(ex), hi_f(v) * ex2(ey));
        prev = s;
    }
}
// a block of a tile as the copy engine left it (row after row), into a plane, rounded
__device__ __forceinline__ void stage_tile(__nv_bfloat16* plane, const __nv_bfloat16* tile, int blk, int lane) {
#pragma unroll
    for (int t = 0; t < kBlock; ++t)
        *reinterpret_cast<uint32_t*>(plane + (blk * kBlock + t) * kRow + 2 * col_word(lane)) = half_pair(tile + (blk * kBlock + t) * N, lane);
}
__device__ __forceinline__ void stage_tile(__nv_bfloat16* plane, const float* tile, int blk, int lane) {
#pragma unroll
    for (int t = 0; t < kBlock; ++t)
        *reinterpret_cast<uint32_t*>(plane + (blk * kBlock + t) * kRow + 2 * col_word(lane)) = half_pair(tile + (blk * kBlock + t) * N, lane);
}
// a block's rows into such a tile, rounded
template <typename T>
__device__ __forceinline__ void keep_rows(unsigned char* tile, const T* p, int C, int rows, int blk, int lane) {
    Pair<T> x[kBlock];
    load_rows<T>(x, p, C, rows, lane);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        uint32_t w[1];
        const float2 v = x[t].get();
        split<1>(v.x, v.y, w);
        *reinterpret_cast<uint32_t*>(tile + raw_word(blk * kBlock + t, lane)) = w[0];
    }
}
__device__ __forceinline__ void scan_tile(Table& tab, const float* tile, int rows, int blk, int lane) {
    float2 run = make_float2(0.f, 0.f);
#pragma unroll
    for (int t = 0; t < kBlock; ++t) {
        const float2 w = *reinterpret_cast<const float2*>(tile + (blk * kBlock + t) * N + 2 * lane);
        run.x += log2_decay(w.x, t < rows);
        run.y += log2_decay(w.y, t < rows);
        *reinterpret_cast<float2*>(&tab[blk * kBlock + t][2 * lane]) = run;
    }
}

// Row-mapped part of y (rows r, columns k) and gv (rows k, columns r): warp (blk, dir) forms its pairs of the token matrix
// and leaves the rows scaled to the chunk's edge (for the entering state) in the planes `edges`.  The two directions of
// a diagonal tile are merged by the masks: dir 0 writes below the diagonal and on it, dir 1 above.
template <int kX, typename RowsOf, typename ColsOf>
__device__ __forceinline__ void pair_rows(RowsOf&& rows_of, ColsOf&& cols_of, const float* u, const Table& tab, const __nv_bfloat16* planes,
                                          __nv_bfloat16* pairs, __nv_bfloat16* edges, int blk, int dir, int lane) {
    const int g = lane >> 2, q = lane & 3;
    const bool safe = block_is_safe(tab, blk, lane);
    Block x;
    rows_of(x);
    AFrag<kX> f;
    {
        float p[2][4] = {}, diag[2] = {0.f, 0.f};
        if (dir == 0 || !safe) {
            Block c;
            cols_of(c);
            if (dir == 0) bonus_terms(x, c, u, q, diag);
            if (!safe) {
                // copies: what a call takes by reference lives in memory, and x stays in registers
                Block xc, cc;
                float pc[2][4] = {};
                copy(xc, x);
                copy(cc, c);
                strong_pairs<kX>(pc, xc, cc, tab, blk, g, q);
#pragma unroll
                for (int i = 0; i < 8; ++i) p[i >> 2][i & 3] = pc[i >> 2][i & 3];
            }
        }
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float e4[4];
                row_exponents(tab, blk, g + 8 * half, dir, safe, kk, q, e4);
#pragma unroll
                for (int e = 0; e < 4; ++e) x[half][kk][e] *= ex2(e4[e]);
            }
        if (safe) {
            f.set(x);
            prod_tokens<kX, kX>(p, f, planes, blk, lane);
            cross_block(x, tab, blk, q);
        }
        // merge with the other direction's half of the tile
#pragma unroll
        for (int nt = 0; nt < 2; ++nt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int row = g + 8 * half, col = 8 * nt + 2 * q;
                if (dir == 0) {
                    if (col == row) p[nt][2 * half] = diag[half];
                    if (col + 1 == row) p[nt][2 * half + 1] = diag[half];
                }
                const bool on0 = dir == 0 ? col <= row : col > row, on1 = dir == 0 ? col + 1 <= row : col + 1 > row;
                uint32_t t[kX];
                split<kX>(p[nt][2 * half], p[nt][2 * half + 1], t);
#pragma unroll
                for (int s = 0; s < kX; ++s) {
                    __nv_bfloat16* d = pairs + s * kPlane + (blk * kBlock + row) * kRow + blk * kBlock + col;
                    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(&t[s]);
                    if (on0 && on1) *reinterpret_cast<uint32_t*>(d) = t[s];
                    else if (on0) d[0] = v.x;
                    else if (on1) d[1] = v.y;
                }
            }
    }
#pragma unroll 1
    for (int j = dir == 0 ? blk - 1 : blk + 1; j >= 0 && j < kBlocks; j += dir == 0 ? -1 : 1) {
        f.set(x);
        float p[2][4] = {};
        prod_tokens<kX, kX>(p, f, planes, j, lane);
        store_tile<kX>(pairs, p, blk, j, g, q);
        cross_block(x, tab, j, q);
    }
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            __nv_bfloat16* d = edges + (blk * kBlock + g + 8 * half) * kRow + 16 * kk + 2 * q;
            uint32_t t[kX];
            split<kX>(x[half][kk][0], x[half][kk][1], t);
#pragma unroll
            for (int s = 0; s < kX; ++s) *reinterpret_cast<uint32_t*>(d + s * kPlane) = t[s];
            split<kX>(x[half][kk][2], x[half][kk][3], t);
#pragma unroll
            for (int s = 0; s < kX; ++s) *reinterpret_cast<uint32_t*>(d + s * kPlane + 8) = t[s];
        }
}
// Slice-mapped part: y[32 tokens x 16 channels] = pairs * values + edge-scaled rows * entering states
template <int kZ, int kX, bool kTrans>
__device__ __forceinline__ void pair_outputs(float (&y)[2][2][4], const __nv_bfloat16* pairs, const __nv_bfloat16* values,
                                             const __nv_bfloat16* edges_left, const __nv_bfloat16* edges_right, const uint4* from_left,
                                             const uint4* from_right, int cs, int th, int lane) {
#pragma unroll
    for (int i = 0; i < 16; ++i) y[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const uint4* st = dir ? from_right : from_left;
        if (st == nullptr) continue;
        const __nv_bfloat16* ed = dir ? edges_right : edges_left;
        uint32_t f[4][kX][4];
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) state_frag<kX, kTrans>(f[kk], st, cs, kk, lane);
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int m = 0; m < 2; ++m)
#pragma unroll
                for (int ia = 0; ia < kX; ++ia) {
                    uint32_t a[4];
                    ldsm4(a, smem_addr(ed + ia * kPlane + (2 * th + m) * kBlock * kRow + 16 * kk + off_a(lane)));
#pragma unroll
                    for (int ib = 0; ib < kX; ++ib)
                        if (Keep<kX, kX>::on(ia, ib)) {
                            mma(y[m][0], a, f[kk][ib][0], f[kk][ib][1]);
                            mma(y[m][1], a, f[kk][ib][2], f[kk][ib][3]);
                        }
                }
    }
#pragma unroll
    for (int b = 0; b < kBlocks; ++b) {
        uint32_t r[kZ][4];      // the values of block b, for both tiles
#pragma unroll
        for (int ib = 0; ib < kZ; ++ib) ldsm4t(r[ib], smem_addr(values + ib * kPlane + b * kBlock * kRow + cs * 16 + off_pos(lane)));
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int ia = 0; ia < kX; ++ia) {
                uint32_t a[4];
                ldsm4(a, smem_addr(pairs + ia * kPlane + (2 * th + m) * kBlock * kRow + b * kBlock + off_a(lane)));
#pragma unroll
                for (int ib = 0; ib < kZ; ++ib)
                    if (Keep<kX, kZ>::on(ia, ib)) {
                        mma(y[m][0], a, r[ib][0], r[ib][1]);
                        mma(y[m][1], a, r[ib][2], r[ib][3]);
                    }
            }
    }
}

// ---- kernel 2 ------------------------------------------------------------------------------------------------
// What bounds it: three or two CTAs of eight warps on an SM (shared memory and registers), each waiting for its own results and its own loads.  Inputs
// come in one set of TMA copies into places that planes take later (B=32, H=12, T=4096, forward / backward us: 661 -> 615 and, where k and r
// also stay, 2302 -> 2060; T=196 47.0 -> 43.1, 155 -> 145).  Each CTA brings the inputs of the one that starts a little later (half
// an SM count of CTAs: before that CTA has started, and so shortly that nothing is evicted) into L2: without that 707 / 2143 where 661 / 2055,
// at a distance of an SM count 667 / 2089.  Tried in the backward: the edge's products while the tiles are under way 2081, states asked for
// a barrier early 2211 (spills).
// The rows of a head's chunk (all 256 threads share the lines):
template <typename T>
__device__ __forceinline__ void prefetch_rows(const T* p, int C, int rows) {
    constexpr int kLines = N * sizeof(T) / 128;
    for (int i = threadIdx.x; i < kChunk * kLines; i += 256)
        if (i / kLines < rows) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(p + static_cast<size_t>(i / kLines) * C) + (i % kLines) * 128));
}
__device__ __forceinline__ void prefetch_bytes(const void* p, int bytes) {
    for (int i = threadIdx.x * 128; i < bytes; i += 256 * 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(p) + i));
}

constexpr uint32_t kRawTile = kChunk * N * 2;


// ---- kernel 2, forward ---------------------------------------------------------------------------------------
struct OutArgs {
    int T, H, n_chunks;
    unsigned ahead;           // CTAs between this one and the one whose inputs it brings into L2
    const void* r;
    const void* k;
    const void* v;
    const float* w;
    const float* u;
    float* y;
    bool scalar;              // y is not 16-byte aligned: 4-byte stores
    const uint4* states;      // [direction][b h][chunk][part][..], rows = value channels
    size_t plane;
    unsigned* status;         // as in StateArgs
    unsigned* mirror;
    unsigned limit;
    unsigned extra;
};

// kX parts of the scaled operands and states, kZ parts of v
template <typename T, int kZ, int kX>
__global__ void __launch_bounds__(256, 3)
wkv6_forward_kernel(const OutArgs a, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mr,
                    const __grid_constant__ CUtensorMap mv) {
    wait_for_launch_before();
    extern __shared__ __align__(1024) unsigned char smem[];
    __nv_bfloat16* kf = reinterpret_cast<__nv_bfloat16*>(smem);       // k towards the right edge of its block, left edge behind it
    __nv_bfloat16* pairs = kf + 2 * kX * kPlane;
    __nv_bfloat16* edges = pairs + kX * kPlane;
    __nv_bfloat16* vs = edges + 2 * kX * kPlane;
    Table& tab = *reinterpret_cast<Table*>(vs + kZ * kPlane);
    // tiles on their way (bfloat16 inputs, by TMA): v and r where k's planes will be, k where the pairs, w where the edges
    uint64_t* bar = reinterpret_cast<uint64_t*>(&tab + 1);
    unsigned char *const v_raw = smem, *const r_raw = smem + kRawTile, *const k_raw = reinterpret_cast<unsigned char*>(pairs),
                  *const w_raw = reinterpret_cast<unsigned char*>(edges);
    static_assert(2 * kPlane * 2 >= 2 * kRawTile && 2 * kPlane * 2 >= kChunk * N * 4 && 2 * kPlane * 2 % 1024 == 0, "room for the tiles");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int n = blockIdx.x % a.n_chunks, bh = blockIdx.x / a.n_chunks;
    const int b = bh / a.H, h = bh - b * a.H, C = a.H * N;
    const size_t base = (static_cast<size_t>(b) * a.T + n * kChunk) * C + static_cast<size_t>(h) * N;
    constexpr bool kRound = sizeof(T) == 4;
    if (sizeof(T) == 2) {
        if (threadIdx.x == 0) {
            sm100::mbar_init(bar, 1);
            sm100::mbar_init_fence();
            sm100::mbar_expect_tx(bar, 3 * kRawTile + kChunk * N * 4 + a.extra);
            sm100::tma_load_3d(w_raw, &mw, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(v_raw, &mv, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(r_raw, &mr, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(k_raw, &mk, bar, h * N, n * kChunk, b);
        }
        __syncthreads();
    }
    if (blockIdx.x + a.ahead < gridDim.x) {
        const int id = blockIdx.x + a.ahead, n2 = id % a.n_chunks, bh2 = id / a.n_chunks, b2 = bh2 / a.H, rows = a.T - n2 * kChunk;
        const size_t at = (static_cast<size_t>(b2) * a.T + n2 * kChunk) * C + static_cast<size_t>(bh2 - b2 * a.H) * N;
        prefetch_rows(static_cast<const T*>(a.k) + at, C, rows);
        prefetch_rows(a.w + at, C, rows);
        prefetch_rows(static_cast<const T*>(a.v) + at, C, rows);
        prefetch_rows(static_cast<const T*>(a.r) + at, C, rows);
        const uint4* st = a.states + static_cast<size_t>(id) * (kX * kStateWords / 4);
        if (n2 > 0) prefetch_bytes(st, kX * kStateWords * 4);
        if (n2 + 1 < a.n_chunks) prefetch_bytes(st + a.plane, kX * kStateWords * 4);
    }
    {
        const int blk = warp & 3, dir = warp >> 2;
        const int rows = a.T - (n * kChunk + blk * kBlock);
        const size_t at0 = base + static_cast<size_t>(blk) * kBlock * C;
        const T* k = static_cast<const T*>(a.k) + at0;
        const T* r = static_cast<const T*>(a.r) + at0;
        __nv_bfloat16* planes = kf + dir * kX * kPlane;
        __nv_bfloat16* mine = edges + dir * kX * kPlane;
        if constexpr (sizeof(T) == 2) {
            if (!sm100::mbar_wait(bar, 0, a.limit)) report_failure(a.status, a.mirror, 2u);
            uint2 rr[2][4], kr[2][4];      // this thread's part of the block, out of the tiles before planes and pairs take their place
#pragma unroll
            for (int i = 0; i < 8; ++i) rr[i >> 2][i & 3] = raw4(r_raw, blk * kBlock + g + 8 * (i >> 2), i & 3, q);
            if (dir == 0) scan_tile(tab, reinterpret_cast<const float*>(w_raw), rows, blk, lane);
            else stage_tile(vs, reinterpret_cast<const __nv_bfloat16*>(v_raw), blk, lane);
            __syncthreads();
            stage_scaled<kX>(planes, k_raw, tab, blk, dir, lane);
#pragma unroll
            for (int i = 0; i < 8; ++i) kr[i >> 2][i & 3] = raw4(k_raw, blk * kBlock + g + 8 * (i >> 2), i & 3, q);
            __syncthreads();
            const auto widen = [](Block& x, const uint2(&raw)[2][4]) {
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint2 v = raw[i >> 2][i & 3];
                    float(&e)[4] = x[i >> 2][i & 3];
                    e[0] = lo_f(v.x); e[1] = hi_f(v.x); e[2] = lo_f(v.y); e[3] = hi_f(v.y);
                }
            };
            pair_rows<kX>([&](Block& x) { widen(x, rr); }, [&](Block& x) { widen(x, kr); }, a.u + h * N, tab, planes, pairs, mine, blk, dir, lane);
        } else {
            Pair<T> kr[kBlock];
            load_rows<T>(kr, k, C, rows, lane);
            if (dir == 0) scan_block(tab, a.w + at0, C, rows, blk, lane);
            else stage_rows<T, kZ, kRound>(vs, static_cast<const T*>(a.v) + at0, C, rows, blk, lane);
            __syncthreads();
            stage_scaled<T, kX, kRound>(planes, kr, tab, blk, dir, lane);
            __syncthreads();
            pair_rows<kX>([&](Block& x) { load_block<T, kRound>(x, r, C, rows, g, q); }, [&](Block& x) { load_block<T, kRound>(x, k, C, rows, g, q); }, a.u + h * N,
                          tab, planes, pairs, mine, blk, dir, lane);
        }
    }
    __syncthreads();
    const int cs = warp & 3, th = warp >> 2;
    const uint4* st = a.states + (static_cast<size_t>(bh) * a.n_chunks + n) * (kX * kStateWords / 4);
    float y[2][2][4];
    pair_outputs<kZ, kX, false>(y, pairs, vs, edges, edges + kX * kPlane, n > 0 ? st : nullptr, n + 1 < a.n_chunks ? st + a.plane : nullptr, cs, th, lane);
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int t = 32 * th + 16 * m + 8 * half + g;
            if (n * kChunk + t < a.T)
                put4(a.scalar, a.y + base + static_cast<size_t>(t) * C + 16 * cs + 4 * q, y[m][0][2 * half], y[m][0][2 * half + 1],
                     y[m][1][2 * half], y[m][1][2 * half + 1]);
        }
    // after a wait that gave up (here and not behind it: there the second loop cost 1.5 % of the forward)
    if (sizeof(T) == 2 && threadIdx.x == 0) sm100::mbar_wait(bar, 0, a.limit / 64);
}

// ---- kernel 2, backward --------------------------------------------------------------------------------------
struct GradArgs {
    int T, H, n_chunks;
    unsigned ahead;           // as in OutArgs
    const void* r;
    const void* k;
    const void* v;
    const void* gy;
    const float* w;
    const float* u;
    void* gr;
    void* gk;
    void* gv;
    float* gw;
    float* gu_part;           // [b][chunk][C]
    bool scalar;              // an output is not 16-byte aligned: element stores
    const uint4* states;      // [pair][direction][b h][chunk][part][..], rows = channels of r, k
    size_t plane;
    unsigned* status;         // as in StateArgs
    unsigned* mirror;
    unsigned limit;
    unsigned extra;
};


// gr (own = gy, partners k, m = gy v^T) or gk (own = v, partners r, m transposed) for 32 tokens x 16 channels:
//   early / late[m tile][row half][e] = sum over earlier / later tokens s of (own_t . other_s) D(t, s) (x) partner_s,
// from the entering state inward: every block the sum crosses decays it, the block's own pairs come last.
template <typename T, int kZ, int kX, bool kTransM, bool kRound>
__device__ __forceinline__ void slice_gradient(float (&out)[2][2][2][4], const __nv_bfloat16* own, const __nv_bfloat16* m, const __nv_bfloat16* planes,
                                               const uint4* from_left, const uint4* from_right, const Table& tab, const T* partner, int C,
                                               int rows, unsigned strong, int cs, int th, int lane) {
    const int g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        float c[2][2][4];
#pragma unroll
        for (int i = 0; i < 16; ++i) c[i >> 3][(i >> 2) & 1][i & 3] = 0.f;
        const uint4* st = dir ? from_right : from_left;
        if (st != nullptr) {
            uint32_t f[4][kX][4];
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) state_frag<kX, false>(f[kk], st, cs, kk, lane);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
#pragma unroll
                    for (int ia = 0; ia < kZ; ++ia) {
                        uint32_t a[4];
                        ldsm4(a, smem_addr(own + ia * kPlane + (2 * th + mt) * kBlock * kRow + 16 * kk + off_a(lane)));
#pragma unroll
                        for (int ib = 0; ib < kX; ++ib)
                            if (Keep<kZ, kX>::on(ia, ib)) {
                                mma(c[mt][0], a, f[kk][ib][0], f[kk][ib][1]);
                                mma(c[mt][1], a, f[kk][ib][2], f[kk][ib][3]);
                            }
                    }
        }
        const __nv_bfloat16* pl = planes + dir * kX * kPlane;
#pragma unroll
        for (int step = 0; step < kBlocks; ++step) {
            const int j = dir == 0 ? step : kBlocks - 1 - step;
            if (dir == 0 ? j > 2 * th + 1 : j < 2 * th) continue;            // beyond both tiles of this warp
            float d[4];
            row4(tab[j * kBlock + kBlock - 1], cs, q, d);
#pragma unroll
            for (int e = 0; e < 4; ++e) d[e] = ex2(d[e]);
            // the partners' rows of block j, for both tiles of this warp: read per tile the backward was 157.3 us, now 154.6
            // (B=32, H=12, T=196; T=4096 2316 and 2304)
            uint32_t r[kX][4];
#pragma unroll
            for (int ib = 0; ib < kX; ++ib) ldsm4t(r[ib], smem_addr(pl + ib * kPlane + j * kBlock * kRow + cs * 16 + off_pos(lane)));
#pragma unroll
            for (int mt = 0; mt < 2; ++mt) {
                const int blk = 2 * th + mt;
                if (dir == 0 ? j > blk : j < blk) continue;
                if (j == blk && ((strong >> blk) & 1u)) continue;
#pragma unroll
                for (int half = 0; half < 2; ++half)
#pragma unroll
                    for (int e = 0; e < 4; ++e) c[mt][e >> 1][2 * half + (e & 1)] *= d[e];
                uint32_t a[kX][4];
#pragma unroll
                for (int ia = 0; ia < kX; ++ia) {
                    if (kTransM) ldsm4t(a[ia], smem_addr(m + ia * kPlane + j * kBlock * kRow + blk * kBlock + off_tok(lane)));
                    else ldsm4(a[ia], smem_addr(m + ia * kPlane + blk * kBlock * kRow + j * kBlock + off_a(lane)));
                    if (j == blk) {
                        // the block's own tile, masked to this direction
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int row = g + 8 * (i & 1), col = 2 * q + 8 * (i >> 1);
                            const uint32_t keep = ((dir == 0 ? col < row : col > row) ? 0x0000ffffu : 0u) |
                                                  ((dir == 0 ? col + 1 < row : col + 1 > row) ? 0xffff0000u : 0u);
                            a[ia][i] &= keep;
                        }
                    }
                }
#pragma unroll
                for (int ib = 0; ib < kX; ++ib)
#pragma unroll
                    for (int ia = 0; ia < kX; ++ia)
                        if (Keep<kX, kX>::on(ia, ib)) {
                            mma(c[mt][0], a[ia], r[ib][0], r[ib][1]);
                            mma(c[mt][1], a[ia], r[ib][2], r[ib][3]);
                        }
            }
        }
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const int blk = 2 * th + mt;
            const bool safe = ((strong >> blk) & 1u) == 0u;
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                float f[4];
                row_exponents(tab, blk, g + 8 * half, dir, safe, cs, q, f);
#pragma unroll
                for (int e = 0; e < 4; ++e) out[dir][mt][half][e] = ex2(f[e]) * c[mt][e >> 1][2 * half + (e & 1)];
            }
            if (!safe) {
                float o[2][4];
#pragma unroll
                for (int i = 0; i < 8; ++i) o[i >> 2][i & 3] = out[dir][mt][i >> 2][i & 3];
                strong_gradients<T, kX, kTransM, kRound>(o, m, partner + static_cast<size_t>(blk) * kBlock * C, C, rows - blk * kBlock, tab, blk, cs,
                                                         dir, lane);
#pragma unroll
                for (int i = 0; i < 8; ++i) out[dir][mt][i >> 2][i & 3] = o[i >> 2][i & 3];
            }
        }
    }
}

// kZ parts of v, gy; kX parts of scaled operands, token products and states; kP parts where only gv is concerned
template <typename T, typename G, typename O, int kZ, int kX, int kP>
__global__ void __launch_bounds__(256, 2) wkv6_backward_kernel(const GradArgs a, const __grid_constant__ CUtensorMap mw, const __grid_constant__ CUtensorMap mk, const __grid_constant__ CUtensorMap mr,
                     const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mg) {
    wait_for_launch_before();
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* const k_raw = smem;               // k and r stay, as bfloat16
    unsigned char* const r_raw = smem + kRawTile;
    __nv_bfloat16* vs = reinterpret_cast<__nv_bfloat16*>(smem + 2 * kRawTile);
    __nv_bfloat16* gs = vs + kZ * kPlane;
    __nv_bfloat16* pf = gs + kZ * kPlane;        // k, then r, towards the right edge of its block, left edge behind it
    __nv_bfloat16* ms = pf + 2 * kX * kPlane;    // gy v^T inside the chunk, later the pairs of gv
    Table& tab = *reinterpret_cast<Table*>(ms + kX * kPlane);
    float* dots = reinterpret_cast<float*>(&tab + 1);       // [kChunk]: gy_t . v_t
    float* edge = dots + N;                                 // [2][N]
    float* gus = edge + 2 * N;                              // [2][N]
    float* seg = gus + 2 * N;                               // [N]: diff over the later half
    uint64_t* bar = reinterpret_cast<uint64_t*>(seg + N);
    // tiles on their way into planes and table: w where m will be, v and gy where the scaled rows will be
    unsigned char *const w_raw = reinterpret_cast<unsigned char*>(ms), *const v_raw = reinterpret_cast<unsigned char*>(pf), *const g_raw = v_raw + kRawTile;
    static_assert(kX == 2, "room for the tiles");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int blk = warp & 3, dir = warp >> 2;              // row-mapped phases
    const int cs = warp & 3, th = warp >> 2;                // slice-mapped phases
    const int n = blockIdx.x % a.n_chunks, bh = blockIdx.x / a.n_chunks;
    const int b = bh / a.H, h = bh - b * a.H, C = a.H * N;
    // a warp whose tokens lie behind the last one forms no gradients (B=32, T=196, H=12, four tokens in every fourth chunk: 143.5 -> 137.5 us)
    const int tokens = a.T - n * kChunk, rows = tokens - blk * kBlock;
    const size_t base = (static_cast<size_t>(b) * a.T + n * kChunk) * C + static_cast<size_t>(h) * N;
    const size_t at0 = base + static_cast<size_t>(blk) * kBlock * C;
    constexpr bool kRound = sizeof(T) == 4, kRoundG = sizeof(G) == 4;
    constexpr int kState = kX * kStateWords / 4;
    // states entering this chunk, [pair (k v | r gy)][from the left | from the right]
    const uint4* st = a.states + (static_cast<size_t>(bh) * a.n_chunks + n) * kState;
    const bool left = n > 0, right = n + 1 < a.n_chunks;
    const uint4 *s_left = left ? st : nullptr, *s_right = right ? st + a.plane : nullptr;
    const uint4 *a_left = left ? st + 2 * a.plane : nullptr, *a_right = right ? st + 3 * a.plane : nullptr;
    const T* rp = static_cast<const T*>(a.r);
    const T* kp = static_cast<const T*>(a.k);

    if (sizeof(T) == 2) {
        if (threadIdx.x == 0) {
            sm100::mbar_init(bar, 1);
            sm100::mbar_init_fence();
            sm100::mbar_expect_tx(bar, 3 * kRawTile + kChunk * N * (4 + sizeof(G)) + a.extra);
            sm100::tma_load_3d(w_raw, &mw, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(g_raw, &mg, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(v_raw, &mv, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(k_raw, &mk, bar, h * N, n * kChunk, b);
            sm100::tma_load_3d(r_raw, &mr, bar, h * N, n * kChunk, b);
        }
        __syncthreads();
    }
    if (blockIdx.x + a.ahead < gridDim.x) {
        const int id = blockIdx.x + a.ahead, n2 = id % a.n_chunks, bh2 = id / a.n_chunks, b2 = bh2 / a.H, rows2 = a.T - n2 * kChunk;
        const size_t at = (static_cast<size_t>(b2) * a.T + n2 * kChunk) * C + static_cast<size_t>(bh2 - b2 * a.H) * N;
        prefetch_rows(kp + at, C, rows2);
        prefetch_rows(a.w + at, C, rows2);
        prefetch_rows(static_cast<const T*>(a.v) + at, C, rows2);
        prefetch_rows(static_cast<const G*>(a.gy) + at, C, rows2);
        prefetch_rows(rp + at, C, rows2);
        const uint4* st2 = a.states + static_cast<size_t>(id) * kState;
        for (int i = 0; i < 4; ++i)      // from the left, from the right, of either pair
            if ((i & 1) ? n2 + 1 < a.n_chunks : n2 > 0) prefetch_bytes(st2 + i * a.plane, kState * 16);
    }
    if (sizeof(T) == 2) {
        if (!sm100::mbar_wait(bar, 0, a.limit)) report_failure(a.status, a.mirror, 2u);
        if (dir == 0) {
            scan_tile(tab, reinterpret_cast<const float*>(w_raw), rows, blk, lane);
        } else {
            stage_tile(vs, reinterpret_cast<const __nv_bfloat16*>(v_raw), blk, lane);
            stage_tile(gs, reinterpret_cast<const G*>(g_raw), blk, lane);
        }
    } else {
        keep_rows<T>(dir == 0 ? k_raw : r_raw, (dir == 0 ? kp : rp) + at0, C, rows, blk, lane);
        if (dir == 0) {
            scan_block(tab, a.w + at0, C, rows, blk, lane);
        } else {
            stage_rows<T, kZ, kRound>(vs, static_cast<const T*>(a.v) + at0, C, rows, blk, lane);
            stage_rows<G, kZ, kRoundG>(gs, static_cast<const G*>(a.gy) + at0, C, rows, blk, lane);
        }
    }
    __syncthreads();
    stage_scaled<kX>(pf + dir * kX * kPlane, k_raw, tab, blk, dir, lane);
    // m = gy v^T: two of the sixteen tiles per warp
    {
        AFrag<kZ> own;
#pragma unroll
        for (int s = 0; s < kZ; ++s)
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) ldsm4(own.w[s][kk], smem_addr(gs + s * kPlane + blk * kBlock * kRow + 16 * kk + off_a(lane)));
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int j = 2 * dir + i;
            float m[2][4] = {};
            prod_tokens<kZ, kZ>(m, own, vs, j, lane);
            store_tile<kX>(ms, m, blk, j, g, q);
            if (j == blk) {
                // diagonal: row g sits in lane (g, g / 2), row g + 8 likewise in the second half
                if (q == (g >> 1)) {
                    dots[blk * kBlock + g] = (g & 1) ? m[0][1] : m[0][0];
                    dots[blk * kBlock + g + 8] = (g & 1) ? m[1][3] : m[1][2];
                }
            }
        }
    }
    // pairs that straddle the chunk's right edge, per channel (see the file header)
    {
        float e0 = 0.f, e1 = 0.f;
        if (right) {
            const uint4* sx = dir == 0 ? st + kState : st + 2 * a.plane + kState;       // passed the edge rightward
            const uint4* sy = dir == 0 ? st + 3 * a.plane : st + a.plane;               // ... leftward
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                float x[8] = {}, y[8] = {};
#pragma unroll
                for (int i = 0; i < kX; ++i) {
                    const int o = i * (kStateWords / 4) + (blk * 4 + kk) * 32 + lane;
                    const uint4 fx = read_behind(sx + o), fy = read_behind(sy + o);
                    const uint32_t wx[4] = {fx.x, fx.y, fx.z, fx.w}, wy[4] = {fy.x, fy.y, fy.z, fy.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        x[2 * j] += lo_f(wx[j]); x[2 * j + 1] += hi_f(wx[j]);
                        y[2 * j] += lo_f(wy[j]); y[2 * j + 1] += hi_f(wy[j]);
                    }
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) { e0 = fmaf(x[j], y[j], e0); e1 = fmaf(x[4 + j], y[4 + j], e1); }
            }
        }
        e0 += __shfl_xor_sync(0xffffffffu, e0, 1); e0 += __shfl_xor_sync(0xffffffffu, e0, 2);
        e1 += __shfl_xor_sync(0xffffffffu, e1, 1); e1 += __shfl_xor_sync(0xffffffffu, e1, 2);
        const int ch = 16 * blk + 4 * (g >> 1) + (g & 1);
        if (q == 0) { edge[dir * N + ch] = e0; edge[dir * N + ch + 2] = e1; }
    }
    unsigned strong = 0u;
#pragma unroll
    for (int j = 0; j < kBlocks; ++j) strong |= block_is_safe(tab, j, lane) ? 0u : 1u << j;
    __syncthreads();

    float mine[2][2][4], diff[2][2][4];          // r gr> + k gk<, and that minus (r gr< + k gk>)
    {
        float u4[4], gu[4] = {0.f, 0.f, 0.f, 0.f};
        row4(a.u + h * N, cs, q, u4);
        float o[2][2][2][4] = {};
        if (32 * th < tokens) slice_gradient<T, kZ, kX, false, kRound>(o, gs, ms, pf, s_left, s_right, tab, kp + base, C, tokens, strong, cs, th, lane);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = 32 * th + 16 * mt + 8 * half + g;
                float r4[4], k4[4];
                const size_t at_t = base + static_cast<size_t>(t) * C + 16 * cs + 4 * q;
                load4(r_raw, t, cs, q, r4);
                load4(k_raw, t, cs, q, k4);
                const float dot = dots[t];
                float g4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float early = o[0][mt][half][e], late = o[1][mt][half][e], kd = k4[e] * dot;
                    g4[e] = early + late + u4[e] * kd;
                    mine[mt][half][e] = r4[e] * early;
                    diff[mt][half][e] = r4[e] * (early - late);
                    gu[e] = fmaf(r4[e], kd, gu[e]);
                }
                if (t < tokens) put4(a.scalar, static_cast<O*>(a.gr) + at_t, g4[0], g4[1], g4[2], g4[3]);
            }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            gu[e] += __shfl_xor_sync(0xffffffffu, gu[e], 4);
            gu[e] += __shfl_xor_sync(0xffffffffu, gu[e], 8);
            gu[e] += __shfl_xor_sync(0xffffffffu, gu[e], 16);
        }
        if (g == 0) put_row4(gus + th * N, cs, q, gu[0], gu[1], gu[2], gu[3]);
    }
    __syncthreads();               // everyone is done with the planes of k
    stage_scaled<kX>(pf + dir * kX * kPlane, r_raw, tab, blk, dir, lane);
    __syncthreads();
    {
        float u4[4];
        row4(a.u + h * N, cs, q, u4);
        float o[2][2][2][4] = {};
        if (32 * th < tokens) slice_gradient<T, kZ, kX, true, kRound>(o, vs, ms, pf, a_left, a_right, tab, rp + base, C, tokens, strong, cs, th, lane);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = 32 * th + 16 * mt + 8 * half + g;
                float r4[4], k4[4];
                const size_t at_t = base + static_cast<size_t>(t) * C + 16 * cs + 4 * q;
                load4(r_raw, t, cs, q, r4);
                load4(k_raw, t, cs, q, k4);
                const float dot = dots[t];
                float g4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float early = o[0][mt][half][e], late = o[1][mt][half][e];
                    g4[e] = early + late + u4[e] * r4[e] * dot;
                    mine[mt][half][e] = fmaf(k4[e], early, mine[mt][half][e]);
                    diff[mt][half][e] = fmaf(k4[e], early - late, diff[mt][half][e]);
                }
                if (t < tokens) put4(a.scalar, static_cast<O*>(a.gk) + at_t, g4[0], g4[1], g4[2], g4[3]);
            }
    }
    // gw: g_m = edge + sum_{t >= m} diff_t - mine_m, from the registers that hold them: a thread has its channels' tokens g of each eight, summed from
    // the last one on over the lanes of a channel and from the later half of the chunk.  (Through tables in shared memory, behind gv,
    // the two arrays were kept in local memory meanwhile, which with this much shared memory means L2.)
    float4 w_own[2][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = 32 * th + 8 * i + g;
        w_own[i >> 1][i & 1] = t < tokens ? read_behind(reinterpret_cast<const float4*>(a.w + base + static_cast<size_t>(t) * C + 16 * cs + 4 * q)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    {
        float carry[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int i = 3; i >= 0; --i)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float& x = diff[i >> 1][i & 1][e];
#pragma unroll
                for (int off = 1; off < 8; off *= 2) {
                    const float later = __shfl_down_sync(0xffffffffu, x, 4 * off);
                    if (g + off < 8) x += later;
                }
                x += carry[e];
                carry[e] = __shfl_sync(0xffffffffu, x, q);      // of the tokens from here on
            }
        if (th == 1 && g == 0) put_row4(seg, cs, q, carry[0], carry[1], carry[2], carry[3]);
    }
    __syncthreads();               // m has been read
    {
        float later[4], e1[4], add[4] = {0.f, 0.f, 0.f, 0.f};
        row4(edge, cs, q, later);
        row4(edge + N, cs, q, e1);
        if (th == 0) row4(seg, cs, q, add);
#pragma unroll
        for (int e = 0; e < 4; ++e) later[e] = (later[e] + e1[e]) + add[e];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = 32 * th + 8 * i + g;
            const float4 w = w_own[i >> 1][i & 1];
            const float w4[4] = {w.x, w.y, w.z, w.w};
            float g4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) g4[e] = (later[e] + (diff[i >> 1][i & 1][e] - mine[i >> 1][i & 1][e])) * decay_slope(w4[e]);
            if (t < tokens) put4(a.scalar, a.gw + base + static_cast<size_t>(t) * C + 16 * cs + 4 * q, g4[0], g4[1], g4[2], g4[3]);
        }
        if (threadIdx.x < N)
            a.gu_part[(static_cast<size_t>(b) * a.n_chunks + n) * C + h * N + threadIdx.x] = gus[threadIdx.x] + gus[N + threadIdx.x];
    }
    if (a.gv != nullptr) {
        // gv: rows are k, columns r, values gy: the forward with exchanged roles.  It needs only the first part of the scaled
        // rows; its edge planes take the room of the second.
        static_assert(kX > kP, "no room for the edge planes");
        __nv_bfloat16* e0 = pf + kP * kPlane;
        __nv_bfloat16* e1 = pf + (kX + kP) * kPlane;
        if (rows > 0) pair_rows<kP>([&](Block& x) { load_block(x, k_raw, blk, g, q); }, [&](Block& x) { load_block(x, r_raw, blk, g, q); }, a.u + h * N, tab,
                      pf + dir * kX * kPlane, ms, dir ? e1 : e0, blk, dir, lane);
        __syncthreads();
        if (32 * th >= tokens) return;
        float y[2][2][4];
        pair_outputs<kZ, kP, true>(y, ms, gs, e0, e1, a_left, a_right, cs, th, lane);
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int t = 32 * th + 16 * mt + 8 * half + g;
                if (t < tokens)
                    put4(a.scalar, static_cast<O*>(a.gv) + base + static_cast<size_t>(t) * C + 16 * cs + 4 * q, y[mt][0][2 * half],
                         y[mt][0][2 * half + 1], y[mt][1][2 * half], y[mt][1][2 * half + 1]);
            }
    }
    if (sizeof(T) == 2 && threadIdx.x == 0) sm100::mbar_wait(bar, 0, a.limit / 64);
}

// gu[c] = sum over batch and chunks of the parts, in a fixed order
__global__ void __launch_bounds__(1024) wkv6_bonus_kernel(int parts, int C, const float* part, float* __restrict__ gu) {
    wait_for_launch_before();
    __shared__ float red[32][33];
    const int c = blockIdx.x * 32 + threadIdx.x;
    float acc = 0.f;
    for (int i = threadIdx.y; i < parts; i += 32) acc += part[static_cast<size_t>(i) * C + c];
    red[threadIdx.y][threadIdx.x] = acc;
    __syncthreads();
    if (threadIdx.y == 0) {
        float t = 0.f;
#pragma unroll
        for (int i = 0; i < 32; ++i) t += red[i][threadIdx.x];
        gu[c] = t;
    }
}

// ---- host side -------------------------------------------------------------------------------------------------
// test mode: barriers wait for 16 bytes that never come, and give up after 2^10 polls
static std::atomic<bool> g_withhold{false};
void set_withhold_test(bool on) { g_withhold.store(on); }
static unsigned wait_limit() { return g_withhold.load() ? 1u << 10 : kWaitLimit; }
static unsigned extra_bytes() { return g_withhold.load() ? 16u : 0u; }

static size_t forward_smem(int kz, int kx) { return static_cast<size_t>(kz + 5 * kx) * kPlane * 2 + sizeof(Table) + 16; }
static size_t backward_smem(int kz, int kx) {
    return 2 * kRawTile + static_cast<size_t>(2 * kz + 3 * kx) * kPlane * 2 + sizeof(Table) + (1 + 2 + 2 + 1) * N * sizeof(float) + 16;
}

static int chunks_of(int T) { return (T + kChunk - 1) / kChunk; }
static size_t state_plane(int B, int T, int H, int parts) {      // uint4 per (pair, direction)
    return static_cast<size_t>(B) * H * chunks_of(T) * parts * (kStateWords / 4);
}
// status word, a copy of u, states (and the parts of gu)
static size_t states_offset(int H) { return 256 + static_cast<size_t>(H) * N * sizeof(float); }
size_t forward_workspace(int B, int T, int H) { return states_offset(H) + 2 * state_plane(B, T, H, 1) * sizeof(uint4); }
size_t backward_workspace(int B, int T, int H) {
    return states_offset(H) + 4 * state_plane(B, T, H, 2) * sizeof(uint4) + static_cast<size_t>(B) * chunks_of(T) * H * N * sizeof(float);
}
// The kernels read u four floats at a time.  A u that starts elsewhere (a view into a parameter buffer) goes through a copy:
// scalar loads in the kernels, or a branch, cost every call 0.5 to 1 %.
static const float* aligned_bonus(const float* u, int H, void* workspace, cudaStream_t stream) {
    if ((reinterpret_cast<uintptr_t>(u) & 15u) == 0) return u;
    float* copy = reinterpret_cast<float*>(static_cast<char*>(workspace) + 256);
    cudaMemcpyAsync(copy, u, static_cast<size_t>(H) * N * sizeof(float), cudaMemcpyDeviceToDevice, stream);
    return copy;
}

// dynamic shared memory above 48 KB is a per-device attribute of each kernel: set the first time the kernel meets the device
static bool allow_smem(const void* kernel, size_t bytes) {
    static std::mutex lock;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> guard(lock);
    if (done.count({dev, kernel})) return true;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes)) != cudaSuccess) return false;
    done.insert({dev, kernel});
    return true;
}
// `ahead` of a launch (see prefetch_rows).  Where the whole call is little more than the device holds at once there is nothing to
// run ahead of: under 16 CTAs per SM the figures are the same within 0.5 % either way, and nothing is fetched.
static unsigned ahead_of(size_t ctas) {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) cudaGetLastError();
    return ctas < 16 * static_cast<size_t>(sms) ? static_cast<unsigned>(ctas) : static_cast<unsigned>(sms / 2);
}
static bool unaligned16(std::initializer_list<const void*> ps) {
    for (const void* p : ps)
        if (reinterpret_cast<uintptr_t>(p) & 15u) return true;
    return false;
}

// launches the first kernel; gy: null for the forward
template <typename T, typename G, int kZ, int kX, bool kRows>
static bool run_states(int B, int T_, int H, const void* r, const void* k, const void* v, const float* w, const void* gy, uint4* states,
                       size_t plane, void* workspace, cudaStream_t stream) {
    constexpr int kPairs = kRows ? 2 : 1;
    static_assert(kZ == 1, "z enters in one part");
    typedef StateSmem<T, T, G, kX, kPairs> S;
    tensor_map::bind_primary_context();   // the tensor-map encoder is a driver call
    const int C = H * N;
    const auto map = [&](CUtensorMap* m, const void* p, bool half) { return tensor_map::make_btc(m, p, B, T_, C, N, kChunk, half); };
    CUtensorMap mw, mk, mv, mr, mg;
    if (!(map(&mw, w, false) && map(&mk, k, sizeof(T) == 2) && map(&mv, v, sizeof(T) == 2))) return false;
    if (kPairs > 1) {
        if (!(map(&mr, r, sizeof(T) == 2) && map(&mg, gy, sizeof(G) == 2))) return false;
    } else {
        mr = mk;
        mg = mv;
    }
    const StateArgs a{T_, H, chunks_of(T_), states, plane, static_cast<unsigned*>(workspace),
                      failure_mirror(kRows ? Op::wkv6_backward : Op::wkv6_forward), wait_limit(), extra_bytes()};
    const auto kernel = wkv6_state_kernel<T, T, G, kX, kRows, kPairs>;
    if (!allow_smem(reinterpret_cast<const void*>(kernel), S::bytes)) return false;
    launch_behind(kernel, dim3(B * H, 2), 128 * kPairs, S::bytes, stream, a, mw, mk, mv, mr, mg);
    return true;
}

template <typename T, int kZ, int kX>
static int run_forward(int B, int T_, int H, const void* r, const void* k, const void* v, const float* w, const float* u, float* y,
                       void* workspace, cudaStream_t stream) {
    uint4* states = reinterpret_cast<uint4*>(static_cast<char*>(workspace) + states_offset(H));
    const size_t plane = state_plane(B, T_, H, kX);
    const int n_chunks = chunks_of(T_);
    int launched = 1;
    if (n_chunks > 1) {
        if (!run_states<T, T, kZ, kX, false>(B, T_, H, nullptr, k, v, w, nullptr, states, plane, workspace, stream)) return -1;
        ++launched;
    }
    OutArgs o{T_, H, n_chunks, ahead_of(static_cast<size_t>(B) * H * n_chunks), r, k, v, w, aligned_bonus(u, H, workspace, stream), y, unaligned16({y}), states, plane,
              static_cast<unsigned*>(workspace), failure_mirror(Op::wkv6_forward), wait_limit(), extra_bytes()};
    tensor_map::bind_primary_context();
    CUtensorMap mw, mk, mr, mv;
    const bool half = sizeof(T) == 2;
    const auto map = [&](CUtensorMap* m, const void* p, bool narrow, bool swizzled) { return tensor_map::make_btc(m, p, B, T_, H * N, N, kChunk, narrow, swizzled); };
    if (!(map(&mw, w, false, false) && map(&mk, k, half, half) && map(&mr, r, half, half) && map(&mv, v, half, false))) return -1;
    const auto kernel = wkv6_forward_kernel<T, kZ, kX>;
    if (!allow_smem(reinterpret_cast<const void*>(kernel), forward_smem(kZ, kX))) return -1;
    launch_behind(kernel, static_cast<unsigned>(B) * H * n_chunks, 256, forward_smem(kZ, kX), stream, o, mw, mk, mr, mv);
    return launched;
}

template <typename T, typename G, typename O, int kZ, int kX, int kP>
static int run_backward(int B, int T_, int H, const void* r, const void* k, const void* v, const float* w, const float* u, const void* gy,
                        void* gr, void* gk, void* gv, float* gw, float* gu, void* workspace, cudaStream_t stream) {
    uint4* states = reinterpret_cast<uint4*>(static_cast<char*>(workspace) + states_offset(H));
    const size_t plane = state_plane(B, T_, H, kX);
    const int n_chunks = chunks_of(T_), C = H * N;
    int launched = 2;
    if (n_chunks > 1) {
        if (!run_states<T, G, kZ, kX, true>(B, T_, H, r, k, v, w, gy, states, plane, workspace, stream)) return -1;
        ++launched;
    }
    float* gu_part = reinterpret_cast<float*>(states + 4 * plane);
    GradArgs o{T_, H, n_chunks, ahead_of(static_cast<size_t>(B) * H * n_chunks), r, k, v, gy, w, aligned_bonus(u, H, workspace, stream), gr, gk, gv, gw, gu_part, unaligned16({gr, gk, gv, gw}), states, plane,
               static_cast<unsigned*>(workspace), failure_mirror(Op::wkv6_backward), wait_limit(), extra_bytes()};
    tensor_map::bind_primary_context();
    CUtensorMap mw, mk, mr, mv, mg;
    const auto map = [&](CUtensorMap* m, const void* p, bool half, bool swizzled) { return tensor_map::make_btc(m, p, B, T_, C, N, kChunk, half, swizzled); };
    if (!(map(&mw, w, false, false) && map(&mk, k, sizeof(T) == 2, sizeof(T) == 2) && map(&mr, r, sizeof(T) == 2, sizeof(T) == 2) &&
          map(&mv, v, sizeof(T) == 2, false) && map(&mg, gy, sizeof(G) == 2, false)))
        return -1;
    const auto kernel = wkv6_backward_kernel<T, G, O, kZ, kX, kP>;
    if (!allow_smem(reinterpret_cast<const void*>(kernel), backward_smem(kZ, kX))) return -1;
    launch_behind(kernel, static_cast<unsigned>(B) * H * n_chunks, 256, backward_smem(kZ, kX), stream, o, mw, mk, mr, mv, mg);
    launch_behind(wkv6_bonus_kernel, C / 32, dim3(32, 32), 0, stream, B * n_chunks, C, gu_part, gu);
    return launched;
}

int forward(int B, int T, int H, const void* r, const void* k, const void* v, const float* w, const float* u, float* y, bool bf16_in,
            void* workspace, cudaStream_t stream) {
    return bf16_in ? run_forward<__nv_bfloat16, 1, 1>(B, T, H, r, k, v, w, u, y, workspace, stream)
                   : run_forward<float, 1, 1>(B, T, H, r, k, v, w, u, y, workspace, stream);
}

int backward(int B, int T, int H, const void* r, const void* k, const void* v, const float* w, const float* u, const void* gy, void* gr,
             void* gk, void* gv, float* gw, float* gu, bool bf16_in, bool gy_bf16, bool bf16_out, void* workspace,
             cudaStream_t stream) {
    typedef __nv_bfloat16 H16;
#define RUN(T_, G_, O_, Z_, X_, P_) run_backward<T_, G_, O_, Z_, X_, P_>(B, T, H, r, k, v, w, u, gy, gr, gk, gv, gw, gu, workspace, stream)
    if (!bf16_in) return RUN(float, float, float, 1, 2, 1);
    if (gy_bf16) return bf16_out ? RUN(H16, H16, H16, 1, 2, 1) : RUN(H16, H16, float, 1, 2, 1);
    return bf16_out ? RUN(H16, float, H16, 1, 2, 1) : RUN(H16, float, float, 1, 2, 1);
#undef RUN
}

}  // namespace wkv6c
