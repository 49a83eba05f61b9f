// WKV6 (head size 64, bidirectional) as exact sequential state sweeps, fp32, any T: what float32 callers get.
//
// Per (batch, head) the operator carries a 64 x 64 state S[key i][value j]
//   rightward  S>_{t+1} = diag(d_t) S>_t + k_t v_t^T      y_t  = r_t^T (S>_t + diag(u) k_t v_t^T)
//   leftward   S<_{t-1} = diag(d_t) S<_t + k_t v_t^T      y_t += r_t^T S<_t
// with d_t = exp(-exp(w_raw_t)).  The gradients need the states S and their adjoints
// A = dL/dS (rightward adjoint runs backwards in time, A>_t = r_t gy_t^T + diag(d_t) A>_{t+1},
// and mirrored for the leftward direction):
//   gr_t = S_t gy_t (+ bonus)   gk_t = A_{t+1} v_t (+ bonus)   gv_t = A_{t+1}^T k_t (+ bonus)
// Every one of these is "read out a 64-vector product of the state, then update the state
// by a decayed rank-1 term", so one sweep engine serves them all: y from a walk of S, gr from a walk
// of S, gk and gv from one walk of A.  A block of two warps owns one state and keeps it in registers, 8 x 8 values per thread.
// Tokens arrive in shared memory 8 at a time through cp.async, double-buffered.  The two
// directions run in two blocks that add into a zeroed output (two addends per element: bit-reproducible).  Where there are too
// few blocks to fill the device, a sequence is walked in several segments at a time (below).
//
// A token's decay enters as the factor d_t alone, never as a difference of summed logarithms, so a token that forgets
// everything (d_t = 0) leaves the others exact.
//
// What bounds it: the float32 pipe and the dependent steps of a token; 51 % of the pipe and 52 % of the issue slots busy in the
// forward, 59 % of either in the backward (B=32, T=196, H=12).  B=32, H=12, forward + backward: T=196 611 us with a row or column of the state per thread, gk and gv in walks of
// their own and (backward) both directions in one block; 491 with 8 x 8 tiles and gk, gv together; 455 with the directions always
// in two blocks (shorter pieces of work spread better over the SMs) and the bonus's scalars only where they are used; T=1024
// 3045 -> 2163.  Sums of eight instead of one chain of 64 also leave half the error (9e-8 for 1.6e-7 in the 2-norm).
// Three-part bfloat16 products in 64-token chunks left ten times that (9e-7).
//
// Decay gradient.  With p_t = r_t * (S_t gy_t) and q_t = k_t * (A_{t+1} v_t) (state parts
// only, elementwise over key channels),
//   d_t * dL/dd_t = sum_{tau>t} p>_tau - sum_{tau>=t} q>_tau + sum_{tau<t} p<_tau - sum_{tau<=t} q<_tau
// (every (source, reader) token pair whose decay product contains d_t, counted from the
// reader side minus the pairs that do not straddle t).  The sweeps write running sums of
// p and q (accumulated in double) to scratch; a last elementwise kernel combines them and
// applies d(d_t)/d(w_raw) = d_t * (-exp(w_raw)), which cancels the division by d_t.  gw is therefore off by the rounding
// of p and q over the whole sequence (5e-6 in the 2-norm at T=1024; sums kept in double to the end: the same).  Where d_t
// is zero in float so is the gradient; the difference is not taken there, since exp(w_raw) would multiply its rounding
// without bound.
//
// Reference being replaced: classification/mmcls_custom/models/backbones/cuda_v6/
// wkv6_cuda.cu:6-97 (forward), :99-346 (backward; its T <= 256 limit does not apply here).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "launch.h"
#include "vrwkv_internal.h"

namespace wkv6 {

constexpr int N = 64;          // head size
constexpr int kBatch = 8;      // tokens per shared-memory batch (two batches of 10 KB and 6 KB of results per block: 8 blocks per SM)
constexpr int kParts = N / kBatch;   // threads that share one token's dot products
constexpr int kVecs = 5;       // r, k, v, gy, decay
enum Kind { KIND_Y = 0, KIND_GR = 1, KIND_GK = 2, KIND_GV = 3 };      // results
enum Walk { WALK_Y, WALK_GR, WALK_GK, WALK_GKV };                    // state S with y or gr read out of it, adjoint A with gk, or gk and gv
enum Vec { V_R = 0, V_K = 1, V_V = 2, V_G = 3, V_D = 4 };

struct Args {
    int B, T, H;
    const float* src[kVecs];   // r, k, v, gy (null in the forward), w_raw  -- (B, T, 64 H)
    const float* u;            // (H, 64)
    float* out[4];             // by kind: y, gr, gk, gv
    float* cum[4];             // running sums: p> (prefix), q> (suffix), p< (suffix), q< (prefix)
    float* gu_part;            // (B, segs, 64 H)
    int segs, seg_len;         // a sequence in segments of seg_len tokens (a multiple of kBatch; the last may be shorter)
    float* states;             // segs > 1: [k v | r gy][time direction][b h][segs - 1] slots of kSlot floats
};
// A slot: the state behind a segment, as element (row i, column j) at j * 64 + i, and the segment's decay of every row.
constexpr int kSlot = N * N + N;

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kPending>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kPending) : "memory");
}

struct Batch {
    float vec[kVecs][kBatch][N];
    float vg[kBatch];    // v_t . gy_t
    float ruk[kBatch];   // sum_i r_t[i] u[i] k_t[i]
};
struct Shared {
    Batch buf[2];
    float out[kBatch][N];         // read-outs of a batch: of the kept dimension,
    float part[2][kBatch][N];     // and of the other one (gv), each warp's share
};
static_assert(sizeof(Shared) <= 48 * 1024, "more shared memory than a kernel has without asking");

__device__ __forceinline__ size_t slot_of(const Args& a, int pair, int dir, int bh, int i) {
    return ((static_cast<size_t>(pair * 2 + dir) * a.B * a.H + bh) * (a.segs - 1) + i) * kSlot;
}

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }
__device__ __forceinline__ void lds8(const float* lo, const float* hi, float2 (&x)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(lo), b = *reinterpret_cast<const float4*>(hi);
    x[0] = make_float2(a.x, a.y); x[1] = make_float2(a.z, a.w); x[2] = make_float2(b.x, b.y); x[3] = make_float2(b.z, b.w);
}
__device__ __forceinline__ float part_of(const float2 (&x)[4], int i) { return i & 1 ? x[i >> 1].y : x[i >> 1].x; }
// Sums of v[0 .. 2 kHalf) over the lanes that differ in bit `mask`; a lane keeps the half that its bit names.
template <int kHalf>
__device__ __forceinline__ void sum_half(float (&v)[8], bool upper, int mask) {
#pragma unroll
    for (int i = 0; i < kHalf; ++i) {
        const float got = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + kHalf], mask);
        v[i] = (upper ? v[i + kHalf] : v[i]) + got;
    }
}

// One walk over a segment (with segs = 1, the whole sequence).  kForward: direction of time.  The two directions run in two
// blocks that add into a zeroed output: exactly two addends per element, so the sum does not depend on their order.  (As a cluster whose
// blocks store the half that they meet first, wait for one another once and add to the other's half they need no clearing, 17 us of 450 at
// B=32, T=196, H=12, but the backward's walks then share the SMs worse: 269 -> 301 us.)
//
// Tile of a thread.  A read-out keeps one dimension of the state and sums over the other; a warp owns 32 of the kept indices
// and all 64 of the summed ones, a thread 8 x 8: kept 32 warp + 8 (lane / 8) + e, summed 4 (lane % 8) + f (f < 4) and the same
// + 32.  So a token costs 8 to 10 16-byte shared loads, none of them in conflict, for 192 to 256 multiply-adds (as pairs, f32x2),
// where a thread with a whole row or column took 32 to 48 for 192 in one chain of sums; the eight lanes' sums are scattered
// (7 shuffles) so that lane l ends with kept index 32 warp + l.  gk (kept: rows) and gv (columns) come from one walk of A: gv's
// sums over a warp's rows meet the other warp's once per batch.
template <int kWalk, bool kForward, bool kSegments>
__device__ __forceinline__ void sweep(const Args& a, Shared& sh, int b, int h, int seg, float u_self, const float* u_smem,
                                      float& gu_acc) {
    constexpr bool kState = kWalk == WALK_Y || kWalk == WALK_GR;               // S, else its adjoint
    constexpr bool kKeepCols = kWalk == WALK_Y, kBoth = kWalk == WALK_GKV;
    constexpr int kKind = kWalk == WALK_Y ? KIND_Y : kWalk == WALK_GR ? KIND_GR : KIND_GK;
    constexpr int kA = kState ? V_K : V_R;                                     // rank-1 update: alpha beta^T
    constexpr int kB_ = kState ? V_V : V_G;
    constexpr int kC = kWalk == WALK_Y ? V_R : kWalk == WALK_GR ? V_G : V_V;   // read-out
    // the rightward state S> runs forward in time, its adjoint A> backward; mirrored for "<"
    constexpr bool kRightward = kState ? kForward : !kForward;
    const int tid = threadIdx.x, lane = tid & 31, kept = tid & ~7, summed = 4 * (lane & 7);
    const int first = kSegments ? seg * a.seg_len : 0, T = kSegments ? min(a.seg_len, a.T - first) : a.T, C = a.H * N;
    const size_t base = (static_cast<size_t>(b) * a.T + first) * C + static_cast<size_t>(h) * N;
    const int n_batches = (T + kBatch - 1) / kBatch;

    auto issue = [&](int bi, Batch* dst) {
        const int bt0 = (kForward ? bi : n_batches - 1 - bi) * kBatch;
#pragma unroll
        for (int vsel = 0; vsel < kVecs; ++vsel) {
            const float* src = a.src[vsel];
            if (src == nullptr) continue;
#pragma unroll
            for (int q = 0; q < (kBatch * N / 4) / N; ++q) {          // 128 chunks of 16 B, 64 threads
                const int chunk = q * N + tid;
                const int row = chunk >> 4, col4 = (chunk & 15) * 4;      // 16 chunks of 16 bytes per token row
                const int t = bt0 + row;
                if (t < T) cp_async16(&dst->vec[vsel][row][col4], src + base + static_cast<size_t>(t) * C + col4);
            }
        }
        cp_async_commit();
    };

    float2 X[8][4];       // [kept e][pairs of summed]
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int f = 0; f < 4; ++f) X[e][f] = dup(0.f);
    const int before = !kSegments ? 0 : kForward ? seg : a.segs - 1 - seg;        // segments this direction has walked
    if (kSegments && before > 0) {
        const float* from = a.states + slot_of(a, kState ? 0 : 1, kForward ? 0 : 1, b * a.H + h, before - 1);
        const auto at = [&](int e, int f) {
            const int p = kept + e, q = summed + (f & 3) + 32 * (f >> 2);
            return kKeepCols ? from[p * N + q] : from[q * N + p];
        };
#pragma unroll
        for (int e = 0; e < 8; ++e)
#pragma unroll
            for (int f = 0; f < 4; ++f) X[e][f] = make_float2(at(e, 2 * f), at(e, 2 * f + 1));
    }
    double run = 0.0;

    issue(0, &sh.buf[0]);
    for (int bi = 0; bi < n_batches; ++bi) {
        Batch* cur = &sh.buf[bi & 1];
        if (bi + 1 < n_batches) {
            issue(bi + 1, &sh.buf[(bi + 1) & 1]);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int bt0 = (kForward ? bi : n_batches - 1 - bi) * kBatch;
        const int rows = min(kBatch, T - bt0);
        // decay in place (rows behind the last token hold anything and are not used)
        float d_t[kBatch];
#pragma unroll
        for (int row = 0; row < kBatch; ++row) d_t[row] = cur->vec[V_D][row][tid];
#pragma unroll
        for (int row = 0; row < kBatch; ++row) cur->vec[V_D][row][tid] = expf(-expf(d_t[row]));
        if (kRightward) {       // per-token scalars of the bonus
            constexpr bool kVg = kWalk != WALK_Y, kRuk = kWalk == WALK_Y || kBoth;
            const int row = tid / kParts, part = tid % kParts;
            float s1 = 0.f, s2 = 0.f;
            if (row < rows) {
                const auto at = [&](const float* x, float2 (&v)[4]) { lds8(x + 4 * part, x + 4 * part + 32, v); };
                float2 x[4], z[4], uu[4];
                if (kVg) {
                    at(cur->vec[V_V][row], x);
                    at(cur->vec[V_G][row], z);
#pragma unroll
                    for (int n = 0; n < 8; ++n) s1 += part_of(x, n) * part_of(z, n);
                }
                if (kRuk) {
                    at(cur->vec[V_R][row], x);
                    at(cur->vec[V_K][row], z);
                    at(u_smem, uu);
#pragma unroll
                    for (int n = 0; n < 8; ++n) s2 += part_of(x, n) * part_of(uu, n) * part_of(z, n);
                }
            }
#pragma unroll
            for (int m = 1; m < kParts; m <<= 1) {
                if (kVg) s1 += __shfl_xor_sync(0xffffffffu, s1, m);
                if (kRuk) s2 += __shfl_xor_sync(0xffffffffu, s2, m);
            }
            if (part == 0) { cur->vg[row] = s1; cur->ruk[row] = s2; }
        }
        __syncthreads();
        // (two or four tokens at a time were slower: twice the code for the walks that share an SM)
#pragma unroll 1
        for (int step = 0; step < rows; ++step) {
            const int row = kForward ? step : rows - 1 - step;
            const auto by_kept = [&](int v, float2 (&x)[4]) { lds8(&cur->vec[v][row][kept], &cur->vec[v][row][kept + 4], x); };
            const auto by_summed = [&](int v, float2 (&x)[4]) { lds8(&cur->vec[v][row][summed], &cur->vec[v][row][summed + 32], x); };
            float out[8];
            float2 c[4];
            by_summed(kC, c);
            if (kKeepCols) {
                float2 d[4], al[4], be[4];
                by_summed(V_D, d);
                by_summed(kA, al);
                by_kept(kB_, be);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 bj = dup(part_of(be, e));
                    float2 o = __fmul2_rn(c[0], X[e][0]);
#pragma unroll
                    for (int f = 1; f < 4; ++f) o = __ffma2_rn(c[f], X[e][f], o);
                    out[e] = o.x + o.y;
#pragma unroll
                    for (int f = 0; f < 4; ++f) X[e][f] = __ffma2_rn(d[f], X[e][f], __fmul2_rn(al[f], bj));
                }
            } else {
                float2 d[4], al[4], be[4], k4[4], g[4];
                by_kept(V_D, d);
                by_kept(kA, al);
                by_summed(kB_, be);
                if (kBoth) {
                    by_kept(V_K, k4);
#pragma unroll
                    for (int f = 0; f < 4; ++f) g[f] = dup(0.f);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float2 di = dup(part_of(d, e)), ai = dup(part_of(al, e));
                    float2 o = __fmul2_rn(c[0], X[e][0]);
#pragma unroll
                    for (int f = 1; f < 4; ++f) o = __ffma2_rn(c[f], X[e][f], o);
                    out[e] = o.x + o.y;
                    if (kBoth) {
                        const float2 ki = dup(part_of(k4, e));
#pragma unroll
                        for (int f = 0; f < 4; ++f) g[f] = __ffma2_rn(ki, X[e][f], g[f]);
                    }
#pragma unroll
                    for (int f = 0; f < 4; ++f) X[e][f] = __ffma2_rn(di, X[e][f], __fmul2_rn(ai, be[f]));
                }
                if (kBoth) {
                    float v[8] = {g[0].x, g[0].y, g[1].x, g[1].y, g[2].x, g[2].y, g[3].x, g[3].y};
                    sum_half<4>(v, (lane & 16) != 0, 16);
                    sum_half<2>(v, (lane & 8) != 0, 8);
                    // columns summed + {0, 1} (+ 2: lane bit 3, + 32: lane bit 4)
                    *reinterpret_cast<float2*>(&sh.part[tid >> 5][row][summed + 2 * ((lane >> 3) & 1) + 32 * (lane >> 4)]) = make_float2(v[0], v[1]);
                }
            }
            sum_half<4>(out, (lane & 4) != 0, 4);
            sum_half<2>(out, (lane & 2) != 0, 2);
            sum_half<1>(out, (lane & 1) != 0, 1);
            sh.out[row][tid] = out[0];
        }
        if (kBoth) __syncthreads();
        // results of the batch, thread = channel: running sums, bonus
#pragma unroll
        for (int step = 0; step < kBatch; ++step) {
            const int row = kForward ? step : kBatch - 1 - step;
            if (row >= rows) continue;
            const size_t idx = base + static_cast<size_t>(bt0 + row) * C + tid;
            float out = sh.out[row][tid];
            // running sums for the decay gradient (state part only)
            if (kKind == KIND_GR) {
                run += static_cast<double>(cur->vec[V_R][row][tid] * out);
                a.cum[kRightward ? 0 : 2][idx] = static_cast<float>(run);
            }
            if (kKind == KIND_GK) {
                run += static_cast<double>(cur->vec[V_K][row][tid] * out);
                a.cum[kRightward ? 1 : 3][idx] = static_cast<float>(run);
            }
            float out_v = kBoth ? sh.part[0][row][tid] + sh.part[1][row][tid] : 0.f;
            // the bonus term lives in the rightward direction only
            if (kRightward) {
                if (kKind == KIND_Y) out += cur->ruk[row] * cur->vec[V_V][row][tid];
                if (kBoth) out_v += cur->ruk[row] * cur->vec[V_G][row][tid];
                if (kKind == KIND_GR) {
                    const float kvg = cur->vec[V_K][row][tid] * cur->vg[row];
                    out += u_self * kvg;
                    gu_acc += cur->vec[V_R][row][tid] * kvg;
                }
                if (kKind == KIND_GK) out += u_self * cur->vec[V_R][row][tid] * cur->vg[row];
            }
            atomicAdd(a.out[kKind] + idx, out);
            if (kBoth) atomicAdd(a.out[KIND_GV] + idx, out_v);
        }
        __syncthreads();   // the batch buffer is refilled two iterations later
    }
}

constexpr int kPerSm = 7;      // blocks, of 128 registers a thread (as fast as 6 of 168, 1 to 4 % faster where there are many)
// grid (b h, walk, direction + 2 segment)
template <bool kBackward, bool kSeg>
__global__ void __launch_bounds__(N, kPerSm) wkv6_sweep_kernel(const Args a) {
    wait_for_launch_before();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Shared& sh = *reinterpret_cast<Shared*>(smem_raw);
    __shared__ __align__(16) float u_smem[N];
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H, seg = kSeg ? blockIdx.z >> 1 : 0;
    const bool forward = (blockIdx.z & 1) != 0;      // in time
    const int tid = threadIdx.x;
    u_smem[tid] = a.u[h * N + tid];
    __syncthreads();
    const float u_self = u_smem[tid];
    float gu = 0.f;
    if (!kBackward) {
        if (forward) sweep<WALK_Y, true, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
        else sweep<WALK_Y, false, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
    } else if (blockIdx.y == 0 && a.out[KIND_GV] != nullptr) {      // the longest walk first
        if (forward) sweep<WALK_GKV, true, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
        else sweep<WALK_GKV, false, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
    } else if (blockIdx.y == 0) {
        if (forward) sweep<WALK_GK, true, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
        else sweep<WALK_GK, false, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
    } else if (forward) {
        sweep<WALK_GR, true, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
        a.gu_part[(static_cast<size_t>(b) * a.segs + seg) * a.H * N + h * N + tid] = gu;            // the bonus lives in this direction
    } else {
        sweep<WALK_GR, false, kSeg>(a, sh, b, h, seg, u_self, u_smem, gu);
    }
}

// ---- sequences in segments -------------------------------------------------------------------------------
// A few sequences leave most of the chip idle, and the walk's latency (0.3 us a token) is all their time.  Such a sequence is
// cut into segments that are walked side by side, still token by token: first the state that each segment would leave
// from zero, and its decay (wkv6_segment_state_kernel: the update without the read-out, a row of the state per thread), then the states
// behind every segment, S_j = decay_j S_{j-1} + own_j (wkv6_segment_scan_kernel), then the sweeps, each from the state
// in front of its segment.  Decays are products of factors here too, so the accuracy is that of the whole walk.
__global__ void __launch_bounds__(N, 9) wkv6_segment_state_kernel(const Args a) {
    wait_for_launch_before();
    __shared__ __align__(16) float buf[2][3][kBatch][N];
    const int tid = threadIdx.x, bh = blockIdx.x, b = bh / a.H, h = bh % a.H;
    const int pair = blockIdx.z >> 1, dir = blockIdx.z & 1, step_i = blockIdx.y;
    const int seg = dir == 0 ? step_i : a.segs - 1 - step_i;
    const int first = seg * a.seg_len, T = min(a.seg_len, a.T - first), C = a.H * N;
    const size_t base = (static_cast<size_t>(b) * a.T + first) * C + static_cast<size_t>(h) * N;
    const int n_batches = (T + kBatch - 1) / kBatch;
    const float* const src[3] = {a.src[pair ? V_R : V_K], a.src[pair ? V_G : V_V], a.src[V_D]};
    const auto issue = [&](int bi) {
        const int bt0 = (dir == 0 ? bi : n_batches - 1 - bi) * kBatch;
#pragma unroll
        for (int v = 0; v < 3; ++v)
#pragma unroll
            for (int q = 0; q < (kBatch * N / 4) / N; ++q) {
                const int chunk = q * N + tid, row = chunk >> 4, col4 = (chunk & 15) * 4, t = bt0 + row;
                if (t < T) cp_async16(&buf[bi & 1][v][row][col4], src[v] + base + static_cast<size_t>(t) * C + col4);
            }
        cp_async_commit();
    };
    float X[N], decay = 1.f;
#pragma unroll
    for (int n = 0; n < N; ++n) X[n] = 0.f;
    issue(0);
    for (int bi = 0; bi < n_batches; ++bi) {
        if (bi + 1 < n_batches) {
            issue(bi + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const auto& cur = buf[bi & 1];
        const int rows = min(kBatch, T - (dir == 0 ? bi : n_batches - 1 - bi) * kBatch);
        for (int step = 0; step < rows; ++step) {
            const int row = dir == 0 ? step : rows - 1 - step;
            const float di = expf(-expf(cur[2][row][tid])), ai = cur[0][row][tid];
            const float4* bv = reinterpret_cast<const float4*>(cur[1][row]);
            decay *= di;
#pragma unroll
            for (int n4 = 0; n4 < N / 4; ++n4) {
                const float4 b4 = bv[n4];
                X[4 * n4 + 0] = fmaf(di, X[4 * n4 + 0], ai * b4.x);
                X[4 * n4 + 1] = fmaf(di, X[4 * n4 + 1], ai * b4.y);
                X[4 * n4 + 2] = fmaf(di, X[4 * n4 + 2], ai * b4.z);
                X[4 * n4 + 3] = fmaf(di, X[4 * n4 + 3], ai * b4.w);
            }
        }
        __syncthreads();   // the buffer is refilled two iterations later
    }
    float* const to = a.states + slot_of(a, pair, dir, bh, step_i);
#pragma unroll
    for (int n = 0; n < N; ++n) to[n * N + tid] = X[n];
    to[N * N + tid] = decay;
}

// the slots of a (pair, direction, batch, head) in walking order: own state -> state behind the segment; a thread per element
__global__ void __launch_bounds__(256) wkv6_segment_scan_kernel(const Args a) {
    wait_for_launch_before();
    float* const slots = a.states + static_cast<size_t>(blockIdx.x) * (a.segs - 1) * kSlot;
    const int e = blockIdx.y * 256 + threadIdx.x, row = e % N;
    constexpr int kAhead = 4;
    float x = 0.f;
    for (int i0 = 0; i0 < a.segs - 1; i0 += kAhead) {
        float own[kAhead], decay[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (i0 + i < a.segs - 1) {
                own[i] = slots[static_cast<size_t>(i0 + i) * kSlot + e];
                decay[i] = slots[static_cast<size_t>(i0 + i) * kSlot + N * N + row];
            }
#pragma unroll
        for (int i = 0; i < kAhead; ++i)
            if (i0 + i < a.segs - 1) {
                x = fmaf(decay[i], x, own[i]);
                slots[static_cast<size_t>(i0 + i) * kSlot + e] = x;
            }
    }
}

// The decay gradient from running sums that begin anew with every segment: a segment's totals are the sums at its last
// token (p>, q<) or first one (p<, q>).  A thread per (batch, segment, kPiece tokens, channel).
constexpr int kPiece = 32;
__global__ void __launch_bounds__(256) wkv6_segment_decay_grad_kernel(const Args a, float* __restrict__ gw) {
    wait_for_launch_before();
    const int C = a.H * N, pieces = (a.seg_len + kPiece - 1) / kPiece;
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<size_t>(a.B) * a.segs * pieces * C) return;
    const int c = static_cast<int>(i % C), piece = static_cast<int>(i / C % pieces);
    const int seg = static_cast<int>(i / C / pieces % a.segs), b = static_cast<int>(i / C / pieces / a.segs);
    const size_t seq = static_cast<size_t>(b) * a.T * C + c;
    const auto head = [&](int j) { return seq + static_cast<size_t>(j) * a.seg_len * C; };
    const auto tail = [&](int j) { return seq + static_cast<size_t>(min((j + 1) * a.seg_len, a.T) - 1) * C; };
    double behind = 0.0, ahead = 0.0;
    for (int j = seg + 1; j < a.segs; ++j) behind += static_cast<double>(a.cum[0][tail(j)]) - a.cum[1][head(j)];
    for (int j = 0; j < seg; ++j) ahead += static_cast<double>(a.cum[2][head(j)]) - a.cum[3][tail(j)];
    const float p_right = a.cum[0][tail(seg)], p_left = a.cum[2][head(seg)];
    const int t0 = seg * a.seg_len + piece * kPiece;
    const int rows = min(min(kPiece, a.seg_len - piece * kPiece), a.T - t0);
#pragma unroll 4
    for (int t = 0; t < rows; ++t) {
        const size_t o = seq + static_cast<size_t>(t0 + t) * C;
        const float right = ((p_right - a.cum[0][o]) - a.cum[1][o]) + static_cast<float>(behind);
        const float left = ((p_left - a.cum[2][o]) - a.cum[3][o]) + static_cast<float>(ahead);
        const float e = expf(a.src[V_D][o]);
        gw[o] = expf(-e) == 0.f ? 0.f : -e * (right + left);
    }
}

// gw_raw = -exp(w_raw) * [ (P>_last - P>_t - Q>_t) + (P<_first - P<_t - Q<_t) ], a thread per 4 channels of a token, per_seq blocks to a
// sequence.  (A thread per element with 64-bit divisions: 25.8 us at B=32, T=196, H=12, now 19.1.)  `scalar`: gw is not
// 16-byte aligned.
__global__ void __launch_bounds__(256) wkv6_decay_grad_kernel(int T, int C, unsigned per_seq, bool scalar, const float* w_raw, const float* cp,
                                                              const float* cq, const float* cp2,
                                                              const float* cq2, float* __restrict__ gw) {
    wait_for_launch_before();
    const unsigned per_row = static_cast<unsigned>(C) / 4, b = blockIdx.x / per_seq, v = (blockIdx.x - b * per_seq) * 256u + threadIdx.x;
    if (v >= per_row * static_cast<unsigned>(T)) return;
    const size_t seq = static_cast<size_t>(b) * T * C, i = seq + static_cast<size_t>(v) * 4;
    const size_t first = seq + v % per_row * 4, last = first + static_cast<size_t>(T - 1) * C;
    const auto at = [](const float* p, size_t o, float (&x)[4]) {
        const float4 t = *reinterpret_cast<const float4*>(p + o);
        x[0] = t.x; x[1] = t.y; x[2] = t.z; x[3] = t.w;
    };
    float p_last[4], p[4], q[4], p_first[4], p2[4], q2[4], w[4], g[4];
    at(cp, i, p); at(cq, i, q); at(cp2, i, p2); at(cq2, i, q2); at(w_raw, i, w);
    at(cp, last, p_last); at(cp2, first, p_first);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float right = (p_last[e] - p[e]) - q[e];
        const float left = (p_first[e] - p2[e]) - q2[e];
        const float x = expf(w[e]);
        g[e] = expf(-x) == 0.f ? 0.f : -x * (right + left);
    }
    if (!scalar) {
        *reinterpret_cast<float4*>(gw + i) = make_float4(g[0], g[1], g[2], g[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) gw[i + e] = g[e];
    }
}

// gu[c] = sum over batch (and segments) of gu_part, fixed order
__global__ void wkv6_bonus_grad_kernel(int B, int C, const float* part, float* __restrict__ gu) {
    wait_for_launch_before();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float acc = 0.f;
#pragma unroll 8
    for (int b = 0; b < B; ++b) acc += part[static_cast<size_t>(b) * C + c];
    gu[c] = acc;
}

// The status word and the results that two directions add into, in one launch: three results of 19 MB took 15 us as memsets, which the launch
// behind them also has to wait for in full.
constexpr int kClearVecs = 8;      // 16-byte stores of a thread
__global__ void __launch_bounds__(256) wkv6_clear_kernel(const Cleared z) {
    wait_for_launch_before();
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && z.status != nullptr) *z.status = 0u;
    float* const p = z.p[blockIdx.y];
    if (p == nullptr) return;
    const bool wide = (reinterpret_cast<uintptr_t>(p) & 15u) == 0;
    const size_t first = static_cast<size_t>(blockIdx.x) * 256 * kClearVecs + threadIdx.x;
#pragma unroll
    for (int i = 0; i < kClearVecs; ++i) {
        const size_t at = (first + static_cast<size_t>(i) * 256) * 4;      // n is a multiple of 64
        if (at >= z.n) return;
        if (wide) {
            *reinterpret_cast<float4*>(p + at) = make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) p[at + e] = 0.f;
        }
    }
}
void clear(const Cleared& z, cudaStream_t stream) {
    const size_t per_block = static_cast<size_t>(256) * kClearVecs * 4;
    launch_behind(wkv6_clear_kernel, dim3(static_cast<unsigned>(std::max<size_t>(1, (z.n + per_block - 1) / per_block)), z.p[1] == nullptr ? 1 : 3), 256, 0, stream, z);
}

struct Plan {
    int segs, len;
};
// How many segments a sequence is walked in, from the sizes alone (so a sequence's last bits may depend on how many others are in
// the call).  Three or four blocks per SM already keep it busy, and the states in front of the segments take two thirds of the time
// of the walks (38 of 60 us at B=3, T=1024, H=12; in the backward, whose walks share them, 69 of 156).  So: segments until there are `fill`
// blocks (counted as if gk and gv had walks of their own), and the whole walk where fewer than three come out or a segment would be
// shorter than a few batches.
// us, whole / segments: forward + backward H=12 B=3 T=1024 770 / 389, B=4 T=400 325 / 236.  Where the line lies: forward, 312
// blocks (B H = 156, T=400) 184 / 172, 432 blocks 186 / 202; backward, 74 to 96 sequences x heads (T=400) within 3 % either way.
static Plan make_plan(int B, int T, int H, int kinds) {
    const long long fill = kinds == 1 ? 1110 : 1332, shortest = kinds == 1 ? 16 : 32, fewest = 3;
    const long long want = std::min(fill / (2LL * B * H * kinds), T / shortest);
    if (want < fewest) return Plan{1, T};
    const int even = static_cast<int>((T + want - 1) / want), len = (even + kBatch - 1) / kBatch * kBatch;
    return Plan{(T + len - 1) / len, len};
}
static size_t state_floats(int B, int H, const Plan& pl, int pairs) {
    return static_cast<size_t>(pairs) * 2 * B * H * (pl.segs - 1) * kSlot;
}
static void run_segment_states(const Args& a, int pairs, cudaStream_t stream) {
    launch_behind(wkv6_segment_state_kernel, dim3(a.B * a.H, a.segs - 1, 2 * pairs), N, 0, stream, a);
    launch_behind(wkv6_segment_scan_kernel, dim3(2 * pairs * a.B * a.H, N * N / 256), 256, 0, stream, a);
}

// status word (which this path never sets), states of segments, running sums, parts of gu
constexpr size_t kHead = 256;
size_t forward_workspace(int B, int T, int H) { return kHead + state_floats(B, H, make_plan(B, T, H, 1), 1) * sizeof(float); }
size_t backward_workspace(int B, int T, int H) {
    const Plan pl = make_plan(B, T, H, 3);
    const size_t E = static_cast<size_t>(B) * T * H * N;
    return kHead + (state_floats(B, H, pl, 2) + 4 * E + static_cast<size_t>(B) * pl.segs * H * N) * sizeof(float);
}

// workspace: forward_workspace() bytes, or null (a sequence is then walked as a whole)
int forward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
            const float* u, float* y, void* workspace, cudaStream_t stream) {
    const Plan pl = workspace ? make_plan(B, T, H, 1) : Plan{1, T};
    Args a{};
    a.B = B; a.T = T; a.H = H;
    a.src[V_R] = r; a.src[V_K] = k; a.src[V_V] = v; a.src[V_G] = nullptr; a.src[V_D] = w_raw;
    a.u = u;
    a.out[KIND_Y] = y;
    a.segs = pl.segs; a.seg_len = pl.len;
    a.states = pl.segs > 1 ? reinterpret_cast<float*>(static_cast<char*>(workspace) + kHead) : nullptr;
    clear(Cleared{{y, nullptr, nullptr}, static_cast<unsigned*>(workspace), static_cast<size_t>(B) * T * H * N}, stream);
    if (pl.segs > 1) run_segment_states(a, 1, stream);
    const auto kernel = pl.segs > 1 ? wkv6_sweep_kernel<false, true> : wkv6_sweep_kernel<false, false>;
    launch_behind(kernel, dim3(B * H, 1, 2 * pl.segs), N, sizeof(Shared), stream, a);
    return pl.segs > 1 ? 3 : 1;
}

int backward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
             const float* u, const float* gy, float* gr, float* gk, float* gv, float* gw, float* gu,
             void* workspace, cudaStream_t stream) {
    const Plan pl = make_plan(B, T, H, 3);
    const int C = H * N;
    const size_t E = static_cast<size_t>(B) * T * C;
    float* ws = reinterpret_cast<float*>(static_cast<char*>(workspace) + kHead);
    Args a{};
    a.B = B; a.T = T; a.H = H;
    a.src[V_R] = r; a.src[V_K] = k; a.src[V_V] = v; a.src[V_G] = gy; a.src[V_D] = w_raw;
    a.u = u;
    a.out[KIND_GR] = gr; a.out[KIND_GK] = gk; a.out[KIND_GV] = gv;
    a.segs = pl.segs; a.seg_len = pl.len;
    a.states = ws;
    ws += state_floats(B, H, pl, 2);
    for (int i = 0; i < 4; ++i) a.cum[i] = ws + i * E;
    a.gu_part = ws + 4 * E;
    clear(Cleared{{gr, gk, gv}, static_cast<unsigned*>(workspace), E}, stream);      // (gv == nullptr: the caller gets gv elsewhere)
    if (pl.segs > 1) run_segment_states(a, 2, stream);
    const auto kernel = pl.segs > 1 ? wkv6_sweep_kernel<true, true> : wkv6_sweep_kernel<true, false>;
    launch_behind(kernel, dim3(B * H, 2, 2 * pl.segs), N, sizeof(Shared), stream, a);
    if (pl.segs > 1) {
        const size_t threads = static_cast<size_t>(B) * pl.segs * ((pl.len + kPiece - 1) / kPiece) * C;
        launch_behind(wkv6_segment_decay_grad_kernel, static_cast<unsigned>((threads + 255) / 256), 256, 0, stream, a, gw);
    } else {
        const unsigned per_seq = static_cast<unsigned>((static_cast<size_t>(T) * C / 4 + 255) / 256);
        launch_behind(wkv6_decay_grad_kernel, per_seq * static_cast<unsigned>(B), 256, 0, stream, T, C, per_seq, (reinterpret_cast<uintptr_t>(gw) & 15u) != 0, w_raw,
                      a.cum[0], a.cum[1], a.cum[2], a.cum[3], gw);
    }
    launch_behind(wkv6_bonus_grad_kernel, (C + 127) / 128, 128, 0, stream, B * pl.segs, C, a.gu_part, gu);
    return pl.segs > 1 ? 5 : 3;
}

}  // namespace wkv6
