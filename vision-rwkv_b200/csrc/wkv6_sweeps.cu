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
// by a decayed rank-1 term", so one sweep engine serves them all.  A block of 64 threads
// owns either the rows (thread = key channel) or the columns (thread = value channel) of
// one state, whichever makes the read-out a sum inside the thread, and keeps its 64 state
// values in registers.  Tokens arrive in shared memory 8 at a time through cp.async,
// double-buffered.  One block runs the rightward pass and then the leftward one of its
// kind and adds the second result to the first itself; while twice the blocks still fit the device in one
// wave, the directions run in two blocks that add into a zeroed output (two addends per element).  Either
// way results are bit-reproducible.  Where there are too few blocks to fill the device, a sequence is walked in several segments
// at a time (below).
//
// A token's decay enters as the factor d_t alone, never as a difference of summed logarithms, so a token that forgets
// everything (d_t = 0) leaves the others exact.  What bounds it is the walk's latency (two warps per block, one token
// after the other).  Three-part bfloat16 products in 64-token chunks took 9.98 ms for forward + backward at B=32, T=4096,
// H=12 against 12.2 ms here and the same 0.61 ms at T=196, but left five times this error (9e-7 for 1.6e-7 in the 2-norm).
//
// Decay gradient.  With p_t = r_t * (S_t gy_t) and q_t = k_t * (A_{t+1} v_t) (state parts
// only, elementwise over key channels),
//   d_t * dL/dd_t = sum_{tau>t} p>_tau - sum_{tau>=t} q>_tau + sum_{tau<t} p<_tau - sum_{tau<=t} q<_tau
// (every (source, reader) token pair whose decay product contains d_t, counted from the
// reader side minus the pairs that do not straddle t).  The sweeps write running sums of
// p and q (accumulated in double) to scratch; a last elementwise kernel combines them and
// applies d(d_t)/d(w_raw) = d_t * (-exp(w_raw)), which cancels the division by d_t.  gw is therefore off by the rounding
// of p and q over the whole sequence (9e-6 in the 2-norm at T=1024; sums kept in double to the end: the same).  Where d_t
// is zero in float so is the gradient; the difference is not taken there, since exp(w_raw) would multiply its rounding
// without bound.
//
// Reference being replaced: classification/mmcls_custom/models/backbones/cuda_v6/
// wkv6_cuda.cu:6-97 (forward), :99-346 (backward; its T <= 256 limit does not apply here).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <mutex>
#include "vrwkv_internal.h"

namespace wkv6 {

constexpr int N = 64;          // head size
constexpr int kBatch = 8;      // tokens per shared-memory batch (two batches of 10 KB per block: 11 blocks per SM)
constexpr int kParts = N / kBatch;   // threads that share one token's dot products
constexpr int kVecs = 5;       // r, k, v, gy, decay
enum Kind { KIND_Y = 0, KIND_GR = 1, KIND_GK = 2, KIND_GV = 3 };
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

__device__ __forceinline__ size_t slot_of(const Args& a, int pair, int dir, int bh, int i) {
    return ((static_cast<size_t>(pair * 2 + dir) * a.B * a.H + bh) * (a.segs - 1) + i) * kSlot;
}

// One pass of one kind over a segment (with segs = 1, the whole sequence).  kRow: thread owns a row (key channel) of
// the state, else a column (value channel).  kForward: direction of time.  kOut: how the result
// meets the other direction's: OUT_WRITE (first pass of a block), OUT_ADD (second pass of the same
// block), OUT_ATOMIC (the two directions run in two blocks and add into a zeroed output: exactly
// two addends per element, so the sum does not depend on their order).
enum OutMode { OUT_WRITE = 0, OUT_ADD = 1, OUT_ATOMIC = 2 };
template <int kKind, bool kForward, int kOut, bool kSegments>
__device__ __forceinline__ void sweep(const Args& a, Batch* buf, int b, int h, int seg, float u_self, const float* u_smem,
                                      float& gu_acc) {
    constexpr bool kRow = (kKind == KIND_GR || kKind == KIND_GK);
    constexpr int kA = (kKind == KIND_Y || kKind == KIND_GR) ? V_K : V_R;   // rank-1 update: alpha beta^T
    constexpr int kB_ = (kKind == KIND_Y || kKind == KIND_GR) ? V_V : V_G;
    constexpr int kC = kKind == KIND_Y ? V_R : kKind == KIND_GR ? V_G : kKind == KIND_GK ? V_V : V_K;   // read-out
    // the rightward state S> runs forward in time, its adjoint A> backward; mirrored for "<"
    constexpr bool kRightward = (kKind == KIND_Y || kKind == KIND_GR) ? kForward : !kForward;
    const int tid = threadIdx.x;
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
            for (int q = 0; q < (kBatch * N / 4) / N; ++q) {          // 256 chunks of 16 B, 64 threads
                const int chunk = q * N + tid;
                const int row = chunk >> 4, col4 = (chunk & 15) * 4;      // 16 chunks of 16 bytes per token row
                const int t = bt0 + row;
                if (t < T) cp_async16(&dst->vec[vsel][row][col4], src + base + static_cast<size_t>(t) * C + col4);
            }
        }
        cp_async_commit();
    };

    float X[N];
#pragma unroll
    for (int n = 0; n < N; ++n) X[n] = 0.f;
    const int before = !kSegments ? 0 : kForward ? seg : a.segs - 1 - seg;        // segments this direction has walked
    if (kSegments && before > 0) {
        constexpr int kPair = (kKind == KIND_Y || kKind == KIND_GR) ? 0 : 1;
        const float* from = a.states + slot_of(a, kPair, kForward ? 0 : 1, b * a.H + h, before - 1);
        if (kRow) {
#pragma unroll
            for (int n = 0; n < N; ++n) X[n] = from[n * N + tid];
        } else {
#pragma unroll
            for (int n4 = 0; n4 < N / 4; ++n4) {
                const float4 x = *reinterpret_cast<const float4*>(from + tid * N + 4 * n4);
                X[4 * n4] = x.x; X[4 * n4 + 1] = x.y; X[4 * n4 + 2] = x.z; X[4 * n4 + 3] = x.w;
            }
        }
    }
    double run = 0.0;

    issue(0, &buf[0]);
    for (int bi = 0; bi < n_batches; ++bi) {
        Batch* cur = &buf[bi & 1];
        if (bi + 1 < n_batches) {
            issue(bi + 1, &buf[(bi + 1) & 1]);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const int bt0 = (kForward ? bi : n_batches - 1 - bi) * kBatch;
        const int rows = min(kBatch, T - bt0);
        // decay in place, per-token scalars
        for (int row = 0; row < rows; ++row) cur->vec[V_D][row][tid] = expf(-expf(cur->vec[V_D][row][tid]));
        {
            const int row = tid / kParts, part = tid % kParts;
            float s1 = 0.f, s2 = 0.f;
            if (row < rows) {
#pragma unroll
                for (int n = part * kBatch; n < part * kBatch + kBatch; ++n) {
                    if (a.src[V_G] != nullptr) s1 += cur->vec[V_V][row][n] * cur->vec[V_G][row][n];
                    s2 += cur->vec[V_R][row][n] * u_smem[n] * cur->vec[V_K][row][n];
                }
            }
#pragma unroll
            for (int m = 1; m < kParts; m <<= 1) {
                s1 += __shfl_xor_sync(0xffffffffu, s1, m);
                s2 += __shfl_xor_sync(0xffffffffu, s2, m);
            }
            if (part == 0 && row < kBatch) { cur->vg[row] = s1; cur->ruk[row] = s2; }
        }
        __syncthreads();
        for (int step = 0; step < rows; ++step) {
            const int row = kForward ? step : rows - 1 - step;
            const int t = bt0 + row;
            const float4* cv = reinterpret_cast<const float4*>(cur->vec[kC][row]);
            float out = 0.f;
            if (kRow) {
                const float di = cur->vec[V_D][row][tid];
                const float ai = cur->vec[kA][row][tid];
                const float4* bv = reinterpret_cast<const float4*>(cur->vec[kB_][row]);
#pragma unroll
                for (int n4 = 0; n4 < N / 4; ++n4) {
                    const float4 c4 = cv[n4], b4 = bv[n4];
                    out += c4.x * X[4 * n4 + 0]; X[4 * n4 + 0] = fmaf(di, X[4 * n4 + 0], ai * b4.x);
                    out += c4.y * X[4 * n4 + 1]; X[4 * n4 + 1] = fmaf(di, X[4 * n4 + 1], ai * b4.y);
                    out += c4.z * X[4 * n4 + 2]; X[4 * n4 + 2] = fmaf(di, X[4 * n4 + 2], ai * b4.z);
                    out += c4.w * X[4 * n4 + 3]; X[4 * n4 + 3] = fmaf(di, X[4 * n4 + 3], ai * b4.w);
                }
            } else {
                const float bj = cur->vec[kB_][row][tid];
                const float4* av = reinterpret_cast<const float4*>(cur->vec[kA][row]);
                const float4* dv = reinterpret_cast<const float4*>(cur->vec[V_D][row]);
#pragma unroll
                for (int n4 = 0; n4 < N / 4; ++n4) {
                    const float4 c4 = cv[n4], a4 = av[n4], d4 = dv[n4];
                    out += c4.x * X[4 * n4 + 0]; X[4 * n4 + 0] = fmaf(d4.x, X[4 * n4 + 0], a4.x * bj);
                    out += c4.y * X[4 * n4 + 1]; X[4 * n4 + 1] = fmaf(d4.y, X[4 * n4 + 1], a4.y * bj);
                    out += c4.z * X[4 * n4 + 2]; X[4 * n4 + 2] = fmaf(d4.z, X[4 * n4 + 2], a4.z * bj);
                    out += c4.w * X[4 * n4 + 3]; X[4 * n4 + 3] = fmaf(d4.w, X[4 * n4 + 3], a4.w * bj);
                }
            }
            const size_t idx = base + static_cast<size_t>(t) * C + tid;
            // running sums for the decay gradient (state part only)
            if (kKind == KIND_GR) {
                run += static_cast<double>(cur->vec[V_R][row][tid] * out);
                a.cum[kRightward ? 0 : 2][idx] = static_cast<float>(run);
            }
            if (kKind == KIND_GK) {
                run += static_cast<double>(cur->vec[V_K][row][tid] * out);
                a.cum[kRightward ? 1 : 3][idx] = static_cast<float>(run);
            }
            // the bonus term lives in the rightward direction only
            if (kRightward) {
                if (kKind == KIND_Y) out += cur->ruk[row] * cur->vec[V_V][row][tid];
                if (kKind == KIND_GV) out += cur->ruk[row] * cur->vec[V_G][row][tid];
                if (kKind == KIND_GR) {
                    const float kvg = cur->vec[V_K][row][tid] * cur->vg[row];
                    out += u_self * kvg;
                    gu_acc += cur->vec[V_R][row][tid] * kvg;
                }
                if (kKind == KIND_GK) out += u_self * cur->vec[V_R][row][tid] * cur->vg[row];
            }
            float* dst = a.out[kKind] + idx;
            if (kOut == OUT_WRITE) *dst = out;
            else if (kOut == OUT_ADD) *dst += out;
            else atomicAdd(dst, out);
        }
        __syncthreads();   // the batch buffer is refilled two iterations later
    }
}

// How the directions (and segments) of a (batch, head, kind) are spread over blocks.
enum Mode {
    WHOLE,         // one block runs both directions in turn
    SPLIT,         // a block per direction (blockIdx.z); both add into a zeroed output
    SEGMENTS,      // a block per direction (blockIdx.z & 1) and segment (blockIdx.z >> 1), likewise
};
template <bool kBackward, Mode kMode>
__global__ void __launch_bounds__(N, 9) wkv6_sweep_kernel(const Args a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Batch* buf = reinterpret_cast<Batch*>(smem_raw);
    __shared__ float u_smem[N];
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H;
    const int kind = kBackward ? 1 + static_cast<int>(blockIdx.y) : 0;
    const int tid = threadIdx.x;
    u_smem[tid] = a.u[h * N + tid];
    __syncthreads();
    const float u_self = u_smem[tid];
    float gu = 0.f;
    constexpr bool kSeg = kMode == SEGMENTS;
    constexpr int kOut1 = kMode == WHOLE ? OUT_WRITE : OUT_ATOMIC, kOut2 = kMode == WHOLE ? OUT_ADD : OUT_ATOMIC;
    const bool first = kMode == WHOLE || (blockIdx.z & 1) == 0, second = kMode == WHOLE || (blockIdx.z & 1) == 1;
    const int seg = kSeg ? blockIdx.z >> 1 : 0;
    if (!kBackward) {
        if (first) sweep<KIND_Y, false, kOut1, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);   // leftward state first
        if (second) sweep<KIND_Y, true, kOut2, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
    } else if (kind == KIND_GR) {
        if (first) {
            sweep<KIND_GR, true, kOut1, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
            a.gu_part[(static_cast<size_t>(b) * a.segs + seg) * a.H * N + h * N + tid] = gu;            // the bonus lives in this direction
        }
        if (second) sweep<KIND_GR, false, kOut2, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
    } else if (kind == KIND_GK) {
        if (first) sweep<KIND_GK, false, kOut1, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);  // rightward adjoint: back in time
        if (second) sweep<KIND_GK, true, kOut2, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
    } else {
        if (first) sweep<KIND_GV, false, kOut1, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
        if (second) sweep<KIND_GV, true, kOut2, kSeg>(a, buf, b, h, seg, u_self, u_smem, gu);
    }
}

// ---- sequences in segments -------------------------------------------------------------------------------
// A few sequences leave most of the chip idle, and the walk's latency (0.5 us a token) is all their time.  Such a sequence is
// cut into segments that are walked side by side, still token by token: first the state that each segment would leave
// from zero, and its decay (wkv6_segment_state_kernel: the update without the read-out, half a token's work), then the states
// behind every segment, S_j = decay_j S_{j-1} + own_j (wkv6_segment_scan_kernel), then the sweeps, each from the state
// in front of its segment.  Decays are products of factors here too, so the accuracy is that of the whole walk.
__global__ void __launch_bounds__(N, 9) wkv6_segment_state_kernel(const Args a) {
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

// gw_raw = -exp(w_raw) * [ (P>_last - P>_t - Q>_t) + (P<_first - P<_t - Q<_t) ]
__global__ void wkv6_decay_grad_kernel(int B, int T, int C, const float* __restrict__ w_raw,
                                       const float* __restrict__ cp, const float* __restrict__ cq,
                                       const float* __restrict__ cp2, const float* __restrict__ cq2,
                                       float* __restrict__ gw) {
    const size_t total = static_cast<size_t>(B) * T * C;
    for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
         i += static_cast<size_t>(gridDim.x) * blockDim.x) {
        const size_t c = i % C;
        const size_t b = i / (static_cast<size_t>(T) * C);
        const size_t first = b * T * C + c, last = first + static_cast<size_t>(T - 1) * C;
        const float right = (cp[last] - cp[i]) - cq[i];
        const float left = (cp2[first] - cp2[i]) - cq2[i];
        const float e = expf(w_raw[i]);
        gw[i] = expf(-e) == 0.f ? 0.f : -e * (right + left);
    }
}

// gu[c] = sum over batch (and segments) of gu_part, fixed order
__global__ void wkv6_bonus_grad_kernel(int B, int C, const float* __restrict__ part, float* __restrict__ gu) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    float acc = 0.f;
    for (int b = 0; b < B; ++b) acc += part[static_cast<size_t>(b) * C + c];
    gu[c] = acc;
}

// Blocks of the sweep kernel that fit the device at once (0 if the kernel cannot be configured).
static int resident_blocks() {
    static std::mutex lock;
    static int cached[64];
    static bool known[64];
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    std::lock_guard<std::mutex> guard(lock);
    if (!known[dev]) {
        const int smem = static_cast<int>(2 * sizeof(Batch));
        bool ok = true;
        for (const auto kernel : {wkv6_sweep_kernel<false, WHOLE>, wkv6_sweep_kernel<false, SPLIT>, wkv6_sweep_kernel<false, SEGMENTS>,
                                  wkv6_sweep_kernel<true, WHOLE>, wkv6_sweep_kernel<true, SPLIT>, wkv6_sweep_kernel<true, SEGMENTS>})
            ok = ok && cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) == cudaSuccess;
        int per_sm = 0, sms = 0;
        ok = ok && cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wkv6_sweep_kernel<true, WHOLE>, N, smem) == cudaSuccess;
        ok = ok && cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
        if (!ok) cudaGetLastError();
        cached[dev] = ok ? per_sm * sms : 0;
        known[dev] = true;
    }
    return cached[dev];
}
static bool configure() { return resident_blocks() > 0; }

// The two directions of a (batch, head, kind) go to two blocks when that still fits the device in
// one wave: the walks are latency-bound, so twice the blocks is close to twice the speed then.
static bool split_directions(int blocks) { return 2 * blocks <= resident_blocks(); }

struct Plan {
    int segs, len;
};
// How many segments a sequence is walked in, from the sizes alone (so a sequence's last bits may depend on how many others are in
// the call).  The device holds nine blocks per SM, but three already hide each other's latency, and the states in front of the
// segments cost half a walk (a third in the backward, whose three kinds share them).  So: segments until there are `fill`
// blocks, and the whole walk where fewer than three come out or a segment would be shorter than a few batches.
// us, whole / segments, forward and forward + backward: H=12 B=1 T=1024 515 / 62, 1053 / 194; T=196 105 / 34, 228 / 116; H=6 B=8
// T=512 264 / 97, 560 / 319.  Where the line lies: forward, 360 blocks (B H = 180, T=400) 223 / 211, 432 blocks 224 / 235;
// backward, 444 blocks (B H = 74, T=800) 867 / 644 for the pair, 720 blocks (B H = 120, T=400) 508 / 599.
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
    wkv6_segment_state_kernel<<<dim3(a.B * a.H, a.segs - 1, 2 * pairs), N, 0, stream>>>(a);
    wkv6_segment_scan_kernel<<<dim3(2 * pairs * a.B * a.H, N * N / 256), 256, 0, stream>>>(a);
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
    if (!configure()) return -1;
    const Plan pl = workspace ? make_plan(B, T, H, 1) : Plan{1, T};
    Args a{};
    a.B = B; a.T = T; a.H = H;
    a.src[V_R] = r; a.src[V_K] = k; a.src[V_V] = v; a.src[V_G] = nullptr; a.src[V_D] = w_raw;
    a.u = u;
    a.out[KIND_Y] = y;
    a.segs = pl.segs; a.seg_len = pl.len;
    a.states = pl.segs > 1 ? reinterpret_cast<float*>(static_cast<char*>(workspace) + kHead) : nullptr;
    const bool split = pl.segs > 1 || split_directions(B * H);
    if (split) cudaMemsetAsync(y, 0, static_cast<size_t>(B) * T * H * N * sizeof(float), stream);
    if (pl.segs > 1) run_segment_states(a, 1, stream);
    const auto kernel = pl.segs > 1 ? wkv6_sweep_kernel<false, SEGMENTS> : split ? wkv6_sweep_kernel<false, SPLIT> : wkv6_sweep_kernel<false, WHOLE>;
    kernel<<<dim3(B * H, 1, split ? 2 * pl.segs : 1), N, 2 * sizeof(Batch), stream>>>(a);
    return pl.segs > 1 ? 3 : 1;
}

int backward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
             const float* u, const float* gy, float* gr, float* gk, float* gv, float* gw, float* gu,
             void* workspace, cudaStream_t stream) {
    if (!configure()) return -1;
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
    const int kinds = gv ? 3 : 2;      // gv == nullptr: the caller gets gv elsewhere (the kinds are gr, gk, gv in this order)
    const bool split = pl.segs > 1 || split_directions(kinds * B * H);
    if (split) {
        cudaMemsetAsync(gr, 0, E * sizeof(float), stream);
        cudaMemsetAsync(gk, 0, E * sizeof(float), stream);
        if (gv) cudaMemsetAsync(gv, 0, E * sizeof(float), stream);
    }
    if (pl.segs > 1) run_segment_states(a, 2, stream);
    const auto kernel = pl.segs > 1 ? wkv6_sweep_kernel<true, SEGMENTS> : split ? wkv6_sweep_kernel<true, SPLIT> : wkv6_sweep_kernel<true, WHOLE>;
    kernel<<<dim3(B * H, kinds, split ? 2 * pl.segs : 1), N, 2 * sizeof(Batch), stream>>>(a);
    if (pl.segs > 1) {
        const size_t threads = static_cast<size_t>(B) * pl.segs * ((pl.len + kPiece - 1) / kPiece) * C;
        wkv6_segment_decay_grad_kernel<<<static_cast<unsigned>((threads + 255) / 256), 256, 0, stream>>>(a, gw);
    } else {
        const int blocks = static_cast<int>(std::min<size_t>((E + 255) / 256, 148 * 16));
        wkv6_decay_grad_kernel<<<blocks, 256, 0, stream>>>(B, T, C, w_raw, a.cum[0], a.cum[1], a.cum[2], a.cum[3], gw);
    }
    wkv6_bonus_grad_kernel<<<(C + 127) / 128, 128, 0, stream>>>(B * pl.segs, C, a.gu_part, gu);
    return pl.segs > 1 ? 5 : 3;
}

}  // namespace wkv6
