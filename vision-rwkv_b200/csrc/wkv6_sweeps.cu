// WKV6 forward (head size 64, bidirectional) as exact sequential state sweeps, fp32, any T, no scratch memory: what
// vrwkv_wkv6_forward_f32, whose signature has no workspace, runs.  (vrwkv_wkv6_forward with exact = 1 gives the same
// accuracy from the chunked kernels of wkv6_chunk.cu, several times faster.)
//
// Per (batch, head) the operator carries a 64 x 64 state S[key i][value j]
//   rightward  S>_{t+1} = diag(d_t) S>_t + k_t v_t^T      y_t  = r_t^T (S>_t + diag(u) k_t v_t^T)
//   leftward   S<_{t-1} = diag(d_t) S<_t + k_t v_t^T      y_t += r_t^T S<_t
// with d_t = exp(-exp(w_raw_t)).  A block of 64 threads owns the columns (thread = value channel) of one
// state, so the read-out is a sum inside the thread, and keeps its 64 state values in registers.  Tokens arrive
// in shared memory 8 at a time through cp.async, double-buffered.  One block runs both directions and
// adds the second result to the first itself; while twice the blocks still fit the device in one wave, the
// directions run in two blocks that add into a zeroed output (two addends per element: bit-reproducible).
//
// Reference being replaced: classification/mmcls_custom/models/backbones/cuda_v6/wkv6_cuda.cu:6-97.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include "vrwkv_internal.h"

namespace wkv6 {

constexpr int N = 64;          // head size
constexpr int kBatch = 8;      // tokens per shared-memory batch
constexpr int kParts = N / kBatch;   // threads that share one token's dot products
constexpr int kVecs = 4;       // r, k, v, decay
enum Vec { V_R = 0, V_K = 1, V_V = 2, V_D = 3 };

struct Args {
    int B, T, H;
    const float* src[kVecs];   // r, k, v, w_raw  -- (B, T, 64 H)
    const float* u;            // (H, 64)
    float* y;
};

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
    float ruk[kBatch];   // sum_i r_t[i] u[i] k_t[i]
};

// One pass over the whole sequence.  kForward: direction of time.  kOut: how the result meets the other
// direction's: OUT_WRITE (first pass of a block), OUT_ADD (second pass of the same block), OUT_ATOMIC (two blocks).
enum OutMode { OUT_WRITE = 0, OUT_ADD = 1, OUT_ATOMIC = 2 };
template <bool kForward, int kOut>
__device__ __forceinline__ void sweep(const Args& a, Batch* buf, int b, int h, const float* u_smem) {
    const int tid = threadIdx.x;
    const int T = a.T, C = a.H * N;
    const size_t base = (static_cast<size_t>(b) * T) * C + static_cast<size_t>(h) * N;
    const int n_batches = (T + kBatch - 1) / kBatch;

    auto issue = [&](int bi, Batch* dst) {
        const int bt0 = (kForward ? bi : n_batches - 1 - bi) * kBatch;
#pragma unroll
        for (int vsel = 0; vsel < kVecs; ++vsel) {
#pragma unroll
            for (int q = 0; q < (kBatch * N / 4) / N; ++q) {
                const int chunk = q * N + tid;
                const int row = chunk >> 4, col4 = (chunk & 15) * 4;      // 16 chunks of 16 bytes per token row
                const int t = bt0 + row;
                if (t < T) cp_async16(&dst->vec[vsel][row][col4], a.src[vsel] + base + static_cast<size_t>(t) * C + col4);
            }
        }
        cp_async_commit();
    };

    float X[N];
#pragma unroll
    for (int n = 0; n < N; ++n) X[n] = 0.f;

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
            float s = 0.f;
            if (row < rows) {
#pragma unroll
                for (int n = part * kBatch; n < part * kBatch + kBatch; ++n) s += cur->vec[V_R][row][n] * u_smem[n] * cur->vec[V_K][row][n];
            }
#pragma unroll
            for (int m = 1; m < kParts; m <<= 1) s += __shfl_xor_sync(0xffffffffu, s, m);
            if (part == 0 && row < kBatch) cur->ruk[row] = s;
        }
        __syncthreads();
        for (int step = 0; step < rows; ++step) {
            const int row = kForward ? step : rows - 1 - step;
            const float4* rv = reinterpret_cast<const float4*>(cur->vec[V_R][row]);
            const float4* kv = reinterpret_cast<const float4*>(cur->vec[V_K][row]);
            const float4* dv = reinterpret_cast<const float4*>(cur->vec[V_D][row]);
            const float vj = cur->vec[V_V][row][tid];
            float out = 0.f;
#pragma unroll
            for (int n4 = 0; n4 < N / 4; ++n4) {
                const float4 r4 = rv[n4], k4 = kv[n4], d4 = dv[n4];
                out += r4.x * X[4 * n4 + 0]; X[4 * n4 + 0] = fmaf(d4.x, X[4 * n4 + 0], k4.x * vj);
                out += r4.y * X[4 * n4 + 1]; X[4 * n4 + 1] = fmaf(d4.y, X[4 * n4 + 1], k4.y * vj);
                out += r4.z * X[4 * n4 + 2]; X[4 * n4 + 2] = fmaf(d4.z, X[4 * n4 + 2], k4.z * vj);
                out += r4.w * X[4 * n4 + 3]; X[4 * n4 + 3] = fmaf(d4.w, X[4 * n4 + 3], k4.w * vj);
            }
            if (kForward) out += cur->ruk[row] * vj;      // the bonus term lives in the rightward direction only
            float* dst = a.y + base + static_cast<size_t>(bt0 + row) * C + tid;
            if (kOut == OUT_WRITE) *dst = out;
            else if (kOut == OUT_ADD) *dst += out;
            else atomicAdd(dst, out);
        }
        __syncthreads();   // the batch buffer is refilled two iterations later
    }
}

// kSplit: blockIdx.z picks the direction and the two blocks of a (batch, head) add into a zeroed
// output; otherwise one block runs both directions in turn.
template <bool kSplit>
__global__ void __launch_bounds__(N, 9) wkv6_sweep_kernel(const Args a) {
    __shared__ __align__(16) Batch buf[2];
    __shared__ float u_smem[N];
    const int b = blockIdx.x / a.H, h = blockIdx.x % a.H;
    u_smem[threadIdx.x] = a.u[h * N + threadIdx.x];
    __syncthreads();
    if (!kSplit || blockIdx.z == 0) sweep<false, kSplit ? OUT_ATOMIC : OUT_WRITE>(a, buf, b, h, u_smem);
    if (!kSplit || blockIdx.z == 1) sweep<true, kSplit ? OUT_ATOMIC : OUT_ADD>(a, buf, b, h, u_smem);
}

// Blocks of the sweep kernel that fit the device at once (0 if it cannot be asked).
static int resident_blocks() {
    static int cached[64];
    static bool known[64];
    int dev = 0;
    cudaGetDevice(&dev);
    dev &= 63;
    if (!known[dev]) {
        int per_sm = 0, sms = 0;
        const bool ok = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, wkv6_sweep_kernel<false>, N, 0) == cudaSuccess &&
                        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess;
        if (!ok) cudaGetLastError();
        cached[dev] = ok ? per_sm * sms : 0;
        known[dev] = true;
    }
    return cached[dev];
}

int forward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
            const float* u, float* y, cudaStream_t stream) {
    const int resident = resident_blocks();
    if (resident <= 0) return -1;
    Args a{B, T, H, {r, k, v, w_raw}, u, y};
    if (2 * B * H <= resident) {
        cudaMemsetAsync(y, 0, static_cast<size_t>(B) * T * H * N * sizeof(float), stream);
        wkv6_sweep_kernel<true><<<dim3(B * H, 1, 2), N, 0, stream>>>(a);
    } else {
        wkv6_sweep_kernel<false><<<dim3(B * H), N, 0, stream>>>(a);
    }
    return 1;
}

}  // namespace wkv6
