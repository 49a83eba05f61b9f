// WKV6 forward on the 5th-generation tensor cores (tcgen05 + TMEM), bf16 operands, fp32 state, for callers of
// vrwkv_wkv6_forward_tc_* whose workspace holds nothing but the status word.  (With the workspace that
// vrwkv_wkv6_forward_workspace_bytes asks for, those entry points run the chunked kernels of wkv6_chunk.cu.)
//
// Per (batch, head) the 64 x 64 state S[key][value] lives in tensor memory as its transpose
// (TMEM lane = value channel, column = key channel, fp32).  The sequence is walked 16 tokens
// at a time; for every 16-token block, with a_t = sum of log-decays of the block's tokens
// before t and A = a_16, all matrix work runs as UMMA instructions (M = 128, fp32 accumulate):
//
//   P (16 x 16)    = Rs (16 x 64) . Kb^T        Rs[t][i] = r_t[i] e^{a_t[i]},  Kb[s][i] = k_s[i] e^{-a_{s+1}[i]}
//                    masked to s < t, the diagonal replaced by the bonus  sum_i r_t[i] u[i] k_t[i]
//   y^T (64 x 16)  = S^T (64 x 64, bf16 copy) . Rs^T  +  V^T (64 x 16) . P^T
//   S^T (64 x 64) += V^T (64 x 16) . Ks         Ks[t][i] = k_t[i] e^{A[i] - a_{t+1}[i]}
//                    after S^T was scaled by e^{A[i]} per key column on its way through registers
//
// The rows of Rs also sit in rows 64..79 of the state operand, so the score product is the same
// instruction shape as the read-out and lands in TMEM lanes 64..79, which an otherwise idle warp
// owns.  e^{-a_{s+1}} grows with the decay; a block whose accumulated log-decay exceeds 80 in any
// channel evaluates its 16 x 16 scores pairwise on the CUDA cores instead (every exponent <= 0
// there), so nothing overflows however strong the decay is.  The leftward direction is the same
// walk over the reversed sequence without the bonus.  The state never leaves the SM: per block it
// makes one round trip TMEM -> registers -> TMEM (decay) and leaves a bf16 copy in shared memory as
// the next A operand.
//
// Data movement: r, k, v, w tiles (16 tokens x 64 channels) arrive by TMA, the next block's while
// the current one is on the tensor core; y tiles leave by TMA reduce-add.  All bf16 operand writes
// are 4-, 8- or 16-byte shared stores, which fixes the thread-to-element maps of the operand phase.
//
// Accuracy is that of bf16 operands with fp32 accumulation (about 1e-2 of max|y|).
//
// Reference being replaced: classification/mmcls_custom/models/backbones/cuda_v6/wkv6_cuda.cu:6-97.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <atomic>
#include <mutex>
#include <cstdint>
#include "launch.h"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"

namespace wkv6tc {

constexpr int N = 64;            // head size
constexpr int SC = 16;           // tokens per block
constexpr uint32_t kWaitLimit = 1u << 20;
constexpr uint32_t kTmemCols = 128;   // S^T: columns 0..63, y^T: 64..79, P^T: 80..95
constexpr float kMaxLogDecay = 80.f;  // per block and channel, for the tensor-core score product

struct Args {
    int B, T, H;
    const float* r;
    const float* k;
    const float* v;
    const float* w;      // raw decay input
    const float* u;      // (H, 64)
    float* y;
    unsigned* status;    // set to 1 if a bounded wait ran out
    unsigned* mirror;    // host-visible copy (may be null)
    unsigned limit;      // polls of a wait
    unsigned extra;      // test only: bytes that the tiles' barriers wait for and no copy brings
};

using sm100::smem_u32;

// log of a token's decay, bounded at -104: e^-104 is zero in float32 already, and so bounded the running sums over a block
// keep their smaller terms to 1e-4 (and stay finite) whatever a token's decay is.  NaN stays NaN.
__device__ __forceinline__ float log_decay(float w) {
    float x;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(x) : "f"(w), "f"(4.6444f));
    return -__expf(x);
}


// canonical K-major, no swizzle: element (row, k) of a [rows x K] bf16 operand
__device__ __forceinline__ int op_index(int rows, int row, int k) { return (k >> 3) * (rows * 8) + row * 8 + (k & 7); }

__device__ __forceinline__ uint64_t make_desc(uint32_t addr, uint32_t lbo_bytes, uint32_t sbo_bytes) {
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3FFF);
    d |= static_cast<uint64_t>((lbo_bytes >> 4) & 0x3FFF) << 16;
    d |= static_cast<uint64_t>((sbo_bytes >> 4) & 0x3FFF) << 32;
    d |= static_cast<uint64_t>(1) << 46;        // descriptor version of this architecture
    return d;
}
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ constexpr uint32_t instr_desc(int m, int n) {
    // fp32 accumulator, bf16 A and B, both K-major
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&x)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7]), "=r"(x[8]),
          "=r"(x[9]), "=r"(x[10]), "=r"(x[11]), "=r"(x[12]), "=r"(x[13]), "=r"(x[14]), "=r"(x[15])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 p = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&p);
}
__device__ __forceinline__ float bf16_round(float x) { return __bfloat162float(__float2bfloat16(x)); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}
// y tile += shared tile (fp32), through the copy engine
__device__ __forceinline__ void tma_reduce_add_3d(const CUtensorMap* map, const void* src, int x, int y, int z) {
    asm volatile("cp.reduce.async.bulk.tensor.3d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4}], [%1];" ::
                     "l"(reinterpret_cast<uint64_t>(map)),
                 "r"(smem_u32(src)), "r"(x), "r"(y), "r"(z)
                 : "memory");
}
// ---- the kernel ---------------------------------------------------------------------------------------
// What must be serial is only
//     state round trip (block n)  ->  read-out / update products (block n)  ->  round trip (n + 1).
// Here one CTA walks one direction of one (batch, head) with nine warps in three roles:
//   producers (warps 3, 6..12, two groups of four): group g prepares the operands of the blocks g, g+2, ...
//       (log-decay sums, scalings, bf16 rounding, the pairwise scores of a strongly decaying block)
//       into operand set g, two block periods ahead of their use;
//   loader (warp 13): the TMA loads of block n+2 as soon as the producers have read block n (issuing
//       the four copies costs several hundred cycles, too many for a thread the others wait for);
//   control (warp 2, owner of TMEM lanes 64..95): issues all tensor-core work; between the score
//       product and the main products it masks the 16 x 16 scores into the P operand;
//   state (warps 0, 1, 4, 5; each owns 32 TMEM lanes x 32 state columns): the round trip, and, while
//       the main products of block n run, the output tile of block n-1 (TMEM -> shared -> TMA
//       reduce-add into y, which the host zeroed; the two directions of a head are two CTAs).
// Hand-overs are mbarriers (operands ready / operand set free / products done) and two named
// barriers; every wait is bounded.
constexpr int kPThreads = 448;    // 4 state warps, 1 control warp, 8 producer warps, 1 loader warp
constexpr int kBarRound = 1;     // named barrier: state + control, 160 threads
constexpr int kBarYTile = 2;     // state, 128 threads
constexpr int kBarProd = 3;      // producer group 0 (128 threads); group 1 uses the next id

struct OpSet {
    __nv_bfloat16 opR[16 * 64];       // B of the read-out; through a base 1 KB lower also the A of the scores (rows 64..79)
    __nv_bfloat16 opKb[16 * 64];      // B of the scores: rows = token s, K = key
    __nv_bfloat16 opK[64 * 16];       // B of the update: rows = key, K = token
    __nv_bfloat16 opV[64 * 16];       // A of the update and of the in-block part (rows 64..127 of the instruction: whatever follows)
    __nv_bfloat16 opP[16 * 16];       // B of the in-block part: rows = token t, K = token s
    float dtot[N];
    float diag[SC];
    uint32_t pairwise;                // the producers wrote opP themselves (strong decay)
    uint32_t pad[15];
};

struct __align__(1024) SmemP {
    __nv_bfloat16 opS[64 * 64];       // A of the read-out: S^T, rows = value, K = key (rows 64..127: the bytes that follow)
    OpSet sets[2];
    float raw[2][4][SC][N];           // r, k, v, w of two blocks in flight
    float ytile[2][SC][N];
    float acum[2][SC + 1][N];         // a_0 .. a_16 per key channel, one array per producer group
    float u[N];
    uint64_t raw_full[2];
    uint64_t raw_free[2];
    uint64_t ops_ready[2];
    uint64_t ops_free[2];
    uint64_t bar_main;
    uint64_t bar_score, drained;
    uint32_t tmem_base;
};

__device__ __forceinline__ bool elect_one() {
    uint32_t pred;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(pred));
    return pred != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool named_bar_or(int id, int threads, bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, %2, %3, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(static_cast<uint32_t>(pred)), "r"(id), "r"(threads)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void tmem_ld8_issue(uint32_t taddr, uint32_t (&x)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(x[0]), "=r"(x[1]), "=r"(x[2]), "=r"(x[3]), "=r"(x[4]), "=r"(x[5]), "=r"(x[6]), "=r"(x[7])
                 : "r"(taddr));
}

// r, k, v staging tiles hold float32 or, for callers whose activations are bfloat16, bfloat16 in the
// first half of the same space (w stays float32).  bfloat16 elements are read as the 32-bit word
// of a channel pair, never as 2-byte accesses.
template <bool kHalfIn>
__device__ __forceinline__ float4 raw_ld4(const float* tile, int row, int c0) {
    if (!kHalfIn) return *reinterpret_cast<const float4*>(tile + row * N + c0);
    const uint2 w = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(tile) + row * N + c0);
    return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                       __uint_as_float(w.y & 0xffff0000u));
}
template <bool kHalfIn>
__device__ __forceinline__ float raw_ld1(const float* tile, int row, int c) {
    if (!kHalfIn) return tile[row * N + c];
    const uint32_t word = reinterpret_cast<const uint32_t*>(tile)[(row * N + c) >> 1];
    return __uint_as_float((c & 1) ? (word & 0xffff0000u) : (word << 16));
}

template <bool kHalfIn>
__global__ void __launch_bounds__(kPThreads, 2)
wkv6_tc_pipelined_kernel(const Args a, const __grid_constant__ CUtensorMap map_r, const __grid_constant__ CUtensorMap map_k,
                         const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_w,
                         const __grid_constant__ CUtensorMap map_y) {
    wait_for_launch_before();
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    SmemP& s = *reinterpret_cast<SmemP*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int bh = blockIdx.x >> 1;
    const bool rightward = (blockIdx.x & 1) == 0;
    const int b = bh / a.H, h = bh % a.H;
    const int T = a.T, C = a.H * N;
    const size_t base = static_cast<size_t>(b) * T * C + static_cast<size_t>(h) * N;
    const int n_steps = (T + SC - 1) / SC;

    const bool is_state = (warp & 3) < 2 && warp < 8;          // warps 0, 1, 4, 5
    const bool is_control = warp == 2;
    const bool is_loader = warp == 13;
    const bool is_producer = !is_state && !is_control && !is_loader;   // warps 3, 6..12
    const int pid = ((warp == 3) ? 0 : warp - 5) * 32 + lane;   // producers: 0..255

    auto tile_start = [&](int step) { return rightward ? step * SC : T - SC * (step + 1); };
    auto row_of = [&](int t) { return rightward ? t : SC - 1 - t; };

    if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            sm100::mbar_init(&s.raw_full[i], 1);
            sm100::mbar_init(&s.raw_free[i], 1);
            sm100::mbar_init(&s.ops_ready[i], 1);
            sm100::mbar_init(&s.ops_free[i], 1);
        }
        sm100::mbar_init(&s.bar_main, 1);
        sm100::mbar_init(&s.bar_score, 1);
        sm100::mbar_init(&s.drained, 1);
        sm100::mbar_init_fence();
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&s.tmem_base)),
                     "r"(kTmemCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    if (tid < N) s.u[tid] = a.u[h * N + tid];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s.tmem_base;
    const uint32_t lane_addr = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);   // this warp's 32 TMEM lanes

    bool failed = false;
    auto wait_on = [&](uint64_t* bar, uint32_t parity) {
        if (!failed && !sm100::mbar_wait(bar, parity, a.limit)) { failed = true; report_failure(a.status, a.mirror, 1u); }
    };

    if (is_producer) {
        // =================================== producers ===================================
        // two groups of four warps; group g prepares the blocks q = g, g + 2, ... into operand set g from staging
        // slot g, with its own running-sum array and named barrier, so that a block has two block periods to get ready
        const int group = pid >> 7, gid = pid & 127;
        const int bar_id = kBarProd + group;
        float(&acum)[SC + 1][N] = s.acum[group];
        OpSet& set = s.sets[group];
        float(&raw)[4][SC][N] = s.raw[group];
        for (int q = group; q < n_steps; q += 2) {
            const uint32_t use_parity = (q >> 1) & 1;
            wait_on(&s.raw_full[group], use_parity);
            // ---- phase A: running sums of the log-decays, a_t[c] for t = 0..16; thread = (key channel, half of the
            //      block), the two halves of a channel in one warp so that the first half's total travels by shuffle ----
            {
                const int c = (gid >> 5) * 16 + (lane & 15), half = lane >> 4;
                float wv[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) wv[j] = raw[3][row_of(half * 8 + j)][c];
                float pre[8], run = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    run += (q * SC + half * 8 + j < T) ? log_decay(wv[j]) : 0.f;
                    pre[j] = run;
                }
                const float up = __shfl_up_sync(0xffffffffu, run, 16);
                const float before = half ? up : 0.f;
                if (half == 0) acum[0][c] = 0.f;
#pragma unroll
                for (int j = 0; j < 8; ++j) acum[half * 8 + j + 1][c] = pre[j] + before;
            }
            if (q >= 2) wait_on(&s.ops_free[group], use_parity ^ 1u);   // the products of block q-2 are done with this set
            sm100::named_bar_sync(bar_id, 128);
            // ---- job 1: work item = (token t, 4 key channels): Rs, Kb, bonus; two items per thread ----
#pragma unroll
            for (int rep = 0; rep < 2; ++rep) {
                const int it = gid + 128 * rep;
                const int t = it >> 4, c0 = (it & 15) * 4, row = row_of(t);
                const float4 rv = raw_ld4<kHalfIn>(&raw[0][0][0], row, c0);
                const float4 kv = raw_ld4<kHalfIn>(&raw[1][0][0], row, c0);
                const float4 at = *reinterpret_cast<const float4*>(&acum[t][c0]);
                const float4 at1 = *reinterpret_cast<const float4*>(&acum[t + 1][c0]);
                const float4 aA = *reinterpret_cast<const float4*>(&acum[SC][c0]);
                const float rvv[4] = {rv.x, rv.y, rv.z, rv.w}, kvv[4] = {kv.x, kv.y, kv.z, kv.w};
                const float a0[4] = {at.x, at.y, at.z, at.w}, a1[4] = {at1.x, at1.y, at1.z, at1.w};
                const float aa[4] = {aA.x, aA.y, aA.z, aA.w};
                float rs[4], kb[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    rs[i] = rvv[i] * __expf(a0[i]);
                    kb[i] = (aa[i] < -kMaxLogDecay) ? 0.f : kvv[i] * __expf(-a1[i]);
                }
                *reinterpret_cast<uint2*>(&set.opR[op_index(16, t, c0)]) = make_uint2(pack_bf16(rs[0], rs[1]), pack_bf16(rs[2], rs[3]));
                *reinterpret_cast<uint2*>(&set.opKb[op_index(16, t, c0)]) = make_uint2(pack_bf16(kb[0], kb[1]), pack_bf16(kb[2], kb[3]));
                if (rightward) {       // the bonus exists in this direction only
                    const float4 uu = *reinterpret_cast<const float4*>(&s.u[c0]);
                    float bonus = (rv.x * uu.x * kv.x + rv.y * uu.y * kv.y) + (rv.z * uu.z * kv.z + rv.w * uu.w * kv.w);
                    bonus += __shfl_xor_sync(0xffffffffu, bonus, 1);
                    bonus += __shfl_xor_sync(0xffffffffu, bonus, 2);
                    bonus += __shfl_xor_sync(0xffffffffu, bonus, 4);
                    bonus += __shfl_xor_sync(0xffffffffu, bonus, 8);
                    if ((it & 15) == 0) set.diag[t] = bonus;
                } else if ((it & 15) == 0) {
                    set.diag[t] = 0.f;
                }
            }
            // ---- job 2: work item = (key channel, quarter of the block): Ks, V^T, e^A; two items per thread ----
            bool big = false;
#pragma unroll
            for (int rep = 0; rep < 2; ++rep) {
                const int it = gid + 128 * rep;
                const int c = it & 63, quarter = it >> 6;
                const float A = acum[SC][c];
                big = big || (A < -kMaxLogDecay);
                float kh[4], vv[4], a1[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int t = quarter * 4 + j, row = row_of(t);
                    a1[j] = acum[t + 1][c];
                    kh[j] = raw_ld1<kHalfIn>(&raw[1][0][0], row, c);
                    vv[j] = raw_ld1<kHalfIn>(&raw[2][0][0], row, c);
                }
                if (quarter == 0) set.dtot[c] = __expf(A);
#pragma unroll
                for (int j = 0; j < 4; ++j) kh[j] *= __expf(A - a1[j]);
                *reinterpret_cast<uint2*>(&set.opK[op_index(64, c, quarter * 4)]) = make_uint2(pack_bf16(kh[0], kh[1]), pack_bf16(kh[2], kh[3]));
                *reinterpret_cast<uint2*>(&set.opV[op_index(64, c, quarter * 4)]) = make_uint2(pack_bf16(vv[0], vv[1]), pack_bf16(vv[2], vv[3]));
            }
            const bool pairwise = named_bar_or(bar_id, 128, big);   // also orders diag before the loop below
            if (pairwise) {
                // ---- strong decay: the 16 x 16 scores pairwise in fp32, every exponent <= 0 ----
                for (int rep = 0; rep < 2; ++rep) {
                    const int it = gid + 128 * rep;
                    const int t = it >> 4, sidx = it & 15;
                    const int row_t = row_of(t), row_s = row_of(sidx);
                    float acc = 0.f;
                    if (sidx < t) {
#pragma unroll 8
                        for (int i = 0; i < N; ++i)
                            acc += raw_ld1<kHalfIn>(&raw[0][0][0], row_t, i) * raw_ld1<kHalfIn>(&raw[1][0][0], row_s, i) *
                                   __expf(acum[t][i] - acum[sidx + 1][i]);
                    } else if (sidx == t) {
                        acc = set.diag[t];
                    }
                    // one 4-byte store per lane pair: 2-byte shared stores are slow
                    const float other = __shfl_xor_sync(0xffffffffu, acc, 1);
                    if ((sidx & 1) == 0) *reinterpret_cast<uint32_t*>(&set.opP[op_index(16, t, sidx)]) = pack_bf16(acc, other);
                }
            }
            if (gid == 0) set.pairwise = pairwise ? 1u : 0u;
            sm100::fence_proxy_async_smem();
            sm100::named_bar_sync(bar_id, 128);
            if (gid == 0) {
                mbar_arrive(&s.ops_ready[group]);
                mbar_arrive(&s.raw_free[group]);              // every producer of the group is done reading this staging slot
            }
        }
    } else if (is_loader) {
        // =================================== loader ===================================
        if (lane == 0) {
            sm100::prefetch_tensormap(&map_r);
            sm100::prefetch_tensormap(&map_k);
            sm100::prefetch_tensormap(&map_v);
            sm100::prefetch_tensormap(&map_w);
            int step = 0;
            for (; step < n_steps; ++step) {
                const int slot = step & 1, y0 = tile_start(step);
                if (step >= 2) {
                    wait_on(&s.raw_free[slot], ((step >> 1) & 1) ^ 1u);
                    wait_on(&s.raw_full[slot], ((step >> 1) & 1) ^ 1u);      // over, unless the readers gave up waiting for it
                }
                if (failed) break;       // nothing is asked for where a copy is missing
                sm100::mbar_expect_tx(&s.raw_full[slot], (kHalfIn ? 3 * 2 + 4 : 4 * 4) * SC * N + a.extra);
                sm100::tma_load_3d(&s.raw[slot][0][0][0], &map_r, &s.raw_full[slot], h * N, y0, b);
                sm100::tma_load_3d(&s.raw[slot][1][0][0], &map_k, &s.raw_full[slot], h * N, y0, b);
                sm100::tma_load_3d(&s.raw[slot][2][0][0], &map_v, &s.raw_full[slot], h * N, y0, b);
                sm100::tma_load_3d(&s.raw[slot][3][0][0], &map_w, &s.raw_full[slot], h * N, y0, b);
            }
            // no copy is left behind
            for (int last = step < 2 ? 0 : step - 2; last < step; ++last) sm100::mbar_wait(&s.raw_full[last & 1], (last >> 1) & 1, failed ? a.limit / 64 : a.limit);
        }
    } else if (is_control) {
        // =================================== control ===================================
        uint32_t score_parity = 0;
        // descriptors are formed by the whole warp (warp-uniform values), one elected lane issues
        const uint64_t d_state = make_desc(smem_u32(s.opS), 1024, 128);
        for (int m = 0; m < n_steps; ++m) {
            const int slot = m & 1;
            OpSet& set = s.sets[slot];
            const uint64_t d_r = make_desc(smem_u32(set.opR), 256, 128);
            const uint64_t d_ra = make_desc(smem_u32(set.opR) - 1024, 256, 128);      // rows 64..79 = Rs
            const uint64_t d_kb = make_desc(smem_u32(set.opKb), 256, 128);
            const uint64_t d_v = make_desc(smem_u32(set.opV), 1024, 128);
            const uint64_t d_p = make_desc(smem_u32(set.opP), 256, 128);
            const uint64_t d_k = make_desc(smem_u32(set.opK), 1024, 128);
            wait_on(&s.ops_ready[slot], (m >> 1) & 1);
            __syncwarp();      // one answer for all lanes, also where a wait ran out
            const bool pairwise = set.pairwise != 0;
            if (!pairwise) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
#pragma unroll
                    for (int ks = 0; ks < N / 16; ++ks)      // a K step of 16 = 512 bytes = 32 descriptor units
                        umma_bf16(tmem + 80, d_ra + 32 * ks, d_kb + 32 * ks, instr_desc(128, 16), ks > 0 ? 1u : 0u);
                    tc_commit(&s.bar_score);
                }
                __syncwarp();
                wait_on(&s.bar_score, score_parity);
                score_parity ^= 1u;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t x[16];
                tmem_ld16_issue(lane_addr + 80, x);
                tmem_ld_wait();
                if (lane < 16) {
                    float pr[16];
                    const float dg = set.diag[lane];
#pragma unroll
                    for (int qq = 0; qq < SC; ++qq) pr[qq] = qq < lane ? __uint_as_float(x[qq]) : (qq == lane ? dg : 0.f);
                    *reinterpret_cast<uint4*>(&set.opP[op_index(16, lane, 0)]) =
                        make_uint4(pack_bf16(pr[0], pr[1]), pack_bf16(pr[2], pr[3]), pack_bf16(pr[4], pr[5]), pack_bf16(pr[6], pr[7]));
                    *reinterpret_cast<uint4*>(&set.opP[op_index(16, lane, 8)]) =
                        make_uint4(pack_bf16(pr[8], pr[9]), pack_bf16(pr[10], pr[11]), pack_bf16(pr[12], pr[13]), pack_bf16(pr[14], pr[15]));
                }
                sm100::fence_proxy_async_smem();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            sm100::named_bar_sync(kBarRound, 160);            // the state warps have finished the round trip of block m
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t ycol = tmem + 64 + 32 * slot;      // y^T of even blocks at columns 64..79, odd at 96..111
            if (elect_one()) {
#pragma unroll
                for (int ks = 0; ks < N / 16; ++ks)          // state operand: a K step of 16 = 2048 bytes = 128 units
                    umma_bf16(ycol, d_state + 128 * ks, d_r + 32 * ks, instr_desc(128, 16), ks > 0 ? 1u : 0u);
                umma_bf16(ycol, d_v, d_p, instr_desc(128, 16), 1u);
                umma_bf16(tmem, d_v, d_k, instr_desc(128, 64), 1u);
                tc_commit(&s.bar_main);
                tc_commit(&s.ops_free[slot]);
            }
            __syncwarp();
        }
        if (elect_one()) tc_commit(&s.drained);
        __syncwarp();
        sm100::mbar_wait(&s.drained, 0, a.limit);      // the tensor memory is given back behind the last products
    } else {
        // =================================== state ===================================
        const int lg = warp & 1, ch = warp >> 2;               // 32 TMEM lanes x 32 state columns per warp
        const int j = lg * 32 + lane;                          // value channel = TMEM lane
        const int sid = ch * 64 + j;                           // 0..127 within the role
        for (int m = 0; m <= n_steps; ++m) {
            if (m >= 1) wait_on(&s.bar_main, (m - 1) & 1);     // products of block m-1 are complete
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (m < n_steps) {
                const OpSet& set = s.sets[m & 1];
                wait_on(&s.ops_ready[m & 1], (m >> 1) & 1);    // dtot of block m
                // ---- round trip of this warp's 32 x 32 piece: bf16 copy for the read-out, decay in place ----
                uint32_t x[2][16];
                if (m > 0) {
                    tmem_ld16_issue(lane_addr + ch * 32, x[0]);
                    tmem_ld16_issue(lane_addr + ch * 32 + 16, x[1]);
                    tmem_ld_wait();
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[0][i] = x[1][i] = 0u;   // the walk starts from the zero state
                }
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    const int c0 = ch * 32 + g * 16;
                    float f[16];
#pragma unroll
                    for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(x[g][i]);
                    *reinterpret_cast<uint4*>(&s.opS[op_index(64, j, c0)]) =
                        make_uint4(pack_bf16(f[0], f[1]), pack_bf16(f[2], f[3]), pack_bf16(f[4], f[5]), pack_bf16(f[6], f[7]));
                    *reinterpret_cast<uint4*>(&s.opS[op_index(64, j, c0 + 8)]) =
                        make_uint4(pack_bf16(f[8], f[9]), pack_bf16(f[10], f[11]), pack_bf16(f[12], f[13]), pack_bf16(f[14], f[15]));
#pragma unroll
                    for (int i = 0; i < 16; ++i) x[g][i] = __float_as_uint(f[i] * set.dtot[c0 + i]);
                    tmem_st16(lane_addr + c0, x[g]);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                sm100::fence_proxy_async_smem();
                if (sid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");   // the y tile of block m-3 has left
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                sm100::named_bar_sync(kBarRound, 160);
            }
            if (m == n_steps) {
                // last pass: no round trip above, so the y slot is released here
                if (sid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");
                sm100::named_bar_sync(kBarYTile, 128);
            }
            if (m >= 1) {
                // ---- y of block m-1, while the products of block m run: this warp takes 8 of the 16 tokens ----
                const int step = m - 1, ys = step & 1;
                uint32_t yt[8];
                tmem_ld8_issue(lane_addr + 64 + 32 * ys + ch * 8, yt);
                tmem_ld_wait();
                const int y0 = tile_start(step);
                if (y0 >= 0) {
#pragma unroll
                    for (int t = 0; t < 8; ++t) s.ytile[ys][row_of(ch * 8 + t)][j] = __uint_as_float(yt[t]);
                    sm100::fence_proxy_async_smem();
                    sm100::named_bar_sync(kBarYTile, 128);
                    if (sid == 0) {
                        tma_reduce_add_3d(&map_y, &s.ytile[ys][0][0], h * N, y0, b);      // rows past T are clipped
                        sm100::tma_store_commit();
                    }
                } else {
                    // ragged last block of the leftward walk: its tile would start before token 0
#pragma unroll
                    for (int t = 0; t < 8; ++t) {
                        const int t_seq = step * SC + ch * 8 + t;
                        if (t_seq < T) atomicAdd(a.y + base + static_cast<size_t>(T - 1 - t_seq) * C + j, __uint_as_float(yt[t]));
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            }
        }
        if (sid == 0) sm100::tma_store_wait_all();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols));
}


// test mode: barriers wait for 16 bytes that never come, and give up after 2^10 polls
static std::atomic<bool> g_withhold{false};
void set_withhold_test(bool on) { g_withhold.store(on); }

// cudaFuncSetAttribute applies to the current device only: one flag per device, under a lock
static bool configure_once() {
    static std::mutex lock;
    static bool done[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> guard(lock);
    bool& configured = done[dev & 63];
    if (!configured) {
        if (cudaFuncSetAttribute(wkv6_tc_pipelined_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(SmemP))) != cudaSuccess ||
            cudaFuncSetAttribute(wkv6_tc_pipelined_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(SmemP))) != cudaSuccess)
            return false;
        configured = true;
    }
    return true;
}

// half_in: r, k, v point at bfloat16; w_raw, u, y are float32 either way
static int launch(int B, int T, int H, const void* r, const void* k, const void* v, const float* w_raw, const float* u,
                  float* y, unsigned* status, bool half_in, cudaStream_t stream) {
    if (!configure_once()) return -1;
    tensor_map::bind_primary_context();   // the tensor-map encoder is a driver call
    const int C = H * N;
    CUtensorMap mr, mk, mv, mw, my;
    if (!(tensor_map::make_btc(&mr, r, B, T, C, N, SC, half_in) && tensor_map::make_btc(&mk, k, B, T, C, N, SC, half_in) &&
          tensor_map::make_btc(&mv, v, B, T, C, N, SC, half_in) && tensor_map::make_btc_f32(&mw, w_raw, B, T, C, N, SC) &&
          tensor_map::make_btc_f32(&my, y, B, T, C, N, SC))) {
        set_error_detail("cuTensorMapEncodeTiled rejected a (C, T, B) tensor map");
        return -1;
    }
    Args a{B, T, H, static_cast<const float*>(r), static_cast<const float*>(k), static_cast<const float*>(v), w_raw, u, y,
           status, failure_mirror(Op::wkv6_forward), g_withhold.load() ? 1u << 10 : kWaitLimit, g_withhold.load() ? 16u : 0u};
    wkv6::clear(wkv6::Cleared{{y}, status, static_cast<size_t>(B) * T * C}, stream);      // both directions add into y
    launch_behind(half_in ? wkv6_tc_pipelined_kernel<true> : wkv6_tc_pipelined_kernel<false>, 2 * B * H, kPThreads, sizeof(SmemP), stream, a, mr, mk, mv, mw, my);
    return 1;
}

int forward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw, const float* u,
            float* y, unsigned* status, cudaStream_t stream) {
    return launch(B, T, H, r, k, v, w_raw, u, y, status, false, stream);
}

int forward_bf16in(int B, int T, int H, const void* r, const void* k, const void* v, const float* w_raw, const float* u,
                   float* y, unsigned* status, cudaStream_t stream) {
    return launch(B, T, H, r, k, v, w_raw, u, y, status, true, stream);
}

}  // namespace wkv6tc
