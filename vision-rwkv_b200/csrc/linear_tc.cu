// out = relu(x W^T)^2 in bfloat16 for an inference pass under bfloat16 autocast: the first half of a channel mix
// (classification/mmcls_custom/models/backbones/vrwkv.py:249-251), as one matrix product on the 5th-generation tensor cores whose
// epilogue rounds, clips and squares.
//
// The product alone is a library's business; what this saves is the pass behind it, which reads and writes the widest activation of
// the network (2 x 154 MB at 256 images of VRWKV-S, C = 384).
//
// A persistent CTA per SM walks 128 x 256 tiles of the result, columns fastest (the rows of x stay in L2).  Warp 0 brings 64-wide slices
// of x and W by TMA (128-byte swizzle, four stages of 48 KB), warp 1 issues tcgen05.mma into one of two accumulators in tensor memory
// (2 x 256 columns, all of it), warps 2 to 5 take the other one through registers and shared memory to a TMA store, so the
// epilogue, about 2 000 cycles, runs under the 3 000 cycles of a tile's products at K = 384.
//
// us, library product / and the pass behind it / this: rows 50176 K=192 N=768 24.7 / 51.4 / 30.9, 384 -> 1536 57.5 / 108.8 / 63.5 (HBM's
// time for x and the result 30, 931 TFLOP/s), 768 -> 3072 180 / 303 / 207, 1024 -> 4096 300 / 469 / 324 (1301 TFLOP/s of a measured 1410);
// rows 12544 768 -> 3072 47.2 / 74.2 / 52.2.  Few tiles, deep products and SMs without a tile in the last round are the library's
// (vrwkv_linear_relu_square_pays).
//
// The same walk over the tiles of several layers of one shape, without the squared ReLU (batch_by_tiles): the layers behind a token shift where
// their weights are too deep to stay in shared memory.  One by one, 12544 x 768 x 768 is a single round of the library's tiles, whose start and
// end nothing covers: four layers 58.1 us, in one launch 50.6; VRWKV6-B on 64 images 8310 -> 8143 us.
//
// Every wait is bounded; one that gives up sets a flag that ends the other roles, and the host-visible word of failures.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <mutex>
#include "../../include/vrwkv_b200.h"
#include "launch.h"
#include "linear_tc.cuh"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"

namespace lineartc {

constexpr int kN = kTile, kK = kSlice, kStages = 4;
constexpr uint32_t kABytes = kM * kK * 2, kStageBytes = kABytes + kN * kK * 2, kBoxBytes = kM * 64 * 2;
constexpr int kThreads = 192;

struct Bars {
    uint64_t full[kStages], empty[kStages], done[2], taken[2], drained;
    uint32_t tmem;
    volatile uint32_t dead;
};
constexpr size_t kSmem = 1024 + kStages * kStageBytes + 2 * kBoxBytes + sizeof(Bars);

// kTest: one role of a CTA withholds what it owes for the first tile, and waits give up early.  A variant of its own: as arguments the two
// cost 1.5 to 2.8 %.
// kSquare: one product and its squared ReLU, else several products as they are, one after the other.
template <bool kSquare, bool kTest>
__global__ void __launch_bounds__(kThreads, 1)
linear_tiles_kernel(const __grid_constant__ Products maps, int tiles, int m_tiles, int n_tiles, int k_blocks, unsigned* mirror) {
    wait_for_launch_before();
    extern __shared__ unsigned char smem_raw[];
    const uint32_t stages = (smem_u32(smem_raw) + 1023u) & ~1023u, out = stages + kStages * kStageBytes;
    Bars& s = *reinterpret_cast<Bars*>(smem_raw + (out + 2 * kBoxBytes - smem_u32(smem_raw)));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    struct Place {
        int product, m0, n0;
    };
    const auto place = [&](int tile) {      // columns fastest, then rows
        const int line = tile / n_tiles, product = kSquare ? 0 : line / m_tiles;
        return Place{product, (line - product * m_tiles) * kM, (tile - line * n_tiles) * kN};
    };
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            sm100::mbar_init(s.full + i, 1);
            sm100::mbar_init(s.empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            sm100::mbar_init(s.done + i, 1);
            sm100::mbar_init(s.taken + i, 4);
        }
        sm100::mbar_init(&s.drained, 1);
        sm100::mbar_init_fence();
        s.dead = 0u;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&s.tmem)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s.tmem;
    constexpr uint32_t limit = kTest ? 1u << 10 : kWaitLimit;
    const int silent = kTest ? static_cast<int>(blockIdx.x % 3) : -1;      // loader, issuer or epilogue
    const auto wait = [&](uint64_t* bar, uint32_t parity) {
        for (uint32_t i = 0; i < limit; ++i) {
            if (sm100::mbar_try_wait(bar, parity)) return true;
            if (i > 64) {
                if (s.dead != 0u) return false;
                __nanosleep(64);
            }
        }
        s.dead = 1u;
        if (mirror != nullptr) *reinterpret_cast<volatile unsigned*>(mirror) = 1u;
        return false;
    };
    if (warp == 0 && lane == 0) {
        uint32_t it = 0;
        bool good = true;
        for (int tile = blockIdx.x; good && tile < tiles; tile += gridDim.x) {
            const Place p = place(tile);
            for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                const uint32_t st = it % kStages;
                good = wait(s.empty + st, (it / kStages & 1u) ^ 1u) && !(kTest && silent == 0 && kb + 1 == k_blocks);
                if (!good) break;
                const uint32_t a = stages + st * kStageBytes;
                sm100::mbar_expect_tx(s.full + st, kStageBytes);
                tma_load_2d(a, maps.x + p.product, s.full + st, kb * kK, p.m0);
                tma_load_2d(a + kABytes, maps.w + p.product, s.full + st, kb * kK, p.n0);
            }
        }
        // nothing of this CTA is in flight when it goes: its products have read every stage, or at least its copies have landed
        for (uint32_t j = it > kStages ? it - kStages : 0u; j < it; ++j) {
            if (good) wait(s.empty + j % kStages, j / kStages & 1u);
            else sm100::mbar_wait(s.full + j % kStages, j / kStages & 1u, kWaitLimit / 64);
        }
    } else if (warp == 1 && lane == 0) {
        uint32_t it = 0, turn = 0;
        bool good = true;
        for (int tile = blockIdx.x; good && tile < tiles; tile += gridDim.x, ++turn) {
            const uint32_t buf = turn & 1u, d = tmem + buf * kN;
            good = wait(s.taken + buf, (turn >> 1 & 1u) ^ 1u);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; good && kb < k_blocks; ++kb, ++it) {
                const uint32_t st = it % kStages;
                good = wait(s.full + st, it / kStages & 1u);
                if (!good) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t a = operand(stages + st * kStageBytes), b = operand(stages + st * kStageBytes + kABytes);
#pragma unroll
                for (int k = 0; k < kK / 16; ++k) mma<kN>(d, a + 2 * k, b + 2 * k, (kb | k) != 0 ? 1u : 0u);      // 16 columns are 32 bytes
                commit(s.empty + st);
            }
            if (good && !(kTest && silent == 1 && turn == 0)) commit(s.done + buf);
        }
        if (!good) {      // products that were issued end before the tensor memory is given back
            commit(&s.drained);
            sm100::mbar_wait(&s.drained, 0, kWaitLimit / 64);
        }
    } else if (warp >= 2) {
        const int quadrant = warp & 3, row = quadrant * 32 + lane;      // of the accumulator, as this warp may read it
        const uint32_t swizzle = row & 7;
        uint32_t turn = 0;
        for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++turn) {
            const Place p = place(tile);
            const uint32_t buf = turn & 1u, d = tmem + (static_cast<uint32_t>(quadrant * 32) << 16) + buf * kN;
            // all four warps go on or none: they share barriers below
            bool good = wait(s.done + buf, turn >> 1 & 1u);
            good = __all_sync(0xffffffffu, good);
            int all;
            asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, 1, 128, p;\n\tselp.s32 %0, 1, 0, q;\n\t}" : "=r"(all) : "r"(good ? 1 : 0) : "memory");
            if (all == 0) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int half = 0; half < 2; ++half) {
                if (threadIdx.x == 64) sm100::tma_store_wait_read();
                sm100::named_bar_sync(1, 128);      // the boxes are free
#pragma unroll
                for (int box = 0; box < 2; ++box) {
                    uint32_t x[64];
#pragma unroll
                    for (int j = 0; j < 4; ++j) load16(d + half * 128 + box * 64 + j * 16, x + j * 16);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
                    for (int j = 0; j < 64; ++j) asm volatile("" : "+r"(x[j]));
                    const uint32_t at = out + box * kBoxBytes + row * 128;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const auto pair = [&](int c) {
                            return kSquare ? relu_square2(x[8 * j + c], x[8 * j + c + 1]) : narrow2(x[8 * j + c], x[8 * j + c + 1]);
                        };
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at + ((j ^ swizzle) << 4)), "r"(pair(0)), "r"(pair(2)), "r"(pair(4)), "r"(pair(6)) : "memory");
                    }
                }
                if (half == 1) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && !(kTest && silent == 2 && turn == 0)) mbar_arrive(s.taken + buf);
                }
                sm100::fence_proxy_async_smem();
                sm100::named_bar_sync(1, 128);
                if (threadIdx.x == 64) {
                    tma_store_2d(maps.out + p.product, out, p.n0 + half * 128, p.m0);
                    tma_store_2d(maps.out + p.product, out + kBoxBytes, p.n0 + half * 128 + 64, p.m0);
                    sm100::tma_store_commit();
                }
            }
        }
        if (threadIdx.x == 64) sm100::tma_store_wait_all();
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

static std::atomic<bool> g_withhold{false};
void set_withhold_test(bool on) { g_withhold.store(on); }
bool withhold_test() { return g_withhold.load(); }

static bool allowed(int* sms) {
    static std::mutex lock;
    static int state[64] = {};      // 0: not asked, -1: no, else SMs
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
    std::lock_guard<std::mutex> guard(lock);
    if (state[dev] == 0) {
        int n = 0;
        const auto allow = [](auto* kernel) {
            return cudaFuncSetAttribute(reinterpret_cast<const void*>(kernel), cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSmem)) == cudaSuccess;
        };
        const bool good = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && tensor_map::encode_fn() != nullptr &&
                          allow(linear_tiles_kernel<true, false>) && allow(linear_tiles_kernel<true, true>) && allow(linear_tiles_kernel<false, false>) &&
                          allow(linear_tiles_kernel<false, true>);
        if (!good) cudaGetLastError();
        state[dev] = good ? n : -1;
    }
    *sms = state[dev];
    return state[dev] > 0;
}

template <bool kSquare>
static int run_tiles(int sms, int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream) {
    const long long m_tiles = (rows + kM - 1) / kM, tiles = m_tiles * (N / kN) * count;
    tensor_map::bind_primary_context();
    Products maps;
    for (int i = 0; i < count; ++i)
        if (!tensor_map::make_rows(maps.x + i, x[i], rows, K, kK, kM) || !tensor_map::make_rows(maps.w + i, w[i], N, K, kK, kN) ||
            !tensor_map::make_rows(maps.out + i, out[i], rows, N, 64, kM)) {
            set_error_detail("cuTensorMapEncodeTiled rejected a matrix");
            return VRWKV_ERR_DEVICE;
        }
    const auto kernel = withhold_test() ? linear_tiles_kernel<kSquare, true> : linear_tiles_kernel<kSquare, false>;
    launch_behind(kernel, static_cast<unsigned>(std::min<long long>(tiles, sms)), kThreads, kSmem, static_cast<cudaStream_t>(stream), maps,
                  static_cast<int>(tiles), static_cast<int>(m_tiles), N / kN, K / kK, failure_mirror(Op::linear));
    return record_launches(1);
}
int tile_sms() {
    int sms = 0;
    return allowed(&sms) ? sms : 0;
}
int batch_by_tiles(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream) {
    int sms = 0;
    return allowed(&sms) ? run_tiles<false>(sms, count, rows, K, N, x, w, out, stream) : VRWKV_ERR_UNSUPPORTED;
}

}  // namespace lineartc

// The GPU's time for a library product and the pass behind it, in a captured loop, over this kernel's, by rounds of tiles: 1.04 and more
// from four rounds on; before that by how full the rounds are: K = 192 0.94 at half, 1.06 at 0.7, 1.15 at 0.8 (1.2 at one full round);
// K = 1024 0.86 at 0.6, 0.96 to 1.02 at 0.7, 1.02 to 1.08 at 0.8.  Rows 1 to 196, K = 64 to 1024: 0.54 to 0.8, of 3 to 8 us (a chain of
// loads; the library splits K).  K = 1536 0.98 to 1.12 at 0.8 and above, K = 4096 0.34 to 0.96 whatever the rows: the library's
// product is the faster one, and the pass is little beside it.
extern "C" int vrwkv_linear_relu_square_pays(long long rows, int K, int N) {
    using namespace lineartc;
    if (rows <= 0 || K <= 0 || N <= 0 || K % kK != 0 || N % kN != 0 || K > kMostTileDepth || rows > (1LL << 30)) return 0;
    const long long tiles = (rows + kM - 1) / kM * (N / kN);
    int sms = 0;
    if (tiles > (1LL << 30) || !allowed(&sms)) return 0;
    const long long rounds = (tiles + sms - 1) / sms;
    return rounds >= 4 || 5 * tiles >= 4 * rounds * sms ? 1 : 0;
}

extern "C" int vrwkv_linear_relu_square(long long rows, int K, int N, const uint16_t* x, const uint16_t* w, uint16_t* out, void* stream) {
    using namespace lineartc;
    if (rows <= 0 || K <= 0 || N <= 0) return VRWKV_ERR_SHAPE;
    if (!x || !w || !out) return VRWKV_ERR_NULL;
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15u) return VRWKV_ERR_ALIGNMENT;
    const long long m_tiles = (rows + kM - 1) / kM, tiles = m_tiles * (N / kN);
    int sms = 0;
    if (K % kK != 0 || N % kN != 0 || rows > (1LL << 30) || tiles > (1LL << 30) || !allowed(&sms)) return VRWKV_ERR_UNSUPPORTED;
    if (square_by_slabs(rows, K, N, slab_sms(true, K))) return run_square_by_slabs(rows, K, N, x, w, out, stream);
    return run_tiles<true>(sms, 1, rows, K, N, &x, &w, &out, stream);
}
