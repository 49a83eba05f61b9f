// Several linear layers of one shape in inference under bfloat16 autocast (the layers behind a token shift:
// classification/mmcls_custom/models/backbones/vrwkv.py:166-168, vrwkv6.py:194-197) as one matrix product on the 5th-generation tensor
// cores, results rounded to bfloat16; and the key layer with its squared ReLU (vrwkv.py:249-251) where it is shallow.  Deeper layers, and columns
// that are no whole slabs, go to the tiles of linear_tc.cu.
//
// Products up to 384 deep are bound by memory.  With slices of W streamed beside those of x (linear_tc.cu) most of what an SM takes from L2
// is W: 240 of 290 KB for 128 x 192 results at a depth of 384.  Here W stays: a persistent CTA holds a slab of 192 of its rows in shared memory
// (147 KB at that depth) and walks 128-row tiles of x, the CTAs of the other slabs beside it on the same tiles, which they find in L2.
// 50176 x 384, three layers: 47.2 us, the library's three products 64.7, HBM's time for x and results 35; figures by size at
// vrwkv_linear_batch_pays.  VRWKV-S on 256 images 5.86 -> 5.68 ms with 24 launches less.
//
// Warp 0 brings slices of x by TMA (and the next tile's into L2), warp 1 issues tcgen05.mma into one of two accumulators in tensor memory,
// sixteen warps take the other one in strips of 64 columns through shared memory to a TMA store.
//
// Tried: the gate sigmoid(x W^T) * y, or the norm and residual behind it, as the epilogue of such a product.  The gate took 32.6 us where product and
// pass take 37.9, but then its product is not one of the three: 68 us for both launches against 70; whole rows for the norm leave no room
// for W to stay, and with W streamed 46.5 us came to 51.4 (gated 73 to 57).
//
// Every wait is bounded; one that gives up sets a flag that ends the other roles, and the host-visible word of failures.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <map>
#include <mutex>
#include <utility>
#include "../../include/vrwkv_b200.h"
#include "launch.h"
#include "linear_tc.cuh"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"

namespace lineartc {

constexpr int kEpilogueWarps = 16, kEpilogueThreads = 32 * kEpilogueWarps, kBatchThreads = 64 + kEpilogueThreads;
constexpr uint32_t kStrip = kM * 64 * 2;       // bytes of 128 rows x 64 bfloat16
constexpr uint32_t kXBytes = kM * kSlice * 2, kWBytes = kSlab * kSlice * 2;

template <int kStages_>
struct Control {
    static constexpr int kStages = kStages_;
    uint64_t full[kStages], empty[kStages], done[2], taken[2], drained;
    uint32_t tmem;
    volatile uint32_t dead;
};
// where a CTA's slab is: the CTAs with equal blockIdx.x % slabs share the row tiles of one
struct Slab {
    const CUtensorMap *x, *w;
    int n0, m_tiles, first, step;
    __device__ __forceinline__ int tiles() const { return first < m_tiles ? (m_tiles - first + step - 1) / step : 0; }
    __device__ __forceinline__ int m0(int i) const { return (first + i * step) * kM; }
};

template <class T>
__device__ __forceinline__ uint32_t start(T& s, int warp) {
    if (threadIdx.x == 0) {
        for (int i = 0; i < T::kStages; ++i) {
            sm100::mbar_init(s.full + i, 1);
            sm100::mbar_init(s.empty + i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            sm100::mbar_init(s.done + i, 1);
            sm100::mbar_init(s.taken + i, kEpilogueWarps);
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
    return s.tmem;
}
__device__ __forceinline__ void finish(uint32_t tmem, int warp) {
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}
// kTest: waits give up early
template <bool kTest, class T>
__device__ __forceinline__ bool wait(T& s, unsigned* mirror, uint64_t* bar, uint32_t parity) {
    constexpr uint32_t limit = kTest ? 1u << 10 : kWaitLimit;
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
}
// `silent` (kTest): the role that withholds what it owes for the first tile: 0 this one, 1 the issuer, 2 the epilogue.
// The slab of W comes with the first tile's slices of x, on the same barriers.
template <bool kTest, class T>
__device__ __forceinline__ void bring_slices(T& s, unsigned* mirror, uint32_t slab, uint32_t stages, const Slab& p, int k_blocks, int silent) {
    const int tiles = p.tiles();
    uint32_t it = 0;
    bool good = true;
    for (int i = 0; good && i < tiles; ++i)
        for (int kb = 0; kb < k_blocks; ++kb, ++it) {
            const uint32_t st = it % T::kStages;
            good = wait<kTest>(s, mirror, s.empty + st, (it / T::kStages & 1u) ^ 1u) && !(kTest && silent == 0 && kb + 1 == k_blocks);
            if (!good) break;
            sm100::mbar_expect_tx(s.full + st, i == 0 ? kXBytes + kWBytes : kXBytes);
            if (i == 0) tma_load_2d(slab + kb * kWBytes, p.w, s.full + st, kb * kSlice, p.n0);
            tma_load_2d(stages + st * kXBytes, p.x, s.full + st, kb * kSlice, p.m0(i));
            if (i + 1 < tiles) tma_prefetch_2d(p.x, kb * kSlice, p.m0(i + 1));
        }
    // nothing of this CTA is in flight when it goes: its products have read every stage, or at least its copies have landed
    for (uint32_t j = it > T::kStages ? it - T::kStages : 0u; j < it; ++j) {
        if (good) wait<kTest>(s, mirror, s.empty + j % T::kStages, j / T::kStages & 1u);
        else sm100::mbar_wait(s.full + j % T::kStages, j / T::kStages & 1u, kWaitLimit / 64);
    }
}
template <bool kTest, class T>
__device__ __forceinline__ void issue_products(T& s, unsigned* mirror, uint32_t slab, uint32_t stages, uint32_t tmem, int tiles, int k_blocks, int silent) {
    uint32_t it = 0;
    bool good = true;
    for (int i = 0; good && i < tiles; ++i) {
        const uint32_t buf = i & 1, d = tmem + buf * 256;
        good = wait<kTest>(s, mirror, s.taken + buf, (i >> 1 & 1u) ^ 1u);
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int kb = 0; good && kb < k_blocks; ++kb, ++it) {
            const uint32_t st = it % T::kStages;
            good = wait<kTest>(s, mirror, s.full + st, it / T::kStages & 1u);
            if (!good) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint64_t a = operand(stages + st * kXBytes), b = operand(slab + kb * kWBytes);
#pragma unroll
            for (int k = 0; k < kSlice / 16; ++k) mma<kSlab>(d, a + 2 * k, b + 2 * k, (kb | k) != 0 ? 1u : 0u);      // 16 columns are 32 bytes
            commit(s.empty + st);
        }
        if (good && !(kTest && silent == 1 && i == 0)) commit(s.done + buf);
    }
    if (!good) {      // products that were issued end before the tensor memory is given back
        commit(&s.drained);
        sm100::mbar_wait(&s.drained, 0, kWaitLimit / 64);
    }
}
// a barrier of some of the epilogue's warps that says whether all of them are well
__device__ __forceinline__ bool all_good(int id, int threads, bool good) {
    int all;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.s32 p, %1, 0;\n\tbar.red.and.pred q, %3, %2, p;\n\tselp.s32 %0, 1, 0, q;\n\t}"
                 : "=r"(all) : "r"(good ? 1 : 0), "r"(threads), "r"(id) : "memory");
    return all != 0;
}
template <int n>
__device__ __forceinline__ void read_sums(uint32_t at, uint32_t (&x)[n]) {
#pragma unroll
    for (int j = 0; j < n; j += 16) load16(at + j, x + j);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < n; ++j) asm volatile("" : "+r"(x[j]));
}
// until all but the last n stores have read shared memory
template <int n>
__device__ __forceinline__ void store_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(n) : "memory"); }
__device__ __forceinline__ void put16(uint32_t at, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(at), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// ---- products as they are ------------------------------------------------------------------------------------------------------
template <int kStages, int kSlots>
static size_t batch_smem(int K) { return K * kSlab * 2 + kStages * kXBytes + kSlots * kStrip + sizeof(Control<kStages>); }

template <int kStages, int kSlots, bool kSquare, bool kTest>
__global__ void __launch_bounds__(kBatchThreads, 1)
linear_batch_kernel(const __grid_constant__ Products maps, int count, int m_tiles, int n_slabs, int k_blocks, unsigned* mirror) {
    wait_for_launch_before();
    constexpr int kPerTile = kSlab / 64;
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t slab = smem_u32(smem), stages = slab + k_blocks * kWBytes, outs = stages + kStages * kXBytes;
    Control<kStages>& s = *reinterpret_cast<Control<kStages>*>(smem + (outs + kSlots * kStrip - slab));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int silent = kTest ? static_cast<int>(blockIdx.x % 3) : -1;
    const int slabs = count * n_slabs, own = blockIdx.x % slabs, product = own / n_slabs;
    const Slab p{maps.x + product, maps.w + product, (own - product * n_slabs) * kSlab, m_tiles, static_cast<int>(blockIdx.x) / slabs, static_cast<int>(gridDim.x) / slabs};
    const int tiles = p.tiles();
    const uint32_t tmem = start(s, warp);
    if (warp == 0) {
        if (lane == 0) bring_slices<kTest>(s, mirror, slab, stages, p, k_blocks, silent);
    } else if (warp == 1) {
        if (lane == 0) issue_products<kTest>(s, mirror, slab, stages, tmem, tiles, k_blocks, silent);
    } else {
        const int quadrant = warp & 3, part = (warp - 2) >> 2, row = quadrant * 32 + lane;      // 16 of a strip's columns
        const uint32_t swizzle = row & 7;
        const bool elected = threadIdx.x == 64;
        uint32_t n = 0;       // strips done
        bool good = true;
        for (int i = 0; good && i < tiles; ++i) {
            const uint32_t buf = i & 1, d = tmem + (static_cast<uint32_t>(quadrant * 32) << 16) + buf * 256 + part * 16;
            good = __all_sync(0xffffffffu, wait<kTest>(s, mirror, s.done + buf, i >> 1 & 1u));
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int strip = 0; strip < kPerTile; ++strip, ++n) {
                uint32_t x[16];
                read_sums(d + strip * 64, x);
                if (strip + 1 == kPerTile) {
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0 && !(kTest && silent == 2 && i == 0)) mbar_arrive(s.taken + buf);
                }
                const uint32_t out = outs + n % kSlots * kStrip + row * 128;
#pragma unroll
                for (int j = 0; j < 2; ++j) {      // 8 columns: 16 bytes of bfloat16
                    const auto pair = [&](int c) {
                        return kSquare ? relu_square2(x[8 * j + c], x[8 * j + c + 1]) : narrow2(x[8 * j + c], x[8 * j + c + 1]);
                    };
                    put16(out + (((2 * part + j) ^ swizzle) << 4), pair(0), pair(2), pair(4), pair(6));
                }
                sm100::fence_proxy_async_smem();
                if (elected) store_wait_read<kSlots - 2>();      // the next strip has its room
                good = all_good(1, kEpilogueThreads, good);
                if (!good) break;
                if (elected) {
                    tma_store_2d(maps.out + product, outs + n % kSlots * kStrip, p.n0 + 64 * strip, p.m0(i));
                    sm100::tma_store_commit();
                }
            }
        }
        if (elected) sm100::tma_store_wait_all();
    }
    finish(tmem, warp);
}

// ---- host --------------------------------------------------------------------------------------------------------------------
// SMs of the current device, 0 where the kernels cannot be had; a kernel's shared memory is set the first time it meets the device
static int prepare(const void* kernel, size_t smem) {
    static std::mutex lock;
    static std::map<std::pair<int, const void*>, int> known;
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> guard(lock);
    const auto at = known.find({dev, kernel});
    if (at != known.end()) return at->second;
    if (tensor_map::encode_fn() == nullptr || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
        cudaGetLastError();
        sms = 0;
    }
    known[{dev, kernel}] = sms;
    return sms;
}
static int refused(const char* why) {
    set_error_detail(why);
    return VRWKV_ERR_DEVICE;
}

template <int kStages, int kSlots, bool kSquare, bool kTest>
static int sms_of() {
    return prepare(reinterpret_cast<const void*>(linear_batch_kernel<kStages, kSlots, kSquare, kTest>), batch_smem<kStages, kSlots>(kStages == 4 ? 256 : kMostSlabDepth));
}
template <int kStages, int kSlots, bool kSquare, bool kTest>
static int run_batch(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream) {
    const auto kernel = linear_batch_kernel<kStages, kSlots, kSquare, kTest>;
    const int sms = sms_of<kStages, kSlots, kSquare, kTest>(), slabs = N / kSlab * count;
    if (sms < slabs) return VRWKV_ERR_UNSUPPORTED;
    tensor_map::bind_primary_context();
    Products maps;
    bool made = true;
    for (int i = 0; i < count; ++i)
        made = made && tensor_map::make_rows(maps.x + i, x[i], rows, K, 64, kM) && tensor_map::make_rows(maps.w + i, w[i], N, K, 64, kSlab) &&
               tensor_map::make_rows(maps.out + i, out[i], rows, N, 64, kM);
    if (!made) return refused("cuTensorMapEncodeTiled rejected a matrix");
    const int m_tiles = static_cast<int>((rows + kM - 1) / kM);
    launch_behind(kernel, std::min(m_tiles, sms / slabs) * slabs, kBatchThreads, batch_smem<kStages, kSlots>(K), static_cast<cudaStream_t>(stream), maps,
                  count, m_tiles, N / kSlab, K / kSlice, failure_mirror(Op::linear));
    return record_launches(1);
}
static bool unaligned(std::initializer_list<const void*> ps) {
    uintptr_t bits = 0;
    for (const void* p : ps) bits |= reinterpret_cast<uintptr_t>(p);
    return (bits & 15u) != 0;
}
// shallow slabs leave room for more slices and strips under way (192 deep, three layers: 22.3 -> 20.8 us at 50176 rows, 85.5 -> 82.7 at 200704)
static bool shallow(int K) { return K <= 256; }
int slab_sms(bool square, int K) {
    if (withhold_test()) return square ? sms_of<4, 4, true, true>() : shallow(K) ? sms_of<4, 4, false, true>() : sms_of<3, 2, false, true>();
    return square ? sms_of<4, 4, true, false>() : shallow(K) ? sms_of<4, 4, false, false>() : sms_of<3, 2, false, false>();
}
int run_square_by_slabs(long long rows, int K, int N, const uint16_t* x, const uint16_t* w, uint16_t* out, void* stream) {
    return (withhold_test() ? run_batch<4, 4, true, true> : run_batch<4, 4, true, false>)(1, rows, K, N, &x, &w, &out, stream);
}
static int run_by_slabs(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream) {
    const auto fn = withhold_test() ? (shallow(K) ? run_batch<4, 4, false, true> : run_batch<3, 2, false, true>)
                                    : (shallow(K) ? run_batch<4, 4, false, false> : run_batch<3, 2, false, false>);
    return fn(count, rows, K, N, x, w, out, stream);
}
static int batch_sms(int K) { return K <= kMostSlabDepth ? slab_sms(false, K) : 0; }

}  // namespace lineartc

extern "C" int vrwkv_linear_batch(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out,
                                  void* stream) {
    using namespace lineartc;
    if (count <= 0 || count > kMostProducts || rows <= 0 || K <= 0 || N <= 0) return VRWKV_ERR_SHAPE;
    if (!x || !w || !out) return VRWKV_ERR_NULL;
    for (int i = 0; i < count; ++i) {
        if (!x[i] || !w[i] || !out[i]) return VRWKV_ERR_NULL;
        if (unaligned({x[i], w[i], out[i]})) return VRWKV_ERR_ALIGNMENT;
    }
    const Route by = batch_route(count, rows, K, N, batch_sms(K), tile_sms());
    if (by == Route::none) return VRWKV_ERR_UNSUPPORTED;
    return (by == Route::slabs ? run_by_slabs : batch_by_tiles)(count, rows, K, N, x, w, out, stream);
}

// Several layers of one shape against as many library products, in a captured loop (us):
//   rows       196 x 384   3136 x 384   12544 x 384   50176 x 384   100352 x 384   196 x 192   12544 x 192   50176 x 192   200704 x 192
//   one        3.0 / 6.7   3.8 / 6.8    6.2 / 9.0     16.9 / 18.6   38.8 / 32.3    2.7 / 5.5   4.2 / 5.6     8.6 / 8.1     26.1 / 27.5
//   two        5.6 / 6.7   7.2 / 6.9    12.1 / 11.4   42.5 / 32.9   77.4 / 59.4    5.1 / 5.4   8.1 / 6.9     17.3 / 12.5   53.2 / 55.6
//   three      8.4 / 6.7   10.8 / 8.4   18.3 / 15.8   64.7 / 47.2   116.0 / 87.6   7.6 / 5.5   11.9 / 6.9    31.2 / 20.8   79.8 / 82.7
//   four       11.1 / 6.7  14.1 / 9.1   26.3 / 19.1   86.1 / 59.6   154.7 / 116.2  9.9 / 5.5   15.9 / 8.1    41.8 / 28.1   106.1 / 108.8
// (a launch saved is worth 2 to 3 us more between other kernels: batch_pays in linear_routes.h); single layers and pairs are the library's.  By tiles (linear_tc.cu), three layers:
//   rows           196          1568         6272         12544        25088         50176         100352
//   256 -> 256     7.7 / 5.6    9.4 / 5.8    11.2 / 6.4   13.9 / 8.7                 38.5 / 28.0   62.9 / 51.4
//   512 -> 512     10.0 / 7.3   10.7 / 7.2   16.9 / 10.8  25.9 / 18.1  46.7 / 38.6   79.1 / 75.4
//   768 -> 768     10.5 / 8.0   13.6 / 8.5   25.2 / 18.8  43.8 / 38.2  76.4 / 76.0   148.0 / 151.1
//   1024 -> 1024   12.5 / 10.3  16.0 / 16.1  39.9 / 29.7  68.0 / 63.0  126.6 / 125.0 247.0 / 249.2
// Four layers gain a little more (12544 x 768 58.1 / 50.6).
extern "C" int vrwkv_linear_batch_pays(int count, long long rows, int K, int N) {
    using namespace lineartc;
    return count <= kMostProducts && batch_pays(count, rows, K, N, batch_sms(K), tile_sms()) ? 1 : 0;
}
