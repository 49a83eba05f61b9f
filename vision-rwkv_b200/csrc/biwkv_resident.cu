// Bi-WKV on sequences of more than 4096 tokens (shorter ones: biwkv_strips.cu).  Many of them: separate launches over independent CTAs,
// see biwkv_chain_kernel.  Few: the whole token range of one (sequence, 32-channel strip) is held in the shared memory of a few
// thread-block clusters while it is scanned in both directions (`linked`).
//
// Work unit: one (sequence b, strip of kCs = 32 channels).  Its T tokens are split into contiguous ranges of n_tok = 32 * n_warps
// tokens, one per CTA, in clusters of `cluster` CTAs.
// Inside a CTA warp s owns the span of 32 tokens [32 s, 32 s + 32); its lower half-warp walks the
// first kL = 16 tokens of the span, its upper half-warp the last 16; lane p of a half-warp owns the
// channel pair (2p, 2p+1).  A thread walks its 16 tokens sequentially with 64-bit shared accesses
// (a half-warp reads one whole 128-byte row), and carries its two channels packed in f32x2
// registers, so one instruction serves both.  One TMA box per tensor and CTA brings the range in
// (zero fill past T and C); outputs overwrite the inputs in place and leave by TMA store (clipped).
//
// A bidirectional scan needs, at each token, the decayed sum over all earlier and all later tokens.
// Per scan level:
//   1. the two half-warps of a warp combine their sub-chunk aggregates by shuffles and post the
//      aggregate of the 32-token span (towards later tokens, and towards earlier ones);
//   2. two warps walk the span aggregates of the CTA serially (one per direction, lane = channel),
//      leave in place the state entering each span from the rest of the CTA, and send the CTA's own
//      aggregate to the CTAs that need it, all warps sharing the sends: st.async into their shared
//      memory, completion counted in bytes on their mbarrier (one hop through the cluster network,
//      no fence, no multicast);
//   3. the same two warps wait (bounded) for the bytes of the other CTAs and combine them;
//   4. every thread adds the outside state, moved to its own position, to its inside state.
// Forward: one level (terms e^{k}[v, 1]).  Backward: a second level for the adjoint pairs
// [gy / Den, gy y / Den]; y and Den are recomputed.
//
// Arithmetic.  Plain floats without any exponent shift: a term is lambda e^{k} [v, 1] with lambda = e^{-w}, recurrences are one packed
// fused multiply-add per token and direction.  That is exact enough whenever 2 max|k| + |u| + |w| + max(-w, 0) T <= 60 (no
// overflow, no harmful underflow in float32).  Every thread checks its own tokens; where one saw otherwise a word in the workspace
// switches on the chunked kernels (biwkv_fused.cu), which stand by and redo the call.  Decay over long distances never comes from
// repeated multiplication by a rounded lambda: the per-channel factors for 16, 32 and n_tok tokens are computed once per CTA in
// double precision and applied as a (high, low) float pair.
//
// Recurrence restated: classification/mmcls_custom/models/backbones/cuda_new/
// bi_wkv_kernel.cu:21-116 (forward), :119-367 (gradients).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <initializer_list>
#include <mutex>
#include "biwkv_math.cuh"
#include "biwkv_pairs.cuh"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"

namespace biwkv {
namespace resident {

using namespace pairs;

constexpr int kL = 16;            // tokens per thread
constexpr int kSpan = 2 * kL;     // tokens per warp
constexpr int kGroup = 4;         // tokens whose loads are issued together (forward)
constexpr int kGroupB = 4;        // ... backward
constexpr int kBatch = 8;         // other CTAs' blocks read together when they are combined
constexpr int kCs = 32;           // channels per strip
constexpr int kMaxWarps = 8;      // spans per CTA
constexpr int kMaxCluster = 16;
constexpr int kMaxThreads = kMaxWarps * 32;
constexpr float kSafeRange = 60.f;
constexpr uint32_t kSpinLimit = 1u << 20;   // ~0.1 s of polling on a barrier

// per-channel constants, computed once per CTA by warp 0 in double precision (rows of kCs floats)
enum ConstRow {
    kLam = 0, kWl2, kCuw, kLam16_hi, kLam16_lo, kLam32_hi, kLam32_lo, kLamC_hi, kLamC_lo, kConstRows
};

// What one launch computes.
enum class Mode {
    linked,     // every level: several clusters hold the sequence, hand-over through global memory
    sums,       // no clusters: the sums of level 1 (forward) or level 2 (backward, level 1 given) of every sub-chunk and CTA
    sums_keep,  // forward: as sums, with the first moments that a backward needs
    spread,     // no clusters: every level given; writes the results
};
template <Mode m>
constexpr bool kUsesCluster = m == Mode::linked;

// rows of kCs floats in the record area behind the data slots
template <bool kMom, bool kBwd>
struct RowsOf {
    static constexpr int kF = kMom ? 4 : 2;       // towards later tokens: a, b (, first moments)
    static constexpr int kR = 2;                  // towards earlier tokens: a, b
    static constexpr int kSub = kF + kR;          // per span
    static constexpr int kLevels = kBwd ? 2 : 1;
    static constexpr int kSlots = kBwd ? 3 : 2;
    static constexpr int kBlockF = kCs * kF + 4;   // floats of a CTA aggregate towards later tokens + flag word (16-byte padded)
    static constexpr int kBlockR = kCs * kR + 4;   // ... towards earlier tokens
    static constexpr int kPeerFloats = (kMaxCluster - 1) * kBlockF;   // one block slot per other rank (ranks above this CTA's shift down by one)
};
template <bool kBwd, Mode kMode = Mode::linked>
using Rows = RowsOf<kBwd || kMode == Mode::sums_keep, kBwd>;
constexpr int kStateRows = 6;      // states that enter a sub-chunk: P (n, d), its first moment (n, d), S (n, d)
constexpr int kPlainRows = 4;      // ... without the moments
// rows of the state that enters the CTA
template <bool kBwd, Mode kMode>
constexpr int kOutsideRows = kUsesCluster<kMode> ? Rows<kBwd, kMode>::kSub : kStateRows;

struct Params {
    int B, T, C;
    int n_strips;
    int cluster;      // CTAs per (sequence, strip)
    int n_warps;      // 32-token spans per CTA
    int n_tok;        // tokens per CTA = n_warps * kSpan
    const float* w;
    const float* u;
    unsigned* status;   // device status word
    unsigned* mirror;   // host-visible copy of a failure (may be null)
    float* partial;     // backward: [grid][2][kCs]
    unsigned* redo_count;   // units that were outside the plain-float range
    uint32_t spin_limit;  // polls before a wait for the other CTAs gives up
    int withhold_rank;    // test only: this rank of every cluster sends nothing (-1: none)
    int ctas;             // CTAs per (sequence, strip)
    // sequences longer than one cluster holds, several clusters: `segs` clusters per (sequence, strip), each with
    // cluster * n_tok tokens, which hand their aggregates to one another through global memory
    int segs;
    float* xseg;          // [unit][seg][level][direction][kSegRec]
    unsigned* xflag;      // same index; zero before launch, 1 (| 2: out of range) once the record is there
    // Without clusters: states that enter sub-chunks, [unit][CTA][sub-chunk][state_rows][kCs], relative to their CTA, and states
    // that enter CTAs, [unit][CTA][state_rows][kCs], which are the CTAs' own sums until biwkv_chain_kernel has run
    float* states1;
    float* ctas1;
    float* states2;       // level 2 (backward)
    float* ctas2;
    int state_rows;       // kStateRows, or kPlainRows where no moments are kept
    unsigned* out_of_range;   // inputs outside the plain-float range were seen
    bool reverse;         // last CTAs first: what the launch before this one read last is still in L2
};

constexpr int kSegRec = 4 * kCs;      // floats per record (forward: 2 rows used)
constexpr int kMaxSegs = 8;

// shared memory: data slots | span records | blocks received from the other CTAs | this CTA's two
// outgoing blocks | state entering this CTA | constants | mbarriers and the flag word
template <bool kBwd, Mode kMode = Mode::linked>
static inline size_t smem_bytes(int n_warps) {
    using R = Rows<kBwd, kMode>;
    const size_t data = static_cast<size_t>(R::kSlots) * n_warps * kSpan * kCs * sizeof(float);
    const size_t rec = (static_cast<size_t>(n_warps) * R::kSub * kCs + (kUsesCluster<kMode> ? R::kPeerFloats : 0) + R::kBlockF + R::kBlockR + kOutsideRows<kBwd, kMode> * kCs + kConstRows * kCs) * sizeof(float);
    return data + rec + 192;
}

// Debug timeline: with -DVRWKV_TIMELINE lane 0 of warps 0 and 5 of the first kTlCtas CTAs and of
// kTlCtas CTAs from the middle of the grid store clock64() at each phase boundary in a buffer of
// 2 * kTlCtas * 2 * kTlMarks words that g_tl_base points to.  Compiled out otherwise.
#ifdef VRWKV_TIMELINE
constexpr int kTlCtas = 64, kTlMarks = 32;
__device__ long long* g_tl_base = nullptr;      // unset: no marks
#define TL_MARK(m)                                                                                         \
    do {                                                                                                   \
        if (tl_slot >= 0 && lane == 0 && (warp == 0 || warp == 5))                                          \
            tl_base[((tl_slot * 2 + (warp ? 1 : 0)) * kTlMarks) + (m)] = clock64();                         \
    } while (0)
#define TL_ARGS , long long* tl_base, int tl_slot
#define TL_PASS , tl_base, tl_slot
#else
#define TL_MARK(m) do { } while (0)
#define TL_ARGS
#define TL_PASS
#endif

struct Ctx {
    float* sub;      // [n_warps][kSub][kCs]; rows 0..kF-1 towards later tokens, kF.. towards earlier
    float* peers;    // [kMaxCluster][kBlockF]: blocks received from the other CTAs (directly behind sub)
    float* stage;    // [kBlockF + kBlockR]: this CTA's outgoing blocks
    unsigned* flag;  // the cluster's out-of-range flag, once known
    float* cta;      // [kSub][kCs]: state entering this CTA from the rest of the cluster
    float* consts;   // [kConstRows][kCs]
    uint64_t* xbar;  // [kLevels] mbarriers counting the bytes the other CTAs send
    unsigned* status;
    unsigned* mirror;
    uint32_t spin_limit;
    bool withhold;   // test only: this CTA sends nothing to the others
    int warp, lane, n_warps, n_tok, cluster, rank;
    int seg, segs, unit;     // this cluster's segment of the sequence
    float* xseg;
    unsigned* xflag;
    float* cta_sums;         // launches without clusters: where this CTA's sums go, [state_rows][kCs]
};

struct Enter {
    Pair2 P, MP, S;   // state (and first moment) entering at the first token; state entering at the last
};

// Element access of a thread's sub-chunk in one data slot.  `area` = the sub-chunk's 16 rows of kCs
// floats (2 KB).  float32 tensors: row i is where it arrived.  bfloat16 tensors: the 16 rows arrive
// dense (64 bytes each) in the upper half of the area and are widened in place as the first pass over
// them walks up the rows: writing float row i (bytes 128 i and up) covers bfloat16 rows <= 2 i - 15
// only, which have been read by then, also when the reads of 4 rows are issued ahead of the writes.
// Results leave as dense bfloat16 rows at the start of the area: row i lands on float rows <= i / 2,
// consumed before it.  Both half-warps of a warp run in lockstep over areas of their own.
constexpr int kHalfRowBytes = kCs * 2;
constexpr int kHalfAreaBytes = kL * kHalfRowBytes;     // 1 KB: the upper half of the 2 KB area
template <bool kHalf>
__device__ __forceinline__ float2 ld_in(const float* area, int i, int pr) {
    if (kHalf) {
        const unsigned char* row = reinterpret_cast<const unsigned char*>(area) + kHalfAreaBytes + i * kHalfRowBytes;
        return __bfloat1622float2(*(reinterpret_cast<const __nv_bfloat162*>(row) + pr));
    }
    return *(reinterpret_cast<const float2*>(area + i * kCs) + pr);
}
template <bool kHalf>
__device__ __forceinline__ void st_out(float* area, int i, int pr, float2 v) {
    if (kHalf) {
        unsigned char* row = reinterpret_cast<unsigned char*>(area) + i * kHalfRowBytes;
        *(reinterpret_cast<__nv_bfloat162*>(row) + pr) = __float22bfloat162_rn(v);
    } else {
        *(reinterpret_cast<float2*>(area + i * kCs) + pr) = v;
    }
}

// ---- sequences of several segments ---------------------------------------------------------------
// Each cluster first completes its own exchange, then its last rank publishes the segment's aggregate
// towards later tokens and its rank 0 the one towards earlier tokens (record, fence, release of a flag
// word), and only then do its CTAs wait (bounded) for the records of the other segments of the same
// (sequence, strip): whoever waits has already published, and clusters are dispatched in index
// order with a unit's segments adjacent, so the records a resident cluster waits for belong to
// clusters that are resident too or next in line.  Decay factors over whole segments are formed in
// double precision from the CTA's (high, low) pair for one CTA's tokens.
__device__ __forceinline__ size_t seg_index(const Ctx& c, int seg, int level, int dir) {
    return ((static_cast<size_t>(c.unit) * c.segs + seg) * 2 + level) * 2 + dir;
}
struct HiLo {
    float2 hi, lo;
};
// lambda^(n_tok * blocks) from the CTA's (high, low) pair for lambda^n_tok, by squaring in double precision
__device__ __forceinline__ HiLo decay_over_blocks(const Ctx& c, int blocks) {
    double base = static_cast<double>(c.consts[kLamC_hi * kCs + c.lane]) + static_cast<double>(c.consts[kLamC_lo * kCs + c.lane]);
    double x = 1.0;
    for (int e = blocks; e > 0; e >>= 1) {
        if (e & 1) x *= base;
        base *= base;
    }
    const float hi = static_cast<float>(x);
    return HiLo{dup(hi), dup(static_cast<float>(x - static_cast<double>(hi)))};
}
// A wait for another CTA ran out.  This one goes no further than the first level: at the second it would send to CTAs that heard
// everything and may have left (out of range).  See stay_for_late_data.
__device__ __forceinline__ void gave_up(const Ctx& c, unsigned bits) {
    report_failure(c.status, c.mirror, bits);
    *reinterpret_cast<volatile unsigned*>(c.flag + 2) = 1u;
}
// Before warp 0 of a CTA goes: one that gave up a wait stays until everything that is sent to it is on its way - every other thread of
// its cluster has gone or come here (a cluster barrier counts the threads that are left) - and then, with a limit, until it is there.
// `phases`: of the cluster barrier that those that go on still pass.
__device__ __forceinline__ void stay_for_late_data(const Ctx& c, int phases, int levels) {
    if (c.warp != 0 || c.flag[2] == 0u) return;
    __syncwarp();
    for (int i = 0; i < phases; ++i) {
        cluster_arrive();
        cluster_wait();
    }
    for (int l = 0; l < levels; ++l) sm100::mbar_wait(c.xbar + l, 0, c.spin_limit);
}
// waits for `count` flags starting at segment `first` (lane j takes segment first + j); returns the OR of their values
__device__ __forceinline__ unsigned seg_wait(const Ctx& c, int first, int count, int level, int dir) {
    unsigned seen = 1u;
    if (c.lane < count) {
        const unsigned* f = c.xflag + seg_index(c, first + c.lane, level, dir);
        seen = 0u;
        for (uint32_t it = 0; it < c.spin_limit; ++it) {
            seen = sm100::flag_relaxed(f);
            if (seen) break;
            __nanosleep(32);
        }
        if (seen) seen = sm100::flag_acquire(f);
    }
    const bool all = __all_sync(0xffffffffu, seen != 0u);
    if (!all && c.lane == 0) gave_up(c, 4u);
    unsigned bits = all ? seen : 2u;
#pragma unroll
    for (int m = 16; m >= 1; m >>= 1) bits |= __shfl_xor_sync(0xffffffffu, bits, m);
    return bits;
}
// Towards later tokens.  In: X, MX = state entering this CTA from the lower ranks of its own cluster; P, M =
// the CTA's own aggregate.  Out: X, MX also hold everything from the earlier segments; flag |= theirs.
template <bool kMom>
__device__ __noinline__ void seg_exchange_forward(const Ctx& c, int level, float2& X, float2& MX, float2 P, float2 M, int& flag) {
    const int lane = c.lane;
    const int seg_tok = c.cluster * c.n_tok;
    if (c.rank == c.cluster - 1 && c.seg + 1 < c.segs) {
        const float2 hi = dup(c.consts[kLamC_hi * kCs + lane]), lo = dup(c.consts[kLamC_lo * kCs + lane]);
        const float2 F = mulc_add(X, hi, lo, P);
        float* rec = c.xseg + seg_index(c, c.seg, level, 0) * kSegRec;
        rec[lane] = F.x; rec[kCs + lane] = F.y;
        if (kMom) {
            const float2 MF = mulc_add(fma2(dup(static_cast<float>(c.n_tok)), X, MX), hi, lo, M);
            rec[2 * kCs + lane] = MF.x; rec[3 * kCs + lane] = MF.y;
        }
        __threadfence();
        __syncwarp();
        if (lane == 0) sm100::flag_release(c.xflag + seg_index(c, c.seg, level, 0), 1u | (flag ? 2u : 0u));
    }
    if (c.seg > 0) {
        const unsigned bits = seg_wait(c, 0, c.seg, level, 0);
        if (bits & 2u) flag = 1;
        const HiLo ls = decay_over_blocks(c, c.cluster);
        const float2 len = dup(static_cast<float>(seg_tok));
        float2 A = f2(0.f, 0.f), MA = f2(0.f, 0.f);
        for (int q = 0; q < c.seg; ++q) {
            const float* rec = c.xseg + seg_index(c, q, level, 0) * kSegRec;
            const float2 f = f2(__ldcg(rec + lane), __ldcg(rec + kCs + lane));
            if (kMom) {
                const float2 mf = f2(__ldcg(rec + 2 * kCs + lane), __ldcg(rec + 3 * kCs + lane));
                MA = mulc_add(fma2(len, A, MA), ls.hi, ls.lo, mf);
            }
            A = mulc_add(A, ls.hi, ls.lo, f);
        }
        // across the lower ranks of this cluster
        const int d = c.rank * c.n_tok;
        const HiLo ld = decay_over_blocks(c, c.rank);
        if (kMom) MX = mulc_add(fma2(dup(static_cast<float>(d)), A, MA), ld.hi, ld.lo, MX);
        X = mulc_add(A, ld.hi, ld.lo, X);
    }
}
// Towards earlier tokens: Y = state entering this CTA from the higher ranks, S = the CTA's own aggregate.
__device__ __noinline__ void seg_exchange_reverse(const Ctx& c, int level, float2& Y, float2 S, int& flag) {
    const int lane = c.lane;
    if (c.rank == 0 && c.seg > 0) {
        const float2 hi = dup(c.consts[kLamC_hi * kCs + lane]), lo = dup(c.consts[kLamC_lo * kCs + lane]);
        const float2 R = mulc_add(Y, hi, lo, S);
        float* rec = c.xseg + seg_index(c, c.seg, level, 1) * kSegRec;
        rec[lane] = R.x; rec[kCs + lane] = R.y;
        __threadfence();
        __syncwarp();
        if (lane == 0) sm100::flag_release(c.xflag + seg_index(c, c.seg, level, 1), 1u | (flag ? 2u : 0u));
    }
    if (c.seg + 1 < c.segs) {
        const unsigned bits = seg_wait(c, c.seg + 1, c.segs - 1 - c.seg, level, 1);
        if (bits & 2u) flag = 1;
        const HiLo ls = decay_over_blocks(c, c.cluster);
        float2 A = f2(0.f, 0.f);
        for (int q = c.segs - 1; q > c.seg; --q) {
            const float* rec = c.xseg + seg_index(c, q, level, 1) * kSegRec;
            A = mulc_add(A, ls.hi, ls.lo, f2(__ldcg(rec + lane), __ldcg(rec + kCs + lane)));
        }
        const HiLo ld = decay_over_blocks(c, c.cluster - 1 - c.rank);
        Y = mulc_add(A, ld.hi, ld.lo, Y);
    }
}
// OR of this CTA's and the other CTAs' out-of-range flags (level 0), from the flag words of the blocks they sent
template <typename RW>
__device__ __forceinline__ int cluster_flag(const Ctx& c, int any) {
    const int lane = c.lane;
    const int other = (lane < c.cluster && lane != c.rank)
                          ? __float_as_int(c.peers[(lane - (lane > c.rank ? 1 : 0)) * RW::kBlockF + kCs * (lane < c.rank ? RW::kF : RW::kR)]) : 0;
    return __any_sync(0xffffffffu, (other | any) != 0) ? 1 : 0;
}

// One exchange level on plain floats (steps 1-4 of the file header).  F / MF: this thread's sub-chunk
// aggregate relative to the first token after its 16 tokens (and its first moment in distance), R:
// relative to the last token before them.  Returns with `unsafe` = OR over the cluster of `unsafe`
// (level 0 only).
//
// kLocal: no cluster; the states returned are relative to the CTA, whose own sums go to memory if anyone needs them.  kLinked: several
// clusters.
template <typename RW, bool kLocal, bool kLinked>
__device__ __forceinline__ Enter fast_exchange(const Ctx& c, int level, Pair2 F, Pair2 MF, Pair2 R, bool& unsafe TL_ARGS) {
    constexpr bool kMom = RW::kF == 4;
    const int lane = c.lane, warp = c.warp, nw = c.n_warps;
    const int p = lane & 15;
    const bool upper = lane >= 16;
    const float2 l16h = *reinterpret_cast<const float2*>(c.consts + kLam16_hi * kCs + 2 * p);
    const float2 l16l = *reinterpret_cast<const float2*>(c.consts + kLam16_lo * kCs + 2 * p);
    const float2 len16 = dup(static_cast<float>(kL));
    // (1) the two halves of the span combine through shuffles; the lower half-warp posts the span record
    Pair2 keepA, keepM;        // what this thread needs of its partner afterwards
    {
        const Pair2 oF{shfl2(F.n, 16), shfl2(F.d, 16)};
        const Pair2 oR{shfl2(R.n, 16), shfl2(R.d, 16)};
        Pair2 oMF{f2(0.f, 0.f), f2(0.f, 0.f)};
        if (kMom) oMF = Pair2{shfl2(MF.n, 16), shfl2(MF.d, 16)};
        keepA = upper ? oF : oR;      // upper half: the lower half's F; lower half: the upper half's R
        keepM = oMF;                  // upper half: the lower half's first moments
        if (!upper) {
            // F, MF, R are the lower half's, oF, oMF, oR the upper half's
            float* s = c.sub + warp * (RW::kSub * kCs) + 2 * p;
            *reinterpret_cast<float2*>(s) = mulc_add(F.n, l16h, l16l, oF.n);
            *reinterpret_cast<float2*>(s + kCs) = mulc_add(F.d, l16h, l16l, oF.d);
            if (kMom) {
                *reinterpret_cast<float2*>(s + 2 * kCs) = mulc_add(fma2(len16, F.n, MF.n), l16h, l16l, oMF.n);
                *reinterpret_cast<float2*>(s + 3 * kCs) = mulc_add(fma2(len16, F.d, MF.d), l16h, l16l, oMF.d);
            }
            *reinterpret_cast<float2*>(s + RW::kF * kCs) = mulc_add(oR.n, l16h, l16l, R.n);
            *reinterpret_cast<float2*>(s + (RW::kF + 1) * kCs) = mulc_add(oR.d, l16h, l16l, R.d);
        }
    }
    const int any = __syncthreads_or(unsafe ? 1 : 0);
    float2 ctaP = f2(0.f, 0.f), ctaM = f2(0.f, 0.f), ctaS = f2(0.f, 0.f);     // the CTA's own aggregates (scan warps)
    TL_MARK(12 + level * 5);
    // (2) serial walk over the spans, one warp per direction, lane = channel, state = (a, b)
    const int scanF = 0, scanR = nw > 1 ? 1 : 0;
    if (warp == scanF) {
        const float2 hi2 = dup(c.consts[kLam32_hi * kCs + lane]), lo2 = dup(c.consts[kLam32_lo * kCs + lane]);
        const float2 len2 = dup(static_cast<float>(kSpan));
        float2 P = f2(0.f, 0.f), M = f2(0.f, 0.f);
        // all loads first, then the dependent chain, storing as it goes: nothing waits on shared memory
        float2 f[kMaxWarps], mf[kMaxWarps];
#pragma unroll
        for (int s = 0; s < kMaxWarps; ++s) {
            f[s] = f2(0.f, 0.f);
            mf[s] = f2(0.f, 0.f);
            if (s < nw) {
                const float* q = c.sub + s * (RW::kSub * kCs) + lane;
                f[s] = f2(q[0], q[kCs]);
                if (kMom) mf[s] = f2(q[2 * kCs], q[3 * kCs]);
            }
        }
        if (level == 1) TL_MARK(22);
#pragma unroll
        for (int s = 0; s < kMaxWarps; ++s) {
            if (s < nw) {
                float* q = c.sub + s * (RW::kSub * kCs) + lane;
                q[0] = P.x; q[kCs] = P.y;
                if (kMom) {
                    q[2 * kCs] = M.x; q[3 * kCs] = M.y;
                    M = mulc_add(fma2(len2, P, M), hi2, lo2, mf[s]);
                }
                P = mulc_add(P, hi2, lo2, f[s]);
            }
        }
        if (level == 1) TL_MARK(23);
        if (kLinked) { ctaP = P; ctaM = M; }
        if (kLocal) {
            c.cta_sums[lane] = P.x; c.cta_sums[kCs + lane] = P.y;
            if (kMom) { c.cta_sums[2 * kCs + lane] = M.x; c.cta_sums[3 * kCs + lane] = M.y; }
        } else {
            // the CTA's aggregate (and its flag) for the higher ranks: into the outgoing block
            float* st = c.stage;
            if (kMom) *reinterpret_cast<float4*>(st + lane * 4) = make_float4(P.x, P.y, M.x, M.y);
            else *reinterpret_cast<float2*>(st + lane * 2) = P;
            if (lane == 0) st[kCs * RW::kF] = __int_as_float(any);
        }
    }
    if (warp == scanR) {
        const float2 hi2 = dup(c.consts[kLam32_hi * kCs + lane]), lo2 = dup(c.consts[kLam32_lo * kCs + lane]);
        float2 S = f2(0.f, 0.f);
        float2 r[kMaxWarps];
#pragma unroll
        for (int s = 0; s < kMaxWarps; ++s) {
            r[s] = f2(0.f, 0.f);
            if (s < nw) {
                const float* q = c.sub + s * (RW::kSub * kCs) + RW::kF * kCs + lane;
                r[s] = f2(q[0], q[kCs]);
            }
        }
#pragma unroll
        for (int s = kMaxWarps - 1; s >= 0; --s) {
            if (s < nw) {
                float* q = c.sub + s * (RW::kSub * kCs) + RW::kF * kCs + lane;
                q[0] = S.x; q[kCs] = S.y;
                S = mulc_add(S, hi2, lo2, r[s]);
            }
        }
        if (kLinked) ctaS = S;
        if (kLocal) {
            c.cta_sums[RW::kF * kCs + lane] = S.x; c.cta_sums[(RW::kF + 1) * kCs + lane] = S.y;
        } else {
            float* st = c.stage + RW::kBlockF;
            *reinterpret_cast<float2*>(st + lane * 2) = S;
            if (lane == 0) st[kCs * RW::kR] = __int_as_float(any);
        }
    }
    // every warp sends the blocks to its share of the other CTAs (rank = warp, warp + n_warps, ...):
    // lane = channel, one record per lane, lane 0 also the flag word
    if (level == 1) TL_MARK(24);
    if (!kLocal) {
        __syncthreads();
    }
    if (level == 1) TL_MARK(25);
    if (!kLocal && !c.withhold) {
        const uint32_t bar_off = sm100::smem_u32(c.xbar + level) - sm100::smem_u32(c.peers);
        for (int r = warp; r < c.cluster; r += nw) {
            if (r == c.rank) continue;
            const uint32_t rb = peer_addr(c.peers, r);
            const uint32_t slot = rb + static_cast<uint32_t>((c.rank - (c.rank > r ? 1 : 0)) * RW::kBlockF) * 4u;
            if (r > c.rank) {
                if (kMom) st_async4(slot + lane * 16u, *reinterpret_cast<const float4*>(c.stage + lane * 4), rb + bar_off);
                else st_async2(slot + lane * 8u, *reinterpret_cast<const float2*>(c.stage + lane * 2), rb + bar_off);
                if (lane == 0) st_async1(slot + kCs * RW::kF * 4u, c.stage[kCs * RW::kF], rb + bar_off);
            } else {
                st_async2(slot + lane * 8u, *reinterpret_cast<const float2*>(c.stage + RW::kBlockF + lane * 2), rb + bar_off);
                if (lane == 0) st_async1(slot + kCs * RW::kR * 4u, c.stage[RW::kBlockF + kCs * RW::kR], rb + bar_off);
            }
        }
    }
    TL_MARK(13 + level * 5);
    // (3) wait for the other CTAs' bytes, combine them
    bool heard = true;
    if (!kLocal && (warp == scanF || warp == scanR)) {
        heard = sm100::mbar_wait(c.xbar + level, 0, c.spin_limit);
        if (!heard && lane == 0) gave_up(c, 1u);
    }
    TL_MARK(14 + level * 5);
    if (!kLocal && warp == scanF) {
        float2 X = f2(0.f, 0.f), MX = f2(0.f, 0.f);
        int flag = any;
        const float2 hi2 = dup(c.consts[kLamC_hi * kCs + lane]), lo2 = dup(c.consts[kLamC_lo * kCs + lane]);
        const float2 len2 = dup(static_cast<float>(c.n_tok));
        for (int r0 = 0; r0 < c.rank; r0 += kBatch) {
            float2 f[kBatch], mf[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                f[j] = f2(0.f, 0.f);
                mf[j] = f2(0.f, 0.f);
                if (r0 + j < c.rank) {
                    const float* q = c.peers + (r0 + j) * RW::kBlockF + lane * RW::kF;      // lower ranks: slot = rank
                    if (kMom) {
                        const float4 t = *reinterpret_cast<const float4*>(q);
                        f[j] = f2(t.x, t.y);
                        mf[j] = f2(t.z, t.w);
                    } else {
                        f[j] = *reinterpret_cast<const float2*>(q);
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                if (r0 + j < c.rank) {
                    if (kMom) MX = mulc_add(fma2(len2, X, MX), hi2, lo2, mf[j]);
                    X = mulc_add(X, hi2, lo2, f[j]);
                }
            }
        }
        if (level == 0) flag = cluster_flag<RW>(c, any || !heard);
        if (kLinked) seg_exchange_forward<kMom>(c, level, X, MX, ctaP, ctaM, flag);
        c.cta[lane] = X.x; c.cta[kCs + lane] = X.y;
        if (kMom) { c.cta[2 * kCs + lane] = MX.x; c.cta[3 * kCs + lane] = MX.y; }
        if (lane == 0) c.flag[0] = static_cast<unsigned>(flag);
    }
    if (!kLocal && warp == scanR) {
        float2 Y = f2(0.f, 0.f);
        const float2 hi2 = dup(c.consts[kLamC_hi * kCs + lane]), lo2 = dup(c.consts[kLamC_lo * kCs + lane]);
        for (int r0 = c.cluster - 1; r0 > c.rank; r0 -= kBatch) {
            float2 f[kBatch];
#pragma unroll
            for (int j = 0; j < kBatch; ++j) {
                f[j] = f2(0.f, 0.f);
                if (r0 - j > c.rank) f[j] = *reinterpret_cast<const float2*>(c.peers + (r0 - j - 1) * RW::kBlockF + lane * 2);
            }
#pragma unroll
            for (int j = 0; j < kBatch; ++j)
                if (r0 - j > c.rank) Y = mulc_add(Y, hi2, lo2, f[j]);
        }
        if (kLinked) {
            int flag = 0;
            if (level == 0) flag = cluster_flag<RW>(c, any || !heard);
            seg_exchange_reverse(c, level, Y, ctaS, flag);
            if (lane == 0) c.flag[1] = static_cast<unsigned>(flag);
        }
        c.cta[RW::kF * kCs + lane] = Y.x; c.cta[(RW::kF + 1) * kCs + lane] = Y.y;
    }
    TL_MARK(15 + level * 5);
    __syncthreads();
    TL_MARK(16 + level * 5);
    // (4) outside state moved to this span's edges + inside state; then to this half's edges
    Enter e;
    {
        const auto row = [](const float* x, int r) { return *reinterpret_cast<const float2*>(x + r * kCs); };
        const float* s = c.sub + warp * (RW::kSub * kCs) + 2 * p;
        Pair2 Pw, MPw{f2(0.f, 0.f), f2(0.f, 0.f)}, Sw;
        if (kLocal) {
            Pw = Pair2{row(s, 0), row(s, 1)};
            if (kMom) MPw = Pair2{row(s, 2), row(s, 3)};
            Sw = Pair2{row(s, RW::kF), row(s, RW::kF + 1)};
        } else {
            const float2 wl2 = row(c.consts + 2 * p, kWl2);
            const float dP = static_cast<float>(kSpan * warp), dS = static_cast<float>(kSpan * (nw - 1 - warp));
            const float2 pP = f2(ex2(-wl2.x * dP), ex2(-wl2.y * dP)), pS = f2(ex2(-wl2.x * dS), ex2(-wl2.y * dS));
            const float* g = c.cta + 2 * p;
            const float2 Xn = row(g, 0), Xd = row(g, 1);
            Pw = Pair2{fma2(pP, Xn, row(s, 0)), fma2(pP, Xd, row(s, 1))};
            if (kMom) {
                const float2 MXn = row(g, 2), MXd = row(g, 3);
                MPw.n = fma2(pP, fma2(dup(dP), Xn, MXn), row(s, 2));
                MPw.d = fma2(pP, fma2(dup(dP), Xd, MXd), row(s, 3));
            }
            const float2 Yn = row(g, RW::kF), Yd = row(g, RW::kF + 1);
            Sw = Pair2{fma2(pS, Yn, row(s, RW::kF)), fma2(pS, Yd, row(s, RW::kF + 1))};
        }
        if (upper) {
            e.P = Pair2{mulc_add(Pw.n, l16h, l16l, keepA.n), mulc_add(Pw.d, l16h, l16l, keepA.d)};
            e.MP = Pair2{mulc_add(fma2(len16, Pw.n, MPw.n), l16h, l16l, keepM.n), mulc_add(fma2(len16, Pw.d, MPw.d), l16h, l16l, keepM.d)};
            e.S = Sw;
        } else {
            e.P = Pw;
            e.MP = MPw;
            e.S = Pair2{mulc_add(Sw.n, l16h, l16l, keepA.n), mulc_add(Sw.d, l16h, l16l, keepA.d)};
        }
        if (level == 0) unsafe = kLocal ? any != 0 : kLinked ? (c.flag[0] | c.flag[1]) != 0u : c.flag[0] != 0u;
    }
    return e;
}

// ---- states kept in memory ---------------------------------------------------------------------
__device__ __forceinline__ void put_state(float* at, int rows, const Enter& e, bool moments) {
    const auto put = [&](int r, float2 v) { *reinterpret_cast<float2*>(at + r * kCs) = v; };
    put(0, e.P.n); put(1, e.P.d);
    if (moments) { put(2, e.MP.n); put(3, e.MP.d); }
    put(rows - 2, e.S.n); put(rows - 1, e.S.d);
}
template <bool kMom>
__device__ __forceinline__ Enter get_state(const float* at, int rows) {
    const auto get = [&](int r) { return __ldg(reinterpret_cast<const float2*>(at + r * kCs)); };
    Enter e;
    e.P = Pair2{get(0), get(1)};
    e.MP = Pair2{f2(0.f, 0.f), f2(0.f, 0.f)};
    if (kMom) e.MP = Pair2{get(2), get(3)};
    e.S = Pair2{get(rows - 2), get(rows - 1)};
    return e;
}
// e: relative to the CTA; g: what enters the CTA, rows of kCs floats in shared memory; dP, dS: tokens between the CTA's edges
// and the sub-chunk's
template <bool kMom>
__device__ __forceinline__ void add_outside(Enter& e, const float* g, int rows, float2 wl2, float dP, float dS) {
    const auto row = [&](int r) { return *reinterpret_cast<const float2*>(g + r * kCs); };
    const float2 pP = f2(ex2(-wl2.x * dP), ex2(-wl2.y * dP)), pS = f2(ex2(-wl2.x * dS), ex2(-wl2.y * dS));
    const float2 Xn = row(0), Xd = row(1);
    e.P = Pair2{fma2(pP, Xn, e.P.n), fma2(pP, Xd, e.P.d)};
    if (kMom) e.MP = Pair2{fma2(pP, fma2(dup(dP), Xn, row(2)), e.MP.n), fma2(pP, fma2(dup(dP), Xd, row(3)), e.MP.d)};
    e.S = Pair2{fma2(pS, row(rows - 2), e.S.n), fma2(pS, row(rows - 1), e.S.d)};
}

// ---- the kernel -----------------------------------------------------------------------------------
// kStash: tokens whose leftward state a thread keeps in registers at a time (16: one reverse sweep
// per sub-chunk; 8: the second half is swept twice, for half the registers).
// kHalf: k, v, gy and the outputs are bfloat16 tensors (float32 arithmetic and shared-memory state all the same).
template <bool kBwd, int kStash, bool kHalf, Mode kMode>
__global__ void __launch_bounds__(kMaxThreads, kBwd ? 2 : 3)
biwkv_resident_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_g,     // backward: gy
                      const __grid_constant__ CUtensorMap map_o0,    // forward: y ; backward: gk
                      const __grid_constant__ CUtensorMap map_o1,    // backward: gv
                      const Params p) {
    using RW = Rows<kBwd, kMode>;
    constexpr bool kCluster = kUsesCluster<kMode>, kLinked = kMode == Mode::linked, kSums = kMode == Mode::sums || kMode == Mode::sums_keep;
    constexpr bool kOwn1 = kCluster || (kSums && !kBwd);        // level 1 is this launch's to sum up; else given
    constexpr bool kOwn2 = kBwd && kMode != Mode::spread;       // level 2 likewise
    constexpr bool kMom1 = RW::kF == 4;                         // level 1 carries first moments
    constexpr bool kResults = !kSums;                           // the launch writes results
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pr = lane & 15, upper = lane >> 4;
    const int nw = p.n_warps;
    const int slot_floats = p.n_tok * kCs;
    float* slot_k = reinterpret_cast<float*>(smem_raw);
    float* slot_v = slot_k + slot_floats;
    float* slot_g = slot_v + slot_floats;                       // backward only
    Ctx c;
    c.sub = slot_k + RW::kSlots * slot_floats;
    c.peers = c.sub + nw * (RW::kSub * kCs);
    c.stage = c.peers + (kCluster ? RW::kPeerFloats : 0);
    c.cta = c.stage + RW::kBlockF + RW::kBlockR;
    c.consts = c.cta + kOutsideRows<kBwd, kMode> * kCs;
    uint64_t* full = reinterpret_cast<uint64_t*>(c.consts + kConstRows * kCs);   // [kMaxWarps]: k, v of one span each
    uint64_t* gfull = full + kMaxWarps;  // [kMaxWarps]: backward, gy of one span each (first needed in pass 2)
    c.xbar = gfull + kMaxWarps;
    c.flag = reinterpret_cast<unsigned*>(c.xbar + 2);
    c.status = p.status;
    c.mirror = p.mirror;
    c.warp = warp; c.lane = lane; c.n_warps = nw; c.n_tok = p.n_tok; c.cluster = p.cluster;
    const int blk_id = kMode == Mode::spread && p.reverse ? static_cast<int>(gridDim.x - 1 - blockIdx.x) : static_cast<int>(blockIdx.x);
    const int unit = blk_id / p.ctas, cta = blk_id - unit * p.ctas;
    c.rank = kCluster ? static_cast<int>(cluster_rank()) : 0;
    c.spin_limit = p.spin_limit;
    c.withhold = c.rank == p.withhold_rank;

#ifdef VRWKV_TIMELINE
    long long* tl_base = g_tl_base;
    int tl_slot = -1;
    if (tl_base != nullptr) {
        const int mid = (static_cast<int>(gridDim.x) / 2 / p.cluster) * p.cluster;
        if (static_cast<int>(blockIdx.x) < kTlCtas) tl_slot = blockIdx.x;
        else if (static_cast<int>(blockIdx.x) >= mid && static_cast<int>(blockIdx.x) < mid + kTlCtas) tl_slot = kTlCtas + blockIdx.x - mid;
        if (tl_slot >= 0 && threadIdx.x == 0) {
            unsigned long long gt; unsigned smid;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(gt));
            asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
            tl_base[(tl_slot * 2) * kTlMarks + 30] = static_cast<long long>(gt);
            tl_base[(tl_slot * 2) * kTlMarks + 31] = smid;
        }
    }
#endif
    TL_MARK(0);
    const int b = unit / p.n_strips, strip = unit - b * p.n_strips;
    const int tok0 = cta * p.n_tok;
    if (kCluster) {      // the segments of a unit are neighbours in launch order
        c.seg = kLinked ? cta / p.cluster : 0; c.segs = kLinked ? p.segs : 1; c.unit = unit;
        c.xseg = p.xseg; c.xflag = p.xflag;
    }
    // this thread's sub-chunk among the kept states, and the CTA's place among those of the CTAs
    const int subs = 2 * nw, sub = 2 * warp + upper;
    const size_t sub_at = ((static_cast<size_t>(blk_id) * subs + sub) * p.state_rows) * kCs + 2 * pr;
    c.cta_sums = kSums ? (kBwd ? p.ctas2 : p.ctas1) + static_cast<size_t>(blk_id) * p.state_rows * kCs : nullptr;

    if (lane == 0) {
        // every warp fetches its own span: one box per tensor, k and v on one barrier, gy on another;
        // the warp starts as soon as its own 32 tokens are there
        constexpr uint32_t kSpanBytes = kSpan * kCs * 4u;
        sm100::mbar_init(full + warp, 1);
        if (kBwd) sm100::mbar_init(gfull + warp, 1);
        sm100::mbar_init_fence();
        if (kHalf) {
            // bfloat16: one box per 16-token sub-chunk, into the upper half of the sub-chunk's own area
            sm100::mbar_expect_tx(full + warp, 4 * kHalfAreaBytes);
            if (kBwd) sm100::mbar_expect_tx(gfull + warp, 2 * kHalfAreaBytes);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = warp * kSpan + h * kL;
                sm100::tma_load_3d(reinterpret_cast<unsigned char*>(slot_k + r * kCs) + kHalfAreaBytes, &map_k, full + warp, strip * kCs, tok0 + r, b);
                sm100::tma_load_3d(reinterpret_cast<unsigned char*>(slot_v + r * kCs) + kHalfAreaBytes, &map_v, full + warp, strip * kCs, tok0 + r, b);
                if (kBwd) sm100::tma_load_3d(reinterpret_cast<unsigned char*>(slot_g + r * kCs) + kHalfAreaBytes, &map_g, gfull + warp, strip * kCs, tok0 + r, b);
            }
        } else {
            sm100::mbar_expect_tx(full + warp, 2 * kSpanBytes);
            sm100::tma_load_3d(slot_k + warp * kSpan * kCs, &map_k, full + warp, strip * kCs, tok0 + warp * kSpan, b);
            sm100::tma_load_3d(slot_v + warp * kSpan * kCs, &map_v, full + warp, strip * kCs, tok0 + warp * kSpan, b);
        }
        if (kBwd && !kHalf) {
            sm100::mbar_expect_tx(gfull + warp, kSpanBytes);
            sm100::tma_load_3d(slot_g + warp * kSpan * kCs, &map_g, gfull + warp, strip * kCs, tok0 + warp * kSpan, b);
        }
    }
    if (threadIdx.x == 0) {
        c.flag[2] = 0u;
        for (int l = 0; l < RW::kLevels; ++l) sm100::mbar_init(c.xbar + l, 1);
        sm100::mbar_init_fence();
        if (kCluster) {
            // bytes the other CTAs will send per level: a block from every lower rank (towards later
            // tokens) and from every higher rank (towards earlier ones)
            const uint32_t bytes = static_cast<uint32_t>(c.rank) * (kCs * RW::kF + 1) * 4u + static_cast<uint32_t>(p.cluster - 1 - c.rank) * (kCs * RW::kR + 1) * 4u;
            sm100::mbar_expect_tx(c.xbar, bytes);
            if (kBwd) sm100::mbar_expect_tx(c.xbar + 1, bytes);
        }
    }
    // given states: fetched while the tiles are on their way.  The rows of the CTA go to c.cta (level 1) and to the unused span
    // records (level 2).
    Enter e1, e2;
    unsigned given_up = 0u;
    if (!kOwn1) {
        e1 = get_state<kBwd && !kSums>(p.states1 + sub_at, p.state_rows);
        given_up = __ldg(p.out_of_range);
        for (int i = threadIdx.x; i < p.state_rows * kCs; i += blockDim.x) {
            c.cta[i] = __ldg(p.ctas1 + static_cast<size_t>(blk_id) * p.state_rows * kCs + i);
            if (kBwd && !kSums) c.sub[i] = __ldg(p.ctas2 + static_cast<size_t>(blk_id) * kStateRows * kCs + i);
        }
    }
    if (kBwd && !kOwn2) e2 = get_state<true>(p.states2 + sub_at, kStateRows);
    {
        // double precision once per channel: a rounded lambda multiplied up over thousands of tokens
        // would drift by distance * 6e-8.  Six exponentials, spread over the warps (lane = channel).
        const int ch = strip * kCs + lane;
        const double wd = (ch < p.C) ? static_cast<double>(p.w[ch]) : 0.0;
        const double ud = (ch < p.C) ? static_cast<double>(p.u[ch]) : 0.0;
        // tasks: 0 lambda (+ w log2 e), 1 e^{u+w}, 2..4 lambda^16, lambda^32, lambda^n_tok as (high, low)
        for (int task = warp; task < 5; task += nw) {
            const double arg = task == 0 ? -wd : task == 1 ? ud + wd : -wd * (task == 2 ? kL : task == 3 ? kSpan : p.n_tok);
            const double x = exp(arg);
            const float hi = static_cast<float>(x);
            const int row = task == 0 ? kLam : task == 1 ? kCuw : task == 2 ? kLam16_hi : task == 3 ? kLam32_hi : kLamC_hi;
            c.consts[row * kCs + lane] = hi;
            if (task >= 2) c.consts[(row + 1) * kCs + lane] = static_cast<float>(x - static_cast<double>(hi));
            if (task == 0) c.consts[kWl2 * kCs + lane] = static_cast<float>(wd * 1.4426950408889634);
        }
    }
    __syncthreads();
    // every CTA of the cluster has initialised its mbarriers before any other CTA sends to them:
    // arrive here, wait once the tiles have landed (long since complete by then)
    // (relaxed: the mbarrier-init fence above is what publishes the initialisation)
    if (kCluster) cluster_arrive_relaxed();
    const int ch0 = strip * kCs + 2 * pr;
    const float2 w2 = (ch0 < p.C) ? *reinterpret_cast<const float2*>(p.w + ch0) : f2(0.f, 0.f);
    const float2 u2 = (ch0 < p.C) ? *reinterpret_cast<const float2*>(p.u + ch0) : f2(0.f, 0.f);
    const float2 lam2 = *reinterpret_cast<const float2*>(c.consts + kLam * kCs + 2 * pr);
    const float2 wl2 = *reinterpret_cast<const float2*>(c.consts + kWl2 * kCs + 2 * pr);
    const float2 c2 = *reinterpret_cast<const float2*>(c.consts + kCuw * kCs + 2 * pr);

    TL_MARK(1);
    if (!sm100::mbar_wait(full + warp, 0, kSpinLimit)) report_failure(p.status, p.mirror, 2u);
    if (kCluster) cluster_wait();
    TL_MARK(2);

    const int row0 = warp * kSpan + upper * kL;
    const int n = max(0, min(kL, p.T - (tok0 + row0)));      // valid tokens of this sub-chunk
    constexpr int kRow = kCs / 2;                              // float2 per row
    float2* k2 = reinterpret_cast<float2*>(slot_k + row0 * kCs) + pr;
    float2* v2 = reinterpret_cast<float2*>(slot_v + row0 * kCs) + pr;
    float2* g2 = reinterpret_cast<float2*>(slot_g + row0 * kCs) + pr;
    float* const area_k = slot_k + row0 * kCs;
    float* const area_v = slot_v + row0 * kCs;
    float* const area_g = slot_g + row0 * kCs;
    // rows past T arrive as zeros; a k of -1e30 makes their terms vanish without any masking below
    if (n < kL)
        for (int i = n; i < kL; ++i) {
            if (kHalf) *(reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<unsigned char*>(area_k) + kHalfAreaBytes + i * kHalfRowBytes) + pr) = __float2bfloat162_rn(-1e30f);
            else k2[i * kRow] = f2(-1e30f, -1e30f);
        }
    __syncwarp();

    // ---- level 1, pass 1: terms z = lambda e^{k} [v, 1] in place of k, v; sub-chunk aggregates ----
    Pair2 F{f2(0.f, 0.f), f2(0.f, 0.f)}, MF{f2(0.f, 0.f), f2(0.f, 0.f)}, R{f2(0.f, 0.f), f2(0.f, 0.f)};
    float2 kmax = f2(0.f, 0.f);
    {
        float2 mu = f2(1.f, 1.f);
        const float2 nwl2 = f2(-wl2.x, -wl2.y), l2e = dup(kLog2e);
        // loads of a group of tokens go first: a store into one slot may not be moved past a later load
        // from another slot by the compiler, so token-by-token code would expose every load's latency
#pragma unroll
        for (int g = 0; g < kL; g += kGroup) {
            float2 kk[kGroup], vv[kGroup];
#pragma unroll
            for (int j = 0; j < kGroup; ++j) { kk[j] = ld_in<kHalf>(area_k, g + j, pr); vv[j] = ld_in<kHalf>(area_v, g + j, pr); }
            if (kHalf) __syncwarp();      // in-place widening: every lane has read these rows before any lane writes over them
#pragma unroll
            for (int j = 0; j < kGroup; ++j) {
                const int i = g + j;
                const float2 k = kk[j], v = vv[j];
                if (kOwn1 && i < n) kmax = f2(fmaxf(kmax.x, fabsf(k.x)), fmaxf(kmax.y, fabsf(k.y)));
                const float2 t = fma2(k, l2e, nwl2);
                const float2 e = f2(ex2(t.x), ex2(t.y));
                const float2 zx = mul2(e, v);
                if (kResults || kBwd) {
                    k2[i * kRow] = zx;
                    v2[i * kRow] = e;
                }
                if (kOwn1) {
                    F.n = fma2(lam2, F.n, zx);
                    F.d = fma2(lam2, F.d, e);
                    if (kMom1) {
                        MF.n = fma2(lam2, MF.n, F.n);
                        MF.d = fma2(lam2, MF.d, F.d);
                    }
                    R.n = fma2(mu, zx, R.n);
                    R.d = fma2(mu, e, R.d);
                    mu = mul2(mu, lam2);
                }
            }
        }
    }
    const float dP = static_cast<float>(kL * sub), dS = static_cast<float>(kL * (subs - 1 - sub));    // tokens to the CTA's edges
    bool unsafe = given_up != 0u;
    TL_MARK(3);
    if (kOwn1) {
        const float Tf = static_cast<float>(p.T);
        unsafe = (2.f * kmax.x + fabsf(u2.x) + fabsf(w2.x) + fmaxf(-w2.x, 0.f) * Tf > kSafeRange) ||
                 (2.f * kmax.y + fabsf(u2.y) + fabsf(w2.y) + fmaxf(-w2.y, 0.f) * Tf > kSafeRange);
        e1 = fast_exchange<RW, kSums, kLinked>(c, 0, F, MF, R, unsafe TL_PASS);
    } else {
        add_outside<kBwd && !kSums>(e1, c.cta + 2 * pr, p.state_rows, wl2, dP, dS);
    }
    TL_MARK(4);
    if (kSums && !kBwd) {
        put_state(p.states1 + sub_at, p.state_rows, e1, kMom1);
        if (unsafe && threadIdx.x == 0) *reinterpret_cast<volatile unsigned*>(p.out_of_range) = 1u;
        return;
    }

    float2 gw = f2(0.f, 0.f), gu = f2(0.f, 0.f);
    if (kBwd && !sm100::mbar_wait(gfull + warp, 0, kSpinLimit)) report_failure(p.status, p.mirror, 2u);
    if (unsafe) {
        // the whole cluster takes this branch together; the count switches on the chunked kernels that stand by, which redo the whole
        // call (without clusters the word that was read does)
        if (kCluster && cta == 0 && threadIdx.x == 0) atomicAdd(p.redo_count, 1u);
        if (kCluster) stay_for_late_data(c, kBwd ? 2 : 1, kBwd ? 2 : 1);
        return;
    }
    if (!kBwd) {
        // ---- forward, pass 2: y = (P + S + e^{u} x) ratio, in place of the numerator term ----
        Pair2 P = e1.P;
#pragma unroll
        for (int blk = 0; blk < kL / kStash; ++blk) {
            Pair2 S = e1.S;
            float2 sn[kStash], sd[kStash];
#pragma unroll
            for (int i = kL - 1; i >= blk * kStash; --i) {
                if (i < (blk + 1) * kStash) { sn[i - blk * kStash] = S.n; sd[i - blk * kStash] = S.d; }
                S.n = fma2(lam2, S.n, k2[i * kRow]);
                S.d = fma2(lam2, S.d, v2[i * kRow]);
            }
#pragma unroll
            for (int g = 0; g < kStash; g += kGroup) {
                float2 zxs[kGroup], zys[kGroup];
#pragma unroll
                for (int j = 0; j < kGroup; ++j) { zxs[j] = k2[(blk * kStash + g + j) * kRow]; zys[j] = v2[(blk * kStash + g + j) * kRow]; }
                if (kHalf) __syncwarp();
#pragma unroll
                for (int j = 0; j < kGroup; ++j) {
                    const int i = blk * kStash + g + j;
                    const float2 zx = zxs[j], zy = zys[j];
                    const float2 nn = fma2(c2, zx, add2(P.n, sn[g + j]));
                    const float2 dd = fma2(c2, zy, add2(P.d, sd[g + j]));
                    const float2 y = mul2(nn, f2(rcp(dd.x), rcp(dd.y)));
                    st_out<kHalf>(area_k, i, pr, y);
                    P.n = fma2(lam2, P.n, zx);
                    P.d = fma2(lam2, P.d, zy);
                }
            }
        }
    } else {
        // the records the other CTAs sent for level 1 have been consumed: tell them (they wait for
        // this before sending level 2 into the same slots).  The reads are complete: their values
        // went into shared memory before the CTA barrier that precedes this point.
        if (kCluster) cluster_arrive_relaxed();
        // ---- backward, pass 2: recompute Den, y; G = gy / Den (in place of gy), -H = -G y (registers);
        //      gu; gw from pairs (output later than input); aggregates of [G, -H] ----
        float2 hn[kL];
        Pair2 rr{f2(0.f, 0.f), f2(0.f, 0.f)}, mr{f2(0.f, 0.f), f2(0.f, 0.f)}, q{f2(0.f, 0.f), f2(0.f, 0.f)};
        float2 gwa = f2(0.f, 0.f);
        {
            Pair2 P = e1.P, PM = e1.MP;
            float2 mu = lam2;
#pragma unroll
            for (int blk = 0; blk < kL / kStash; ++blk) {
                Pair2 S = e1.S;
                float2 sn[kStash], sd[kStash];
#pragma unroll
                for (int i = kL - 1; i >= blk * kStash; --i) {
                    if (i < (blk + 1) * kStash) { sn[i - blk * kStash] = S.n; sd[i - blk * kStash] = S.d; }
                    S.n = fma2(lam2, S.n, k2[i * kRow]);
                    S.d = fma2(lam2, S.d, v2[i * kRow]);
                }
#pragma unroll
                for (int g = 0; g < kStash; g += kGroupB) {
                    float2 zxs[kGroupB], zys[kGroupB], gys[kGroupB];
#pragma unroll
                    for (int j = 0; j < kGroupB; ++j) {
                        const int i = blk * kStash + g + j;
                        zxs[j] = k2[i * kRow]; zys[j] = v2[i * kRow]; gys[j] = ld_in<kHalf>(area_g, i, pr);
                    }
                    if (kHalf) __syncwarp();
#pragma unroll
                    for (int j = 0; j < kGroupB; ++j) {
                        const int i = blk * kStash + g + j;
                        const float2 zx = zxs[j], zy = zys[j];
                        const float2 nn = fma2(c2, zx, add2(P.n, sn[g + j]));
                        const float2 dd = fma2(c2, zy, add2(P.d, sd[g + j]));
                        // rows past T: gy = 0 must stay 0 whatever the denominator
                        const float2 inv = f2(rcp(fmaxf(dd.x, 1e-37f)), rcp(fmaxf(dd.y, 1e-37f)));
                        const float2 ny = f2(nn.x * -inv.x, nn.y * -inv.y);
                        const float2 g_ = mul2(gys[j], inv);
                        const float2 h = mul2(g_, ny);                  // -H
                        if (kResults) {
                            g2[i * kRow] = g_;
                            hn[i] = h;
                            gu = fma2(zx, g_, gu);
                            gu = fma2(zy, h, gu);
                            gwa = fma2(g_, PM.n, gwa);
                            gwa = fma2(h, PM.d, gwa);
                        }
                        P.n = fma2(lam2, P.n, zx);
                        P.d = fma2(lam2, P.d, zy);
                        if (kResults) {
                            PM.n = fma2(lam2, PM.n, P.n);
                            PM.d = fma2(lam2, PM.d, P.d);
                        }
                        if (!kOwn2) continue;
                        rr.n = fma2(lam2, rr.n, g_);
                        rr.d = fma2(lam2, rr.d, h);
                        mr.n = fma2(lam2, mr.n, rr.n);
                        mr.d = fma2(lam2, mr.d, rr.d);
                        q.n = fma2(mu, g_, q.n);
                        q.d = fma2(mu, h, q.d);
                        mu = mul2(mu, lam2);
                    }
                }
            }
            gu = mul2(gu, c2);
            rr.n = mul2(rr.n, lam2); rr.d = mul2(rr.d, lam2);
            mr.n = mul2(mr.n, lam2); mr.d = mul2(mr.d, lam2);
        }
        bool ignored = false;
        TL_MARK(5);
        if (kCluster) cluster_wait();
        if (kOwn2) e2 = fast_exchange<RW, kSums, kLinked>(c, 1, rr, mr, q, ignored TL_PASS);
        else add_outside<true>(e2, c.sub + 2 * pr, kStateRows, wl2, dP, dS);
        if (kSums) {
            put_state(p.states2 + sub_at, kStateRows, e2, true);
            return;
        }
        TL_MARK(6);
        // ---- backward, pass 3: gk, gv in place of the terms; gw from pairs (output earlier than input).
        //      Adjoint states are kept divided by lambda, so that [G, -H] enter without a multiply. ----
        {
            const float2 il2 = f2(rcp(lam2.x), rcp(lam2.y));
            Pair2 Rp{mul2(e2.P.n, il2), mul2(e2.P.d, il2)}, MRp{mul2(e2.MP.n, il2), mul2(e2.MP.d, il2)};
            const Pair2 Qin{mul2(e2.S.n, il2), mul2(e2.S.d, il2)};
#pragma unroll
            for (int blk = 0; blk < kL / kStash; ++blk) {
                Pair2 Q = Qin;
                float2 sn[kStash], sd[kStash];
#pragma unroll
                for (int i = kL - 1; i >= blk * kStash; --i) {
                    if (i < (blk + 1) * kStash) { sn[i - blk * kStash] = Q.n; sd[i - blk * kStash] = Q.d; }
                    Q.n = fma2(lam2, Q.n, g2[i * kRow]);
                    Q.d = fma2(lam2, Q.d, hn[i]);
                }
#pragma unroll
                for (int g = 0; g < kStash; g += kGroupB) {
                    float2 zxs[kGroupB], zys[kGroupB], gs_[kGroupB];
#pragma unroll
                    for (int j = 0; j < kGroupB; ++j) {
                        const int i = blk * kStash + g + j;
                        zxs[j] = k2[i * kRow]; zys[j] = v2[i * kRow]; gs_[j] = g2[i * kRow];
                    }
                    if (kHalf) __syncwarp();
#pragma unroll
                    for (int j = 0; j < kGroupB; ++j) {
                        const int i = blk * kStash + g + j;
                        const float2 g_ = gs_[j], h = hn[i];
                        const float2 zx = zxs[j], zy = zys[j];
                        const float2 AG = fma2(c2, g_, add2(sn[g + j], Rp.n));
                        const float2 AH = fma2(c2, h, add2(sd[g + j], Rp.d));      // -A^H
                        st_out<kHalf>(area_v, i, pr, mul2(zy, AG));
                        st_out<kHalf>(area_k, i, pr, fma2(zx, AG, mul2(zy, AH)));
                        gwa = fma2(zx, MRp.n, gwa);
                        gwa = fma2(zy, MRp.d, gwa);
                        Rp.n = fma2(lam2, Rp.n, g_);
                        Rp.d = fma2(lam2, Rp.d, h);
                        MRp.n = fma2(lam2, MRp.n, Rp.n);
                        MRp.d = fma2(lam2, MRp.d, Rp.d);
                    }
                }
            }
        }
        gw = f2(-gwa.x, -gwa.y);
    }
    TL_MARK(7);

    if (kBwd) {
        // this thread's own rows of the gy slot are free now: park its gw, gu there for the CTA sum
        g2[0] = gw;
        g2[kRow] = gu;
    }
    sm100::fence_proxy_async_smem();
    __syncthreads();
    if (kHalf) {
        // one box per sub-chunk (its 16 dense bfloat16 rows), issued by the warp that wrote them
        if (lane == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int r = warp * kSpan + h * kL;
                if (tok0 + r < p.T) {
                    sm100::tma_store_3d(&map_o0, slot_k + r * kCs, strip * kCs, tok0 + r, b);
                    if (kBwd) sm100::tma_store_3d(&map_o1, slot_v + r * kCs, strip * kCs, tok0 + r, b);
                }
            }
            sm100::tma_store_commit();
        }
    } else if (threadIdx.x == 0 && (!kLinked || tok0 < p.T)) {
        sm100::tma_store_3d(&map_o0, slot_k, strip * kCs, tok0, b);
        if (kBwd) sm100::tma_store_3d(&map_o1, slot_v, strip * kCs, tok0, b);
        sm100::tma_store_commit();
    }
    if (kBwd && warp < 2) {
        for (int j = warp; j < 2; j += min(nw, 2)) {
            float acc = 0.f;
            for (int s = 0; s < 2 * nw; ++s) acc += slot_g[(s * kL + j) * kCs + lane];
            p.partial[(static_cast<size_t>(blk_id) * 2 + j) * kCs + lane] = acc;
        }
    }
    TL_MARK(8);
    if (kHalf ? lane == 0 : threadIdx.x == 0) sm100::tma_store_wait_read();   // shared memory may go once the stores have read it
    TL_MARK(9);
    if (kCluster) stay_for_late_data(c, 1, kBwd ? 2 : 1);
}

// out[j][c] = sum over sequences and cluster ranks of partial[cta][j][c % 32], fixed order
__global__ void __launch_bounds__(1024)
reduce_partials(Params p, float* __restrict__ out) {
    __shared__ float red[32][33];
    const int strip = blockIdx.x, j = blockIdx.y, lane = threadIdx.x;
    const int ch = strip * kCs + lane;
    if (*p.out_of_range != 0u) return;       // the chunked kernels redo the whole call and write gw, gu
    const int per_unit = p.ctas;
    const int rows = p.B * per_unit;
    float acc = 0.f;
    for (int r = threadIdx.y; r < rows; r += 32) {
        const int b = r / per_unit, rank = r - b * per_unit;
        const size_t cta = (static_cast<size_t>(b) * p.n_strips + strip) * per_unit + rank;
        acc += p.partial[(cta * 2 + j) * kCs + lane];
    }
    red[threadIdx.y][lane] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && ch < p.C) {
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) total += red[r][lane];
        out[static_cast<size_t>(j) * p.C + ch] = total;
    }
}

// Sequences longer than one cluster holds, where there are enough of them.
//   forward                  k, v -> sums of every 16 tokens and of every CTA (sums); the CTAs' sums chained along the sequence
//                            (this kernel); k, v and both -> y (spread)
//   backward                 the first two steps with first moments, unless the forward kept their results; k, v, gy and these
//                            -> sums of the adjoint pairs (sums); chained; everything -> gk, gv, gw, gu (spread)
// The launches are plain grids of independent CTAs, so each runs at the rate of HBM (5.9 to 6.9 TB/s for the bytes that it has to
// move, some of them from L2; the states of every 16 tokens are 1 to 1.5 bytes per element and level).  That is 22 bytes per element
// forward (23 with states kept) where k, v, y are 12, and 38 backward from kept states (47.5 without) where 20 are necessary, but nothing
// waits for another CTA.  Several clusters per sequence (linked) move the necessary bytes and spend more on the skew between their
// starts.  Forward + backward, float32: B=8, T=16384, C=768 1927 us linked, 1128 us so; B=16, T=4200 899 and 591 us.  (The latter move
// by 1 to 2 % with the board and with where the buffers lie.)  In one launch these steps were slower, beside 1060 us for separate launches of the same build: with a
// barrier of all CTAs between them and tiles handed out one by one 1228 us, taken by tickets in the order of the steps 1428 us, and so
// with neighbouring sequences' steps side by side, so that the second reads come from L2, 1224 us.
//
// This kernel: a warp takes one of four parts of a unit - towards later or earlier tokens, numerators or denominators -, lane =
// channel, T / 256 steps over a few KB.  In double precision: rounded to float at every step, the results were a third further
// from a float64 evaluation at T=32768.
// `seen` / `kept_seen`: the word for inputs out of range goes with states that are kept.
__global__ void __launch_bounds__(128)
biwkv_chain_kernel(float* __restrict__ sums, const float* __restrict__ w, int n_strips, int n_ctas, int n_tok, int rows, int C,
                   const unsigned* seen, unsigned* kept_seen) {
    constexpr int kStep = 16;
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 5, unit = blockIdx.x, ch = (unit % n_strips) * kCs + lane;
    if (kept_seen != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *kept_seen = *seen;
    const double x = exp(-(ch < C ? static_cast<double>(w[ch]) : 0.0) * n_tok), len = n_tok;
    const bool back = part >= 2, moments = !back && rows == kStateRows;
    const int step = (back ? -rows : rows) * kCs;
    float* at = sums + (static_cast<size_t>(unit) * n_ctas + (back ? n_ctas - 1 : 0)) * rows * kCs + ((part & 1) + (back ? rows - 2 : 0)) * kCs + lane;
    double P = 0.0, M = 0.0;
    for (int c0 = 0; c0 < n_ctas; c0 += kStep, at += kStep * step) {
        float f[kStep], m[kStep];
#pragma unroll
        for (int j = 0; j < kStep; ++j) {
            f[j] = c0 + j < n_ctas ? at[j * step] : 0.f;
            m[j] = moments && c0 + j < n_ctas ? at[j * step + 2 * kCs] : 0.f;
        }
#pragma unroll
        for (int j = 0; j < kStep; ++j)
            if (c0 + j < n_ctas) {
                at[j * step] = static_cast<float>(P);
                if (moments) {
                    at[j * step + 2 * kCs] = static_cast<float>(M);
                    M = fma(fma(len, P, M), x, static_cast<double>(m[j]));
                }
                P = fma(P, x, static_cast<double>(f[j]));
            }
    }
}

// ---- host side ------------------------------------------------------------------------------------
constexpr int kFwdStash = 8;
constexpr int kBwdStash = 8;

// test mode: rank 1 of every cluster withholds its sends and waits give up after 2^10 polls, so that
// the bounded waits can be seen to run out (status bit 0) without anything hanging
static std::atomic<bool> g_withhold{false};
void set_withhold_test(bool on) { g_withhold.store(on); }

struct Plan {
    int cluster = 0, segs = 1, n_warps = 0, n_tok = 0, ctas = 0;
    bool split = false;      // in separate launches
};

// How many CTAs hold a sequence, and in how many clusters.
//
// Up to 4096 tokens: not here (biwkv_strips.cu).
//
// Above, separate launches (see biwkv_chain_kernel) from kSplitCtas CTAs of 256 tokens on.  Below that one launch of linked
// clusters is as fast or faster, being fewer launches (forward / backward us, float32): B=1, C=192, T=8192 (192 CTAs) linked 25 /
// 45, separate 27 / 53; T=16384 (384) 29 / 73 and 31 / 72; T=32768 (768) 56 / 178 and 43 / 111; B=2, C=768, T=4200 (816) 49 / 114
// and 38 / 94.  At the line itself, forward + backward, linked / separate, replayed from a graph: B=2, T=8192, C=256 (512) float32 101 /
// 80, bfloat16 k, v with float32 w 112 / 92, with bfloat16 w 105 / 86; B=6, T=4200, C=192 (612) 116 / 88, 129 / 106, 122 / 96.  Called
// one by one such steps are host time either way, 112 to 150 us, of which the four more launches take 5 to 10 (B=4, T=4200, C=256, all
// bfloat16: 143 / 150).
// Linked clusters: about 2048 tokens (8 CTAs) each, since clusters of 8 fill more SMs than clusters of 16, up to kMaxSegs of
// them; the CTAs of a cluster follow from the tokens.
constexpr long long kSplitCtas = 512;
static bool make_plan(int B, int T, int C, Plan& pl) {
    if (C % 4 != 0) return false;      // no tensor maps over such rows, in either type
    constexpr int kCtaMax = kMaxWarps * kSpan;              // tokens one CTA holds
    constexpr int kSegMax = kMaxCluster * kCtaMax;          // tokens one cluster holds
    const auto up = [](int a, int b) { return (a + b - 1) / b; };
    if (T <= kSegMax) return false;
    pl.segs = std::max(up(T, kSegMax), std::min(kMaxSegs, (T + 1024) / 2048));
    if (pl.segs > kMaxSegs) return false;
    pl.split = static_cast<long long>(B) * up(C, kCs) * up(T, kCtaMax) >= kSplitCtas;
    if (pl.split) {
        pl.segs = pl.cluster = 1;
        pl.ctas = up(T, kCtaMax);
    } else {
        pl.cluster = up(up(T, pl.segs), kCtaMax);
        pl.ctas = pl.segs * pl.cluster;
    }
    pl.n_warps = up(up(T, pl.ctas), kSpan);
    pl.n_tok = pl.n_warps * kSpan;
    // every CTA owns a token, or at least every segment
    return static_cast<long long>(pl.split ? pl.ctas - 1 : (pl.segs - 1) * pl.cluster) * pl.n_tok < T;
}

struct DeviceState {
    bool probed = false, ok = false;
    // [tensor types][bwd][cluster][n_warps]: 0 unknown, 1 launchable, -1 not
    signed char fits[2][2][kMaxCluster + 1][kMaxWarps + 1] = {};
};
static std::mutex g_mutex;
static DeviceState g_dev[64];

template <bool kBwd, Types kTypes, Mode kMode>
static auto kernel() { return biwkv_resident_kernel<kBwd, kBwd ? kBwdStash : kFwdStash, kTypes != Types::f32, kMode>; }
template <typename F>
static bool allow(F* fn, size_t smem, bool cluster) {
    const void* f = reinterpret_cast<const void*>(fn);
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) == cudaSuccess &&
           (!cluster || cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
}
template <bool kBwd, Types kTypes, Mode kMode>
static bool allow_kernel() { return allow(kernel<kBwd, kTypes, kMode>(), smem_bytes<kBwd, kMode>(kMaxWarps), kUsesCluster<kMode>); }
template <bool kBwd, Types kTypes>
static bool allow_types() {
    return allow_kernel<kBwd, kTypes, Mode::linked>() && allow_kernel<kBwd, kTypes, Mode::sums>() && allow_kernel<kBwd, kTypes, Mode::spread>() &&
           allow_kernel<false, kTypes, Mode::sums_keep>();
}

template <bool kBwd, Types kTypes>
static bool fits(const Plan& pl) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lock(g_mutex);
    DeviceState& d = g_dev[dev & 63];
    if (!d.probed) {
        d.probed = true;
        int cl = 0;
        cudaDeviceGetAttribute(&cl, cudaDevAttrClusterLaunch, dev);
        d.ok = cl != 0 && tensor_map::encode_fn() != nullptr && allow_types<false, Types::f32>() && allow_types<false, Types::bf16>() &&
               allow_types<true, Types::f32>() && allow_types<true, Types::bf16>();
        if (!d.ok) cudaGetLastError();
    }
    if (!d.ok || pl.split) return d.ok;
    signed char& slot = d.fits[static_cast<int>(kTypes)][kBwd ? 1 : 0][pl.cluster][pl.n_warps];
    if (slot == 0) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(pl.cluster);
        cfg.blockDim = dim3(pl.n_warps * 32);
        cfg.dynamicSmemBytes = smem_bytes<kBwd>(pl.n_warps);
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeClusterDimension;
        at[0].val.clusterDim.x = pl.cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        int n = 0;
        const cudaError_t err = cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(kernel<kBwd, kTypes, Mode::linked>()), &cfg);
        if (err != cudaSuccess) cudaGetLastError();
        slot = (err == cudaSuccess && n > 0) ? 1 : -1;
    }
    return slot > 0;
}

bool eligible(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, Types types) {
    if (C % (types != Types::f32 ? 8 : 4) != 0) return false;                     // TMA row pitch must be 16-byte
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) & 15u) return false;    // TMA base alignment
    Plan pl;
    if (!make_plan(B, T, C, pl)) return false;
    const long long ctas = static_cast<long long>(B) * ((C + kCs - 1) / kCs) * pl.ctas;
    if (ctas > (1LL << 30)) return false;
    if (types == Types::wide) return false;      // the kernels that stand by have no such form
    if (types == Types::bf16) return bwd ? fits<true, Types::bf16>(pl) : fits<false, Types::bf16>(pl);
    return bwd ? fits<true, Types::f32>(pl) : fits<false, Types::f32>(pl);
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// states of sub-chunks and CTAs: out-of-range word | of the CTAs | of the sub-chunks
struct StatesCarve {
    size_t off_ctas, off_subs, total;
};
static StatesCarve carve_states(size_t units, const Plan& pl, int rows) {
    StatesCarve cv;
    cv.off_ctas = 256;
    cv.off_subs = cv.off_ctas + align_up(units * pl.ctas * rows * kCs * sizeof(float), 256);
    cv.total = cv.off_subs + align_up(units * pl.ctas * 2 * pl.n_warps * rows * kCs * sizeof(float), 256);
    return cv;
}
static size_t units_of(int B, int C) { return static_cast<size_t>(B) * ((C + kCs - 1) / kCs); }

// workspace: status block (256 B) | longer sequences: segment flags, workspace of the kernels that stand by (all of that but the
// end of the last to be cleared) | redo list | backward partials | copies of w, u | segment records | states of level 2, of level 1 (the
// last not where they are kept)
constexpr size_t kStatusBytes = 256;
struct Carve {
    size_t off_flags, off_stand_by, cleared, off_partial, off_vectors, off_records, off_states2, off_states1, total;
};
static Carve carve(int B, int T, int C, const Plan& pl, bool bwd) {
    const size_t units = units_of(B, C), recs = pl.segs > 1 ? units * pl.segs * 4 : 0;
    Carve cv;
    cv.off_flags = kStatusBytes;
    cv.off_stand_by = cv.off_flags + align_up(recs * sizeof(unsigned), 256);
    cv.cleared = cv.off_stand_by + fused::cleared_bytes(B, T, C, bwd);
    cv.off_partial = cv.off_stand_by + align_up(fused::workspace_bytes(B, T, C, bwd), 256);
    cv.off_vectors = cv.off_partial + (bwd ? align_up(units * pl.ctas * 2 * kCs * sizeof(float), 256) : 0);
    cv.off_records = cv.off_vectors + align_up(2 * static_cast<size_t>(C) * sizeof(float), 256);
    cv.off_states2 = cv.off_records + align_up(recs * kSegRec * sizeof(float), 256);
    cv.off_states1 = cv.off_states2 + (pl.split && bwd ? carve_states(units, pl, kStateRows).total : 0);
    cv.total = cv.off_states1 + (pl.split ? carve_states(units, pl, bwd ? kStateRows : kPlainRows).total : 0);
    return cv;
}

size_t workspace_bytes(int B, int T, int C, bool bwd, bool kept) {
    Plan pl;
    if (!make_plan(B, T, C, pl)) return 256;
    const Carve cv = carve(B, T, C, pl, bwd);
    return kept ? cv.off_states1 : cv.total;
}

size_t kept_bytes(int B, int T, int C) {
    Plan pl;
    if (!make_plan(B, T, C, pl) || !pl.split) return 0;
    return carve_states(units_of(B, C), pl, kStateRows).total;
}

struct Maps {
    CUtensorMap k, v, g, o0, o1;
};
template <bool kBwd, Types kTypes, Mode kMode>
static bool run(const Params& p, const Maps& m, size_t grid, cudaStream_t stream) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(p.n_warps * 32);
    cfg.dynamicSmemBytes = smem_bytes<kBwd, kMode>(p.n_warps);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = p.cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = kUsesCluster<kMode> ? 1 : 0;
    const cudaError_t err = cudaLaunchKernelEx(&cfg, kernel<kBwd, kTypes, kMode>(), m.k, m.v, m.g, m.o0, m.o1, p);
    if (err == cudaSuccess) return true;
    set_error_detail(cudaGetErrorName(err));
    return false;
}

// kept: forward: where to leave what a backward needs (may be null); backward: what a forward left (may be null)
template <bool kBwd, Types kTypes>
static int launch(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy,
                  void* o0, void* o1, float* gwgu, void* workspace, void* kept, cudaStream_t stream) {
    constexpr bool kHalf = kTypes != Types::f32;
    Plan pl;
    if (!make_plan(B, T, C, pl)) return -1;
    Params p{};
    p.B = B; p.T = T; p.C = C;
    p.n_strips = (C + kCs - 1) / kCs;
    p.cluster = pl.cluster; p.n_warps = pl.n_warps; p.n_tok = pl.n_tok; p.ctas = pl.ctas;
    unsigned char* ws = static_cast<unsigned char*>(workspace);
    p.status = reinterpret_cast<unsigned*>(ws);
    p.mirror = failure_mirror(kBwd ? Op::biwkv_backward : Op::biwkv_forward);
    const size_t units = units_of(B, C), grid = units * pl.ctas;
    const Carve cv = carve(B, T, C, pl, kBwd);
    p.redo_count = reinterpret_cast<unsigned*>(ws) + 1;
    p.segs = pl.segs;
    p.xflag = reinterpret_cast<unsigned*>(ws + cv.off_flags);
    p.xseg = reinterpret_cast<float*>(ws + cv.off_records);
    p.partial = reinterpret_cast<float*>(ws + cv.off_partial);
    float* const vectors = reinterpret_cast<float*>(ws + cv.off_vectors);
    p.w = paired(w, C, vectors, stream);
    p.u = paired(u, C, vectors + C, stream);
    p.spin_limit = g_withhold.load() ? (1u << 10) : kSpinLimit;
    p.withhold_rank = g_withhold.load() ? 1 : -1;
    p.state_rows = kBwd || kept ? kStateRows : kPlainRows;
    p.out_of_range = p.redo_count;
    if (pl.split) {
        unsigned char* base = kept ? static_cast<unsigned char*>(kept) : ws + cv.off_states1;
        StatesCarve sc = carve_states(units, pl, p.state_rows);
        if (kBwd && kept) p.out_of_range = reinterpret_cast<unsigned*>(base);
        p.ctas1 = reinterpret_cast<float*>(base + sc.off_ctas);
        p.states1 = reinterpret_cast<float*>(base + sc.off_subs);
        if (kBwd) {
            sc = carve_states(units, pl, kStateRows);
            p.ctas2 = reinterpret_cast<float*>(ws + cv.off_states2 + sc.off_ctas);
            p.states2 = reinterpret_cast<float*>(ws + cv.off_states2 + sc.off_subs);
        }
    }
    tensor_map::bind_primary_context();   // the tensor-map encoder is a driver call
    Maps m;
    // float32: loads one box per 32-token span, stores one box per CTA; bfloat16: one box per 16-token sub-chunk both ways
    const int box_in = kHalf ? kL : kSpan, box_g = kHalf ? kL : kSpan, box_out = kHalf ? kL : pl.n_tok;
    bool ok = tensor_map::make_btc(&m.k, k, B, T, C, kCs, box_in, kHalf) && tensor_map::make_btc(&m.v, v, B, T, C, kCs, box_in, kHalf) &&
              tensor_map::make_btc(&m.o0, o0, B, T, C, kCs, box_out, kHalf);
    if (kBwd) {
        ok = ok && tensor_map::make_btc(&m.g, gy, B, T, C, kCs, box_g, kHalf) && tensor_map::make_btc(&m.o1, o1, B, T, C, kCs, box_out, kHalf);
    } else {
        m.g = m.k;       // not used
        m.o1 = m.o0;
    }
    if (!ok) {
        set_error_detail("cuTensorMapEncodeTiled rejected a (C, T, B) tensor map");
        return -1;
    }
    cudaMemsetAsync(ws, 0, cv.cleared, stream);
    int launched = 0;
    bool done = true;
    if (pl.split) {
        unsigned* const kept_seen = !kBwd && kept ? static_cast<unsigned*>(kept) : nullptr;
        const auto chain = [&](float* sums, int rows) {
            biwkv_chain_kernel<<<static_cast<unsigned>(units), 128, 0, stream>>>(sums, p.w, p.n_strips, pl.ctas, pl.n_tok, rows, C, p.out_of_range, kept_seen);
        };
        if (!kBwd || !kept) {
            done = p.state_rows == kStateRows ? run<false, kTypes, Mode::sums_keep>(p, m, grid, stream) : run<false, kTypes, Mode::sums>(p, m, grid, stream);
            chain(p.ctas1, p.state_rows);
            launched += 2;
        }
        if (kBwd) {
            done = done && run<kBwd, kTypes, Mode::sums>(p, m, grid, stream);
            chain(p.ctas2, kStateRows);
            launched += 2;
        }
        p.reverse = true;
        done = done && run<kBwd, kTypes, Mode::spread>(p, m, grid, stream);
    } else {
        done = run<kBwd, kTypes, Mode::linked>(p, m, grid, stream);
    }
    if (!done) return -1;
    ++launched;
    if (kBwd) {
        reduce_partials<<<dim3(p.n_strips, 2), dim3(32, 32), 0, stream>>>(p, gwgu);
        ++launched;
    }
    void* const stand_by = ws + cv.off_stand_by;
    int n;
    if constexpr (kHalf) {
        n = kBwd ? fused::backward_bf16(B, T, C, w, u, k, v, gy, gwgu, o0, o1, stand_by, stream, p.out_of_range)
                 : fused::forward_bf16(B, T, C, w, u, k, v, o0, stand_by, stream, p.out_of_range);
    } else {
        const auto in = [](const void* x) { return static_cast<const float*>(x); };
        const auto out = [](void* x) { return static_cast<float*>(x); };
        n = kBwd ? fused::backward(B, T, C, w, u, in(k), in(v), in(gy), gwgu, out(o0), out(o1), stand_by, stream, p.out_of_range)
                 : fused::forward(B, T, C, w, u, in(k), in(v), out(o0), stand_by, stream, p.out_of_range);
    }
    return n < 0 ? n : launched + n;
}

int forward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, Types types,
            void* workspace, cudaStream_t stream, void* keep) {
    const auto fn = types == Types::f32 ? launch<false, Types::f32> : launch<false, Types::bf16>;
    return fn(B, T, C, w, u, k, v, nullptr, y, nullptr, nullptr, workspace, keep, stream);
}

int backward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy, float* gwgu,
             void* gk, void* gv, Types types, void* workspace, cudaStream_t stream, const void* kept) {
    const auto fn = types == Types::f32 ? launch<true, Types::f32> : launch<true, Types::bf16>;
    return fn(B, T, C, w, u, k, v, gy, gk, gv, gwgu, workspace, const_cast<void*>(kept), stream);
}

}  // namespace resident
}  // namespace biwkv
