// Bi-WKV on sequences that one CTA or one cluster holds: narrow strips of channels.
//
// Work unit: one (sequence b, strip of kCs = 2 P channels).  One CTA, or a cluster of up to 16, holds all T tokens of the unit in
// shared memory while they are scanned in both directions, so every element of k, v (and gy) crosses HBM once in and every
// output once out.  P lanes of a warp, a channel pair each, walk L tokens one after the other; a warp has kW = 32 / P such
// walkers, its span is kW L tokens, and the spans of a CTA's warps and the CTAs of a cluster follow one another.
//
// Why narrow: what bounds these kernels is a CTA's chain of latencies (tile, sums, hand-over, results, twice in the backward), and
// the hand-over between CTAs is its longest link.  A CTA's shared memory holds about 8700 elements of k, v and gy whatever their
// shape; with strips of 32 channels that is 272 tokens, with 8 channels 1088, so four times fewer CTAs hand over to one another and
// most sequences need one (make_plan).  Rows of 32 or 64 bytes cost little: loads and stores of a backward's tiles alone, B=32, T=4096,
// C=768: float32 320, 315, 333 us with 32, 16, 8 channels; bfloat16 k, v beside float32 gy 183, 194, 301 us.
//
// Odd L keeps the walkers of a half-warp in different banks: their rows lie L rows of 8 P bytes apart.
//
// Per scan level (forward: one, over the terms e^{k}[v, 1]; backward: a second over the adjoint pairs [gy / Den, gy y / Den]):
//   1. every walker sums up its L tokens, towards later ones and towards earlier ones;
//   2. the walkers of a warp combine by shuffles, in rounds of pairs: the last walker of a group holds its sum towards later
//      tokens, the first the one towards earlier tokens;
//   3. warp 0 chains the spans of the CTA, and in a cluster sends the CTA's own sums to the others (st.async: data and
//      notification in one hop), waits (bounded) for theirs and chains them;
//   4. every thread adds what lies outside its group, moved to its own position.
// y, Den are recomputed in the backward; nothing is kept from the forward.
//
// Within a walker the tokens go in four groups (L - 12, 4, 4, 4).  A walk towards later tokens also leaves the groups' sums towards
// earlier ones in registers, so that the next pass knows the state at every group's far end and reads its terms once: walking back
// over the tokens first read them two and a half times.
//
// Instructions are what it is worth to save: an SM's 16 warps issue in 40 % of the cycles, each waiting for its own results most of the
// time.  Hence no first moments (biwkv_backward_kernel), one read of the terms, single factors instead of (high, low) pairs within a
// warp, constants by products.
//
// Measured, calls in captured loops (all their kernels), forward / backward us at 100.7 M elements (C = 768), float32, beside the kernels
// with strips of 32 channels and 16 tokens per walker that were here: T=64 190 / 375 (181 / 398), 196 179 / 354 (203 / 488), 576
// 201 / 388 (233 / 574), 1024 192 / 380 (208 / 490), 4096 219 / 487 (258 / 654), 16384 285 / 658 (358 / 688); bfloat16 k, v beside float32
// y, gy: T=196 157 / 370 (228 / 488), 576 196 / 400 (242 / 563), 4096 222 / 512 (268 / 641), 16384 281 / 738 (545 / 718).  At the rate of a
// plain copy float32 would take 185 / 308, bfloat16 123 / 185; a forward, which reads twice what it writes, can be a little faster than
// that (T=196).  Where a sequence fills less than a warp's span, CTAs of one warp are started and ended faster than they work: 256
// sequences of 2 to 30 tokens, C = 1024, 27.5 to 29 / 55 to 58 us (24.6 / 47 to 51).
// A persistent kernel that kept the terms in tensor memory, so that tiles of the next unit arrived meanwhile, was slower (T=1024
// backward 530 for 431 of the kernel it was made from): not the tiles are waited for but the steps of the arithmetic.
//
// Arithmetic, exactness and the exact kernel: plain floats without exponent shift, safe whenever 2 max|k| + |u| + |w| + max(-w, 0) T
// <= 60 (and rows past T grow by little, kSafePast); each thread checks its own tokens, the first exchange carries the OR, and every CTA
// leaves a word that says whether its unit is left to biwkv_exact_kernel (per-token max-shifted arithmetic, launched behind).  Decays over
// half a walker and more come from double precision, as one float within a warp, as (high, low) pairs between warps and CTAs.  That and
// the chain of a cluster's CTAs in float32 (it was in double) cost no accuracy: for weights as the models start from, 2-norm errors
// against float64 at T = 17 .. 17408 are below those of the kernels that were here in every result, at T = 16384 y 2.1e-7 for 2.4e-7, gw
// 5.7e-7 for 6.3e-7.  (With max(-w, 0) T of 30 to 40 at T = 4096 gk and gv are 3.1e-7 for 2.9e-7, all else below there too.)
//
// Recurrence restated: classification/mmcls_custom/models/backbones/cuda_new/bi_wkv_kernel.cu:21-116 (forward), :119-367
// (gradients).
#include <cuda_bf16.h>
#include <algorithm>
#include <atomic>
#include <mutex>
#include "biwkv_math.cuh"
#include "biwkv_pairs.cuh"
#include "launch.h"
#include "sm100_async.cuh"
#include "tensor_map.h"
#include "vrwkv_internal.h"

namespace biwkv {
namespace strips {

using resident::Types;
using namespace pairs;

constexpr int kMaxWarps = 8;                // of a CTA
constexpr int kMaxCluster = 16;
constexpr int kBatch = 8;                   // other CTAs' blocks read together
constexpr uint32_t kSpinLimit = 1u << 20;   // ~0.1 s of polling on a barrier
constexpr float kSafeRange = 60.f;

// P channel pairs, L tokens per walker
template <int P_, int L_>
struct Strip {
    static constexpr int P = P_, L = L_;
    static constexpr int kCs = 2 * P;               // channels
    static constexpr int kW = 32 / P;               // walkers per warp
    static constexpr int kSpan = kW * L;            // tokens per warp
    static constexpr int kAreaFloats = 64 * L;      // of a warp, per tensor
    // a walker's groups of tokens
    static constexpr int kFirst = L % 4 == 1 ? 5 : L % 4 == 0 ? 4 : L % 4;
    static constexpr int kGroups = 4;
    static_assert(L == kFirst + 12, "four groups");
    static constexpr int kGroup = kFirst > 4 ? kFirst : 4;      // the longest
    static __host__ __device__ constexpr int at(int g) { return g == 0 ? 0 : kFirst + 4 * (g - 1); }
    static __host__ __device__ constexpr int len(int g) { return g == 0 ? kFirst : 4; }
    static constexpr int kConstRows = 13 + kW + 2;
};
// per-channel constants in rows of kCs floats, computed once per CTA in double precision
enum ConstRow { kLam = 0, kWl2, kCuw, kLam4, kLamFirst, kLamHalf, kFixLo, kFixHi, kLimit, kLamS_hi, kLamS_lo, kLamC_hi, kLamC_lo, kLamL };      // kLamL: lambda^(L d), d = 0..kW, and zero

// A CTA's sums as sent to another: [channel][a, b] and a flag word
template <class St>
constexpr int kBlock = 2 * St::kCs + 4;
// Rows past T, up to a whole walker, hold zeros, but what the walks carry grows on over them, and must stay finite to vanish against the
// zeros: e^kSafePast beyond what valid rows may reach is left alone (e^68, and e^20 = 5e8 for T times the inputs' size).
constexpr float kSafePast = 8.f;
constexpr int kRecRows = 4;      // of kCs floats, per span: towards later tokens a, b; towards earlier ones a, b

struct Params {
    int B, T, C;
    int n_strips, c_padded, units;
    int cluster;      // CTAs per unit
    int n_warps, n_tok;      // warps and tokens per unit and CTA
    const float* w;
    const float* u;
    void* o0;         // results
    void* o1;
    unsigned* status;
    unsigned* mirror;
    float* partial;         // backward: [b][rank][gw | gu][c_padded]
    unsigned* words;        // one per CTA, from the fast kernel to the exact one: kRedo, bits of waits that gave up
    uint32_t spin_limit;
    int withhold_rank;      // test only: this rank of every cluster sends nothing (-1: none)
};

// What a CTA leaves in its word: its unit is the exact kernel's; status bits of its waits, shifted.  Every CTA writes its own, so nothing
// has to be cleared before the launch (a memset took 1.5 us of the GPU and as much of the host, in a forward of one image 14).
constexpr unsigned kRedo = 1u, kFailedShift = 8;
// what may be launched behind this grid need not wait for its end any longer; what a dependent grid reads of the one before it
__device__ __forceinline__ void launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

struct Ctx {
    float* sub;      // [n_warps][kRecRows][kCs]
    float* peers;    // [levels][cluster - 1][kBlock]: received (ranks above this CTA's shift down by one)
    float* stage;    // [2][kBlock]: this CTA's
    float* cta;      // [kRecRows][kCs]: state entering this CTA from the cluster
    float* consts;
    uint64_t* xbar;  // [levels]: bytes the other CTAs send
    unsigned* flag;  // [0]: the unit's, out of range; [1]: this CTA's waits that gave up
    uint32_t spin_limit;
    bool withhold;
    int warp, lane, n_warps, n_tok, cluster, rank;
};
// a wait gave up
__device__ __forceinline__ void failed(const Ctx& c, unsigned bits) { atomicOr(c.flag + 1, bits); }

struct Enter {
    Pair2 P, S;   // state entering at the first token, at the last
};

__device__ __forceinline__ Pair2 zero() { return Pair2{f2(0.f, 0.f), f2(0.f, 0.f)}; }
__device__ __forceinline__ float2 at2(const float* row) { return *reinterpret_cast<const float2*>(row); }
__device__ __forceinline__ float2 shfl_from(float2 a, int src) {
    return f2(__shfl_sync(0xffffffffu, a.x, src), __shfl_sync(0xffffffffu, a.y, src));
}
__device__ __forceinline__ float2 widen(uint32_t x) { return f2(__uint_as_float(x << 16), __uint_as_float(x & 0xffff0000u)); }

// Constants of a strip, by the CTA's first 2 kCs threads, in double precision (a rounded lambda multiplied up over thousands of tokens
// would drift by distance * 6e-8).  The powers are products, 1e-16 each; an exponential of each, spread over the CTA, was more work
// than everything else where a CTA is one warp.
template <class St, bool kSingle>
__device__ __forceinline__ void strip_constants(float* consts, const Params& p, int strip) {
    constexpr int kCs = St::kCs;
    if (threadIdx.x >= 2 * kCs) return;
    const int ch = threadIdx.x & (kCs - 1), at = strip * kCs + ch;
    const float w = at < p.C ? p.w[at] : 0.f, u = at < p.C ? p.u[at] : 0.f;
    // no infinity: what lies past the end of a sequence is zero and has to stay so
    const auto put = [&](int row, double x) { consts[row * kCs + ch] = static_cast<float>(x > 1e38 ? 1e38 : x); };
    const double wd = w;
    const bool own = threadIdx.x >= kCs;      // the second half: e^{u + w}
    double x = exp(own ? static_cast<double>(u) + wd : -wd);
    if (own) {
        put(kCuw, x);
        const float grows = fmaxf(-w, 0.f), whole = static_cast<float>((p.T + St::L - 1) / St::L * St::L);
        consts[kLimit * kCs + ch] = kSafeRange - (fabsf(u) + fabsf(w) + fmaxf(grows * static_cast<float>(p.T), grows * whole - kSafePast));
        put(kLamL + St::kW + 1, 0.0);
        return;
    }
    put(kLam, x);
    put(kWl2, wd * 1.4426950408889634);
    // Within half a walker (two groups) powers of the rounded lambda, which the walks multiply by: a token's weight in a denominator and
    // in the sums of gradients then has the same error, and the two cancel (with powers of lambda itself for one of the two, gk and gv
    // were off by 3.8e-7 for 2.4e-7).  Across a half lambda itself: what the walk has in excess is taken off (kFixLo, kFixHi).
    const double r = static_cast<float>(x), r2 = r * r, r4 = r2 * r2, r_first = St::kFirst == 5 ? r4 * r : St::kFirst == 3 ? r2 * r : r4;
    const double x2 = x * x, x4 = x2 * x2, x8 = x4 * x4, x_first = St::kFirst == 5 ? x4 * x : St::kFirst == 3 ? x2 * x : x4;
    put(kLam4, r4);
    put(kLamFirst, r_first);
    put(kLamHalf, x_first * x4);
    put(kFixLo, x_first * x4 - r_first * r4);
    put(kFixHi, x8 - r4 * r4);
    const double xl = x_first * x4 * x8;
    double y = 1.0;
#pragma unroll
    for (int d = 0; d <= St::kW; ++d) {
        put(kLamL + d, y);
        if (d < St::kW) y *= xl;
    }
    const auto put_pair = [&](int row, double v) {
        put(row, v);
        put(row + 1, v > 1e38 ? 0.0 : v - static_cast<double>(static_cast<float>(v)));
    };
    put_pair(kLamS_hi, y);      // over a warp's span
    if (!kSingle) {
        double z = y;
        for (int s = 1; s < p.n_warps; ++s) z *= y;
        put_pair(kLamC_hi, z);
    }
}

// One exchange (steps 2-4 of the file header).  F: the walker's sum relative to the first token after its L, R: relative to the last
// token before them.  `unsafe`: level 0, OR over the unit.
template <class St, bool kSingle>
__device__ __forceinline__ Enter exchange(const Ctx& c, int level, Pair2 F, Pair2 R, bool& unsafe) {
    constexpr int P = St::P, kCs = St::kCs, kW = St::kW, kB = kBlock<St>;
    const int lane = c.lane, warp = c.warp, nw = c.n_warps;
    const int pr = lane % P, wk = lane / P;
    const float* const cst = c.consts + 2 * pr;
    // lambda^(L d) rounded; row kW + 1 is zero
    const auto pow = [&](int d) { return at2(cst + (kLamL + d) * kCs); };
    // (2) `tot`: in the last walker of a group its sum towards later tokens, in the first the one towards earlier tokens.  In a round the
    // later one of two groups receives the former from the other, the earlier one the latter; what a walker does not receive it adds
    // times zero.
    Enter e;
    Pair2 tot;
#pragma unroll
    for (int g = 1; g < kW; g *= 2) {
        const bool up = (wk & g) != 0;
        const float2 over = pow(g);
        if (g == 1) {
            const Pair2 in{shfl2(sel2(up, R.n, F.n), P), shfl2(sel2(up, R.d, F.d), P)};
            e.P = Pair2{sel2(up, in.n, f2(0.f, 0.f)), sel2(up, in.d, f2(0.f, 0.f))};
            e.S = Pair2{sel2(up, f2(0.f, 0.f), in.n), sel2(up, f2(0.f, 0.f), in.d)};
            tot = Pair2{fma2(over, in.n, sel2(up, F.n, R.n)), fma2(over, in.d, sel2(up, F.d, R.d))};
        } else {
            const int src = ((wk & ~(2 * g - 1)) + (up ? g - 1 : g)) * P + pr;
            const Pair2 in{shfl_from(tot.n, src), shfl_from(tot.d, src)};
            const int d = wk & (g - 1);      // walkers of the own group on the near side: d, or g - 1 - d
            const float2 to_P = pow(up ? d : kW + 1), to_S = pow(up ? kW + 1 : g - 1 - d);
            e.P = Pair2{fma2(to_P, in.n, e.P.n), fma2(to_P, in.d, e.P.d)};
            e.S = Pair2{fma2(to_S, in.n, e.S.n), fma2(to_S, in.d, e.S.d)};
            tot = Pair2{fma2(over, in.n, tot.n), fma2(over, in.d, tot.d)};
        }
    }
    float* const rec = c.sub + warp * (kRecRows * kCs) + 2 * pr;
    if (wk == kW - 1 || wk == 0) {
        float* const at = rec + (wk == 0 ? 2 * kCs : 0);
        *reinterpret_cast<float2*>(at) = tot.n;
        *reinterpret_cast<float2*>(at + kCs) = tot.d;
    }
    const int any = __syncthreads_or(unsafe ? 1 : 0);
    // (3) lane = channel, first kCs lanes towards later tokens, next kCs towards earlier ones; state = (a, b)
    const bool back = (lane & kCs) != 0;
    const int ch = lane & (kCs - 1);
    if (warp == 0 && lane < 2 * kCs) {
        float* const q0 = c.sub + (back ? ((nw - 1) * kRecRows + 2) * kCs : 0) + ch;
        const int step = back ? -kRecRows * kCs : kRecRows * kCs;
        const float2 hi2 = dup(c.consts[kLamS_hi * kCs + ch]), lo2 = dup(c.consts[kLamS_lo * kCs + ch]);
        float2 X = f2(0.f, 0.f), f[kMaxWarps];
#pragma unroll
        for (int s = 0; s < kMaxWarps; ++s) {
            f[s] = f2(0.f, 0.f);
            if (s < nw) f[s] = f2(q0[s * step], q0[s * step + kCs]);
        }
#pragma unroll
        for (int s = 0; s < kMaxWarps; ++s) {
            if (s < nw) {
                q0[s * step] = X.x; q0[s * step + kCs] = X.y;
                X = mulc_add(X, hi2, lo2, f[s]);
            }
        }
        if (!kSingle) {
            float* const st = c.stage + (back ? kB : 0);
            *reinterpret_cast<float2*>(st + ch * 2) = X;
            if (ch == 0) st[2 * kCs] = __int_as_float(any);
        }
    }
    __syncthreads();
    if (!kSingle) {
        // every warp sends the blocks to its share of the other CTAs: lane = channel, lane 0 also the flag word
        float* const peers = c.peers + level * (c.cluster - 1) * kB;
        if (!c.withhold) {
            const uint32_t bar_off = sm100::smem_u32(c.xbar + level) - sm100::smem_u32(peers);
            for (int r = warp; r < c.cluster; r += nw) {
                if (r == c.rank || lane >= kCs) continue;
                const uint32_t rb = peer_addr(peers, r);
                const uint32_t slot = rb + static_cast<uint32_t>((c.rank - (c.rank > r ? 1 : 0)) * kB) * 4u;
                const float* const st = c.stage + (r > c.rank ? 0 : kB);
                st_async2(slot + lane * 8u, at2(st + lane * 2), rb + bar_off);
                if (lane == 0) st_async1(slot + 2 * kCs * 4u, st[2 * kCs], rb + bar_off);
            }
        }
        __syncwarp();
        if (warp == 0) {
            const bool heard = sm100::mbar_wait(c.xbar + level, 0, c.spin_limit);
            if (!heard && lane == 0) failed(c, 1u);
            if (level == 0) {
                // A CTA that gave up goes no further either: at the next level it would send to CTAs that heard everything and may have left.
                const int other = (lane < c.cluster && lane != c.rank) ? __float_as_int(peers[(lane - (lane > c.rank ? 1 : 0)) * kB + 2 * kCs]) : 0;
                const int flag = __any_sync(0xffffffffu, !heard || (other | any) != 0) ? 1 : 0;
                if (lane == 0) c.flag[0] = static_cast<unsigned>(flag);
            }
            if (lane < 2 * kCs) {
                // lower ranks' blocks lie at their rank, higher ones' one below
                const int count = back ? c.cluster - 1 - c.rank : c.rank;
                const float* const q0 = peers + (back ? (c.cluster - 2) * kB : 0) + ch * 2;
                const int step = back ? -kB : kB;
                const float2 hi2 = dup(c.consts[kLamC_hi * kCs + ch]), lo2 = dup(c.consts[kLamC_lo * kCs + ch]);
                float2 X = f2(0.f, 0.f);
                for (int r0 = 0; r0 < count; r0 += kBatch) {
                    float2 f[kBatch];
#pragma unroll
                    for (int j = 0; j < kBatch; ++j) {
                        f[j] = f2(0.f, 0.f);
                        if (r0 + j < count) f[j] = at2(q0 + (r0 + j) * step);
                    }
#pragma unroll
                    for (int j = 0; j < kBatch; ++j)
                        if (r0 + j < count) X = mulc_add(X, hi2, lo2, f[j]);
                }
                float* const o = c.cta + (back ? 2 * kCs : 0) + ch;
                o[0] = X.x; o[kCs] = X.y;
            }
        }
        __syncthreads();
    }
    // (4)
    Pair2 Pw{at2(rec), at2(rec + kCs)}, Sw{at2(rec + 2 * kCs), at2(rec + 3 * kCs)};
    if (!kSingle) {
        const float2 wl2 = at2(cst + kWl2 * kCs);
        const float dP = static_cast<float>(St::kSpan * warp), dS = static_cast<float>(St::kSpan * (nw - 1 - warp));
        const float2 pP = f2(ex2(-wl2.x * dP), ex2(-wl2.y * dP)), pS = f2(ex2(-wl2.x * dS), ex2(-wl2.y * dS));
        const float* const o = c.cta + 2 * pr;
        Pw = Pair2{fma2(pP, at2(o), Pw.n), fma2(pP, at2(o + kCs), Pw.d)};
        Sw = Pair2{fma2(pS, at2(o + 2 * kCs), Sw.n), fma2(pS, at2(o + 3 * kCs), Sw.d)};
    }
    const float2 to_P = pow(wk), to_S = pow(kW - 1 - wk);
    e.P = Pair2{fma2(to_P, Pw.n, e.P.n), fma2(to_P, Pw.d, e.P.d)};
    e.S = Pair2{fma2(to_S, Sw.n, e.S.n), fma2(to_S, Sw.d, e.S.d)};
    if (level == 0) unsafe = kSingle ? any != 0 : c.flag[0] != 0u;
    return e;
}

// The states at the groups' far ends, from the state behind the last group and the groups' own sums
__device__ __forceinline__ void group_ends(Pair2 (&S)[4], const Pair2 (&r)[4], Pair2 in, float2 lam4, float2 fix_hi) {
    const auto before = [&](Pair2 s, Pair2 t) { return Pair2{fma2(lam4, s.n, t.n), fma2(lam4, s.d, t.d)}; };
    S[3] = in;
    S[2] = before(in, r[3]);
    S[1] = before(S[2], Pair2{fma2(fix_hi, in.n, r[2].n), fma2(fix_hi, in.d, r[2].d)});
    S[0] = before(S[1], r[1]);
}
// the walker's sum towards earlier tokens from its groups'
__device__ __forceinline__ Pair2 group_sum(const Pair2 (&r)[4], float2 lam4, const float* cst, int cs) {
    const float2 first = at2(cst + kLamFirst * cs), half = at2(cst + kLamHalf * cs);
    const auto sum = [](float2 f, Pair2 s, Pair2 t) { return Pair2{fma2(f, s.n, t.n), fma2(f, s.d, t.d)}; };
    return sum(half, sum(lam4, r[3], r[2]), sum(first, r[1], r[0]));
}
// a state at the end of a half that it entered as `in`
__device__ __forceinline__ void past_half(Pair2& s, Pair2 in, float2 fix) { s = Pair2{fma2(fix, in.n, s.n), fma2(fix, in.d, s.d)}; }
// a group's sum towards earlier tokens: sum_j lambda^j [n_j, d_j]
template <int N>
__device__ __forceinline__ Pair2 horner(const float2 (&n)[N], const float2 (&d)[N], int len, float2 lam2) {
    Pair2 r{n[len - 1], d[len - 1]};
#pragma unroll
    for (int j = N - 2; j >= 0; --j)
        if (j < len - 1) r = Pair2{fma2(lam2, r.n, n[j]), fma2(lam2, r.d, d[j])};
    return r;
}
// the states at a group's tokens from the one at its far end: s_j = lambda s_{j+1} + term_{j+1}
template <int N>
__device__ __forceinline__ void walk_back(float2 (&sn)[N], float2 (&sd)[N], Pair2 end, const float2 (&n)[N], const float2 (&d)[N], int len, float2 lam2) {
    sn[len - 1] = end.n;
    sd[len - 1] = end.d;
#pragma unroll
    for (int j = N - 2; j >= 0; --j)
        if (j < len - 1) { sn[j] = fma2(lam2, sn[j + 1], n[j + 1]); sd[j] = fma2(lam2, sd[j + 1], d[j + 1]); }
}

// shared memory: tiles of k, v (gy) | span records | blocks received, per level | outgoing blocks | state entering this CTA | constants |
// mbarriers and the flag word
template <class St, bool kBwd>
static inline size_t smem_bytes(int n_warps, int cluster) {
    const size_t peers = cluster > 1 ? ((kBwd ? 2 : 1) * static_cast<size_t>(cluster - 1) + 2) * kBlock<St> + kRecRows * St::kCs : 0;
    return ((kBwd ? 3 : 2) * static_cast<size_t>(n_warps) * St::kAreaFloats + static_cast<size_t>(n_warps) * kRecRows * St::kCs + peers +
            St::kConstRows * St::kCs) * sizeof(float) + (2 * kMaxWarps + 4) * 8;
}
// what follows the tiles; returns the mbarriers of the tiles
template <class St, bool kBwd, bool kSingle>
__device__ __forceinline__ uint64_t* carve_smem(Ctx& c, float* at, const Params& p) {
    c.warp = threadIdx.x >> 5; c.lane = threadIdx.x & 31; c.n_warps = p.n_warps; c.n_tok = p.n_tok;
    c.cluster = kSingle ? 1 : p.cluster;
    c.rank = kSingle ? 0 : static_cast<int>(cluster_rank());
    c.spin_limit = p.spin_limit;
    c.withhold = c.rank == p.withhold_rank;
    c.sub = at;
    c.peers = c.sub + p.n_warps * (kRecRows * St::kCs);
    c.stage = c.peers + (kSingle ? 0 : (kBwd ? 2 : 1) * (p.cluster - 1) * kBlock<St>);
    c.cta = c.stage + (kSingle ? 0 : 2 * kBlock<St>);
    c.consts = c.cta + (kSingle ? 0 : kRecRows * St::kCs);
    uint64_t* const bars = reinterpret_cast<uint64_t*>(c.consts + St::kConstRows * St::kCs);
    c.xbar = bars + 2 * kMaxWarps;
    c.flag = reinterpret_cast<unsigned*>(c.xbar + 2);
    if (threadIdx.x == 0) c.flag[1] = 0u;      // a CTA barrier follows before anyone waits for anything
    return bars;
}
// behind a CTA barrier that follows the last wait
__device__ __forceinline__ void leave_word(const Ctx& c, const Params& p, unsigned redo) {
    launch_dependents();
    if (threadIdx.x == 0) {
        const unsigned bits = c.flag[1];
        p.words[blockIdx.x] = redo | bits << kFailedShift;
        if (bits != 0u && p.mirror != nullptr) *reinterpret_cast<volatile unsigned*>(p.mirror) = bits;
        if (blockIdx.x == 0) *p.status = 0u;      // the exact kernel collects the bits
    }
}
// Before warp 0 of a CTA goes.  A CTA whose waits for the others all ended has everything that is ever sent to it.  One that gave up
// stays until every other thread of its cluster has gone or come here, so that all that is sent is on its way (a cluster barrier counts
// the threads that are left), and then for that to arrive, again with a limit.
template <bool kBwd>
__device__ __forceinline__ void stay_for_late_data(const Ctx& c) {
    if (c.warp != 0 || c.flag[1] == 0u) return;
    __syncwarp();
    cluster_arrive();
    cluster_wait();
    for (int l = 0; l < (kBwd ? 2 : 1); ++l) sm100::mbar_wait(c.xbar + l, 0, c.spin_limit);
}
// the mbarriers of the hand-over between CTAs: a block from every other one, per level
template <class St, bool kBwd>
__device__ __forceinline__ void arm_hand_over(const Ctx& c) {
    for (int l = 0; l < (kBwd ? 2 : 1); ++l) sm100::mbar_init(c.xbar + l, 1);
    sm100::mbar_init_fence();
    for (int l = 0; l < (kBwd ? 2 : 1); ++l) sm100::mbar_expect_tx(c.xbar + l, static_cast<uint32_t>(c.cluster - 1) * (2 * St::kCs + 1) * 4u);
}

// A walker's rows in a bfloat16 result; byte offsets within a sequence are 32-bit (eligible)
struct RowsOut {
    char* base;
    uint32_t at, pitch;
    __device__ __forceinline__ RowsOut(void* out, const Params& p, int b, int row, int ch)
        : base(static_cast<char*>(out) + static_cast<size_t>(b) * p.T * p.C * 2), at(static_cast<uint32_t>(row) * p.C * 2 + ch * 2), pitch(p.C * 2) {}
    __device__ __forceinline__ void put(int i, float2 v) const { *reinterpret_cast<__nv_bfloat162*>(base + (at + static_cast<uint32_t>(i) * pitch)) = __float22bfloat162_rn(v); }
};

// Pass 1: terms z = lambda e^{k} [v, 1] in place of k, v; the walker's sum F towards later tokens and its groups' sums r towards
// earlier ones; whether an input is outside the plain-float range.
template <class St, bool kHalfIn>
__device__ __forceinline__ void terms(float* slot_k, float* slot_v, int row0, int pr, int n, const float* cst, float2 lam2, Pair2& F,
                                      Pair2 (&r)[St::kGroups], bool& unsafe) {
    constexpr int L = St::L, kCs = St::kCs, kRow = kCs / 2, kG = St::kGroup;
    float2* const k2 = reinterpret_cast<float2*>(slot_k + row0 * kCs) + pr;
    float2* const v2 = reinterpret_cast<float2*>(slot_v + row0 * kCs) + pr;
    float2 kmax = f2(0.f, 0.f);
    Pair2 F_half;
    uint32_t kr[kHalfIn ? L : 1], vr[kHalfIn ? L : 1];
    if (kHalfIn) {
        const uint32_t* const hk = reinterpret_cast<const uint32_t*>(slot_k + St::kAreaFloats / 2) + row0 * kRow + pr;
        const uint32_t* const hv = reinterpret_cast<const uint32_t*>(slot_v + St::kAreaFloats / 2) + row0 * kRow + pr;
#pragma unroll
        for (int i = 0; i < L; ++i) { kr[i] = hk[i * kRow]; vr[i] = hv[i * kRow]; }
        __syncwarp();
    }
    const float2 wl2 = at2(cst + kWl2 * kCs);
    const float2 nwl2 = f2(-wl2.x, -wl2.y), l2e = dup(kLog2e);
#pragma unroll
    for (int g = 0; g < St::kGroups; ++g) {
        // loads of a group go first: a store into one slot may not be moved past a later load from another by the compiler
        float2 kk[kG], vv[kG];
#pragma unroll
        for (int j = 0; j < St::len(g); ++j) {
            const int i = St::at(g) + j;
            if (kHalfIn) { kk[j] = widen(kr[i]); vv[j] = widen(vr[i]); }
            else { kk[j] = k2[i * kRow]; vv[j] = v2[i * kRow]; }
            kmax = f2(fmaxf(kmax.x, fabsf(kk[j].x)), fmaxf(kmax.y, fabsf(kk[j].y)));
        }
        // rows past T arrive as zeros; a k of -1e30 makes their terms vanish
        if (n < L) {
#pragma unroll
            for (int j = 0; j < St::len(g); ++j)
                if (St::at(g) + j >= n) kk[j] = dup(-1e30f);
        }
#pragma unroll
        for (int j = 0; j < St::len(g); ++j) {
            const int i = St::at(g) + j;
            const float2 t = fma2(kk[j], l2e, nwl2);
            kk[j] = f2(ex2(t.x), ex2(t.y));        // the denominators' term
            vv[j] = mul2(kk[j], vv[j]);
            k2[i * kRow] = vv[j];
            v2[i * kRow] = kk[j];
            F.n = fma2(lam2, F.n, vv[j]);
            F.d = fma2(lam2, F.d, kk[j]);
        }
        r[g] = horner(vv, kk, St::len(g), lam2);
        if (g == 1) F_half = F;
    }
    past_half(F, F_half, at2(cst + kFixHi * kCs));
    const float2 limit = at2(cst + kLimit * kCs);
    unsafe = 2.f * kmax.x > limit.x || 2.f * kmax.y > limit.y;
}

// ---- forward ---------------------------------------------------------------------------------------
// kTypes as in resident::Types.  bfloat16 tensors arrive by TMA as well, dense in the upper half of the warp's area: a thread
// takes all its rows into registers before the warp writes its (float) terms over them.  bfloat16 results leave from registers:
// a warp's store writes whole 32- or 16-byte pieces of rows.
template <class St, Types kTypes, bool kSingle>
__global__ void __launch_bounds__(kMaxWarps * 32, 3)
biwkv_forward_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                     const __grid_constant__ CUtensorMap map_y,     // float32 results
                     const Params p) {
    wait_for_launch_before();
    constexpr int P = St::P, L = St::L, kCs = St::kCs, kSpan = St::kSpan, kArea = St::kAreaFloats, kG = St::kGroup, kGroups = St::kGroups;
    constexpr bool kHalf = kTypes != Types::f32, kHalfOut = kTypes == Types::bf16;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pr = lane % P, wk = lane / P;
    const int nw = p.n_warps;
    float* const slot_k = reinterpret_cast<float*>(smem_raw) + warp * kArea;       // this warp's areas
    float* const slot_v = slot_k + nw * kArea;
    Ctx c;
    uint64_t* const full = carve_smem<St, false, kSingle>(c, reinterpret_cast<float*>(smem_raw) + 2 * nw * kArea, p);   // k, v of one span each
    const int unit = kSingle ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) / p.cluster;
    const int b = unit / p.n_strips, strip = unit - b * p.n_strips;
    const int tok0 = c.rank * p.n_tok + warp * kSpan;      // of this warp
    if (lane == 0) {
        // every warp fetches its own span and starts as soon as it is there
        sm100::mbar_init(full + warp, 1);
        sm100::mbar_init_fence();
        constexpr int kIn = kHalf ? kArea / 2 : 0;      // where the tile lands in the area
        sm100::mbar_expect_tx(full + warp, 2 * (kArea - kIn) * 4);
        sm100::tma_load_3d(slot_k + kIn, &map_k, full + warp, strip * kCs, tok0, b);
        sm100::tma_load_3d(slot_v + kIn, &map_v, full + warp, strip * kCs, tok0, b);
    }
    if (!kSingle && threadIdx.x == 0) arm_hand_over<St, false>(c);
    strip_constants<St, kSingle>(c.consts, p, strip);
    __syncthreads();
    // every CTA of the cluster has initialised its mbarriers before any other sends to them: arrive here, wait once the tiles have
    // landed (relaxed: the mbarrier-init fence above publishes the initialisation)
    if (!kSingle) cluster_arrive_relaxed();
    const int ch0 = strip * kCs + 2 * pr;
    const float* const cst = c.consts + 2 * pr;
    const float2 lam2 = at2(cst + kLam * kCs), c2 = at2(cst + kCuw * kCs), lam4 = at2(cst + kLam4 * kCs);
    if (!sm100::mbar_wait(full + warp, 0, kSpinLimit)) failed(c, 2u);
    if (!kSingle) cluster_wait();

    const int row0 = wk * L;                                       // of this walker in the warp's areas
    const int n = max(0, min(L, p.T - (tok0 + row0)));             // valid tokens
    constexpr int kRow = kCs / 2;                                  // float2 per row
    float2* const k2 = reinterpret_cast<float2*>(slot_k + row0 * kCs) + pr;
    float2* const v2 = reinterpret_cast<float2*>(slot_v + row0 * kCs) + pr;

    Pair2 F = zero(), r[kGroups];
    bool unsafe;
    terms<St, kHalf>(slot_k, slot_v, row0, pr, n, cst, lam2, F, r, unsafe);
    // nothing valid lies behind the end of the sequence: weights that grow with distance must not overflow there
    if (n < L) F = zero();
    Enter e1 = exchange<St, kSingle>(c, 0, F, group_sum(r, lam4, cst, kCs), unsafe);
    if (n == 0) e1 = Enter{zero(), zero()};
    if (unsafe) {
        // The whole cluster takes this branch together, but for the others of a CTA that gave up a wait: the unit is left to the exact
        // kernel, which runs right behind.
        __syncthreads();
        leave_word(c, p, kRedo);
        if (!kSingle) stay_for_late_data<false>(c);
        return;
    }
    leave_word(c, p, 0u);      // the last wait of this CTA lies behind its barrier in the exchange
    // ---- pass 2: y = (P + S + e^{u} x) ratio, in place of the numerator term ----
    const int n_out = ch0 < p.C ? n : 0;
    const RowsOut y(p.o0, p, b, tok0 + row0, ch0);
    Pair2 S[kGroups], Pt = e1.P;
    group_ends(S, r, e1.S, lam4, at2(cst + kFixHi * kCs));
#pragma unroll
    for (int g = 0; g < kGroups; ++g) {
        if (g == 2) past_half(Pt, e1.P, at2(cst + kFixLo * kCs));
        float2 zx[kG], zy[kG], sn[kG], sd[kG];
#pragma unroll
        for (int j = 0; j < St::len(g); ++j) { zx[j] = k2[(St::at(g) + j) * kRow]; zy[j] = v2[(St::at(g) + j) * kRow]; }
        walk_back(sn, sd, S[g], zx, zy, St::len(g), lam2);
#pragma unroll
        for (int j = 0; j < St::len(g); ++j) {
            const int i = St::at(g) + j;
            const float2 nn = fma2(c2, zx[j], add2(Pt.n, sn[j]));
            const float2 dd = fma2(c2, zy[j], add2(Pt.d, sd[j]));
            const float2 o = mul2(nn, f2(rcp(dd.x), rcp(dd.y)));
            if (kHalfOut) {
                if (i < n_out) y.put(i, o);
            } else {
                k2[i * kRow] = kHalf ? round2(o) : o;
            }
            Pt.n = fma2(lam2, Pt.n, zx[j]);
            Pt.d = fma2(lam2, Pt.d, zy[j]);
        }
    }
    if (!kHalfOut) {
        sm100::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && tok0 < p.T) {
            sm100::tma_store_3d(&map_y, slot_k, strip * kCs, tok0, b);
            sm100::tma_store_commit();
            sm100::tma_store_wait_read();   // shared memory may go once the stores have read it
        }
    }
}

// ---- backward --------------------------------------------------------------------------------------
// The decay's gradient counts, for every pair of tokens and for every place between them, the pair's term once: summed over places it
// is the product of the state that enters a token with the adjoint state from that token on, in both directions.  So no first moments
// are carried, neither by the walks nor by the hand-overs (they were two of the walks' six states and a third of what was handed
// over).  Towards later tokens both factors are known in pass 3.  Towards earlier ones pass 2 has the state of k, v and the walker's
// own part of the adjoint one; what enters the walker multiplies a sum that pass 2 leaves.
template <class St, Types kTypes, bool kSingle>
__global__ void __launch_bounds__(kMaxWarps * 32, 2)
biwkv_backward_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                      const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_gk,     // float32 results
                      const __grid_constant__ CUtensorMap map_gv, const Params p) {
    wait_for_launch_before();
    constexpr int P = St::P, L = St::L, kCs = St::kCs, kSpan = St::kSpan, kArea = St::kAreaFloats, kG = St::kGroup, kGroups = St::kGroups;
    constexpr bool kHalf = kTypes != Types::f32, kHalfG = kTypes == Types::bf16;            // bfloat16 k, v, gk, gv ; gy
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pr = lane % P, wk = lane / P;
    const int nw = p.n_warps;
    float* const slot_k = reinterpret_cast<float*>(smem_raw) + warp * kArea;       // this warp's areas
    float* const slot_v = slot_k + nw * kArea;
    float* const slot_g = slot_v + nw * kArea;
    Ctx c;
    uint64_t* const full = carve_smem<St, true, kSingle>(c, reinterpret_cast<float*>(smem_raw) + 3 * nw * kArea, p);   // k, v of one span each
    uint64_t* const gfull = full + kMaxWarps;                                                                         // gy (first needed in pass 2)
    const int unit = kSingle ? static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x) / p.cluster;
    const int b = unit / p.n_strips, strip = unit - b * p.n_strips;
    const int tok0 = c.rank * p.n_tok + warp * kSpan;      // of this warp
    if (lane == 0) {
        sm100::mbar_init(full + warp, 1);
        sm100::mbar_init(gfull + warp, 1);
        sm100::mbar_init_fence();
        constexpr int kIn = kHalf ? kArea / 2 : 0, kInG = kHalfG ? kArea / 2 : 0;
        sm100::mbar_expect_tx(full + warp, 2 * (kArea - kIn) * 4);
        sm100::tma_load_3d(slot_k + kIn, &map_k, full + warp, strip * kCs, tok0, b);
        sm100::tma_load_3d(slot_v + kIn, &map_v, full + warp, strip * kCs, tok0, b);
        sm100::mbar_expect_tx(gfull + warp, (kArea - kInG) * 4);
        sm100::tma_load_3d(slot_g + kInG, &map_g, gfull + warp, strip * kCs, tok0, b);
    }
    if (!kSingle && threadIdx.x == 0) arm_hand_over<St, true>(c);
    strip_constants<St, kSingle>(c.consts, p, strip);
    __syncthreads();
    if (!kSingle) cluster_arrive_relaxed();      // as in the forward
    const int ch0 = strip * kCs + 2 * pr;
    const float* const cst = c.consts + 2 * pr;
    const float2 lam2 = at2(cst + kLam * kCs), lam4 = at2(cst + kLam4 * kCs);
    if (!sm100::mbar_wait(full + warp, 0, kSpinLimit)) failed(c, 2u);
    if (!kSingle) cluster_wait();

    const int row0 = wk * L;                                       // of this walker in the warp's areas
    const int n = max(0, min(L, p.T - (tok0 + row0)));             // valid tokens
    constexpr int kRow = kCs / 2;                                  // float2 per row
    float2* const k2 = reinterpret_cast<float2*>(slot_k + row0 * kCs) + pr;
    float2* const v2 = reinterpret_cast<float2*>(slot_v + row0 * kCs) + pr;
    float2* const g2 = reinterpret_cast<float2*>(slot_g + row0 * kCs) + pr;

    // ---- pass 1: terms z = lambda e^{k} [v, 1] in place of k, v; the walker's sums ----
    Pair2 F = zero(), r[kGroups];
    bool unsafe;
    terms<St, kHalf>(slot_k, slot_v, row0, pr, n, cst, lam2, F, r, unsafe);
    // nothing valid lies behind the end of the sequence: weights that grow with distance must not overflow there
    if (n < L) F = zero();
    Enter e1 = exchange<St, kSingle>(c, 0, F, group_sum(r, lam4, cst, kCs), unsafe);
    if (n == 0) e1 = Enter{zero(), zero()};
    if (!sm100::mbar_wait(gfull + warp, 0, kSpinLimit)) failed(c, 2u);
    if (unsafe) {      // as in the forward
        __syncthreads();
        leave_word(c, p, kRedo);
        if (!kSingle) stay_for_late_data<true>(c);
        return;
    }
    if (kHalfG) {
        const uint32_t* const hg = reinterpret_cast<const uint32_t*>(slot_g + kArea / 2) + row0 * kRow + pr;
        uint32_t gr[L];
#pragma unroll
        for (int i = 0; i < L; ++i) gr[i] = hg[i * kRow];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < L; ++i) g2[i * kRow] = widen(gr[i]);
    }
    // ---- pass 2: recompute Den, y; G = gy / Den (in place of gy), -H = -G y (registers); gu; sums of [G, -H] ----
    const float2 c2 = at2(cst + kCuw * kCs);
    float2 hn[L];
    Pair2 S[kGroups], rr = zero(), q[kGroups], W = zero();
    float2 gwa = f2(0.f, 0.f), gu = f2(0.f, 0.f);
    {
        group_ends(S, r, e1.S, lam4, at2(cst + kFixHi * kCs));
        Pair2 Pt = e1.P, rr_half;
        float2 ahead = f2(1.f, 1.f);      // lambda^(tokens of the walker before the group)
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            if (g == 2) {
                past_half(Pt, e1.P, at2(cst + kFixLo * kCs));
                rr_half = rr;
                ahead = at2(cst + kLamHalf * kCs);
            }
            float2 zx[kG], zy[kG], gg[kG], hh[kG], sn[kG], sd[kG];
#pragma unroll
            for (int j = 0; j < St::len(g); ++j) {
                const int i = St::at(g) + j;
                zx[j] = k2[i * kRow]; zy[j] = v2[i * kRow]; gg[j] = g2[i * kRow];
                if (kTypes == Types::wide) gg[j] = round2(gg[j]);
            }
            walk_back(sn, sd, S[g], zx, zy, St::len(g), lam2);
            Pair2 w_;      // sum over the group's tokens of lambda^j times the state from that token on
#pragma unroll
            for (int j = St::len(g) - 1; j >= 0; --j) {
                // the state from token j on is the one behind token j - 1
                const Pair2 from = j > 0 ? Pair2{sn[j > 0 ? j - 1 : 0], sd[j > 0 ? j - 1 : 0]} : Pair2{fma2(lam2, sn[0], zx[0]), fma2(lam2, sd[0], zy[0])};
                w_ = j == St::len(g) - 1 ? from : Pair2{fma2(lam2, w_.n, from.n), fma2(lam2, w_.d, from.d)};
            }
            W = Pair2{fma2(ahead, w_.n, W.n), fma2(ahead, w_.d, W.d)};
            if (g == 0) ahead = at2(cst + kLamFirst * kCs);
            if (g == 2) ahead = mul2(ahead, lam4);
            Pair2 from{fma2(lam2, sn[0], zx[0]), fma2(lam2, sd[0], zy[0])};
#pragma unroll
            for (int j = 0; j < St::len(g); ++j) {
                const int i = St::at(g) + j;
                const float2 nn = fma2(c2, zx[j], add2(Pt.n, sn[j]));
                const float2 dd = fma2(c2, zy[j], add2(Pt.d, sd[j]));
                float2 inv = f2(rcp(dd.x), rcp(dd.y));
                if (n < L && i >= n) inv = f2(0.f, 0.f);      // rows past T: their denominator may be zero
                const float2 ny = f2(nn.x * -inv.x, nn.y * -inv.y);
                gg[j] = mul2(gg[j], inv);
                hh[j] = mul2(gg[j], ny);               // -H
                g2[i * kRow] = gg[j];
                hn[i] = hh[j];
                gu = fma2(zx[j], gg[j], gu);
                gu = fma2(zy[j], hh[j], gu);
                gwa = fma2(from.n, rr.n, gwa);
                gwa = fma2(from.d, rr.d, gwa);
                from = Pair2{sn[j], sd[j]};
                Pt.n = fma2(lam2, Pt.n, zx[j]);
                Pt.d = fma2(lam2, Pt.d, zy[j]);
                rr.n = fma2(lam2, rr.n, gg[j]);
                rr.d = fma2(lam2, rr.d, hh[j]);
            }
            q[g] = horner(gg, hh, St::len(g), lam2);
        }
        past_half(rr, rr_half, at2(cst + kFixHi * kCs));
        gu = mul2(gu, c2);
    }
    Enter e2;
    {
        Pair2 Q = group_sum(q, lam4, cst, kCs);
        bool ignored = false;
        if (n < L) rr = zero();
        e2 = exchange<St, kSingle>(c, 1, rr, Q, ignored);      // sums and states are those of the adjoint pairs divided by lambda
        if (n == 0) e2 = Enter{zero(), zero()};
    }
    // ---- pass 3: gk, gv in place of the terms; gw ----
    {
        gwa = fma2(e2.P.n, W.n, gwa);
        gwa = fma2(e2.P.d, W.d, gwa);
        Pair2 Rp = e2.P, Pt = e1.P;
        group_ends(S, q, e2.S, lam4, at2(cst + kFixHi * kCs));
        const int n_out = ch0 < p.C ? n : 0;
        const RowsOut gk(p.o0, p, b, tok0 + row0, ch0), gv(p.o1, p, b, tok0 + row0, ch0);
#pragma unroll
        for (int g = 0; g < kGroups; ++g) {
            if (g == 2) {
                past_half(Pt, e1.P, at2(cst + kFixLo * kCs));
                past_half(Rp, e2.P, at2(cst + kFixLo * kCs));
            }
            float2 zx[kG], zy[kG], gg[kG], hh[kG], sn[kG], sd[kG];
#pragma unroll
            for (int j = 0; j < St::len(g); ++j) {
                const int i = St::at(g) + j;
                zx[j] = k2[i * kRow]; zy[j] = v2[i * kRow]; gg[j] = g2[i * kRow]; hh[j] = hn[i];
            }
            walk_back(sn, sd, S[g], gg, hh, St::len(g), lam2);
            Pair2 from{fma2(lam2, sn[0], gg[0]), fma2(lam2, sd[0], hh[0])};
#pragma unroll
            for (int j = 0; j < St::len(g); ++j) {
                const int i = St::at(g) + j;
                const float2 AG = fma2(c2, gg[j], add2(sn[j], Rp.n));
                const float2 AH = fma2(c2, hh[j], add2(sd[j], Rp.d));      // -A^H
                const float2 ov = mul2(zy[j], AG), ok = fma2(zx[j], AG, mul2(zy[j], AH));
                if (kHalf) {
                    if (i < n_out) { gk.put(i, ok); gv.put(i, ov); }
                } else {
                    v2[i * kRow] = ov;
                    k2[i * kRow] = ok;
                }
                gwa = fma2(Pt.n, from.n, gwa);
                gwa = fma2(Pt.d, from.d, gwa);
                from = Pair2{sn[j], sd[j]};
                Pt.n = fma2(lam2, Pt.n, zx[j]);
                Pt.d = fma2(lam2, Pt.d, zy[j]);
                Rp.n = fma2(lam2, Rp.n, gg[j]);
                Rp.d = fma2(lam2, Rp.d, hh[j]);
            }
        }
    }
    if (!kHalf) {
        sm100::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && tok0 < p.T) {
            sm100::tma_store_3d(&map_gk, slot_k, strip * kCs, tok0, b);
            sm100::tma_store_3d(&map_gv, slot_v, strip * kCs, tok0, b);
            sm100::tma_store_commit();
        }
    }
    // gw, gu of the warp into its span record, whose states it has read
    float2 gw = f2(-gwa.x, -gwa.y);
#pragma unroll
    for (int m = P; m < 32; m *= 2) { gw = add2(gw, shfl2(gw, m)); gu = add2(gu, shfl2(gu, m)); }
    if (wk == 0) {
        float* const rec = c.sub + warp * (kRecRows * kCs) + 2 * pr;
        *reinterpret_cast<float2*>(rec) = gw;
        *reinterpret_cast<float2*>(rec + kCs) = gu;
    }
    __syncthreads();
    leave_word(c, p, 0u);
    if (threadIdx.x < 2 * kCs) {
        const int j = threadIdx.x / kCs, ch = threadIdx.x & (kCs - 1);
        float acc = 0.f;
        for (int s = 0; s < nw; ++s) acc += c.sub[(s * kRecRows + j) * kCs + ch];
        p.partial[((static_cast<size_t>(b) * c.cluster + c.rank) * 2 + j) * p.c_padded + strip * kCs + ch] = acc;
    }
    if (!kHalf && lane == 0) sm100::tma_store_wait_read();   // shared memory may go once the stores have read it
    if (!kSingle) stay_for_late_data<true>(c);
}

// ---- the exact kernel ----------------------------------------------------------------------------
// Serves the units that the kernel above left behind (normally none: one load and out): same tiles, same split of the work,
// (value, exponent) records, any exponent range.  Slow and simple.
struct ExactCtx {
    float* area;     // [n_sub][5][kCs], then reused
    float* agg;      // [5][kCs]
    int n_sub, n_tok, cluster, rank;
};
struct Entering {
    Acc4 left;    // state entering the walker at its first token (with first moments)
    Acc2 right;   // state entering it at its last position
};
__device__ __forceinline__ void cluster_or_cta_sync(const ExactCtx& c) {
    __syncwarp();
    if (c.cluster > 1) {
        cluster_arrive();
        cluster_wait();
    } else {
        __syncthreads();
    }
}
// One channel per thread and call.  Two rounds (one per direction) over the same record area; every thread walks the records it
// needs itself and reads the other CTAs' sums out of their shared memory.  Each record is moved to its reader in one step: moved
// along record by record, up to 63 times, exponents of a hundred lost 5e-6 at every step.  kMom = false (forward): no first moments.
template <class St, bool kMom>
__device__ __noinline__ Entering exact_exchange(const ExactCtx& c, int sub, int ch, float w, const Acc4 own_right, const Acc2 own_left) {
    constexpr int kRec = kMom ? 5 : 3, kCs = St::kCs, L = St::L;
    Entering out;
    {
        float* s = c.area + sub * kRec * kCs + ch;
        s[0] = own_right.a; s[kCs] = own_right.b; s[(kRec - 1) * kCs] = own_right.o;
        if (kMom) { s[2 * kCs] = own_right.ma; s[3 * kCs] = own_right.mb; }
        __syncwarp();
        __syncthreads();
        Acc4 X = acc4_zero();
        for (int j = 0; j < sub; ++j) {
            const float* q = c.area + j * kRec * kCs + ch;
            Acc4 t{q[0], q[kCs], kMom ? q[2 * kCs] : 0.f, kMom ? q[3 * kCs] : 0.f, q[(kRec - 1) * kCs]};
            acc4_decay(t, w, static_cast<float>(L * (sub - 1 - j)));
            X = acc4_merge(X, t);
        }
        if (sub == c.n_sub - 1) {
            Acc4 t = X;
            acc4_decay(t, w, static_cast<float>(L));
            t = acc4_merge(t, own_right);
            c.agg[ch] = t.a; c.agg[kCs + ch] = t.b; c.agg[(kRec - 1) * kCs + ch] = t.o;
            if (kMom) { c.agg[2 * kCs + ch] = t.ma; c.agg[3 * kCs + ch] = t.mb; }
        }
        cluster_or_cta_sync(c);
        Acc4 Y = acc4_zero();
        for (int r = 0; r < c.rank; ++r) {
            const uint32_t a = peer_addr(c.agg + ch, r);
            Acc4 t{ld_peer(a), ld_peer(a + kCs * 4), kMom ? ld_peer(a + 2 * kCs * 4) : 0.f, kMom ? ld_peer(a + 3 * kCs * 4) : 0.f,
                   ld_peer(a + (kRec - 1) * kCs * 4)};
            acc4_decay(t, w, static_cast<float>(c.n_tok * (c.rank - 1 - r)));
            Y = acc4_merge(Y, t);
        }
        acc4_decay(Y, w, static_cast<float>(L * sub));
        out.left = acc4_merge(Y, X);
        cluster_or_cta_sync(c);
    }
    {
        float* s = c.area + sub * 3 * kCs + ch;
        s[0] = own_left.a; s[kCs] = own_left.b; s[2 * kCs] = own_left.o;
        __syncwarp();
        __syncthreads();
        Acc2 Z = acc2_zero();
        for (int j = c.n_sub - 1; j > sub; --j) {
            const float* q = c.area + j * 3 * kCs + ch;
            Acc2 t{q[0], q[kCs], q[2 * kCs]};
            acc2_decay(t, w, static_cast<float>(L * (j - 1 - sub)));
            Z = acc2_merge(Z, t);
        }
        if (sub == 0) {
            Acc2 t = Z;
            acc2_decay(t, w, static_cast<float>(L));
            t = acc2_merge(t, own_left);
            c.agg[ch] = t.a; c.agg[kCs + ch] = t.b; c.agg[2 * kCs + ch] = t.o;
        }
        cluster_or_cta_sync(c);
        Acc2 Y = acc2_zero();
        for (int r = c.cluster - 1; r > c.rank; --r) {
            const uint32_t a = peer_addr(c.agg + ch, r);
            Acc2 t{ld_peer(a), ld_peer(a + kCs * 4), ld_peer(a + 2 * kCs * 4)};
            acc2_decay(t, w, static_cast<float>(c.n_tok * (r - 1 - c.rank)));
            Y = acc2_merge(Y, t);
        }
        acc2_decay(Y, w, static_cast<float>(L * (c.n_sub - 1 - sub)));
        out.right = acc2_merge(Y, Z);
        cluster_or_cta_sync(c);
    }
    return out;
}

// One channel of one walker: ks / vs / gs point at its first token (stride kCs), n = valid tokens.  Sweeps are position-anchored
// (biwkv_math.cuh).  Forward: y into ks.  Backward: gk into ks, gv into vs, the thread's gw / gu shares returned.
template <class St, bool kBwd>
__device__ __noinline__ void exact_walk(const ExactCtx& c, int sub, int ch, float* ks, float* vs, float* gs, int n, float w, float u,
                                        float& gw_out, float& gu_out) {
    constexpr int kCs = St::kCs, L = St::L;
    const float last = static_cast<float>(n - 1);
    Acc4 right = acc4_zero();
    Acc2 left = acc2_zero();
    for (int i = 0; i < n; ++i) acc4_absorb(right, ks[i * kCs] + w * static_cast<float>(i), vs[i * kCs], 1.f);
    for (int i = n - 1; i >= 0; --i) acc2_add(left, ks[i * kCs] - w * static_cast<float>(i), vs[i * kCs], 1.f);
    // a short walk still spans L positions for its right-hand neighbours
    right.o -= w * static_cast<float>(n);
    acc4_decay(right, w, static_cast<float>(L - n));
    left.o -= w;
    const Entering e1 = exact_exchange<St, kBwd>(c, sub, ch, w, right, left);
    const Acc4 P4 = e1.left;                        // anchored at token 0
    Acc2 S = e1.right;
    acc2_decay(S, w, static_cast<float>(L - n));    // given at position L-1; anchor it at token n-1
    Acc2 stash[L];
    for (int i = n - 1; i >= 0; --i) {
        const float d = last - static_cast<float>(i);
        stash[i] = acc2_at(S, w, d);
        acc2_add(S, ks[i * kCs] + w * d, vs[i * kCs], 1.f);
    }
    if (!kBwd) {
        Acc2 Pt{P4.a, P4.b, P4.o};
        for (int i = 0; i < n; ++i) {
            const float k = ks[i * kCs], v = vs[i * kCs], d = static_cast<float>(i);
            const TokenOut o = token_out(acc2_at(Pt, w, d), stash[i], k, v, u);
            ks[i * kCs] = o.y;
            acc2_add(Pt, k + w * d, v, 1.f);
        }
        return;
    }
    // backward: G e^{m}, H e^{m}, -m per token; gw from pairs (output later than input)
    float gg[L], hh[L], xo[L];
    float gw = 0.f, gu = 0.f;
    Acc4 PM = P4;   // prefix state with first moments
    for (int i = 0; i < n; ++i) {
        const float k = ks[i * kCs], v = vs[i * kCs], d = static_cast<float>(i);
        const Acc2 Pi{PM.a, PM.b, PM.o - w * d};
        const TokenOut o = token_out(Pi, stash[i], k, v, u);
        gg[i] = gs[i * kCs] * o.inv_den;
        hh[i] = gg[i] * o.y;
        xo[i] = -o.m;
        gw -= wkv_exp(Pi.o + xo[i]) * (gg[i] * PM.ma - hh[i] * PM.mb);
        acc4_absorb(PM, k + w * d, v, 1.f);
    }
    Acc4 later = acc4_zero();
    Acc2 earlier = acc2_zero();
    for (int i = 0; i < n; ++i) acc4_absorb(later, xo[i] + w * static_cast<float>(i), gg[i], hh[i]);
    for (int i = n - 1; i >= 0; --i) acc2_add(earlier, xo[i] - w * static_cast<float>(i), gg[i], hh[i]);
    later.o -= w * static_cast<float>(n);
    acc4_decay(later, w, static_cast<float>(L - n));
    earlier.o -= w;
    const Entering e2 = exact_exchange<St, kBwd>(c, sub, ch, w, later, earlier);
    Acc4 Rt = e2.left;                              // anchored at token 0
    Acc2 Q = e2.right;
    acc2_decay(Q, w, static_cast<float>(L - n));    // anchored at token n-1
    float pk[L], pv[L];
    for (int i = n - 1; i >= 0; --i) {
        const float d = last - static_cast<float>(i);
        const float e = wkv_exp(ks[i * kCs] + Q.o - w * d);
        pv[i] = e * Q.a;
        pk[i] = e * (Q.a * vs[i * kCs] - Q.b);
        acc2_add(Q, xo[i] + w * d, gg[i], hh[i]);
    }
    for (int i = 0; i < n; ++i) {
        const float k = ks[i * kCs], v = vs[i * kCs], d = static_cast<float>(i);
        const float e = wkv_exp(k + Rt.o - w * d);
        const float es = wkv_exp(u + k + xo[i]);
        const float self = es * (v * gg[i] - hh[i]);
        vs[i * kCs] = pv[i] + e * Rt.a + es * gg[i];
        ks[i * kCs] = pk[i] + e * (Rt.a * v - Rt.b) + self;
        gu += self;
        gw -= e * (Rt.ma * v - Rt.mb);
        acc4_absorb(Rt, xo[i] + w * d, gg[i], hh[i]);
    }
    gw_out = gw;
    gu_out = gu;
}

template <class St, bool kBwd>
static inline size_t exact_smem(int n_warps) {
    const size_t data = static_cast<size_t>(kBwd ? 3 : 2) * n_warps * St::kAreaFloats;
    return (data + static_cast<size_t>(n_warps) * St::kW * 5 * St::kCs + 5 * St::kCs) * sizeof(float) + 16;
}

template <class St, bool kBwd, Types kTypes>
__global__ void __launch_bounds__(kMaxWarps * 32, 1)
biwkv_exact_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_o0,
                   const __grid_constant__ CUtensorMap map_o1, const Params p) {
    launch_dependents();
    wait_for_launch_before();
    constexpr int P = St::P, L = St::L, kCs = St::kCs, kSpan = St::kSpan, kArea = St::kAreaFloats;
    constexpr bool kHalf = kTypes != Types::f32, kHalfG = kTypes == Types::bf16;
    constexpr bool kHalfOut = kBwd ? kHalf : kTypes == Types::bf16;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const int n_clusters = static_cast<int>(gridDim.x) / p.cluster, mine = static_cast<int>(blockIdx.x) / p.cluster;
    const int rank = p.cluster > 1 ? static_cast<int>(cluster_rank()) : 0;
    // this cluster's units: mine, mine + n_clusters, ..; all their CTAs wrote the same kRedo
    bool any = false;
    unsigned bits = 0u;
    for (int u = mine + static_cast<int>(threadIdx.x) * n_clusters; u < p.units; u += static_cast<int>(blockDim.x) * n_clusters) {
        any = any || (__ldcg(p.words + static_cast<size_t>(u) * p.cluster) & kRedo) != 0u;
        bits |= __ldcg(p.words + static_cast<size_t>(u) * p.cluster + rank) >> kFailedShift;
    }
    if (bits != 0u) atomicOr(p.status, bits);
    if (!__syncthreads_or(any ? 1 : 0)) return;       // the same for every CTA of a cluster
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int pr = lane % P, wk = lane / P;
    const int nw = p.n_warps;
    float* const slot_k = reinterpret_cast<float*>(smem_raw) + warp * kArea;
    float* const slot_v = slot_k + nw * kArea;
    float* const slot_g = slot_v + nw * kArea;
    ExactCtx c;
    c.n_sub = nw * St::kW; c.n_tok = p.n_tok; c.cluster = p.cluster;
    c.area = reinterpret_cast<float*>(smem_raw) + (kBwd ? 3 : 2) * nw * kArea;
    c.agg = c.area + c.n_sub * 5 * kCs;
    c.rank = rank;
    uint64_t* const full = reinterpret_cast<uint64_t*>(c.agg + 5 * kCs);
    if (threadIdx.x == 0) {
        sm100::mbar_init(full, 1);
        sm100::mbar_init_fence();
    }
    __syncthreads();
    const int cta0 = c.rank * p.n_tok, tok0 = cta0 + warp * kSpan, row0 = wk * L, sub = warp * St::kW + wk;
    const int n = max(0, min(L, p.T - (tok0 + row0)));
    float* const ks = slot_k + row0 * kCs + 2 * pr;
    float* const vs = slot_v + row0 * kCs + 2 * pr;
    float* const gs = slot_g + row0 * kCs + 2 * pr;
    uint32_t phase = 0;
    for (int unit = mine; unit < p.units; unit += n_clusters) {
        if ((__ldcg(p.words + static_cast<size_t>(unit) * p.cluster) & kRedo) == 0u) continue;
        const int b = unit / p.n_strips, strip = unit - b * p.n_strips;
        constexpr int kIn = kHalf ? kArea / 2 : 0, kInG = kHalfG ? kArea / 2 : 0;
        if (threadIdx.x == 0) {
            sm100::mbar_expect_tx(full, static_cast<uint32_t>(nw) * (2 * (kArea - kIn) + (kBwd ? kArea - kInG : 0)) * 4u);
            for (int s = 0; s < nw; ++s) {
                sm100::tma_load_3d(slot_k + s * kArea + kIn, &map_k, full, strip * kCs, cta0 + s * kSpan, b);
                sm100::tma_load_3d(slot_v + s * kArea + kIn, &map_v, full, strip * kCs, cta0 + s * kSpan, b);
                if (kBwd) sm100::tma_load_3d(slot_g + s * kArea + kInG, &map_g, full, strip * kCs, cta0 + s * kSpan, b);
            }
        }
        const int ch0 = strip * kCs + 2 * pr;
        const float2 w2 = ch0 < p.C ? at2(p.w + ch0) : f2(0.f, 0.f), u2 = ch0 < p.C ? at2(p.u + ch0) : f2(0.f, 0.f);
        if (!sm100::mbar_wait(full, phase, kSpinLimit)) report_failure(p.status, p.mirror, 2u);
        phase ^= 1u;
        const auto widen_rows = [&](float* area) {      // all of the warp's rows are read before any is written over
            uint32_t x[L];
            for (int i = 0; i < L; ++i) x[i] = (reinterpret_cast<const uint32_t*>(area + kArea / 2) + (row0 + i) * P)[pr];
            __syncwarp();
            for (int i = 0; i < L; ++i) *reinterpret_cast<float2*>(area + (row0 + i) * kCs + 2 * pr) = f2(__uint_as_float(x[i] << 16), __uint_as_float(x[i] & 0xffff0000u));
            __syncwarp();
        };
        if (kHalf) { widen_rows(slot_k); widen_rows(slot_v); }
        if (kBwd && kHalfG) widen_rows(slot_g);
        if (kBwd && kTypes == Types::wide)
            for (int i = 0; i < L; ++i) *reinterpret_cast<float2*>(gs + i * kCs) = round2(at2(gs + i * kCs));
        float2 gw = f2(0.f, 0.f), gu = f2(0.f, 0.f);
        exact_walk<St, kBwd>(c, sub, 2 * pr, ks, vs, gs, n, w2.x, u2.x, gw.x, gu.x);
        exact_walk<St, kBwd>(c, sub, 2 * pr + 1, ks + 1, vs + 1, gs + 1, n, w2.y, u2.y, gw.y, gu.y);
        if (kHalfOut) {
            const size_t at = (static_cast<size_t>(b) * p.T + tok0 + row0) * p.C + ch0;
            for (int i = 0; i < (ch0 < p.C ? n : 0); ++i) {
                *reinterpret_cast<__nv_bfloat162*>(static_cast<__nv_bfloat16*>(p.o0) + at + static_cast<size_t>(i) * p.C) = __float22bfloat162_rn(at2(ks + i * kCs));
                if (kBwd) *reinterpret_cast<__nv_bfloat162*>(static_cast<__nv_bfloat16*>(p.o1) + at + static_cast<size_t>(i) * p.C) = __float22bfloat162_rn(at2(vs + i * kCs));
            }
        } else {
            if (kHalf)
                for (int i = 0; i < L; ++i) *reinterpret_cast<float2*>(ks + i * kCs) = round2(at2(ks + i * kCs));
            sm100::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0 && tok0 < p.T) {
                sm100::tma_store_3d(&map_o0, slot_k, strip * kCs, tok0, b);
                if (kBwd) sm100::tma_store_3d(&map_o1, slot_v, strip * kCs, tok0, b);
                sm100::tma_store_commit();
            }
        }
        if (kBwd) {
            *reinterpret_cast<float2*>(gs) = gw;
            *reinterpret_cast<float2*>(gs + kCs) = gu;
            __syncthreads();
            if (threadIdx.x < 2 * kCs) {
                const int jj = threadIdx.x / kCs, ch = threadIdx.x & (kCs - 1);
                const float* const g0 = reinterpret_cast<const float*>(smem_raw) + 2 * nw * kArea + ch;
                float acc = 0.f;
                for (int s = 0; s < c.n_sub; ++s) acc += g0[(s / St::kW) * kArea + ((s % St::kW) * L + jj) * kCs];
                p.partial[((static_cast<size_t>(b) * c.cluster + c.rank) * 2 + jj) * p.c_padded + strip * kCs + ch] = acc;
            }
        }
        if (!kHalfOut && lane == 0) sm100::tma_store_wait_read();
        // the slots are free for the next unit; the next tiles are written through the async proxy
        sm100::fence_proxy_async_smem();
        __syncthreads();
    }
}

// out[j][c] = sum over sequences and ranks of the partials, fixed order
__global__ void __launch_bounds__(1024) reduce_partials(int rows, int c_padded, int C, const float* partial, float* __restrict__ out) {
    wait_for_launch_before();
    __shared__ float red[32][33];
    const int j = blockIdx.y, lane = threadIdx.x, ch = blockIdx.x * 32 + lane;
    float acc = 0.f;
    if (ch < C)
        for (int r = threadIdx.y; r < rows; r += 32) acc += __ldcg(partial + (static_cast<size_t>(r) * 2 + j) * c_padded + ch);
    red[threadIdx.y][lane] = acc;
    __syncthreads();
    if (threadIdx.y == 0 && ch < C) {
        float total = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) total += red[r][lane];
        out[static_cast<size_t>(j) * C + ch] = total;
    }
}

// ---- host side ------------------------------------------------------------------------------------
// test mode: rank 1 of every cluster withholds its sends and waits give up after 2^10 polls, so that the bounded waits can be seen
// to run out (status bit 0) without anything hanging
static std::atomic<bool> g_withhold{false};
void set_withhold_test(bool on) { g_withhold.store(on); }

// How a call is split: which strips, CTAs per unit, warps per CTA.
struct Plan {
    int strip = 0, cluster = 1, n_warps = 0;
    int cs = 0, n_tok = 0;
};
// f(Strip) for the one that a plan names
template <class F>
static auto with_strip(int strip, F&& f) {
    switch (strip) {
        case 0: return f(Strip<8, 17>());
        case 1: return f(Strip<4, 17>());
        case 2: return f(Strip<8, 15>());
        default: return f(Strip<4, 15>());
    }
}
constexpr int kStrips = 4;
// The sequences that are served here.  Up to 4096 tokens all.  Above, where there are at least kManyCtas CTAs' worth (of 256 tokens and
// 32 channels, as biwkv_resident.cu counts them), up to kMostTokens, 16 CTAs of the narrow strips; with every tensor bfloat16 up to
// kMostHalf, 16 of the others.  Training pairs through autograd, us, separate launches with kept states / here: float32 B=16, T=4200,
// C=768 546 / 382; 16 x 8192 1022 / 801; 8 x 16384 1053 / 952; bfloat16 k, v beside float32 y, gy 710 / 383, 1286 / 868, 1295 / 1033;
// all bfloat16 551 / 408, 952 / 915, but 11 x 12000 971 / 1085 (rows of 16 bytes, and two passes over half the bytes are cheap).
// Below kManyCtas this is faster as well (B=2, T=4200, C=384: forward 31 / 23, backward 65 / 34): the line is not one of speed.  The routes
// there keep the shapes at which their tests count launches and kept states.
constexpr int kAnyTokens = 4096, kMostTokens = kMaxCluster * kMaxWarps * Strip<4, 17>::kSpan, kMostHalf = kMaxCluster * kMaxWarps * Strip<8, 17>::kSpan;
constexpr long long kManyCtas = 768;
bool in_range(int B, int T, int C, Types types) {
    if (C % (types != Types::f32 ? 8 : 4) != 0) return false;      // TMA row pitch must be 16-byte
    if (T <= kAnyTokens) return true;
    return T <= (types == Types::bf16 ? kMostHalf : kMostTokens) && static_cast<long long>(B) * ((C + 31) / 32) * ((T + 255) / 256) >= kManyCtas;
}

// A plan's time for a token, up to a factor: token slots taken, the warps that an SM then has in hand (registers: 16 of the backward,
// 24 of the forward), the hand-over between a cluster's CTAs, narrow rows.
static float plan_cost(int T, bool bwd, Types types, const Plan& pl) {
    // clusters of 1 to 8 CTAs; strips of 16 channels, tokens a multiple of 544, us at 100.7 M elements: float32 backward 352, 423, 459, 449,
    // (2304 tokens) 479, 478, -, 500; forward, bfloat16, 164, 191, 206, 206, 220, 208, -, 221
    static const float kBackward[] = {1.f, 1.2f, 1.3f, 1.27f, 1.39f, 1.36f, 1.42f, 1.41f}, kForward[] = {1.f, 1.13f, 1.2f, 1.2f, 1.26f, 1.24f, 1.3f, 1.3f};
    const int most = bwd ? 16 : 24, held = most / pl.n_warps * pl.n_warps;
    const float waste = static_cast<float>(pl.cluster * pl.n_tok) / static_cast<float>(T);
    const float idle = 1.f + 0.4f * static_cast<float>(most - held) / static_cast<float>(most);
    // more CTAs: float32 backward of 10, 12, 16 CTAs 544 (5000 tokens), 593, 633; forward 226, 241, 259
    const float* const by_cluster = bwd ? kBackward : kForward;
    const int most_listed = 8, listed = pl.cluster < most_listed ? pl.cluster : most_listed;
    const float hand_over = by_cluster[listed - 1] + (bwd ? 0.05f : 0.025f) * static_cast<float>(pl.cluster - listed);
    const float narrow = pl.cs == 16 ? 1.f : types == Types::f32 ? (bwd ? 1.04f : 1.19f) : (bwd ? 1.14f : 1.09f);
    return waste * idle * hand_over * narrow;
}
static bool make_plan(int B, int T, int C, bool bwd, Types types, Plan& best) {
    if (!in_range(B, T, C, types)) return false;
    const auto up = [](int a, int b) { return (a + b - 1) / b; };
    float least = 0.f;
    best.strip = -1;
    for (int i = 0; i < kStrips; ++i) {
        Plan pl;
        pl.strip = i;
        int span = 0;
        with_strip(i, [&](auto st) { span = decltype(st)::kSpan; pl.cs = decltype(st)::kCs; });
        pl.cluster = up(T, kMaxWarps * span);
        pl.n_warps = up(up(T, pl.cluster), span);
        pl.n_tok = pl.n_warps * span;
        if (pl.cluster > kMaxCluster) continue;      // every CTA owns a token: T > (cluster - 1) kMaxWarps span
        if (g_withhold.load() && pl.cluster == 1 && i != 0) continue;      // the test wants a hand-over where there can be one
        const float cost = plan_cost(T, bwd, types, pl);
        if (best.strip < 0 || cost < least) {
            best = pl;
            least = cost;
        }
    }
    return best.strip >= 0;
}

template <class St, Types kTypes>
static auto forward_kernel(bool single) { return single ? biwkv_forward_kernel<St, kTypes, true> : biwkv_forward_kernel<St, kTypes, false>; }
template <class St, Types kTypes>
static auto backward_kernel(bool single) { return single ? biwkv_backward_kernel<St, kTypes, true> : biwkv_backward_kernel<St, kTypes, false>; }
constexpr int kMostSmem = 227 * 1024;
template <typename F>
static bool allow(F* fn, bool cluster) {
    const void* f = reinterpret_cast<const void*>(fn);
    return cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem) == cudaSuccess &&
           (!cluster || cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess);
}
template <class St, Types kTypes>
static bool allow_all() {
    return allow(forward_kernel<St, kTypes>(true), false) && allow(forward_kernel<St, kTypes>(false), true) &&
           allow(backward_kernel<St, kTypes>(true), false) && allow(backward_kernel<St, kTypes>(false), true) &&
           allow(biwkv_exact_kernel<St, false, kTypes>, true) && allow(biwkv_exact_kernel<St, true, kTypes>, true);
}
template <class St>
static bool allow_types() { return allow_all<St, Types::f32>() && allow_all<St, Types::bf16>() && allow_all<St, Types::wide>(); }

static bool allow_strips() {
    for (int i = 0; i < kStrips; ++i)
        if (!with_strip(i, [](auto st) { return allow_types<decltype(st)>(); })) return false;
    return true;
}

struct DeviceState {
    bool probed = false, ok = false;
    // [strip][tensor types][bwd][cluster][n_warps]: 0 unknown, 1 launchable, -1 not
    signed char fits[kStrips][3][2][kMaxCluster + 1][kMaxWarps + 1] = {};
};
static std::mutex g_mutex;
static DeviceState g_dev[64];

template <typename F>
static bool cluster_fits(F* fn, int cluster, int threads, size_t smem) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(cluster);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster; at[0].val.clusterDim.y = 1; at[0].val.clusterDim.z = 1;
    cfg.attrs = at; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, reinterpret_cast<const void*>(fn), &cfg) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return n > 0;
}
template <class St, bool kBwd, Types kTypes>
static bool fits(const Plan& pl) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lock(g_mutex);
    DeviceState& d = g_dev[dev & 63];
    if (!d.probed) {
        d.probed = true;
        int cl = 0;
        cudaDeviceGetAttribute(&cl, cudaDevAttrClusterLaunch, dev);
        d.ok = cl != 0 && tensor_map::encode_fn() != nullptr && allow_strips();
        if (!d.ok) cudaGetLastError();
    }
    if (!d.ok || pl.cluster == 1) return d.ok;
    signed char& slot = d.fits[pl.strip][static_cast<int>(kTypes)][kBwd ? 1 : 0][pl.cluster][pl.n_warps];
    if (slot == 0) {
        const int threads = pl.n_warps * 32;
        const size_t smem = smem_bytes<St, kBwd>(pl.n_warps, pl.cluster);
        bool good;
        if constexpr (kBwd) good = cluster_fits(backward_kernel<St, kTypes>(false), pl.cluster, threads, smem);
        else good = cluster_fits(forward_kernel<St, kTypes>(false), pl.cluster, threads, smem);
        slot = good && cluster_fits(biwkv_exact_kernel<St, kBwd, kTypes>, pl.cluster, threads, exact_smem<St, kBwd>(pl.n_warps)) ? 1 : -1;
    }
    return slot > 0;
}
template <class St>
static bool fits(const Plan& pl, bool bwd, Types types) {
    if (types == Types::wide) return bwd ? fits<St, true, Types::wide>(pl) : fits<St, false, Types::wide>(pl);
    if (types == Types::bf16) return bwd ? fits<St, true, Types::bf16>(pl) : fits<St, false, Types::bf16>(pl);
    return bwd ? fits<St, true, Types::f32>(pl) : fits<St, false, Types::f32>(pl);
}
static size_t strips_of(int C, const Plan& pl) { return (C + pl.cs - 1) / pl.cs; }

bool eligible(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, Types types) {
    for (const void* q : ptrs)
        if (reinterpret_cast<uintptr_t>(q) & 15u) return false;    // TMA base alignment
    Plan pl;
    if (!make_plan(B, T, C, bwd, types, pl) || B * strips_of(C, pl) * pl.cluster > (1u << 30)) return false;
    if (static_cast<long long>(T) * C > (1LL << 30)) return false;      // 32-bit offsets within a sequence
    return with_strip(pl.strip, [&](auto st) { return fits<decltype(st)>(pl, bwd, types); });
}

static size_t align_up(size_t x, size_t a) { return (x + a - 1) / a * a; }
// workspace: status block (256 B) | a word per CTA | backward partials | copies of w, u
struct Carve {
    size_t off_words, off_partial, off_vectors, total;
};
static Carve carve(int B, int C, const Plan& pl, bool bwd) {
    Carve cv;
    cv.off_words = 256;
    cv.off_partial = cv.off_words + align_up(B * strips_of(C, pl) * pl.cluster * sizeof(unsigned), 256);
    cv.off_vectors = cv.off_partial + (bwd ? align_up(static_cast<size_t>(B) * pl.cluster * 2 * strips_of(C, pl) * pl.cs * sizeof(float), 256) : 0);
    cv.total = cv.off_vectors + align_up(2 * static_cast<size_t>(C) * sizeof(float), 256);
    return cv;
}
size_t workspace_bytes(int B, int T, int C, bool bwd, Types types) {
    Plan pl;
    return make_plan(B, T, C, bwd, types, pl) ? carve(B, C, pl, bwd).total : 0;
}

template <class St, bool kBwd, Types kTypes>
static int launch(const Plan& pl, int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy,
                  void* o0, void* o1, float* gwgu, void* workspace, cudaStream_t stream) {
    constexpr bool kHalf = kTypes != Types::f32, kHalfOut = kBwd ? kHalf : kTypes == Types::bf16;
    constexpr int kCs = St::kCs, kSpan = St::kSpan;
    unsigned char* const ws = static_cast<unsigned char*>(workspace);
    const Carve cv = carve(B, C, pl, kBwd);
    float* const vectors = reinterpret_cast<float*>(ws + cv.off_vectors);
    Params p{};
    p.B = B; p.T = T; p.C = C;
    p.n_strips = static_cast<int>(strips_of(C, pl)); p.c_padded = p.n_strips * kCs; p.units = B * p.n_strips;
    p.cluster = pl.cluster; p.n_warps = pl.n_warps; p.n_tok = pl.n_tok;
    p.w = paired(w, C, vectors, stream);
    if (T == 1) {      // a single token is not decayed: whatever w is, the rows that fill up its walker must not grow with it
        cudaMemsetAsync(vectors, 0, static_cast<size_t>(C) * sizeof(float), stream);
        p.w = vectors;
    }
    p.u = paired(u, C, vectors + C, stream);
    p.o0 = o0; p.o1 = o1;
    p.status = reinterpret_cast<unsigned*>(ws);
    p.mirror = failure_mirror(kBwd ? Op::biwkv_backward : Op::biwkv_forward);
    p.partial = reinterpret_cast<float*>(ws + cv.off_partial);
    p.words = reinterpret_cast<unsigned*>(ws + cv.off_words);
    p.spin_limit = g_withhold.load() ? (1u << 10) : kSpinLimit;
    p.withhold_rank = g_withhold.load() ? 1 : -1;
    tensor_map::bind_primary_context();   // the tensor-map encoder is a driver call
    CUtensorMap mk, mv, mg, m0, m1;
    bool ok = tensor_map::make_btc(&mk, k, B, T, C, kCs, kSpan, kHalf) && tensor_map::make_btc(&mv, v, B, T, C, kCs, kSpan, kHalf);
    mg = m0 = m1 = mk;      // where not used
    if (kBwd) ok = ok && tensor_map::make_btc(&mg, gy, B, T, C, kCs, kSpan, kTypes == Types::bf16);
    if (!kHalfOut) ok = ok && tensor_map::make_btc(&m0, o0, B, T, C, kCs, kSpan, false) && (!kBwd || tensor_map::make_btc(&m1, o1, B, T, C, kCs, kSpan, false));
    if (!ok) {
        set_error_detail("cuTensorMapEncodeTiled rejected a (C, T, B) tensor map");
        return -1;
    }
    // `behind`: launched behind the kernel before it, which it waits for by itself (wait_for_launch_before)
    const auto run = [&](auto* fn, bool behind, size_t clusters, size_t smem, auto... args) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(clusters * pl.cluster));
        cfg.blockDim = dim3(pl.n_warps * 32);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute at[2];
        unsigned n = 0;
        if (behind) {
            at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            at[n++].val.programmaticStreamSerializationAllowed = 1;
        }
        if (pl.cluster > 1) {
            at[n].id = cudaLaunchAttributeClusterDimension;
            at[n].val.clusterDim.x = pl.cluster; at[n].val.clusterDim.y = 1; at[n++].val.clusterDim.z = 1;
        }
        cfg.attrs = at; cfg.numAttrs = n;
        const cudaError_t err = cudaLaunchKernelEx(&cfg, fn, args..., p);
        if (err != cudaSuccess) set_error_detail(cudaGetErrorName(err));
        return err == cudaSuccess;
    };
    const size_t units = p.units;
    const size_t smem = smem_bytes<St, kBwd>(pl.n_warps, pl.cluster);
    bool done;
    // Behind the kernel before it where a CTA holds whole sequences: 256 x 196 x 384 in bfloat16 36.9 -> 36.5 us.  Clusters start when enough SMs of
    // one group are free, and those that start while the kernel before ends lie worse: 16 x 4200 x 768 408.6 -> 411.5, 8 x 16384 x 768 950.7 -> 956.5.
    const bool early = pl.cluster == 1;
    if constexpr (kBwd) done = run(backward_kernel<St, kTypes>(pl.cluster == 1), early, units, smem, mk, mv, mg, m0, m1);
    else done = run(forward_kernel<St, kTypes>(pl.cluster == 1), early, units, smem, mk, mv, m0);
    if (!done) return -1;
    // the exact kernel: a few clusters that serve whatever the fast kernel left behind
    if (!run(biwkv_exact_kernel<St, kBwd, kTypes>, true, std::min<size_t>(units, std::max(16, 128 / pl.cluster)), exact_smem<St, kBwd>(pl.n_warps), mk, mv, mg, m0, m1)) return -1;
    if (kBwd) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((C + 31) / 32, 2);
        cfg.blockDim = dim3(32, 32);
        cfg.stream = stream;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at; cfg.numAttrs = 1;
        cudaLaunchKernelEx(&cfg, reduce_partials, B * pl.cluster, p.c_padded, C, static_cast<const float*>(p.partial), gwgu);
    }
    return kBwd ? 3 : 2;
}
template <bool kBwd, Types kTypes>
static int launch(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy, void* o0, void* o1,
                  float* gwgu, void* workspace, cudaStream_t stream) {
    Plan pl;
    if (!make_plan(B, T, C, kBwd, kTypes, pl)) return -1;
    return with_strip(pl.strip, [&](auto st) { return launch<decltype(st), kBwd, kTypes>(pl, B, T, C, w, u, k, v, gy, o0, o1, gwgu, workspace, stream); });
}

int forward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, Types types, void* workspace,
            cudaStream_t stream) {
    const auto fn = types == Types::f32 ? launch<false, Types::f32> : types == Types::bf16 ? launch<false, Types::bf16> : launch<false, Types::wide>;
    return fn(B, T, C, w, u, k, v, nullptr, y, nullptr, nullptr, workspace, stream);
}
int backward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy, float* gwgu, void* gk,
             void* gv, Types types, void* workspace, cudaStream_t stream) {
    const auto fn = types == Types::f32 ? launch<true, Types::f32> : types == Types::bf16 ? launch<true, Types::bf16> : launch<true, Types::wide>;
    return fn(B, T, C, w, u, k, v, gy, gk, gv, gwgu, workspace, stream);
}

}  // namespace strips
}  // namespace biwkv
