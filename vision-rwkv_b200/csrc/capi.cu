// C ABI of the library: argument validation, path selection, launch accounting.
// The contract of every function is stated in include/vrwkv_b200.h.
#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <mutex>
#include "vrwkv_b200.h"
#include "vrwkv_internal.h"

using biwkv::resident::Types;

namespace {
std::atomic<unsigned long long> g_launches{0};
std::atomic<int> g_path{0};   // 0 auto (resident, else fused, else generic), 1 generic only, 2 skip the resident path

thread_local char g_detail[256] = "";   // per calling thread: no lock needed

inline bool misaligned4(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 3u) != 0; }

int check_shape(int B, int T, int C) {
    if (B <= 0 || T <= 0 || C <= 0) return VRWKV_ERR_SHAPE;
    if (B > 65535) return VRWKV_ERR_SHAPE;                       // gridDim.z
    if (static_cast<long long>(T) > 4000000LL) return VRWKV_ERR_SHAPE;
    return VRWKV_OK;
}

int finish(int launched) {
    if (launched < 0) { cudaGetLastError(); return VRWKV_ERR_DEVICE; }
    g_launches.fetch_add(static_cast<unsigned long long>(launched), std::memory_order_relaxed);
    const cudaError_t err = cudaGetLastError();
    if (err == cudaSuccess) return VRWKV_OK;
    set_error_detail(cudaGetErrorName(err));
    return VRWKV_ERR_LAUNCH;
}
}  // namespace

void set_error_detail(const char* text) {
    std::strncpy(g_detail, text ? text : "", sizeof(g_detail) - 1);
    g_detail[sizeof(g_detail) - 1] = 0;
}

int record_launches(int launched) { return finish(launched); }

// One word per device and operator in pinned, mapped host memory: kernels write it only when a bounded wait runs out, the host
// reads it as ordinary memory, so watching for failures costs neither a copy nor an event per launch.
namespace {
constexpr int kMirrorDevices = 64, kMirrorOps = 5;
std::atomic<unsigned*> g_mirror{nullptr};
std::mutex g_mirror_mutex;
}  // namespace

// the words, set up by the first call; null where that fails
static unsigned* mirror_base() {
    unsigned* base = g_mirror.load(std::memory_order_acquire);
    if (base != nullptr) return base;
    std::lock_guard<std::mutex> lock(g_mirror_mutex);
    base = g_mirror.load(std::memory_order_acquire);
    if (base != nullptr) return base;
    // not an operation a stream capture may contain: leave the thread's capture mode out of it
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    void* p = nullptr;
    const cudaError_t err = cudaHostAlloc(&p, kMirrorDevices * kMirrorOps * sizeof(unsigned), cudaHostAllocPortable | cudaHostAllocMapped);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (err != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::memset(p, 0, kMirrorDevices * kMirrorOps * sizeof(unsigned));
    base = static_cast<unsigned*>(p);
    g_mirror.store(base, std::memory_order_release);
    return base;
}

unsigned* failure_mirror(Op op) {
    // a linear layer has no workspace whose status word would tell: its word is there from its first launch on
    unsigned* base = op == Op::linear ? mirror_base() : g_mirror.load(std::memory_order_acquire);
    int dev = 0;
    if (base == nullptr || cudaGetDevice(&dev) != cudaSuccess || dev >= kMirrorDevices) return nullptr;
    return base + dev * kMirrorOps + static_cast<int>(op);
}

extern "C" {

int vrwkv_version(void) { return 100; }

const char* vrwkv_last_error_detail(void) { return g_detail; }

const char* vrwkv_status_string(int status) {
    switch (status) {
        case VRWKV_OK: return "ok";
        case VRWKV_ERR_SHAPE: return "bad shape: B, T, C must be positive, B <= 65535, T <= 4000000";
        case VRWKV_ERR_NULL: return "null pointer argument";
        case VRWKV_ERR_WORKSPACE: return "workspace smaller than the *_workspace_bytes value";
        case VRWKV_ERR_ALIGNMENT: return "pointer alignment: data 4 bytes (WKV6 inputs 16 bytes), workspace 256 bytes";
        case VRWKV_ERR_LAUNCH: return "CUDA reported an error after a kernel launch";
        case VRWKV_ERR_DEVICE: return "required driver entry point or device attribute unavailable";
        case VRWKV_ERR_HEAD_SIZE: return "WKV6 requires C == 64 * H";
        case VRWKV_ERR_UNSUPPORTED: return "shape or alignment not covered by this entry point's kernels; use the plain f32 entry points";
        default: return "unknown status";
    }
}

unsigned long long vrwkv_launch_count(void) { return g_launches.load(std::memory_order_relaxed); }

int vrwkv_set_path(int path) {
    if (path < 0 || path > 3) return VRWKV_ERR_SHAPE;
    biwkv::resident::set_withhold_test(path == 3);
    biwkv::strips::set_withhold_test(path == 3);
    lineartc::set_withhold_test(path == 3);
    wkv6c::set_withhold_test(path == 3);
    wkv6tc::set_withhold_test(path == 3);
    g_path.store(path == 3 ? 0 : path);
    return VRWKV_OK;
}

int vrwkv_workspace_status(const void* workspace, void* stream, unsigned* status_out) {
    if (!workspace || !status_out) return VRWKV_ERR_NULL;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (cudaMemcpyAsync(status_out, workspace, sizeof(unsigned), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        cudaGetLastError();
        return VRWKV_ERR_LAUNCH;
    }
    return VRWKV_OK;
}

unsigned vrwkv_take_failures(int device) {
    unsigned* const base = mirror_base();
    if (base == nullptr) return 0;
    if (device < 0 || device >= kMirrorDevices) return 0;
    unsigned bits = 0;
    for (int op = 0; op < kMirrorOps; ++op) {
        volatile unsigned* word = base + device * kMirrorOps + op;
        const unsigned seen = *word;
        if (seen == 0) continue;
        *word = 0;
        bits |= seen | 1u << (8 + op);
    }
    return bits;
}

// Whether the narrow-strip kernels serve the call.
static bool strips_serve(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, Types types) {
    return g_path.load() == 0 && biwkv::strips::eligible(B, T, C, ptrs, bwd, types);
}
// The workspace that a call must bring: where those kernels serve it, no room for the others' paths.
static size_t scratch_bytes(bool one_pass, int B, int T, int C, Types types, bool bwd) {
    if (one_pass) return biwkv::strips::workspace_bytes(B, T, C, bwd, types);
    return bwd ? vrwkv_biwkv_backward_workspace_bytes(B, T, C) : vrwkv_biwkv_forward_workspace_bytes(B, T, C);
}
// Whether the kernels for long sequences serve the call, with what stands by behind them.
static bool resident_serves(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, Types types) {
    return g_path.load() == 0 && biwkv::resident::eligible(B, T, C, ptrs, bwd, types) && biwkv::fused::eligible(B, T, C, ptrs, types == Types::bf16);
}

static size_t one_pass_most(int B, int T, int C, bool bwd) {
    size_t most = 0;
    for (Types types : {Types::f32, Types::bf16, Types::wide}) most = std::max(most, biwkv::strips::workspace_bytes(B, T, C, bwd, types));
    return most;
}

size_t vrwkv_biwkv_forward_workspace_bytes(int B, int T, int C) {
    if (check_shape(B, T, C) != VRWKV_OK) return 0;
    return std::max({biwkv::generic_forward_workspace(B, T, C) + 256, biwkv::fused::workspace_bytes(B, T, C, false),
                     biwkv::resident::workspace_bytes(B, T, C, false), one_pass_most(B, T, C, false)});
}

int vrwkv_biwkv_forward_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                            const float* v, float* y, void* workspace, size_t workspace_bytes,
                            void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !y || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(k) || misaligned4(v) || misaligned4(y) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, y}, false, Types::f32);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::f32, false)) return VRWKV_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (one_pass) return finish(biwkv::strips::forward(B, T, C, w, u, k, v, y, Types::f32, workspace, s));
    if (resident_serves(B, T, C, {k, v, y}, false, Types::f32))
        return finish(biwkv::resident::forward(B, T, C, w, u, k, v, y, Types::f32, workspace, s));
    if (g_path.load() != 1 && biwkv::fused::eligible(B, T, C, {k, v, y}))
        return finish(biwkv::fused::forward(B, T, C, w, u, k, v, y, workspace, s));
    // generic path: status word (first 256 bytes) is cleared, scratch follows
    cudaMemsetAsync(workspace, 0, 256, s);
    return finish(biwkv::generic_forward(B, T, C, w, u, k, v, y, static_cast<char*>(workspace) + 256, s));
}

size_t vrwkv_biwkv_backward_workspace_bytes(int B, int T, int C) {
    if (check_shape(B, T, C) != VRWKV_OK) return 0;
    return std::max({biwkv::generic_backward_workspace(B, T, C) + 256, biwkv::fused::workspace_bytes(B, T, C, true),
                     biwkv::resident::workspace_bytes(B, T, C, true), one_pass_most(B, T, C, true)});
}

int vrwkv_biwkv_backward_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                             const float* v, const float* gy, float* gwgu, float* gk, float* gv,
                             void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !gy || !gwgu || !gk || !gv || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(k) || misaligned4(v) || misaligned4(gy) ||
        misaligned4(gwgu) || misaligned4(gk) || misaligned4(gv) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, gy, gk, gv}, true, Types::f32);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::f32, true)) return VRWKV_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (one_pass)
        return finish(biwkv::strips::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, Types::f32, workspace, s));
    if (resident_serves(B, T, C, {k, v, gy, gk, gv}, true, Types::f32))
        return finish(biwkv::resident::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, Types::f32, workspace, s));
    if (g_path.load() != 1 && biwkv::fused::eligible(B, T, C, {k, v, gy, gk, gv}))
        return finish(biwkv::fused::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, workspace, s));
    cudaMemsetAsync(workspace, 0, 256, s);
    return finish(biwkv::generic_backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv,
                                          static_cast<char*>(workspace) + 256, s));
}

static bool types_of(int types, Types& t) {
    if (types < VRWKV_TENSORS_F32 || types > VRWKV_TENSORS_BF16_WIDE) return false;
    t = types == VRWKV_TENSORS_F32 ? Types::f32 : types == VRWKV_TENSORS_BF16 ? Types::bf16 : Types::wide;
    return true;
}

int vrwkv_biwkv_one_pass(int B, int T, int C, int tensors) {
    Types types;
    return check_shape(B, T, C) == VRWKV_OK && types_of(tensors, types) && biwkv::strips::in_range(B, T, C, types) ? 1 : 0;
}

size_t vrwkv_biwkv_one_pass_workspace_bytes(int B, int T, int C, int tensors, int backward) {
    Types types;
    return check_shape(B, T, C) == VRWKV_OK && types_of(tensors, types) ? biwkv::strips::workspace_bytes(B, T, C, backward != 0, types) : 0;
}

size_t vrwkv_biwkv_kept_bytes(int B, int T, int C) {
    if (check_shape(B, T, C) != VRWKV_OK) return 0;
    return biwkv::resident::kept_bytes(B, T, C);
}

size_t vrwkv_biwkv_kept_workspace_bytes(int B, int T, int C, int backward) {
    return vrwkv_biwkv_kept_bytes(B, T, C) == 0 ? 0 : biwkv::resident::workspace_bytes(B, T, C, backward != 0, true);
}

int vrwkv_biwkv_forward_keep(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, int tensors,
                             void* kept, size_t kept_bytes, void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    Types types;
    if (!types_of(tensors, types)) return VRWKV_ERR_UNSUPPORTED;
    if (!w || !u || !k || !v || !y || !kept || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(kept)) & 255u)) return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < vrwkv_biwkv_kept_workspace_bytes(B, T, C, 0)) return VRWKV_ERR_WORKSPACE;
    if (!resident_serves(B, T, C, {k, v, y}, false, types)) return VRWKV_ERR_UNSUPPORTED;
    if (biwkv::resident::kept_bytes(B, T, C) == 0) return VRWKV_ERR_UNSUPPORTED;
    if (kept_bytes < biwkv::resident::kept_bytes(B, T, C)) return VRWKV_ERR_WORKSPACE;
    return finish(biwkv::resident::forward(B, T, C, w, u, k, v, y, types, workspace, static_cast<cudaStream_t>(stream), kept));
}

int vrwkv_biwkv_backward_kept(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy,
                              float* gwgu, void* gk, void* gv, int tensors, const void* kept, size_t kept_bytes, void* workspace,
                              size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    Types types;
    if (!types_of(tensors, types)) return VRWKV_ERR_UNSUPPORTED;
    if (!w || !u || !k || !v || !gy || !gwgu || !gk || !gv || !kept || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(gwgu) || ((reinterpret_cast<uintptr_t>(workspace) | reinterpret_cast<uintptr_t>(kept)) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < vrwkv_biwkv_kept_workspace_bytes(B, T, C, 1)) return VRWKV_ERR_WORKSPACE;
    if (!resident_serves(B, T, C, {k, v, gy, gk, gv}, true, types)) return VRWKV_ERR_UNSUPPORTED;
    if (biwkv::resident::kept_bytes(B, T, C) == 0) return VRWKV_ERR_UNSUPPORTED;
    if (kept_bytes < biwkv::resident::kept_bytes(B, T, C)) return VRWKV_ERR_WORKSPACE;
    return finish(biwkv::resident::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, types, workspace, static_cast<cudaStream_t>(stream), kept));
}

int vrwkv_biwkv_forward_save_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                                 const float* v, float* y, float* logden, void* workspace,
                                 size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !y || !logden || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || (reinterpret_cast<uintptr_t>(workspace) & 255u)) return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < vrwkv_biwkv_forward_workspace_bytes(B, T, C)) return VRWKV_ERR_WORKSPACE;
    if (!biwkv::fused::eligible(B, T, C, {k, v, y, logden})) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::fused::forward_save(B, T, C, w, u, k, v, y, logden, workspace, static_cast<cudaStream_t>(stream)));
}

int vrwkv_biwkv_backward_saved_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                                   const float* v, const float* gy, const float* y, const float* logden,
                                   float* gwgu, float* gk, float* gv, void* workspace,
                                   size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !gy || !y || !logden || !gwgu || !gk || !gv || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(gwgu) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < vrwkv_biwkv_backward_workspace_bytes(B, T, C)) return VRWKV_ERR_WORKSPACE;
    if (!biwkv::fused::eligible_saved(B, T, C, {k, v, gy, y, logden, gk, gv})) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::fused::backward_saved(B, T, C, w, u, k, v, gy, y, logden, gwgu, gk, gv, workspace,
                                               static_cast<cudaStream_t>(stream)));
}

int vrwkv_biwkv_forward_bf16(int B, int T, int C, const float* w, const float* u, const uint16_t* k,
                             const uint16_t* v, uint16_t* y, void* workspace, size_t workspace_bytes,
                             void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !y || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || (reinterpret_cast<uintptr_t>(workspace) & 255u)) return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, y}, false, Types::bf16);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::bf16, false)) return VRWKV_ERR_WORKSPACE;
    if (one_pass)
        return finish(biwkv::strips::forward(B, T, C, w, u, k, v, y, Types::bf16, workspace, static_cast<cudaStream_t>(stream)));
    if (resident_serves(B, T, C, {k, v, y}, false, Types::bf16))
        return finish(biwkv::resident::forward(B, T, C, w, u, k, v, y, Types::bf16, workspace, static_cast<cudaStream_t>(stream)));
    if (!biwkv::fused::eligible(B, T, C, {k, v, y}, true)) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::fused::forward_bf16(B, T, C, w, u, k, v, y, workspace, static_cast<cudaStream_t>(stream)));
}

int vrwkv_biwkv_backward_bf16(int B, int T, int C, const float* w, const float* u, const uint16_t* k,
                              const uint16_t* v, const uint16_t* gy, float* gwgu, uint16_t* gk,
                              uint16_t* gv, void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !gy || !gwgu || !gk || !gv || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(gwgu) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, gy, gk, gv}, true, Types::bf16);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::bf16, true)) return VRWKV_ERR_WORKSPACE;
    if (one_pass)
        return finish(biwkv::strips::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, Types::bf16, workspace, static_cast<cudaStream_t>(stream)));
    if (resident_serves(B, T, C, {k, v, gy, gk, gv}, true, Types::bf16))
        return finish(biwkv::resident::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, Types::bf16, workspace, static_cast<cudaStream_t>(stream)));
    if (!biwkv::fused::eligible(B, T, C, {k, v, gy, gk, gv}, true)) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::fused::backward_bf16(B, T, C, w, u, k, v, gy, gwgu, gk, gv, workspace,
                                              static_cast<cudaStream_t>(stream)));
}

int vrwkv_biwkv_forward_bf16_wide(int B, int T, int C, const float* w, const float* u, const uint16_t* k, const uint16_t* v, float* y,
                                  void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !y || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || (reinterpret_cast<uintptr_t>(workspace) & 255u)) return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, y}, false, Types::wide);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::wide, false)) return VRWKV_ERR_WORKSPACE;
    if (!one_pass) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::strips::forward(B, T, C, w, u, k, v, y, Types::wide, workspace, static_cast<cudaStream_t>(stream)));
}

int vrwkv_biwkv_backward_bf16_wide(int B, int T, int C, const float* w, const float* u, const uint16_t* k, const uint16_t* v,
                                   const float* gy, float* gwgu, uint16_t* gk, uint16_t* gv, void* workspace, size_t workspace_bytes,
                                   void* stream) {
    if (int st = check_shape(B, T, C)) return st;
    if (!w || !u || !k || !v || !gy || !gwgu || !gk || !gv || !workspace) return VRWKV_ERR_NULL;
    if (misaligned4(w) || misaligned4(u) || misaligned4(gwgu) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    const bool one_pass = strips_serve(B, T, C, {k, v, gy, gk, gv}, true, Types::wide);
    if (workspace_bytes < scratch_bytes(one_pass, B, T, C, Types::wide, true)) return VRWKV_ERR_WORKSPACE;
    if (!one_pass) return VRWKV_ERR_UNSUPPORTED;
    return finish(biwkv::strips::backward(B, T, C, w, u, k, v, gy, gwgu, gk, gv, Types::wide, workspace, static_cast<cudaStream_t>(stream)));
}

// ---- WKV6 ---------------------------------------------------------------------------------------
static int check_wkv6(int B, int T, int C, int H) {
    if (B <= 0 || T <= 0 || C <= 0 || H <= 0) return VRWKV_ERR_SHAPE;
    if (C != 64 * H) return VRWKV_ERR_HEAD_SIZE;
    if (static_cast<long long>(B) * H > 1000000000LL || T > 4000000) return VRWKV_ERR_SHAPE;   // 2*B*H is a grid dimension
    return VRWKV_OK;
}
static inline bool misaligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) != 0; }

size_t vrwkv_wkv6_backward_workspace_bytes(int B, int T, int C, int H) {
    if (check_wkv6(B, T, C, H) != VRWKV_OK) return 0;
    return wkv6::backward_workspace(B, T, H);
}

size_t vrwkv_wkv6_forward_workspace_bytes(int B, int T, int C, int H, int exact) {
    if (check_wkv6(B, T, C, H) != VRWKV_OK) return 0;
    return exact ? wkv6::forward_workspace(B, T, H) : wkv6c::forward_workspace(B, T, H);
}

int vrwkv_wkv6_forward(int B, int T, int C, int H, const void* r, const void* k, const void* v, int in_bf16, int exact,
                       const float* w_raw, const float* u, float* y, void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_wkv6(B, T, C, H)) return st;
    if (!r || !k || !v || !w_raw || !u || !y || !workspace) return VRWKV_ERR_NULL;
    if (in_bf16 && exact) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned16(r) || misaligned16(k) || misaligned16(v) || misaligned16(w_raw) || misaligned4(u) || misaligned4(y) ||
        (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < vrwkv_wkv6_forward_workspace_bytes(B, T, C, H, exact)) return VRWKV_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (exact)      // clears the status word itself
        return finish(wkv6::forward(B, T, H, static_cast<const float*>(r), static_cast<const float*>(k), static_cast<const float*>(v), w_raw, u,
                                    y, workspace, s));
    wkv6::clear(wkv6::Cleared{{}, static_cast<unsigned*>(workspace), 0}, s);
    return finish(wkv6c::forward(B, T, H, r, k, v, w_raw, u, y, in_bf16 != 0, workspace, s));
}

int vrwkv_wkv6_forward_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                           const float* w_raw, const float* u, float* y, void* stream) {
    if (int st = check_wkv6(B, T, C, H)) return st;
    if (!r || !k || !v || !w_raw || !u || !y) return VRWKV_ERR_NULL;
    if (misaligned16(r) || misaligned16(k) || misaligned16(v) || misaligned16(w_raw) || misaligned4(u) ||
        misaligned4(y))
        return VRWKV_ERR_ALIGNMENT;
    return finish(wkv6::forward(B, T, H, r, k, v, w_raw, u, y, nullptr, static_cast<cudaStream_t>(stream)));
}

int vrwkv_wkv6_forward_tc_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                              const float* w_raw, const float* u, float* y, void* workspace,
                              size_t workspace_bytes, void* stream) {
    if (int st = check_wkv6(B, T, C, H)) return st;
    if (!r || !k || !v || !w_raw || !u || !y || !workspace) return VRWKV_ERR_NULL;
    if (misaligned16(r) || misaligned16(k) || misaligned16(v) || misaligned16(w_raw) || misaligned4(u) ||
        misaligned16(y) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < 256) return VRWKV_ERR_WORKSPACE;
    if (g_path.load() != 1 && workspace_bytes >= wkv6c::forward_workspace(B, T, H))
        return vrwkv_wkv6_forward(B, T, C, H, r, k, v, 0, 0, w_raw, u, y, workspace, workspace_bytes, stream);
    return finish(wkv6tc::forward(B, T, H, r, k, v, w_raw, u, y, static_cast<unsigned*>(workspace), static_cast<cudaStream_t>(stream)));
}

int vrwkv_wkv6_forward_tc_bf16(int B, int T, int C, int H, const uint16_t* r, const uint16_t* k,
                               const uint16_t* v, const float* w_raw, const float* u, float* y,
                               void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_wkv6(B, T, C, H)) return st;
    if (!r || !k || !v || !w_raw || !u || !y || !workspace) return VRWKV_ERR_NULL;
    if (misaligned16(r) || misaligned16(k) || misaligned16(v) || misaligned16(w_raw) || misaligned4(u) ||
        misaligned16(y) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < 256) return VRWKV_ERR_WORKSPACE;
    if (g_path.load() != 1 && workspace_bytes >= wkv6c::forward_workspace(B, T, H))
        return vrwkv_wkv6_forward(B, T, C, H, r, k, v, 1, 0, w_raw, u, y, workspace, workspace_bytes, stream);
    return finish(wkv6tc::forward_bf16in(B, T, H, r, k, v, w_raw, u, y, static_cast<unsigned*>(workspace),
                                         static_cast<cudaStream_t>(stream)));
}

static int wkv6_backward(int B, int T, int C, int H, const void* r, const void* k, const void* v, bool in_bf16, bool exact,
                         const float* w_raw, const float* u, const void* gy, bool gy_bf16, void* gr, void* gk, void* gv, bool out_bf16,
                         float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream) {
    if (int st = check_wkv6(B, T, C, H)) return st;
    if (!r || !k || !v || !w_raw || !u || !gy || !gr || !gk || !gw || !gu || !workspace) return VRWKV_ERR_NULL;      // gv may be NULL
    if ((in_bf16 || gy_bf16 || out_bf16) && exact) return VRWKV_ERR_UNSUPPORTED;
    if (!in_bf16 && (gy_bf16 || out_bf16)) return VRWKV_ERR_UNSUPPORTED;
    if (misaligned16(r) || misaligned16(k) || misaligned16(v) || misaligned16(w_raw) || misaligned16(gy) || misaligned4(u) ||
        misaligned4(gw) || misaligned4(gu) || (reinterpret_cast<uintptr_t>(workspace) & 255u))
        return VRWKV_ERR_ALIGNMENT;
    for (const void* p : {static_cast<const void*>(gr), static_cast<const void*>(gk), static_cast<const void*>(gv)})
        if (reinterpret_cast<uintptr_t>(p) & (out_bf16 ? 1u : 3u)) return VRWKV_ERR_ALIGNMENT;
    if (workspace_bytes < (exact ? wkv6::backward_workspace(B, T, H) : wkv6c::backward_workspace(B, T, H))) return VRWKV_ERR_WORKSPACE;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (exact) {      // clears the status word itself
        const auto in = [](const void* p) { return static_cast<const float*>(p); };
        const auto out = [](void* p) { return static_cast<float*>(p); };
        return finish(wkv6::backward(B, T, H, in(r), in(k), in(v), w_raw, u, in(gy), out(gr), out(gk), out(gv), gw, gu, workspace, s));
    }
    wkv6::clear(wkv6::Cleared{{}, static_cast<unsigned*>(workspace), 0}, s);
    return finish(wkv6c::backward(B, T, H, r, k, v, w_raw, u, gy, gr, gk, gv, gw, gu, in_bf16, gy_bf16, out_bf16, workspace, s));
}

size_t vrwkv_wkv6_backward_bytes(int B, int T, int C, int H, int exact) {
    if (check_wkv6(B, T, C, H) != VRWKV_OK) return 0;
    return exact ? wkv6::backward_workspace(B, T, H) : wkv6c::backward_workspace(B, T, H);
}

int vrwkv_wkv6_backward(int B, int T, int C, int H, const void* r, const void* k, const void* v, int in_bf16, int exact,
                        const float* w_raw, const float* u, const void* gy, int gy_bf16, void* gr, void* gk, void* gv, int out_bf16,
                        float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream) {
    return wkv6_backward(B, T, C, H, r, k, v, in_bf16 != 0, exact != 0, w_raw, u, gy, gy_bf16 != 0, gr, gk, gv, out_bf16 != 0, gw, gu,
                         workspace, workspace_bytes, stream);
}

int vrwkv_wkv6_backward_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                            const float* w_raw, const float* u, const float* gy, float* gr, float* gk,
                            float* gv, float* gw, float* gu, void* workspace, size_t workspace_bytes,
                            void* stream) {
    return wkv6_backward(B, T, C, H, r, k, v, false, true, w_raw, u, gy, false, gr, gk, gv, false, gw, gu, workspace, workspace_bytes,
                         stream);
}

size_t vrwkv_wkv6_backward_tc_workspace_bytes(int B, int T, int C, int H) {
    if (check_wkv6(B, T, C, H) != VRWKV_OK) return 0;
    return wkv6c::backward_workspace(B, T, H);
}

int vrwkv_wkv6_backward_tc_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                               const float* w_raw, const float* u, const float* gy, float* gr, float* gk, float* gv,
                               float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream) {
    return wkv6_backward(B, T, C, H, r, k, v, false, false, w_raw, u, gy, false, gr, gk, gv, false, gw, gu, workspace, workspace_bytes,
                         stream);
}

int vrwkv_wkv6_backward_tc_bf16(int B, int T, int C, int H, const uint16_t* r, const uint16_t* k, const uint16_t* v,
                                const float* w_raw, const float* u, const uint16_t* gy, float* gr, float* gk, float* gv,
                                float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream) {
    return wkv6_backward(B, T, C, H, r, k, v, true, false, w_raw, u, gy, true, gr, gk, gv, false, gw, gu, workspace, workspace_bytes,
                         stream);
}

}  // extern "C"
