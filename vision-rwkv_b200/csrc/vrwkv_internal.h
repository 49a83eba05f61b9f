// Declarations shared between the C-ABI translation unit and the kernel files.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>
#include <initializer_list>

// Remember a one-line explanation of the most recent failure (read by vrwkv_last_error_detail).
void set_error_detail(const char* text);
// Add `launched` kernels to the process-wide count and turn the CUDA error state into a status.
int record_launches(int launched);
// Host-visible word of the current device and operator that kernels set when a bounded wait runs out (pinned, mapped;
// null until vrwkv_take_failures() has been called once, but for Op::linear).  It costs a successful launch nothing.
enum class Op { biwkv_forward, biwkv_backward, wkv6_forward, wkv6_backward, linear };
unsigned* failure_mirror(Op op);

namespace lineartc {
void set_withhold_test(bool on);   // test only: one role of every CTA withholds an arrival, waits give up early
bool withhold_test();
}

#ifdef __CUDACC__
// A bounded wait ran out: `status` is the launch's own device word, `mirror` the host-visible one (may be null).
__device__ __forceinline__ void report_failure(unsigned* status, unsigned* mirror, unsigned bits) {
    atomicOr(status, bits);
    if (mirror != nullptr) *reinterpret_cast<volatile unsigned*>(mirror) = bits;
}
#endif

namespace biwkv {
// Each launcher returns the number of kernels it enqueued.
size_t generic_forward_workspace(int B, int T, int C);
size_t generic_backward_workspace(int B, int T, int C);
int generic_forward(int B, int T, int C, const float* w, const float* u, const float* k,
                    const float* v, float* y, void* workspace, cudaStream_t stream);
int generic_backward(int B, int T, int C, const float* w, const float* u, const float* k,
                     const float* v, const float* gy, float* gwgu, float* gk, float* gv,
                     void* workspace, cudaStream_t stream);
namespace resident {
// Long sequences (biwkv_resident.cu): 4096 < T <= 32768, C % 4 == 0 (f32) or C % 8 == 0 (bf16; wide: not here), 16-byte aligned
// tensors.  The chunked kernels stand by for inputs outside the plain-float range: fused::eligible has to hold too.
// w, u, gwgu are float32 always, arithmetic and shared-memory state too.
enum class Types {
    f32,      // every tensor float32
    bf16,     // k, v, y, gy, gk, gv bfloat16
    wide,     // k, v, gk, gv bfloat16; gy float32, rounded as it is read; y float32 holding bfloat16 values
};
// True when it can serve this call on the current device.
bool eligible(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, Types types);
void set_withhold_test(bool on);   // test only: one rank per cluster sends nothing, waits give up early
// kept: of a call that leaves or starts from kept states
size_t workspace_bytes(int B, int T, int C, bool bwd, bool kept = false);
// What a forward leaves for the backward: the states entering every 16 tokens, 1.5 bytes per element, and a flag; 0
// where the backward takes nothing (T <= 4096, or few tokens in all).
size_t kept_bytes(int B, int T, int C);
int forward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, Types types,
            void* workspace, cudaStream_t stream, void* keep = nullptr);
int backward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy, float* gwgu,
             void* gk, void* gv, Types types, void* workspace, cudaStream_t stream, const void* kept = nullptr);
}  // namespace resident
namespace strips {
// Narrow strips, whole sequences in one CTA or cluster (biwkv_strips.cu), all types; 16-byte aligned tensors of these sizes:
bool in_range(int B, int T, int C, resident::Types types);
// ... and the current device can launch them
bool eligible(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bwd, resident::Types types);
void set_withhold_test(bool on);
size_t workspace_bytes(int B, int T, int C, bool bwd, resident::Types types);      // 0 outside in_range
int forward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, resident::Types types,
            void* workspace, cudaStream_t stream);
int backward(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy, float* gwgu,
             void* gk, void* gv, resident::Types types, void* workspace, cudaStream_t stream);
}  // namespace strips
namespace fused {
// True when the fused TMA path can serve this call on the current device.
bool eligible(int B, int T, int C, std::initializer_list<const void*> ptrs, bool bf16 = false);
size_t workspace_bytes(int B, int T, int C, bool bwd);
// run_if: when set, every kernel of the launch returns at once while that device word is zero; the caller then has cleared the
// first cleared_bytes of the workspace.
size_t cleared_bytes(int B, int T, int C, bool bwd);
int forward(int B, int T, int C, const float* w, const float* u, const float* k, const float* v,
            float* y, void* workspace, cudaStream_t stream, const unsigned* run_if = nullptr);
int backward(int B, int T, int C, const float* w, const float* u, const float* k, const float* v,
             const float* gy, float* gwgu, float* gk, float* gv, void* workspace,
             cudaStream_t stream, const unsigned* run_if = nullptr);
// Forward that also writes log Den (one float per element), and the backward that starts from the
// saved y and log Den: one exchange level instead of two.
bool eligible_saved(int B, int T, int C, std::initializer_list<const void*> ptrs);
int forward_save(int B, int T, int C, const float* w, const float* u, const float* k, const float* v, float* y,
                 float* logden, void* workspace, cudaStream_t stream);
int backward_saved(int B, int T, int C, const float* w, const float* u, const float* k, const float* v,
                   const float* gy, const float* y, const float* logden, float* gwgu, float* gk, float* gv,
                   void* workspace, cudaStream_t stream);
// k, v, y, gy, gk, gv hold bfloat16; w, u, gwgu stay float; arithmetic is the float kernels'.
int forward_bf16(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y,
                 void* workspace, cudaStream_t stream, const unsigned* run_if = nullptr);
int backward_bf16(int B, int T, int C, const float* w, const float* u, const void* k, const void* v,
                  const void* gy, float* gwgu, void* gk, void* gv, void* workspace, cudaStream_t stream,
                  const unsigned* run_if = nullptr);
}  // namespace fused
}  // namespace biwkv

namespace wkv6 {
// What a launch finds at zero: the status word, and results of n floats each that its blocks add into.  In the place of memsets, and like
// them not among the kernels that a launcher counts.
struct Cleared {
    float* p[3];           // null: none
    unsigned* status;      // may be null
    size_t n;
};
void clear(const Cleared& z, cudaStream_t stream);
// float32 state sweeps (wkv6_sweeps.cu); gv may be null, and the forward's workspace
size_t forward_workspace(int B, int T, int H);
int forward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
            const float* u, float* y, void* workspace, cudaStream_t stream);
size_t backward_workspace(int B, int T, int H);
int backward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
             const float* u, const float* gy, float* gr, float* gk, float* gv, float* gw, float* gu,
             void* workspace, cudaStream_t stream);
}  // namespace wkv6

namespace wkv6tc {
void set_withhold_test(bool on);   // test only: as in wkv6c
// Tensor-core forward (bf16 operands, fp32 state) without scratch memory.  `status` points at 4 writable device bytes.
int forward(int B, int T, int H, const float* r, const float* k, const float* v, const float* w_raw,
            const float* u, float* y, unsigned* status, cudaStream_t stream);
// r, k, v in bfloat16 (read as such by the kernel: no widening pass), w_raw, u, y float32.
int forward_bf16in(int B, int T, int H, const void* r, const void* k, const void* v, const float* w_raw,
                   const float* u, float* y, unsigned* status, cudaStream_t stream);
}  // namespace wkv6tc

namespace wkv6c {
// Chunked tensor-core kernels (wkv6_chunk.cu): bfloat16 operands (r, k, v, gy in bfloat16, or float32 rounded on the way
// in), scaled operands of gr, gk, gw carried to 16 bits.  gv may be null.
void set_withhold_test(bool on);   // test only: barriers wait for more than is copied, and give up early
size_t forward_workspace(int B, int T, int H);
size_t backward_workspace(int B, int T, int H);
int forward(int B, int T, int H, const void* r, const void* k, const void* v, const float* w, const float* u, float* y,
            bool bf16_in, void* workspace, cudaStream_t stream);
int backward(int B, int T, int H, const void* r, const void* k, const void* v, const float* w, const float* u, const void* gy,
             void* gr, void* gk, void* gv, float* gw, float* gu, bool bf16_in, bool gy_bf16, bool bf16_out, void* workspace,
             cudaStream_t stream);
}  // namespace wkv6c
