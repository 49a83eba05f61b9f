/* vrwkv_b200 -- C ABI of the B200 (sm_100a) token-mixing kernels of Vision-RWKV.
 *
 * Every entry point takes plain device pointers and sizes, launches on the CUDA
 * stream it is given (a cudaStream_t passed as void*; NULL is the legacy default
 * stream), never synchronises, never allocates, and returns a status code
 * (VRWKV_OK == 0).  The caller owns every buffer, including the scratch
 * "workspace" (256-byte aligned), whose size the matching *_workspace_bytes function
 * reports.
 * Outputs need no initialisation: every element is written.
 *
 * Layouts: k, v, y, gy, gk, gv, r, gr, w_raw, gw_raw are (B, T, C) row-major,
 * channel fastest (the backbones' token-major layout).  All data are fp32, as in
 * the reference, whose Python wrappers cast to fp32 before calling the kernels.
 *
 * Each declaration names the reference interface it stands in for, by path inside
 * the OpenGVLab/Vision-RWKV tree ("CLS/" = classification/mmcls_custom/models/
 * backbones/, "MAE/" = classification/mae/).
 */
#ifndef VRWKV_B200_H_
#define VRWKV_B200_H_

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum vrwkv_status {
    VRWKV_OK = 0,
    VRWKV_ERR_SHAPE = 1,       /* a dimension is <= 0 or beyond what a launch can index   */
    VRWKV_ERR_NULL = 2,        /* a required pointer is NULL                               */
    VRWKV_ERR_WORKSPACE = 3,   /* workspace_bytes is smaller than *_workspace_bytes says   */
    VRWKV_ERR_ALIGNMENT = 4,   /* data pointer not 4-byte / workspace not 256-byte aligned */
    VRWKV_ERR_LAUNCH = 5,      /* cudaGetLastError() reported a failure after a launch     */
    VRWKV_ERR_DEVICE = 6,      /* driver entry point or device attribute unavailable       */
    VRWKV_ERR_HEAD_SIZE = 7,   /* WKV6: C != 64 * H                                        */
    VRWKV_ERR_UNSUPPORTED = 8  /* bf16 and saved-result entry points: shape or alignment outside
                                  what their kernels cover; nothing ran, use the plain f32
                                  entry points                                               */
};

/* Library version, major*10000 + minor*100 + patch. */
int vrwkv_version(void);
/* Human-readable text for a status code (static storage). */
const char* vrwkv_status_string(int status);
/* One line about the most recent non-zero status of the calling thread (for instance the name
 * of the CUDA error behind VRWKV_ERR_LAUNCH).  Thread-local storage.  Diagnostic. */
const char* vrwkv_last_error_detail(void);
/* Number of kernels this library has launched in the calling process so far, but for two that stand for what others did before and that was
 * not counted: the clearing of the status word and of results that WKV6's directions add into (memsets), and vrwkv_narrow (casts). */
unsigned long long vrwkv_launch_count(void);

/* Kernel path selection, for tests and measurements: 0 = automatic (default: Bi-WKV takes the
 * kernels that hold sequences in shared memory when T <= 32768, C % 4 == 0 (bfloat16: C % 8 == 0) and the
 * tensors are 16-byte aligned - one CTA or cluster per sequence strip where vrwkv_biwkv_one_pass is 1, else several
 * clusters or, for many tokens in all, separate launches -,
 * else the persistent tile kernels, else the generic multi-launch path), 1 = the
 * first-generation kernels (Bi-WKV: the generic multi-launch path; vrwkv_wkv6_forward_tc_*: the walk
 * that needs no scratch memory, whatever the workspace holds), 2 = Bi-WKV skips the
 * cluster-resident kernels (persistent tile kernels where eligible), 3 = test of the bounded
 * device-side waits: as 0, but one CTA of every cluster withholds what it owes the others and
 * the waits give up after about a thousand polls, so the call returns promptly with bit 0 of the
 * status word set and meaningless results (nothing hangs, nothing faults); the linear layers likewise, one role of each CTA, and
 * WKV6 on the tensor cores, whose barriers wait for more than is copied (bit 1).  Process-wide.
 * No reference counterpart. */
int vrwkv_set_path(int path);
/* Copies the device status word kept in the first 4 bytes of a workspace to *status_out
 * after synchronising `stream`.  0 means no bounded device-side wait ran out; bit 0 = a
 * hand-over between CTAs (tile-exchange flag, cluster mbarrier) never arrived, bit 1 = a TMA load never
 * completed, bit 2 = a record of another segment of a long sequence never arrived.  Diagnostic only;
 * no reference counterpart (the reference never checks its launches). */
int vrwkv_workspace_status(const void* workspace, void* stream, unsigned* status_out);

/* Failure bits (as in vrwkv_workspace_status) that launches on `device` have reported since the last call, and
 * clears them; 0 if none.  Bits 8 to 12 say whose launches: Bi-WKV forward, Bi-WKV backward, WKV6 forward, WKV6
 * backward, vrwkv_linear_relu_square.  Kernels that give up a bounded wait write a word of mapped host memory, so the
 * call reads host memory: no synchronisation, no copy.  A launch that is still running reports later:
 * synchronise first to see its result.  The first call (per process) sets the word up; launches made before it
 * report through their workspace only (vrwkv_linear_relu_square, which has none, sets the word up by itself: after a
 * synchronisation this call tells whether its result is whole). */
unsigned vrwkv_take_failures(int device);

/* ---- Bi-WKV --------------------------------------------------------------------
 * y[b,t,c] = sum_j p_tj v[b,j,c] / sum_j p_tj,  log p_tj = k[b,j,c] - w[c]|t-j| for
 * j != t and u[c] + k[b,t,c] for j == t.  w, u: (C,).
 *
 * vrwkv_biwkv_forward_f32 replaces
 *   cuda_forward(int B,int T,int C,float*w,float*u,float*k,float*v,float*y)
 *       MAE/vrwkv/cuda/wkv_op.cpp:3,6-8  (kernel MAE/vrwkv/cuda/wkv_cuda.cu:332-338)
 *   bi_wkv_cuda_forward(w,u,k,v) -> y
 *       CLS/cuda_new/bi_wkv.cpp:11-15,23-33 (kernel CLS/cuda_new/bi_wkv_kernel.cu:370-399)
 * without their T <= T_MAX, C >= 32 and B*C % 32 == 0 restrictions.
 */
size_t vrwkv_biwkv_forward_workspace_bytes(int B, int T, int C);
int vrwkv_biwkv_forward_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                            const float* v, float* y, void* workspace, size_t workspace_bytes,
                            void* stream);

/* vrwkv_biwkv_backward_f32 replaces
 *   cuda_backward(int B,int T,int C,float*w,float*u,float*k,float*v,float*gy,
 *                 float*gw,float*gu,float*gk,float*gv)
 *       MAE/vrwkv/cuda/wkv_op.cpp:4,9-11 (kernel MAE/vrwkv/cuda/wkv_cuda.cu:340-345)
 *   bi_wkv_cuda_backward(w,u,k,v,gy) -> {gw,gu,gk,gv}
 *       CLS/cuda_new/bi_wkv.cpp:17-21,35-47 (kernel CLS/cuda_new/bi_wkv_kernel.cu:401-443)
 * gwgu is (2, C): row 0 = gw, row 1 = gu, already summed over batch and tokens in
 * a fixed order (no atomics), contiguous so one all-reduce covers both.  Nothing
 * per-token is kept from the forward: the backward recomputes from k, v, gy.
 */
size_t vrwkv_biwkv_backward_workspace_bytes(int B, int T, int C);
int vrwkv_biwkv_backward_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                             const float* v, const float* gy, float* gwgu, float* gk, float* gv,
                             void* workspace, size_t workspace_bytes, void* stream);

/* Forward that keeps what the backward needs, and the backward that uses it.  The reference's
 * backward rebuilds y, 1/Den and the shift per token inside its kernel and holds them in three
 * scratch tensors (bi_wkv_kernel.cu:259-302, 415-417).  Here the forward can write log Den_t next
 * to y (one extra float per element), and vrwkv_biwkv_backward_saved_f32 takes k, v, gy and the
 * saved y, log Den: it needs one cross-tile exchange instead of two, at the price of keeping logden
 * (B*T*C floats) from forward to backward.  The pair runs on the tile kernels; where vrwkv_biwkv_one_pass
 * is 1 vrwkv_biwkv_forward_f32 + vrwkv_biwkv_backward_f32, which keep nothing, are
 * about twice as fast.  Results agree with the recomputing pair to float32 rounding.  Same workspace sizes.  Both are
 * served by the single-pass TMA kernels only (C % 4 == 0, 16-byte aligned tensors, T below about
 * 37 000); otherwise they return VRWKV_ERR_UNSUPPORTED and nothing ran. */
int vrwkv_biwkv_forward_save_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                                 const float* v, float* y, float* logden, void* workspace,
                                 size_t workspace_bytes, void* stream);
int vrwkv_biwkv_backward_saved_f32(int B, int T, int C, const float* w, const float* u, const float* k,
                                   const float* v, const float* gy, const float* y, const float* logden,
                                   float* gwgu, float* gk, float* gv, void* workspace,
                                   size_t workspace_bytes, void* stream);

/* bfloat16 activations: k, v, y, gy, gk, gv are bfloat16 bit patterns (uint16_t), w, u and
 * gwgu stay float, arithmetic is the f32 kernels' (inputs widened in shared memory, results
 * rounded to nearest-even on the way out).  They replace the float casts around the extension
 * calls in WKV.forward / WKV.backward (CLS/vrwkv.py:34-37, 51-55: `k.float().contiguous()` ...)
 * together with the calls themselves.  Workspace sizes are those of the f32 entry points.
 * Served by the single-pass TMA kernels only: C % 8 == 0, 16-byte aligned tensors and
 * ceil(T / 128) below the number of resident thread blocks (about T < 37 000); anything else
 * returns VRWKV_ERR_UNSUPPORTED before launching, and the caller casts and uses the f32 calls.
 */
int vrwkv_biwkv_forward_bf16(int B, int T, int C, const float* w, const float* u, const uint16_t* k,
                             const uint16_t* v, uint16_t* y, void* workspace, size_t workspace_bytes,
                             void* stream);
int vrwkv_biwkv_backward_bf16(int B, int T, int C, const float* w, const float* u, const uint16_t* k,
                              const uint16_t* v, const uint16_t* gy, float* gwgu, uint16_t* gk,
                              uint16_t* gv, void* workspace, size_t workspace_bytes, void* stream);
/* The same with float32 y and gy, what autograd has when w, u are float32 parameters and k, v come out of autocast
 * (CLS/vrwkv.py:42-44, 56-61 widen y and cast gy there): y holds the bfloat16 result widened, gy is rounded to bfloat16 as it is read.
 * Sizes for which vrwkv_biwkv_one_pass(.., VRWKV_TENSORS_BF16_WIDE) is 1; anything else, and tensors that are not 16-byte aligned,
 * returns VRWKV_ERR_UNSUPPORTED before launching. */
int vrwkv_biwkv_forward_bf16_wide(int B, int T, int C, const float* w, const float* u, const uint16_t* k, const uint16_t* v, float* y,
                                  void* workspace, size_t workspace_bytes, void* stream);
int vrwkv_biwkv_backward_bf16_wide(int B, int T, int C, const float* w, const float* u, const uint16_t* k, const uint16_t* v,
                                   const float* gy, float* gwgu, uint16_t* gk, uint16_t* gv, void* workspace, size_t workspace_bytes,
                                   void* stream);

/* 1 where calls of these sizes (`tensors`: enum below) go through the kernels that read and write every element once, forward and
 * backward: T <= 4096, and longer sequences up to 17 408 tokens where there are many.  A training pair has nothing to gain there from
 * kept states (next comment). */
int vrwkv_biwkv_one_pass(int B, int T, int C, int tensors);
/* Workspace with which the entry points above serve such calls: at most a few bytes per sequence and channel, where their own queries
 * have room for every path (up to 8.1 bytes per element).  0 where vrwkv_biwkv_one_pass is 0; too small for calls that go another way
 * all the same (tensors off a 16-byte boundary, vrwkv_set_path): VRWKV_ERR_WORKSPACE, nothing ran. */
size_t vrwkv_biwkv_one_pass_workspace_bytes(int B, int T, int C, int tensors, int backward);

/* The training pair for long sequences: a forward that leaves the states entering every 16 tokens (1.5 bytes per element, in a
 * caller-owned buffer of vrwkv_biwkv_kept_bytes bytes, 256-byte aligned), and a backward that starts from them instead of
 * rebuilding them: two passes over the inputs instead of three.  vrwkv_biwkv_kept_bytes is 0 where a backward has no use for
 * them (T <= 4096, or few tokens in all); where vrwkv_biwkv_one_pass is 1 the entry points above are faster.
 * w, u, k, v of the backward must be those of the forward.  `tensors` says what k, v, y, gy, gk, gv hold (enum below, as in the
 * entry points above; VRWKV_TENSORS_BF16_WIDE is refused: only the kernels that keep nothing take it).  The workspaces hold neither
 * the states nor room for the other paths: vrwkv_biwkv_kept_workspace_bytes bytes, 0 where nothing is kept (those of the other entry
 * points are larger and serve too).  VRWKV_ERR_UNSUPPORTED: outside the cluster-resident
 * kernels (shape, alignment, vrwkv_set_path), nothing ran, use the other entry points; a forward may succeed and the backward
 * still return it (for an unaligned gy).  Results agree with the pair that keeps nothing to float32 rounding (where
 * vrwkv_biwkv_one_pass is 0, y bit for bit).
 * No reference counterpart (its backward rebuilds everything, bi_wkv_kernel.cu:259-302). */
enum vrwkv_tensors { VRWKV_TENSORS_F32 = 0, VRWKV_TENSORS_BF16 = 1, VRWKV_TENSORS_BF16_WIDE = 2 };
size_t vrwkv_biwkv_kept_bytes(int B, int T, int C);
size_t vrwkv_biwkv_kept_workspace_bytes(int B, int T, int C, int backward);
int vrwkv_biwkv_forward_keep(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, void* y, int tensors,
                             void* kept, size_t kept_bytes, void* workspace, size_t workspace_bytes, void* stream);
int vrwkv_biwkv_backward_kept(int B, int T, int C, const float* w, const float* u, const void* k, const void* v, const void* gy,
                              float* gwgu, void* gk, void* gv, int tensors, const void* kept, size_t kept_bytes, void* workspace,
                              size_t workspace_bytes, void* stream);

/* vrwkv_biwkv_forward_f32_noalloc has no counterpart in the reference.  It is
 * vrwkv_biwkv_forward_f32 for callers that cannot allocate device memory and so have no
 * workspace to pass (a host that owns all device memory and lends only inputs and outputs,
 * a loop running under a frozen memory plan, code inside a region where allocation is
 * forbidden).  Its scratch is a 16 MiB array built into the library's device image, present
 * once on every GPU that loads the library until the process exits.
 *   - A shape is accepted when B * ceil(T / 16) * 24 * C bytes fit in 16 MiB (for example
 *     B=2, T=196, C=192, or B=4, T=1024, C=768); larger shapes return VRWKV_ERR_WORKSPACE.
 *   - The first call on a device also looks up the array's device address; make that call
 *     before starting any stream capture.  No call allocates or frees.
 *   - All calls on a device share the array: two calls that can overlap on the GPU (different
 *     streams with no ordering between them) race; calls on one stream do not.
 * Results equal vrwkv_biwkv_forward_f32's generic path bit for bit. */
int vrwkv_biwkv_forward_f32_noalloc(int B, int T, int C, const float* w, const float* u,
                                    const float* k, const float* v, float* y, void* stream);

/* ---- WKV6 (bidirectional, head size 64) ---------------------------------------------
 * Per (batch, head), state S in R^{64x64} [key][value], d_t = exp(-exp(w_raw_t)):
 *   S>_{t+1} = diag(d_t) S>_t + k_t v_t^T,  S<_{t-1} = diag(d_t) S<_t + k_t v_t^T
 *   y_t = r_t^T (S>_t + diag(u) k_t v_t^T) + r_t^T S<_t
 * r, k, v, w_raw, y, gy and the gradients are (B, T, C) with C = 64 H; u and gu are (H, 64).
 * Inputs must be 16-byte aligned.
 *
 * vrwkv_wkv6_forward_f32 replaces
 *   cuda_forward(int B,int T,int C,int H,float*r,float*k,float*v,float*w,float*u,float*y)
 *       CLS/cuda_v6/wkv6_op.cpp:4,7-9 (kernel CLS/cuda_v6/wkv6_cuda.cu:6-97,348-353)
 * It takes the raw decay input and forms -exp(w_raw) itself, where the reference's Python
 * wrapper does that in a separate pass (CLS/vrwkv6.py:48).  It needs no scratch memory.
 */
int vrwkv_wkv6_forward_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                           const float* w_raw, const float* u, float* y, void* stream);

/* vrwkv_wkv6_forward.  exact = 1: float32 r, k, v and float32 accuracy, as vrwkv_wkv6_forward_f32, but a few sequences
 * are walked in several segments at a time (at most 19 MB of scratch, none where the sequences fill the device).  exact = 0: 64-token chunks on the tensor cores (the states that enter each chunk, then all chunks in parallel):
 * r, k, v enter the matrix products as bfloat16 (in_bf16 = 1: they are bfloat16 bit patterns and are read as such; 0:
 * float32, rounded on the way in), sums are fp32; results agree with exact = 1 to about 1e-2 of max|y|.  w_raw, u and y are
 * float32.
 * Replaces the same reference entry point, and with in_bf16 the `.float()` passes in front of the reference's call
 * (CLS/vrwkv6.py:220 hands whatever dtype the projections produced to a kernel that reads float). */
size_t vrwkv_wkv6_forward_workspace_bytes(int B, int T, int C, int H, int exact);
int vrwkv_wkv6_forward(int B, int T, int C, int H, const void* r, const void* k, const void* v, int in_bf16, int exact,
                       const float* w_raw, const float* u, float* y, void* workspace, size_t workspace_bytes, void* stream);

/* vrwkv_wkv6_forward_tc_f32 / _bf16: vrwkv_wkv6_forward with exact = 0 for float32 / bfloat16 r, k, v.  A workspace of
 * 256 bytes (256-byte aligned; its first word is a status word as in vrwkv_workspace_status) is enough: they then walk
 * the sequence with the state in tensor memory, which is slower than the chunks they run when the workspace has
 * vrwkv_wkv6_forward_workspace_bytes(B, T, C, H, 0) bytes. */
int vrwkv_wkv6_forward_tc_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                              const float* w_raw, const float* u, float* y, void* workspace,
                              size_t workspace_bytes, void* stream);
int vrwkv_wkv6_forward_tc_bf16(int B, int T, int C, int H, const uint16_t* r, const uint16_t* k,
                               const uint16_t* v, const float* w_raw, const float* u, float* y,
                               void* workspace, size_t workspace_bytes, void* stream);

/* vrwkv_wkv6_backward_f32 replaces
 *   cuda_backward(int B,int T,int C,int H,float*r,...,float*gy,float*gr,float*gk,float*gv,
 *                 float*gw,float*gu)
 *       CLS/cuda_v6/wkv6_op.cpp:5,10-12 (kernels CLS/cuda_v6/wkv6_cuda.cu:99-346,355-362)
 * without its T <= 256 limit.  gw is the gradient w.r.t. w_raw (as in the reference, whose
 * kernels multiply by -exp(w_raw)); gu is already summed over batch (the reference returns
 * (B, C) and sums in Python, CLS/vrwkv6.py:69).  gv may be NULL: the value gradient is then left
 * out; by the symmetry of the operator it equals the forward applied to (r, k, v) := (k, r, gy).
 */
size_t vrwkv_wkv6_backward_workspace_bytes(int B, int T, int C, int H);
int vrwkv_wkv6_backward_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                            const float* w_raw, const float* u, const float* gy, float* gr, float* gk,
                            float* gv, float* gw, float* gu, void* workspace, size_t workspace_bytes,
                            void* stream);

/* The general form of the backward.  exact = 1: float32 tensors and accuracy (vrwkv_wkv6_backward_f32).  exact = 0, for
 * callers whose activations are half precision anyway: r, k, v, gy enter the matrix products as bfloat16, sums are fp32;
 * gv agrees with exact = 1 to about 1e-2 of its maximum, gr, gk, gw, gu (whose scaled operands are carried to 16 bits)
 * to about 1e-4 for bfloat16 inputs.  in_bf16: r, k, v are bfloat16 bit patterns; gy_bf16: gy is (needs in_bf16; else
 * gy is float32 and rounded on the way in); out_bf16: gr, gk, gv are written as bfloat16 (needs in_bf16).  gw, gu are
 * float32.  gv may be NULL. */
size_t vrwkv_wkv6_backward_bytes(int B, int T, int C, int H, int exact);
int vrwkv_wkv6_backward(int B, int T, int C, int H, const void* r, const void* k, const void* v, int in_bf16, int exact,
                        const float* w_raw, const float* u, const void* gy, int gy_bf16, void* gr, void* gk, void* gv, int out_bf16,
                        float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream);

/* vrwkv_wkv6_backward with exact = 0 and float32 gradients, for float32 / bfloat16 r, k, v, gy. */
size_t vrwkv_wkv6_backward_tc_workspace_bytes(int B, int T, int C, int H);
int vrwkv_wkv6_backward_tc_f32(int B, int T, int C, int H, const float* r, const float* k, const float* v,
                               const float* w_raw, const float* u, const float* gy, float* gr, float* gk, float* gv,
                               float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream);
int vrwkv_wkv6_backward_tc_bf16(int B, int T, int C, int H, const uint16_t* r, const uint16_t* k, const uint16_t* v,
                                const float* w_raw, const float* u, const uint16_t* gy, float* gr, float* gk, float* gv,
                                float* gw, float* gu, void* workspace, size_t workspace_bytes, void* stream);

/* ---- Q-Shift + token-mix interpolation (the step in front of the K/V/R projections) ----
 * x is (B, H*W, C), tokens in raster order.  xx = x with channel group g (`group` channels
 * each, group = int(C * channel_gamma)) moved by `shift` pixels: g=0 right, g=1 left, g=2 down,
 * g=3 up, zero fill at the image border, channels beyond 4*group copied.  Outputs
 * out[m] = x * mix[m] + xx * (1 - mix[m]), m < n_out (1..3), mix[m] of shape (C,).
 * `mix`, `out`, `gout`, `gmix` are host arrays of n_out device pointers.
 *
 * Replaces the tensor-op sequence q_shift(...) followed by the n_out lerps of
 *   VRWKV_SpatialMix.jit_func   CLS/vrwkv.py:156-164  (n_out = 3: xk, xv, xr)
 *   VRWKV_ChannelMix.forward    CLS/vrwkv.py:247-250  (n_out = 2: xk, xr)
 *   q_shift                     CLS/vrwkv.py:68-79
 * The backward returns gx and gmix[m] (C,), the latter summed over batch and tokens in a
 * fixed order. */
int vrwkv_qshift_mix_forward_f32(int B, int H, int W, int C, int group, int shift, int n_out,
                                 const float* x, const float* const* mix, float* const* out,
                                 void* stream);
size_t vrwkv_qshift_mix_backward_workspace_bytes(int B, int H, int W, int C, int n_out);
int vrwkv_qshift_mix_backward_f32(int B, int H, int W, int C, int group, int shift, int n_out,
                                  const float* x, const float* const* mix, const float* const* gout,
                                  float* gx, float* const* gmix, void* workspace, size_t workspace_bytes,
                                  void* stream);

/* The per-head shift of VRWKV6 (q_shift_multihead, CLS/vrwkv6.py:75-101) fused with the same
 * interpolations (VRWKV_ChannelMix of vrwkv6.py: xk, xr): within every head of head_dim channels
 * the four quarters take the left, right, upper and lower neighbour.  head_dim is a multiple of 4
 * that divides C.  Workspace of the backward: vrwkv_qshift_mix_backward_workspace_bytes. */
int vrwkv_qshift_multihead_mix_forward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out,
                                           const float* x, const float* const* mix, float* const* out,
                                           void* stream);
int vrwkv_qshift_multihead_mix_backward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out,
                                            const float* x, const float* const* mix,
                                            const float* const* gout, float* gx, float* const* gmix,
                                            void* workspace, size_t workspace_bytes, void* stream);

/* Either forward with bfloat16 outputs, what the linear layers behind it round them to under autocast (head_dim 0:
 * `group` as in vrwkv_qshift_mix_forward_f32, else the per-head form and `group` is ignored). */
int vrwkv_qshift_mix_forward_bf16out(int B, int H, int W, int C, int group, int head_dim, int shift, int n_out, const float* x,
                                     const float* const* mix, uint16_t* const* out, void* stream);

/* The per-head shift fused with the data-dependent interpolations of the VRWKV6 spatial mix
 * (CLS/vrwkv6.py:75-100, 180-193):  out_j = x + (q_shift_multihead(x) - x) * (maa_j[c] + m_j[b,t,c]),
 * j < n_out <= 5.  maa: n_out device pointers to (C,) float vectors; m: n_out device pointers to
 * (B, H*W, C) per-token offsets, float32 or (m_is_bf16 != 0) bfloat16 bit patterns, any of them NULL
 * for "no offset" (n_out = 1 with m[0] = NULL is xxx = x + xx * time_maa_x; n_out = 5 gives the inputs
 * of the w, k, v, r, g branches).  head_dim: a multiple of 16 that divides C.  The backward returns gx,
 * the offset gradients gm_j (dtype of m; NULL exactly where m_j is NULL) and the (C,) gradients gmaa_j,
 * summed in a fixed order.  All tensors 16-byte aligned (bfloat16 ones 8). */
int vrwkv_qshift_ddlerp_forward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out, const float* x,
                                    const float* const* maa, const void* const* m, int m_is_bf16, float* const* out,
                                    void* stream);
/* ... with bfloat16 outputs */
int vrwkv_qshift_ddlerp_forward_bf16out(int B, int H, int W, int C, int head_dim, int shift, int n_out, const float* x,
                                        const float* const* maa, const void* const* m, int m_is_bf16, uint16_t* const* out,
                                        void* stream);
size_t vrwkv_qshift_ddlerp_backward_workspace_bytes(int B, int H, int W, int C, int n_out);
int vrwkv_qshift_ddlerp_backward_f32(int B, int H, int W, int C, int head_dim, int shift, int n_out, const float* x,
                                     const float* const* maa, const void* const* m, int m_is_bf16,
                                     const float* const* gout, float* gx, void* const* gm, float* const* gmaa,
                                     void* workspace, size_t workspace_bytes, void* stream);

/* Inference-only steps between the matrix products of a block.  No reference counterpart as kernels: tensor-op chains there.
 *   vrwkv_sigmoid_gate: out = sigmoid(r) * y, out in the type of r (CLS/vrwkv.py:182-187, 253-257); bfloat16 y needs bfloat16 r;
 *     _f32out: the bfloat16 result widened
 *   vrwkv_relu_square: out = relu(x)^2 in the type of x (CLS/vrwkv.py:251); _f32out: of bfloat16 x in float32 (exact)
 *   vrwkv_linear_relu_square: out (rows, N) = relu(x W^T)^2 of x (rows, K) and W (N, K), the product rounded to bfloat16 first
 *     (CLS/vrwkv.py:250-251); K % 64 == 0, N % 256 == 0, else VRWKV_ERR_UNSUPPORTED; _pays: 1 where it takes less of the current
 *     device's time than a library's product and vrwkv_relu_square
 *   vrwkv_linear_batch: out_i (rows, N) = x_i W_i^T rounded to bfloat16, i < count <= 4, in one launch (the layers behind a token shift,
 *     CLS/vrwkv.py:166-168, vrwkv6.py:194-197); K % 64 == 0 and K <= 384, N % 192 == 0, N <= 1536 or K <= 1024, N % 256 == 0, else
 *     VRWKV_ERR_UNSUPPORTED; _pays: 1 where it takes less of the current device's time than a library's products
 *   vrwkv_norm_residual: out = x + gamma * (normalise(a) * weight + bias) over rows of C <= 1024 channels, C % 4 == 0;
 *     weight and bias NULL: out = x + gamma * a; gamma NULL: 1 (CLS/vrwkv.py:297-318)
 *   vrwkv_layer_norm: out = normalise(x) * weight + bias over such rows
 *   vrwkv_gated_norm_residual: the same as norm_residual with a = sigmoid(r) * y, all bfloat16
 *   vrwkv_head_norm_gate_bf16out: vrwkv_normgate_forward_f32 with group 64, the result rounded to bfloat16
 *   vrwkv_add_rows: out[i] = table[i mod period] + a[i], a bfloat16, float32 result; period a multiple of 8 that divides n
 *     (CLS/vrwkv.py:392, CLS/vrwkv6.py:200)
 *   vrwkv_widen: out = a as float32; n a multiple of 8
 *   vrwkv_narrow: out_i = src_i rounded to bfloat16, n_i values each, i < count <= 16, in one launch (which, like the casts
 *     that it stands for, vrwkv_launch_count does not count: a network's count does not depend on who casts its weights)
 *   vrwkv_patch_rows: img (B, channels, H, W) to (B, H / patch, W / patch, channels, patch, patch) in bfloat16, whole patches only;
 *     patch % 8 == 0, W % 4 == 0 (the operand of the patch embedding, CLS/vrwkv.py:357)
 * Sigmoid, its product and y are rounded to bfloat16 where r is.  All tensors 16-byte aligned. */
int vrwkv_sigmoid_gate(long long n, const void* r, int r_is_bf16, const void* y, int y_is_bf16, void* out, void* stream);
int vrwkv_sigmoid_gate_f32out(long long n, const uint16_t* r, const uint16_t* y, float* out, void* stream);
int vrwkv_relu_square(long long n, const void* x, int is_bf16, void* out, void* stream);
int vrwkv_relu_square_f32out(long long n, const uint16_t* x, float* out, void* stream);
int vrwkv_linear_relu_square_pays(long long rows, int K, int N);
int vrwkv_linear_relu_square(long long rows, int K, int N, const uint16_t* x, const uint16_t* w, uint16_t* out, void* stream);
int vrwkv_linear_batch_pays(int count, long long rows, int K, int N);
int vrwkv_linear_batch(int count, long long rows, int K, int N, const uint16_t* const* x, const uint16_t* const* w, uint16_t* const* out, void* stream);
int vrwkv_add_rows(long long n, long long period, const float* table, const uint16_t* a, float* out, void* stream);
int vrwkv_narrow(int count, const float* const* src, const long long* n, uint16_t* const* out, void* stream);
int vrwkv_widen(long long n, const uint16_t* a, float* out, void* stream);
int vrwkv_patch_rows(int B, int channels, int H, int W, int patch, const float* img, uint16_t* out, void* stream);
int vrwkv_layer_norm(int rows, int C, float eps, const float* x, const float* weight, const float* bias, float* out, void* stream);
int vrwkv_norm_residual(int rows, int C, float eps, const void* a, int a_is_bf16, const float* weight, const float* bias,
                        const float* gamma, const float* x, float* out, void* stream);
int vrwkv_gated_norm_residual(int rows, int C, float eps, const uint16_t* r, const uint16_t* y, const float* weight, const float* bias,
                              const float* gamma, const float* x, float* out, void* stream);
int vrwkv_head_norm_gate_bf16out(int rows, int C, float eps, const float* x, const void* gate, int gate_is_bf16, int gate_act,
                                 const float* gamma, const float* beta, uint16_t* out, void* stream);

/* Normalise-and-gate epilogue behind the two operators, one pass forward and one backward:
 *   out = (normalise(x) * gamma + beta) * gate
 * over rows of C channels; group == C is the LayerNorm + sigmoid gate behind Bi-WKV in the large
 * backbone (key_norm, then sr * x: CLS/vrwkv.py:184-186), group == 64 the per-head GroupNorm + SiLU
 * gate behind WKV6 (ln_x, then x * g: CLS/vrwkv6.py:133, 205-212).  The reference runs them as a
 * normalisation pass and a multiply pass (and an activation pass before them).  `gate` holds, float32 or
 * (gate_is_bf16 != 0) bfloat16 bit patterns, the gate itself (gate_act 0), or the projection whose sigmoid
 * (gate_act 1) or SiLU (gate_act 2) is the gate - the backward then returns the gradient of that projection; x, out, gamma, beta float32; mean and rstd receive
 * rows * C / group floats each for the backward.  group must be a multiple of 64, at most 1024, and
 * divide C (else VRWKV_ERR_UNSUPPORTED); pointers 8-byte aligned.  Biased variance, eps inside the
 * square root, as torch.nn.LayerNorm / GroupNorm.  The backward returns gx, ggate (dtype of gate) and
 * ggamma | gbeta as one (2, C) float buffer, summed in a fixed order. */
int vrwkv_normgate_forward_f32(int rows, int C, int group, float eps, const float* x, const void* gate,
                               int gate_is_bf16, int gate_act, const float* gamma, const float* beta, float* out,
                               float* mean, float* rstd, void* stream);
size_t vrwkv_normgate_backward_workspace_bytes(int rows, int C, int group);
int vrwkv_normgate_backward_f32(int rows, int C, int group, const float* gout, const float* x, const void* gate,
                                int gate_is_bf16, int gate_act, const float* gamma, const float* beta, const float* mean,
                                const float* rstd, float* gx, void* ggate, float* ggamma_gbeta, void* workspace,
                                size_t workspace_bytes, void* stream);

#ifdef __cplusplus
}
#endif
#endif /* VRWKV_B200_H_ */
