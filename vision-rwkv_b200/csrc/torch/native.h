// Shared by the translation units of the torch extension: argument checks, error reporting, workspaces.
#pragma once
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/Exceptions.h>
#include "vrwkv_b200.h"

namespace vrwkv {

using at::Tensor;

// Raises the package's VrwkvError (from a thread that may or may not hold the interpreter lock).
[[noreturn]] void raise(const std::string& text);
[[noreturn]] void raise_status(int status, const char* what);

inline void check(int status, const char* what) {
    if (status != VRWKV_OK) raise_status(status, what);
}
// A bounded device-side wait that ran out in an earlier launch surfaces here: one read of a host word.
void raise_failures(int device, const char* what);

inline void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }
inline Tensor workspace(size_t bytes, const Tensor& like) {
    return at::empty({static_cast<int64_t>(bytes < 16 ? 16 : bytes)}, like.options().dtype(at::kByte));
}
inline Tensor f32(const Tensor& t) { return t.scalar_type() == at::kFloat ? t.contiguous() : t.to(at::kFloat).contiguous(); }
inline float* fp(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }
inline bool is_bf16(const Tensor& t) { return t.scalar_type() == at::kBFloat16; }
// Forward-mode tangents: the autograd nodes refuse them, and a call that does without a node must not drop them.
inline bool has_tangent(const Tensor& t) { return t._fw_grad(/*level=*/0).defined(); }
inline void refuse_tangents(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts) TORCH_CHECK_NOT_IMPLEMENTED(!has_tangent(*t), "forward-mode differentiation is not implemented for this operator");
}
inline void refuse_tangents(const std::vector<Tensor>& ts) {
    for (const Tensor& t : ts) refuse_tangents({&t});
}
// whether the call needs its autograd node
inline bool any_requires_grad(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (has_tangent(*t)) return true;
    if (!at::GradMode::is_enabled()) return false;
    for (const Tensor* t : ts)
        if (t->requires_grad()) return true;
    return false;
}

}  // namespace vrwkv
