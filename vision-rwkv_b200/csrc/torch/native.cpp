// Host path of the operators as a torch extension: the checks, allocations, dtype rules and autograd
// nodes that sit between a model's call and the C ABI, in C++.
//
// A call on a small input is all host time: through ctypes and a Python autograd Function a forward took
// 65 us of which the GPU worked 11.  The rules are those of the reference's Python wrappers
// (classification/mmcls_custom/models/backbones/vrwkv.py:29-65, vrwkv6.py:22-73); the Python modules
// above this file keep the public names.
#include <torch/csrc/utils/pybind.h>
#include "glue.h"
#include "native.h"

namespace vrwkv {

namespace {
PyObject* g_error_class = nullptr;     // vision_rwkv_b200._lib.VrwkvError
}

void raise(const std::string& text) {
    pybind11::gil_scoped_acquire gil;
    PyErr_SetString(g_error_class ? g_error_class : PyExc_RuntimeError, text.c_str());
    python_error e;
    e.persist();
    throw e;
}

void raise_status(int status, const char* what) {
    std::string text = std::string(what) + " failed with status " + std::to_string(status) + ": " + vrwkv_status_string(status);
    const char* detail = vrwkv_last_error_detail();
    if (detail && *detail) text += std::string(" [") + detail + "]";
    raise(text);
}

void raise_failures(int device, const char* what) {
    const unsigned bits = vrwkv_take_failures(device);
    if (bits == 0) return;
    static const char* const kNames[] = {"Bi-WKV forward", "Bi-WKV backward", "WKV6 forward", "WKV6 backward", "linear"};
    std::string names;
    for (int i = 0; i < 5; ++i)
        if (bits >> (8 + i) & 1u) names += (names.empty() ? "" : ", ") + std::string(kNames[i]);
    char word[16];
    snprintf(word, sizeof(word), "%#x", bits & 0xffu);
    raise(std::string("device status word ") + word + ", seen at " + what + " (a bounded device-side wait ran out in an earlier launch, " +
          names + ": its outputs, and everything computed from them, are invalid)");
}

namespace {

void check_cuda(const Tensor& t, const char* name, const Tensor& like) {
    TORCH_CHECK(t.is_cuda(), name, " must be a CUDA tensor");
    TORCH_CHECK(t.device() == like.device(), name, " is on ", t.device(), ", expected ", like.device());
}

// ---- Bi-WKV ------------------------------------------------------------------------------------
void check_biwkv(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
    check_cuda(k, "k", k);
    check_cuda(v, "v", k);
    check_cuda(w, "w", k);
    check_cuda(u, "u", k);
    TORCH_CHECK(k.dim() == 3, "k must be (B, T, C), got ", k.sizes());
    TORCH_CHECK(v.sizes() == k.sizes(), "k, v (and gy) must have the same shape");
    TORCH_CHECK(w.numel() == k.size(2) && u.numel() == k.size(2), "w and u must hold C=", k.size(2), " values");
}

at::ScalarType result_dtype(const Tensor& w) {
    return w.scalar_type() == at::kHalf || w.scalar_type() == at::kBFloat16 ? w.scalar_type() : at::kFloat;
}

// The forward that keeps states for the backward, into `kept`; false (and an undefined `kept`) where it does not serve the call.
bool biwkv_forward_keep(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, const Tensor& y, Tensor* kept) {
    const int B = k.size(0), T = k.size(1), C = k.size(2);
    const int types = is_bf16(k) ? VRWKV_TENSORS_BF16 : VRWKV_TENSORS_F32;
    const size_t bytes = vrwkv_biwkv_kept_bytes(B, T, C);
    if (bytes == 0 || vrwkv_biwkv_one_pass(B, T, C, types)) return false;
    *kept = workspace(bytes, k);
    const Tensor ws = workspace(vrwkv_biwkv_kept_workspace_bytes(B, T, C, 0), k);
    const int st = vrwkv_biwkv_forward_keep(B, T, C, fp(w), fp(u), k.data_ptr(), v.data_ptr(), y.data_ptr(),
                                            types, kept->data_ptr(), kept->numel(), ws.data_ptr(),
                                            ws.numel(), stream_of(k));
    if (st != VRWKV_OK) kept->reset();
    if (st == VRWKV_ERR_UNSUPPORTED) return false;
    check(st, "vrwkv_biwkv_forward_keep");
    return true;
}

// A Bi-WKV entry point with the scratch memory it needs: little where the one-pass kernels serve the sizes, all of it where they cannot
// be had for these tensors after all.  call(workspace) returns a status; the last one is the result.
template <typename F>
int with_scratch(const Tensor& k, int types, bool backward, F&& call) {
    const int B = k.size(0), T = k.size(1), C = k.size(2);
    const size_t bytes = vrwkv_biwkv_one_pass_workspace_bytes(B, T, C, types, backward);
    if (bytes != 0) {
        const int st = call(workspace(bytes, k));
        if (st != VRWKV_ERR_WORKSPACE) return st;
    }
    return call(workspace(backward ? vrwkv_biwkv_backward_workspace_bytes(B, T, C) : vrwkv_biwkv_forward_workspace_bytes(B, T, C), k));
}

// k, v float32 or both bfloat16, contiguous; y in their dtype.  kept: null, or receives the states for a backward (left
// undefined where none are kept).
Tensor biwkv_forward_raw(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, Tensor* kept = nullptr) {
    const int B = k.size(0), T = k.size(1), C = k.size(2);
    Tensor y = at::empty_like(k);
    if (k.numel() == 0) return y;
    if (kept && biwkv_forward_keep(w, u, k, v, y, kept)) {
        raise_failures(k.get_device(), "vrwkv_biwkv_forward");
        return y;
    }
    if (is_bf16(k)) {
        const int st = with_scratch(k, VRWKV_TENSORS_BF16, false, [&](const Tensor& ws) {
            return vrwkv_biwkv_forward_bf16(B, T, C, fp(w), fp(u), static_cast<uint16_t*>(k.data_ptr()), static_cast<uint16_t*>(v.data_ptr()),
                                            static_cast<uint16_t*>(y.data_ptr()), ws.data_ptr(), ws.numel(), stream_of(k));
        });
        if (st == VRWKV_ERR_UNSUPPORTED) return biwkv_forward_raw(w, u, f32(k), f32(v)).to(at::kBFloat16);
        check(st, "vrwkv_biwkv_forward_bf16");
    } else {
        check(with_scratch(k, VRWKV_TENSORS_F32, false, [&](const Tensor& ws) {
                  return vrwkv_biwkv_forward_f32(B, T, C, fp(w), fp(u), fp(k), fp(v), fp(y), ws.data_ptr(), ws.numel(), stream_of(k));
              }), "vrwkv_biwkv_forward_f32");
    }
    raise_failures(k.get_device(), "vrwkv_biwkv_forward");
    return y;
}

// whether the entry points with float32 y, gy beside bfloat16 k, v are for calls of this size
bool wide_serves(const Tensor& k) { return vrwkv_biwkv_one_pass(k.size(0), k.size(1), k.size(2), VRWKV_TENSORS_BF16_WIDE) != 0; }

// k, v bfloat16, contiguous; y float32 holding bfloat16 values.  Undefined where the kernel does not cover the call.
Tensor biwkv_forward_wide(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
    if (k.numel() != 0 && !wide_serves(k)) return Tensor();
    const int B = k.size(0), T = k.size(1), C = k.size(2);
    Tensor y = at::empty_like(k, k.options().dtype(at::kFloat));
    if (k.numel() == 0) return y;
    const int st = with_scratch(k, VRWKV_TENSORS_BF16_WIDE, false, [&](const Tensor& ws) {
        return vrwkv_biwkv_forward_bf16_wide(B, T, C, fp(w), fp(u), static_cast<uint16_t*>(k.data_ptr()), static_cast<uint16_t*>(v.data_ptr()), fp(y),
                                             ws.data_ptr(), ws.numel(), stream_of(k));
    });
    if (st == VRWKV_ERR_UNSUPPORTED) return Tensor();
    check(st, "vrwkv_biwkv_forward_bf16_wide");
    raise_failures(k.get_device(), "vrwkv_biwkv_forward");
    return y;
}

Tensor biwkv_forward(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, bool bf16_io, Tensor* kept = nullptr) {
    const c10::cuda::CUDAGuard guard(k.device());
    const bool half = bf16_io && is_bf16(k) && is_bf16(v);
    if (half && result_dtype(w) == at::kFloat) {
        // float32 w, u under autocast: the kernel writes the widened result itself
        const Tensor y = biwkv_forward_wide(f32(w), f32(u), k.contiguous(), v.contiguous());
        if (y.defined()) return y;
    }
    const Tensor y = half ? biwkv_forward_raw(f32(w), f32(u), k.contiguous(), v.contiguous(), kept)
                          : biwkv_forward_raw(f32(w), f32(u), f32(k), f32(v), kept);
    return y.to(result_dtype(w));
}

// What a saved-tensor hook hands back for the kept states need not be what the forward left: the states are taken where it is still
// a buffer of bytes of that size on this device, copied if it starts off the kernels' boundary, and rebuilt (undefined) otherwise.
Tensor usable_states(const Tensor& kept, const Tensor& k) {
    if (!kept.defined() || kept.scalar_type() != at::kByte || kept.device() != k.device() || kept.layout() != at::kStrided || kept.dim() != 1 ||
        static_cast<size_t>(kept.numel()) != vrwkv_biwkv_kept_bytes(k.size(0), k.size(1), k.size(2)))
        return Tensor();
    const bool placed = kept.is_contiguous() && (reinterpret_cast<uintptr_t>(kept.data_ptr()) & 255u) == 0;
    return placed ? kept : at::empty_like(kept, at::MemoryFormat::Contiguous).copy_(kept);
}

// k, v float32, or bfloat16 (then gy in either type); all contiguous.  kept: what the forward left, or undefined.
std::array<Tensor, 4> biwkv_backward_raw(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, const Tensor& gy,
                                         const Tensor& kept = Tensor()) {
    // no kernels for a float32 gy: narrowed before anything is allocated
    if (k.numel() != 0 && is_bf16(k) && !is_bf16(gy) && !wide_serves(k)) return biwkv_backward_raw(w, u, k, v, gy.to(at::kBFloat16), kept);
    const int B = k.size(0), T = k.size(1), C = k.size(2);
    Tensor gk = at::empty_like(k), gv = at::empty_like(k);
    Tensor gwgu = at::empty({2, C}, k.options().dtype(at::kFloat));
    if (k.numel() == 0) {
        gwgu.zero_();
        return {gwgu.select(0, 0), gwgu.select(0, 1), gk, gv};
    }
    int resumed = VRWKV_ERR_UNSUPPORTED;
    if (kept.defined()) {
        const Tensor ws = workspace(vrwkv_biwkv_kept_workspace_bytes(B, T, C, 1), k);
        resumed = vrwkv_biwkv_backward_kept(B, T, C, fp(w), fp(u), k.data_ptr(), v.data_ptr(), gy.data_ptr(), fp(gwgu), gk.data_ptr(),
                                            gv.data_ptr(), is_bf16(k) ? VRWKV_TENSORS_BF16 : VRWKV_TENSORS_F32, kept.data_ptr(), kept.numel(), ws.data_ptr(), ws.numel(), stream_of(k));
        if (resumed != VRWKV_ERR_UNSUPPORTED) check(resumed, "vrwkv_biwkv_backward_kept");
    }
    const auto half = [](const Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()); };
    if (resumed == VRWKV_OK) {
        // done
    } else if (is_bf16(k) && !is_bf16(gy)) {
        const int st = with_scratch(k, VRWKV_TENSORS_BF16_WIDE, true, [&](const Tensor& ws) {
            return vrwkv_biwkv_backward_bf16_wide(B, T, C, fp(w), fp(u), half(k), half(v), fp(gy), fp(gwgu), half(gk), half(gv), ws.data_ptr(), ws.numel(), stream_of(k));
        });
        if (st == VRWKV_ERR_UNSUPPORTED) return biwkv_backward_raw(w, u, k, v, gy.to(at::kBFloat16));
        check(st, "vrwkv_biwkv_backward_bf16_wide");
    } else if (is_bf16(k)) {
        const int st = with_scratch(k, VRWKV_TENSORS_BF16, true, [&](const Tensor& ws) {
            return vrwkv_biwkv_backward_bf16(B, T, C, fp(w), fp(u), half(k), half(v), half(gy), fp(gwgu), half(gk), half(gv), ws.data_ptr(), ws.numel(), stream_of(k));
        });
        if (st == VRWKV_ERR_UNSUPPORTED) {
            auto g = biwkv_backward_raw(w, u, f32(k), f32(v), f32(gy));
            return {g[0], g[1], g[2].to(at::kBFloat16), g[3].to(at::kBFloat16)};
        }
        check(st, "vrwkv_biwkv_backward_bf16");
    } else {
        check(with_scratch(k, VRWKV_TENSORS_F32, true, [&](const Tensor& ws) {
                  return vrwkv_biwkv_backward_f32(B, T, C, fp(w), fp(u), fp(k), fp(v), fp(gy), fp(gwgu), fp(gk), fp(gv), ws.data_ptr(), ws.numel(), stream_of(k));
              }), "vrwkv_biwkv_backward_f32");
    }
    raise_failures(k.get_device(), "vrwkv_biwkv_backward");
    return {gwgu.select(0, 0), gwgu.select(0, 1), gk, gv};
}

struct BiWkv : torch::autograd::Function<BiWkv> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& w, const Tensor& u, const Tensor& k,
                          const Tensor& v, bool bf16_io) {
        Tensor kept;
        Tensor y = biwkv_forward(w, u, k, v, bf16_io, &kept);
        ctx->save_for_backward({w, u, k, v, kept});
        ctx->saved_data["bf16_io"] = bf16_io;
        return y;
    }
    static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &w = saved[0], &u = saved[1], &k = saved[2], &v = saved[3], &gy = grads[0];
        const c10::cuda::CUDAGuard guard(k.device());
        const at::NoGradGuard no_grad;
        const Tensor kept = usable_states(saved[4], k);
        const at::ScalarType out = result_dtype(w);
        const bool half = ctx->saved_data["bf16_io"].toBool() && is_bf16(k) && is_bf16(v);
        auto g = half ? biwkv_backward_raw(f32(w), f32(u), k.contiguous(), v.contiguous(), is_bf16(gy) ? gy.contiguous() : f32(gy), kept)
                      : biwkv_backward_raw(f32(w), f32(u), f32(k), f32(v), f32(gy), kept);
        // on the bfloat16 path gk, gv stay bfloat16 (what autograd hands to a bfloat16 k anyway) unless w is half
        if (!half || out == at::kHalf) { g[2] = g[2].to(out); g[3] = g[3].to(out); }
        return {g[0].to(out), g[1].to(out), g[2], g[3], Tensor()};
    }
};

// bfloat16 k, v to a bfloat16 y whatever the dtype of w: the values that biwkv widens where w is float32
Tensor biwkv_half(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
    check_biwkv(w, u, k, v);
    TORCH_CHECK(is_bf16(k) && is_bf16(v), "k, v must be bfloat16");
    refuse_tangents({&w, &u, &k, &v});
    const c10::cuda::CUDAGuard guard(k.device());
    return biwkv_forward_raw(f32(w), f32(u), k.contiguous(), v.contiguous());
}

Tensor biwkv(const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, bool bf16_io) {
    check_biwkv(w, u, k, v);
    if (!any_requires_grad({&w, &u, &k, &v})) return biwkv_forward(w, u, k, v, bf16_io);
    return BiWkv::apply(w, u, k, v, bf16_io);
}

// ---- WKV6 --------------------------------------------------------------------------------------
bool all_bf16(std::initializer_list<const Tensor*> ts) {
    for (const Tensor* t : ts)
        if (!is_bf16(*t)) return false;
    return true;
}

void check_wkv6(int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
                const Tensor& u) {
    check_cuda(r, "r", r);
    check_cuda(k, "k", r);
    check_cuda(v, "v", r);
    check_cuda(w, "w", r);
    check_cuda(u, "u", r);
    TORCH_CHECK(r.dim() == 3 && r.size(0) == B && r.size(1) == T && r.size(2) == C, "r has shape ", r.sizes(), ", expected (", B, ", ",
                T, ", ", C, ")");
    TORCH_CHECK(k.sizes() == r.sizes(), "k must have the shape of r");
    TORCH_CHECK(v.sizes() == r.sizes(), "v must have the shape of r");
    TORCH_CHECK(w.sizes() == r.sizes(), "w must have the shape of r");
    TORCH_CHECK(C == 64 * H, "head size must be 64: C=", C, ", H=", H);
    TORCH_CHECK(u.numel() == C, "u must hold C=", C, " values");
}

Tensor wkv6_forward(int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w_, const Tensor& u_,
                    bool tensor_cores) {
    const c10::cuda::CUDAGuard guard(r.device());
    const int B = r.size(0), T = r.size(1), C = r.size(2);
    const Tensor w = f32(w_), u = f32(u_);
    Tensor y = at::empty({B, T, C}, r.options().dtype(at::kFloat));
    if (y.numel() == 0) return y;
    const bool half = tensor_cores && all_bf16({&r, &k, &v});
    const Tensor r_ = half ? r.contiguous() : f32(r), k_ = half ? k.contiguous() : f32(k), v_ = half ? v.contiguous() : f32(v);
    Tensor ws = workspace(vrwkv_wkv6_forward_workspace_bytes(B, T, C, H, !tensor_cores), r);
    check(vrwkv_wkv6_forward(B, T, C, H, r_.data_ptr(), k_.data_ptr(), v_.data_ptr(), half, !tensor_cores, fp(w), fp(u), fp(y), ws.data_ptr(),
                             ws.numel(), stream_of(r)),
          "vrwkv_wkv6_forward");
    raise_failures(r.get_device(), "vrwkv_wkv6_forward");
    return y;
}

// The walk in 16-token blocks (vrwkv_wkv6_forward_tc_bf16 without scratch memory): slower than wkv6_forward, other roundings.
Tensor wkv6_walk(const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w_, const Tensor& u_) {
    const int B = r.size(0), T = r.size(1), C = r.size(2), H = C / 64;
    check_wkv6(B, T, C, H, r, k, v, w_, u_);
    TORCH_CHECK(all_bf16({&r, &k, &v}), "r, k, v must be bfloat16");
    refuse_tangents({&r, &k, &v, &w_, &u_});
    const c10::cuda::CUDAGuard guard(r.device());
    const Tensor w = f32(w_), u = f32(u_), r_ = r.contiguous(), k_ = k.contiguous(), v_ = v.contiguous();
    Tensor y = at::empty({B, T, C}, r.options().dtype(at::kFloat));
    if (y.numel() == 0) return y;
    Tensor ws = workspace(256, r);
    check(vrwkv_wkv6_forward_tc_bf16(B, T, C, H, static_cast<uint16_t*>(r_.data_ptr()), static_cast<uint16_t*>(k_.data_ptr()),
                                     static_cast<uint16_t*>(v_.data_ptr()), fp(w), fp(u), fp(y), ws.data_ptr(), 256, stream_of(r)),
          "vrwkv_wkv6_forward_tc_bf16");
    raise_failures(r.get_device(), "vrwkv_wkv6_forward_tc_bf16");
    return y;
}

struct Wkv6 : torch::autograd::Function<Wkv6> {
    static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
                          const Tensor& u, int64_t H, bool tensor_cores) {
        Tensor y = wkv6_forward(H, r, k, v, w, u, tensor_cores);
        ctx->save_for_backward({r, k, v, w, u});
        ctx->saved_data["H"] = H;
        ctx->saved_data["tc"] = tensor_cores;
        return y;
    }
    static torch::autograd::tensor_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::tensor_list grads) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &r = saved[0], &k = saved[1], &v = saved[2], &gy = grads[0];
        const c10::cuda::CUDAGuard guard(r.device());
        const at::NoGradGuard no_grad;
        const int64_t H = ctx->saved_data["H"].toInt();
        const int B = r.size(0), T = r.size(1), C = r.size(2);
        const Tensor w = f32(saved[3]), u = f32(saved[4]);
        const auto opt = r.options().dtype(at::kFloat);
        const bool exact = !ctx->saved_data["tc"].toBool(), half = !exact && all_bf16({&r, &k, &v});
        // bfloat16 r, k, v take their gradients in bfloat16 (what autograd would round them to); gy is read as it comes
        const auto out = half ? r.options() : opt;
        Tensor gr = at::empty({B, T, C}, out), gk = at::empty({B, T, C}, out), gv = at::empty({B, T, C}, out),
               gw = at::empty({B, T, C}, opt), gu = at::empty({H, C / H}, opt);
        if (gr.numel() == 0) {
            gu.zero_();
        } else {
            const Tensor r_ = half ? r.contiguous() : f32(r), k_ = half ? k.contiguous() : f32(k), v_ = half ? v.contiguous() : f32(v);
            const Tensor g = half && is_bf16(gy) ? gy.contiguous() : f32(gy);
            Tensor ws = workspace(vrwkv_wkv6_backward_bytes(B, T, C, H, exact), r);
            check(vrwkv_wkv6_backward(B, T, C, H, r_.data_ptr(), k_.data_ptr(), v_.data_ptr(), half, exact, fp(w), fp(u), g.data_ptr(),
                                      is_bf16(g), gr.data_ptr(), gk.data_ptr(), gv.data_ptr(), half, fp(gw), fp(gu), ws.data_ptr(),
                                      ws.numel(), stream_of(r)),
                  "vrwkv_wkv6_backward");
            raise_failures(r.get_device(), "vrwkv_wkv6_backward");
        }
        return {gr, gk, gv, gw, gu.view({H, C / H}), Tensor(), Tensor()};
    }
};

Tensor wkv6(int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
            const Tensor& u, bool tensor_cores) {
    check_wkv6(B, T, C, H, r, k, v, w, u);
    if (!any_requires_grad({&r, &k, &v, &w, &u})) return wkv6_forward(H, r, k, v, w, u, tensor_cores);
    return Wkv6::apply(r, k, v, w, u, H, tensor_cores);
}

// python_error carries its exception through C++; hand it back to the interpreter at the boundary
template <typename F>
auto guarded(F f) {
    return [f](auto... args) {
        try {
            pybind11::gil_scoped_release release;
            return f(args...);
        } catch (python_error& e) {
            e.restore();
            throw pybind11::error_already_set();
        }
    };
}

}  // namespace
}  // namespace vrwkv

PYBIND11_MODULE(_native, m) {
    using at::Tensor;
    m.def("set_error_class", [](pybind11::object cls) { vrwkv::g_error_class = cls.release().ptr(); });
    m.def("biwkv", [](const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v, bool bf16_io) {
        return vrwkv::guarded([&] { return vrwkv::biwkv(w, u, k, v, bf16_io); })();
    });
    m.def("qshift_mix", [](const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group, bool per_head) {
        return vrwkv::guarded([&] { return vrwkv::qshift_mix(x, mixes, H, W, shift, group, per_head); })();
    });
    m.def("qshift_ddlerp", [](const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H, int64_t W,
                              int64_t shift, int64_t head_dim) {
        return vrwkv::guarded([&] { return vrwkv::qshift_ddlerp(x, maas, offsets, H, W, shift, head_dim); })();
    });
    m.def("biwkv_half", [](const Tensor& w, const Tensor& u, const Tensor& k, const Tensor& v) {
        return vrwkv::guarded([&] { return vrwkv::biwkv_half(w, u, k, v); })();
    });
    m.def("sigmoid_gate", [](const Tensor& r, const Tensor& y, bool wide) { return vrwkv::guarded([&] { return vrwkv::sigmoid_gate(r, y, wide); })(); });
    m.def("relu_square", [](const Tensor& x, bool wide) { return vrwkv::guarded([&] { return vrwkv::relu_square(x, wide); })(); });
    m.def("linear_relu_square", [](const Tensor& x, const Tensor& weight) { return vrwkv::guarded([&] { return vrwkv::linear_relu_square(x, weight); })(); });
    m.def("key_layer", [](const Tensor& x, const Tensor& weight) { return vrwkv::guarded([&] { return vrwkv::key_layer(x, weight); })(); });
    m.def("autocast_copy", [](const Tensor& t) { return vrwkv::guarded([&] { return vrwkv::autocast_copy(t); })(); });
    m.def("narrow", [](std::vector<Tensor> weights) { return vrwkv::guarded([&] { return vrwkv::narrow(weights); })(); });
    m.def("linear_batch", [](std::vector<Tensor> xs, std::vector<Tensor> weights) { return vrwkv::guarded([&] { return vrwkv::linear_batch(xs, weights); })(); });
    m.def("add_rows", [](const Tensor& table, const Tensor& a) { return vrwkv::guarded([&] { return vrwkv::add_rows(table, a); })(); });
    m.def("patch_rows", [](const Tensor& img, int64_t patch) { return vrwkv::guarded([&] { return vrwkv::patch_rows(img, patch); })(); });
    m.def("widen", [](const Tensor& a) { return vrwkv::guarded([&] { return vrwkv::widen(a); })(); });
    m.def("layer_norm", [](const Tensor& x, const Tensor& weight, const Tensor& bias, double eps) {
        return vrwkv::guarded([&] { return vrwkv::layer_norm(x, weight, bias, eps); })();
    });
    m.def("norm_residual", [](const Tensor& x, const Tensor& a, std::optional<Tensor> weight, std::optional<Tensor> bias,
                              std::optional<Tensor> gamma, double eps) {
        return vrwkv::guarded([&] { return vrwkv::norm_residual(x, a, weight, bias, gamma, eps); })();
    });
    m.def("gated_norm_residual", [](const Tensor& x, const Tensor& r, const Tensor& y, std::optional<Tensor> weight, std::optional<Tensor> bias,
                                    std::optional<Tensor> gamma, double eps) {
        return vrwkv::guarded([&] { return vrwkv::gated_norm_residual(x, r, y, weight, bias, gamma, eps); })();
    });
    m.def("head_norm_gate_half", [](const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, double eps, int64_t act) {
        return vrwkv::guarded([&] { return vrwkv::head_norm_gate_half(x, gate, weight, bias, eps, act); })();
    });
    m.def("qshift_mix_half", [](const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group, bool per_head) {
        return vrwkv::guarded([&] { return vrwkv::qshift_mix_half(x, mixes, H, W, shift, group, per_head); })();
    });
    m.def("qshift_ddlerp_half", [](const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H, int64_t W,
                                   int64_t shift, int64_t head_dim) {
        return vrwkv::guarded([&] { return vrwkv::qshift_ddlerp_half(x, maas, offsets, H, W, shift, head_dim); })();
    });
    m.def("norm_gate", [](const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, int64_t group, double eps, int64_t act) {
        return vrwkv::guarded([&] { return vrwkv::norm_gate(x, gate, weight, bias, group, eps, act); })();
    });
    m.def("wkv6_walk", [](const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w, const Tensor& u) {
        return vrwkv::guarded([&] { return vrwkv::wkv6_walk(r, k, v, w, u); })();
    });
    m.def("wkv6", [](int64_t B, int64_t T, int64_t C, int64_t H, const Tensor& r, const Tensor& k, const Tensor& v, const Tensor& w,
                     const Tensor& u, bool tensor_cores) {
        return vrwkv::guarded([&] { return vrwkv::wkv6(B, T, C, H, r, k, v, w, u, tensor_cores); })();
    });
}
