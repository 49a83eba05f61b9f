// Host path of the inference-only steps between a block's matrix products (csrc/mixer_epilogue.cu).  The rules that decide
// whether a call may come here are epilogue.py's.
#include <ATen/autocast_mode.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include "glue.h"

namespace vrwkv {

namespace {
// contiguous and 16-byte aligned (a view may start anywhere)
Tensor flat(const Tensor& t) {
    const Tensor c = t.contiguous();
    return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15u) ? c.clone() : c;
}
void same_place(const Tensor& t, const Tensor& like, const char* name) {
    TORCH_CHECK(t.is_cuda() && t.device() == like.device(), name, " must be on ", like.device());
    refuse_tangents({&t, &like});
}
}  // namespace

Tensor sigmoid_gate(const Tensor& r_, const Tensor& y_, bool wide) {
    same_place(y_, r_, "y");
    TORCH_CHECK(r_.sizes() == y_.sizes(), "r and y must have the same shape");
    const c10::cuda::CUDAGuard guard(r_.device());
    const Tensor r = flat(r_), y = flat(y_);
    TORCH_CHECK(!wide || (is_bf16(r) && is_bf16(y)), "only bfloat16 is widened");
    Tensor out = at::empty(r.sizes(), wide ? r.options().dtype(at::kFloat) : r.options());
    if (r.numel() == 0) return out;
    if (wide)
        check(vrwkv_sigmoid_gate_f32out(r.numel(), static_cast<uint16_t*>(r.data_ptr()), static_cast<uint16_t*>(y.data_ptr()), fp(out), stream_of(r)),
              "vrwkv_sigmoid_gate_f32out");
    else
        check(vrwkv_sigmoid_gate(r.numel(), r.data_ptr(), is_bf16(r), y.data_ptr(), is_bf16(y), out.data_ptr(), stream_of(r)), "vrwkv_sigmoid_gate");
    return out;
}

Tensor relu_square(const Tensor& x_, bool wide) {
    same_place(x_, x_, "x");
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = flat(x_);
    TORCH_CHECK(!wide || is_bf16(x), "only bfloat16 is widened");
    Tensor out = at::empty(x.sizes(), wide ? x.options().dtype(at::kFloat) : x.options());
    if (x.numel() == 0) return out;
    if (wide) check(vrwkv_relu_square_f32out(x.numel(), static_cast<uint16_t*>(x.data_ptr()), fp(out), stream_of(x)), "vrwkv_relu_square_f32out");
    else check(vrwkv_relu_square(x.numel(), x.data_ptr(), is_bf16(x), out.data_ptr(), stream_of(x)), "vrwkv_relu_square");
    return out;
}

Tensor linear_relu_square(const Tensor& x_, const Tensor& weight_) {
    same_place(x_, weight_, "x");
    const c10::cuda::CUDAGuard guard(x_.device());
    TORCH_CHECK(is_bf16(x_) && weight_.dim() == 2 && x_.dim() >= 1 && x_.size(-1) == weight_.size(1), "x must be bfloat16 rows of the weight's width");
    const Tensor x = flat(x_), weight = flat(at::autocast::cached_cast(at::kBFloat16, weight_, at::kCUDA));      // autocast's own cast, and its cache
    auto sizes = x.sizes().vec();
    sizes.back() = weight.size(0);
    Tensor out = at::empty(sizes, x.options());
    if (x.numel() == 0) return out;
    const auto p = [](const Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()); };
    check(vrwkv_linear_relu_square(x.numel() / x.size(-1), weight.size(1), weight.size(0), p(x), p(weight), p(out), stream_of(x)), "vrwkv_linear_relu_square");
    raise_failures(x.get_device(), "vrwkv_linear_relu_square");
    return out;
}

std::vector<Tensor> linear_batch(std::vector<Tensor> xs, std::vector<Tensor> weights) {
    TORCH_CHECK(!xs.empty() && xs.size() <= 4 && xs.size() == weights.size(), "one to four layers");
    const c10::cuda::CUDAGuard guard(xs[0].device());
    const int64_t depth = xs[0].dim() >= 1 ? xs[0].size(-1) : 0, rows = depth ? xs[0].numel() / depth : 0;
    std::vector<Tensor> outs;
    if (weights[0].dim() != 2 || !vrwkv_linear_batch_pays(xs.size(), rows, depth, weights[0].size(0))) {
        for (size_t i = 0; i < xs.size(); ++i) outs.push_back(at::linear(xs[i], weights[i]));
        return outs;
    }
    const uint16_t *x[4], *w[4];
    uint16_t* out[4];
    const auto p = [](const Tensor& t) { return static_cast<uint16_t*>(t.data_ptr()); };
    for (size_t i = 0; i < xs.size(); ++i) {
        same_place(xs[i], xs[0], "x");
        same_place(weights[i], xs[0], "weight");
        TORCH_CHECK(is_bf16(xs[i]) && xs[i].sizes() == xs[0].sizes() && weights[i].sizes() == weights[0].sizes() && weights[0].size(1) == depth,
                    "the layers must be of one shape, on bfloat16 rows of their weights' width");
        xs[i] = flat(xs[i]);
        weights[i] = flat(at::autocast::cached_cast(at::kBFloat16, weights[i], at::kCUDA));      // autocast's own cast, and its cache
        auto sizes = xs[i].sizes().vec();
        sizes.back() = weights[i].size(0);
        outs.push_back(at::empty(sizes, xs[i].options()));
        x[i] = p(xs[i]); w[i] = p(weights[i]); out[i] = p(outs[i]);
    }
    check(vrwkv_linear_batch(xs.size(), rows, depth, weights[0].size(0), x, w, out, stream_of(xs[0])), "vrwkv_linear_batch");
    raise_failures(xs[0].get_device(), "vrwkv_linear_batch");
    return outs;
}

constexpr int64_t kOneByOne = 128 * 128 * 256;      // elements of a result: 128 tiles, less than one to an SM

Tensor key_layer(const Tensor& x, const Tensor& weight) {
    same_place(x, weight, "x");
    TORCH_CHECK(weight.dim() == 2 && x.dim() >= 1, "x must be rows of the weight's width");
    const c10::cuda::CUDAGuard guard(x.device());
    if (x.numel() == 0) return linear_relu_square(x, weight);
    const int64_t rows = x.numel() / x.size(-1);
    if (vrwkv_linear_relu_square_pays(rows, weight.size(1), weight.size(0))) return linear_relu_square(x, weight);
    // Small calls one by one cost the host more than the GPU: 16 us more for torch's product and the pass, where this kernel's GPU time
    // is 5 to 11 us and theirs 3 to 8 (one image, VRWKV-T to -B: 3.40 ms a forward, else 3.55).  A captured call costs the GPU's time alone.
    if (weight.size(1) <= 1024 && rows * weight.size(0) <= kOneByOne && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None)
        return linear_relu_square(x, weight);
    return relu_square(at::linear(x, weight), false);
}

Tensor autocast_copy(const Tensor& t) { return at::autocast::cached_cast(at::kBFloat16, t, at::kCUDA); }

std::vector<Tensor> narrow(std::vector<Tensor> weights) {
    TORCH_CHECK(!weights.empty() && weights.size() <= 16, "one to sixteen weights");
    const c10::cuda::CUDAGuard guard(weights[0].device());
    const float* src[16];
    uint16_t* out[16];
    long long n[16];
    std::vector<Tensor> outs;
    for (const Tensor& w : weights)
        if (has_tangent(w)) return {};
    for (size_t i = 0; i < weights.size(); ++i) {
        same_place(weights[i], weights[0], "a weight");
        TORCH_CHECK(weights[i].scalar_type() == at::kFloat && weights[i].is_contiguous() && weights[i].numel() > 0, "weights must be float32 and contiguous");
        outs.push_back(at::empty(weights[i].sizes(), weights[i].options().dtype(at::kBFloat16)));
        src[i] = fp(weights[i]);
        out[i] = static_cast<uint16_t*>(outs[i].data_ptr());
        n[i] = weights[i].numel();
    }
    check(vrwkv_narrow(weights.size(), src, n, out, stream_of(weights[0])), "vrwkv_narrow");
    return outs;
}

Tensor add_rows(const Tensor& table_, const Tensor& a_) {
    same_place(table_, a_, "table");
    TORCH_CHECK(is_bf16(a_) && table_.scalar_type() == at::kFloat, "a must be bfloat16 and the table float32");
    TORCH_CHECK(table_.numel() > 0 && a_.numel() % table_.numel() == 0, "a must hold whole tables");
    const c10::cuda::CUDAGuard guard(a_.device());
    const Tensor a = flat(a_), table = flat(table_);
    Tensor out = at::empty(a.sizes(), table.options());
    if (a.numel() != 0)
        check(vrwkv_add_rows(a.numel(), table.numel(), fp(table), static_cast<uint16_t*>(a.data_ptr()), fp(out), stream_of(a)), "vrwkv_add_rows");
    return out;
}

Tensor widen(const Tensor& a_) {
    same_place(a_, a_, "a");
    TORCH_CHECK(is_bf16(a_), "a must be bfloat16");
    const c10::cuda::CUDAGuard guard(a_.device());
    const Tensor a = flat(a_);
    Tensor out = at::empty(a.sizes(), a.options().dtype(at::kFloat));
    if (a.numel() != 0) check(vrwkv_widen(a.numel(), static_cast<uint16_t*>(a.data_ptr()), fp(out), stream_of(a)), "vrwkv_widen");
    return out;
}

Tensor patch_rows(const Tensor& img_, int64_t patch) {
    same_place(img_, img_, "img");
    TORCH_CHECK(img_.dim() == 4 && img_.scalar_type() == at::kFloat && patch > 0, "img must be (B, channels, H, W) in float32");
    const c10::cuda::CUDAGuard guard(img_.device());
    const Tensor img = flat(img_);
    const int64_t B = img.size(0), c = img.size(1), H = img.size(2), W = img.size(3);
    Tensor out = at::empty({B, (H / patch) * (W / patch), c * patch * patch}, img.options().dtype(at::kBFloat16));
    if (out.numel() != 0)
        check(vrwkv_patch_rows(B, c, H, W, patch, fp(img), static_cast<uint16_t*>(out.data_ptr()), stream_of(img)), "vrwkv_patch_rows");
    return out;
}

namespace {
// r_: null, or a gate's operand (a_ is then what it gates)
Tensor norm_residual_of(const Tensor& x_, const Tensor& a_, const Tensor* r_, const std::optional<Tensor>& weight, const std::optional<Tensor>& bias,
                        const std::optional<Tensor>& gamma, double eps) {
    same_place(a_, x_, "a");
    const int64_t C = x_.size(-1), rows = C ? x_.numel() / C : 0;
    TORCH_CHECK(a_.sizes() == x_.sizes(), "a must have the shape of x");
    if (r_) {
        same_place(*r_, x_, "r");
        TORCH_CHECK(r_->sizes() == x_.sizes() && is_bf16(*r_) && is_bf16(a_), "r and y must be bfloat16 of the shape of x");
    }
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = flat(x_), a = flat(a_), r = r_ ? flat(*r_) : Tensor();
    Tensor kept[3];
    const std::optional<Tensor>* given[3] = {&weight, &bias, &gamma};
    const float* p[3] = {};
    for (int i = 0; i < 3; ++i)
        if (given[i]->has_value()) {
            same_place(**given[i], x_, "a parameter");
            kept[i] = flat(f32(**given[i]));
            TORCH_CHECK(kept[i].numel() == C, "parameters must hold C values");
            p[i] = fp(kept[i]);
        }
    Tensor out = at::empty(x.sizes(), x.options());
    if (x.numel() != 0 && r_)
        check(vrwkv_gated_norm_residual(rows, C, static_cast<float>(eps), static_cast<uint16_t*>(r.data_ptr()), static_cast<uint16_t*>(a.data_ptr()),
                                        p[0], p[1], p[2], fp(x), fp(out), stream_of(x)),
              "vrwkv_gated_norm_residual");
    else if (x.numel() != 0)
        check(vrwkv_norm_residual(rows, C, static_cast<float>(eps), a.data_ptr(), is_bf16(a), p[0], p[1], p[2], fp(x), fp(out), stream_of(x)),
              "vrwkv_norm_residual");
    return out;
}

}  // namespace

Tensor layer_norm(const Tensor& x_, const Tensor& weight_, const Tensor& bias_, double eps) {
    same_place(weight_, x_, "weight");
    same_place(bias_, x_, "bias");
    const int64_t C = x_.size(-1), rows = C ? x_.numel() / C : 0;
    TORCH_CHECK(x_.scalar_type() == at::kFloat && weight_.numel() == C && bias_.numel() == C, "x must be float32; weight and bias must hold C values");
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = flat(x_), weight = flat(f32(weight_)), bias = flat(f32(bias_));
    Tensor out = at::empty(x.sizes(), x.options());
    if (x.numel() != 0) check(vrwkv_layer_norm(rows, C, static_cast<float>(eps), fp(x), fp(weight), fp(bias), fp(out), stream_of(x)), "vrwkv_layer_norm");
    return out;
}

Tensor norm_residual(const Tensor& x, const Tensor& a, const std::optional<Tensor>& weight, const std::optional<Tensor>& bias,
                     const std::optional<Tensor>& gamma, double eps) {
    return norm_residual_of(x, a, nullptr, weight, bias, gamma, eps);
}
Tensor gated_norm_residual(const Tensor& x, const Tensor& r, const Tensor& y, const std::optional<Tensor>& weight,
                           const std::optional<Tensor>& bias, const std::optional<Tensor>& gamma, double eps) {
    return norm_residual_of(x, y, &r, weight, bias, gamma, eps);
}

Tensor head_norm_gate_half(const Tensor& x_, const Tensor& gate_, const Tensor& weight_, const Tensor& bias_, double eps, int64_t act) {
    same_place(gate_, x_, "gate");
    same_place(weight_, x_, "weight");
    same_place(bias_, x_, "bias");
    const int64_t C = x_.size(-1), rows = C ? x_.numel() / C : 0;
    TORCH_CHECK(gate_.sizes() == x_.sizes() && weight_.numel() == C && bias_.numel() == C,
                "gate must have the shape of x; gamma and beta must hold C values");
    const c10::cuda::CUDAGuard guard(x_.device());
    const Tensor x = flat(f32(x_)), gate = flat(is_bf16(gate_) ? gate_ : f32(gate_)), weight = flat(f32(weight_)), bias = flat(f32(bias_));
    Tensor out = at::empty(x.sizes(), x.options().dtype(at::kBFloat16));
    if (x.numel() != 0)
        check(vrwkv_head_norm_gate_bf16out(rows, C, static_cast<float>(eps), fp(x), gate.data_ptr(), is_bf16(gate), act, fp(weight), fp(bias),
                                           static_cast<uint16_t*>(out.data_ptr()), stream_of(x)),
              "vrwkv_head_norm_gate_bf16out");
    return out;
}

}  // namespace vrwkv
