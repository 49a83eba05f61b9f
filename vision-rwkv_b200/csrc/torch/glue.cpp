// Host path of the kernels around the operators: token shift with its interpolations (qshift_mix, qshift_ddlerp)
// and the normalise-and-gate step behind them.  Rules as in qshift.py / normgate.py, whose functions call these.
#include "glue.h"

namespace vrwkv {

namespace {

using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;

constexpr int kMost = 5;

struct Grid {
    int B, H, W, C;
};
Grid grid_of(const Tensor& x, int64_t H, int64_t W) {
    TORCH_CHECK(x.is_cuda(), "x must be a CUDA tensor");
    TORCH_CHECK(x.dim() == 3, "x must be (B, T, C), got ", x.sizes());
    TORCH_CHECK(H * W == x.size(1), "patch resolution ", H, "x", W, " does not match T=", x.size(1));
    return Grid{static_cast<int>(x.size(0)), static_cast<int>(H), static_cast<int>(W), static_cast<int>(x.size(2))};
}
void check_vectors(const std::vector<Tensor>& ts, const Tensor& x) {
    for (const Tensor& t : ts) {
        TORCH_CHECK(t.device() == x.device(), "mix vectors are on ", t.device(), ", expected ", x.device());
        TORCH_CHECK(t.numel() == x.size(2), "mix vectors must hold C=", x.size(2), " values");
    }
}
template <typename P>
struct Pointers {
    P at[kMost] = {};
    void set(size_t i, const Tensor& t) { at[i] = t.defined() ? static_cast<P>(t.data_ptr()) : nullptr; }
};
std::vector<Tensor> flat_f32(at::TensorList ts) {
    std::vector<Tensor> out;
    for (const Tensor& t : ts) out.push_back(f32(t).view(-1));
    return out;
}

// ---- q_shift + interpolations ------------------------------------------------------------------
struct QShiftArgs {
    int64_t H, W, shift, group;   // group: channels per shifted group, or per head
    bool per_head;
};

std::vector<Tensor> qshift_forward(const Tensor& xf, const std::vector<Tensor>& mixes, const QShiftArgs& a, bool half_out = false) {
    const Grid g = grid_of(xf, a.H, a.W);
    std::vector<Tensor> outs;
    Pointers<const float*> pm;
    Pointers<float*> po;
    Pointers<uint16_t*> ph;
    for (size_t i = 0; i < mixes.size(); ++i) {
        outs.push_back(at::empty_like(xf, half_out ? xf.options().dtype(at::kBFloat16) : xf.options()));
        pm.set(i, mixes[i]);
        po.set(i, outs[i]);
        ph.set(i, outs[i]);
    }
    if (xf.numel() == 0) return outs;
    if (half_out) {
        check(vrwkv_qshift_mix_forward_bf16out(g.B, g.H, g.W, g.C, a.per_head ? 0 : a.group, a.per_head ? a.group : 0, a.shift, mixes.size(),
                                               fp(xf), pm.at, ph.at, stream_of(xf)),
              "vrwkv_qshift_mix_forward_bf16out");
        return outs;
    }
    const auto entry = a.per_head ? vrwkv_qshift_multihead_mix_forward_f32 : vrwkv_qshift_mix_forward_f32;
    check(entry(g.B, g.H, g.W, g.C, a.group, a.shift, mixes.size(), fp(xf), pm.at, po.at, stream_of(xf)), "vrwkv_qshift_mix_forward_f32");
    return outs;
}

struct QShiftMix : torch::autograd::Function<QShiftMix> {
    static variable_list forward(AutogradContext* ctx, const Tensor& x, at::TensorList mixes, int64_t H, int64_t W, int64_t shift,
                                 int64_t group, bool per_head) {
        const QShiftArgs a{H, W, shift, group, per_head};
        const Tensor xf = f32(x);
        const std::vector<Tensor> flat = flat_f32(mixes);
        variable_list saved{xf};
        saved.insert(saved.end(), flat.begin(), flat.end());
        saved.insert(saved.end(), mixes.begin(), mixes.end());
        ctx->save_for_backward(saved);
        ctx->saved_data["n"] = static_cast<int64_t>(mixes.size());
        ctx->saved_data["geometry"] = std::vector<int64_t>{H, W, shift, group, per_head ? 1 : 0};
        ctx->saved_data["dtype"] = static_cast<int64_t>(x.scalar_type());
        variable_list outs = qshift_forward(xf, flat, a);
        for (Tensor& o : outs) o = o.to(x.scalar_type());
        return outs;
    }
    static variable_list backward(AutogradContext* ctx, variable_list gouts) {
        const auto saved = ctx->get_saved_variables();
        const size_t n = ctx->saved_data["n"].toInt();
        const auto geo = ctx->saved_data["geometry"].toIntVector();
        const Tensor& x = saved[0];
        const c10::cuda::CUDAGuard guard(x.device());
        const at::NoGradGuard no_grad;
        const Grid g = grid_of(x, geo[0], geo[1]);
        Tensor gx = at::empty_like(x);
        Tensor gmix = at::empty({static_cast<int64_t>(n), g.C}, x.options());
        std::vector<Tensor> gs;
        Pointers<const float*> pm, pg;
        Pointers<float*> po;
        for (size_t i = 0; i < n; ++i) {
            gs.push_back(f32(gouts[i]));
            pm.set(i, saved[1 + i]);
            pg.set(i, gs[i]);
            po.at[i] = fp(gmix) + i * g.C;
        }
        if (x.numel() == 0) {
            gmix.zero_();
        } else {
            Tensor ws = workspace(vrwkv_qshift_mix_backward_workspace_bytes(g.B, g.H, g.W, g.C, n), x);
            const auto entry = geo[4] ? vrwkv_qshift_multihead_mix_backward_f32 : vrwkv_qshift_mix_backward_f32;
            check(entry(g.B, g.H, g.W, g.C, geo[3], geo[2], n, fp(x), pm.at, pg.at, fp(gx), po.at, ws.data_ptr(), ws.numel(), stream_of(x)),
                  "vrwkv_qshift_mix_backward_f32");
        }
        variable_list out{gx.to(static_cast<at::ScalarType>(ctx->saved_data["dtype"].toInt()))};
        for (size_t i = 0; i < n; ++i) out.push_back(gmix.select(0, i).view(saved[1 + n + i].sizes()));
        out.resize(out.size() + 16);     // the arguments that are no tensors
        return out;
    }
};

// ---- per-head shift + data-dependent interpolations ----------------------------------------------
struct QShiftDdlerp : torch::autograd::Function<QShiftDdlerp> {
    // rest = maas, then the offsets that are given; present[j] says whether output j has one
    static variable_list forward(AutogradContext* ctx, const Tensor& x, at::TensorList rest, std::vector<int64_t> present, int64_t H,
                                 int64_t W, int64_t shift, int64_t head_dim) {
        const size_t n = present.size();
        const Tensor xf = f32(x);
        const Grid g = grid_of(xf, H, W);
        const std::vector<Tensor> maas(rest.begin(), rest.begin() + n);
        std::vector<Tensor> given(rest.begin() + n, rest.end());
        bool half = !given.empty();
        for (const Tensor& m : given) half = half && is_bf16(m);
        const std::vector<Tensor> flat = flat_f32(maas);
        variable_list saved{xf};
        saved.insert(saved.end(), flat.begin(), flat.end());
        std::vector<int64_t> dtypes;
        for (Tensor& m : given) {
            TORCH_CHECK(m.sizes() == x.sizes() && m.device() == x.device(), "offsets must have the shape of x and be on its device");
            dtypes.push_back(static_cast<int64_t>(m.scalar_type()));
            m = half ? m.contiguous() : f32(m);
            saved.push_back(m);
        }
        saved.insert(saved.end(), maas.begin(), maas.end());
        ctx->save_for_backward(saved);
        ctx->saved_data["present"] = present;
        ctx->saved_data["dtypes"] = dtypes;
        ctx->saved_data["geometry"] = std::vector<int64_t>{H, W, shift, head_dim, half ? 1 : 0};
        ctx->saved_data["dtype"] = static_cast<int64_t>(x.scalar_type());
        variable_list outs;
        Pointers<const float*> pa;
        Pointers<const void*> pm;
        Pointers<float*> po;
        size_t at_m = 0;
        for (size_t i = 0; i < n; ++i) {
            outs.push_back(at::empty_like(xf));
            pa.set(i, flat[i]);
            po.set(i, outs[i]);
            if (present[i]) pm.set(i, given[at_m++]);
        }
        if (x.numel() == 0) return outs;
        check(vrwkv_qshift_ddlerp_forward_f32(g.B, g.H, g.W, g.C, head_dim, shift, n, fp(xf), pa.at, pm.at, half, po.at, stream_of(xf)),
              "vrwkv_qshift_ddlerp_forward_f32");
        return outs;
    }
    static variable_list backward(AutogradContext* ctx, variable_list gouts) {
        const auto saved = ctx->get_saved_variables();
        const auto present = ctx->saved_data["present"].toIntVector();
        const auto dtypes = ctx->saved_data["dtypes"].toIntVector();
        const auto geo = ctx->saved_data["geometry"].toIntVector();
        const size_t n = present.size(), n_given = dtypes.size();
        const Tensor& x = saved[0];
        const c10::cuda::CUDAGuard guard(x.device());
        const at::NoGradGuard no_grad;
        const Grid g = grid_of(x, geo[0], geo[1]);
        Tensor gx = at::empty_like(x);
        Tensor gmaa = at::zeros({static_cast<int64_t>(n), g.C}, x.options());
        std::vector<Tensor> gs, gms;
        Pointers<const float*> pa, pg;
        Pointers<const void*> pm;
        Pointers<void*> pgm;
        Pointers<float*> po;
        size_t at_m = 0;
        for (size_t i = 0; i < n; ++i) {
            gs.push_back(f32(gouts[i]));
            pa.set(i, saved[1 + i]);
            pg.set(i, gs[i]);
            po.at[i] = fp(gmaa) + i * g.C;
            if (present[i]) {
                const Tensor& m = saved[1 + n + at_m++];
                gms.push_back(at::empty_like(m));
                pm.set(i, m);
                pgm.set(i, gms.back());
            }
        }
        if (x.numel() != 0) {
            Tensor ws = workspace(vrwkv_qshift_ddlerp_backward_workspace_bytes(g.B, g.H, g.W, g.C, n), x);
            check(vrwkv_qshift_ddlerp_backward_f32(g.B, g.H, g.W, g.C, geo[3], geo[2], n, fp(x), pa.at, pm.at, geo[4], pg.at, fp(gx), pgm.at,
                                                   po.at, ws.data_ptr(), ws.numel(), stream_of(x)),
                  "vrwkv_qshift_ddlerp_backward_f32");
        }
        variable_list out{gx.to(static_cast<at::ScalarType>(ctx->saved_data["dtype"].toInt()))};
        for (size_t i = 0; i < n; ++i) {
            const Tensor& maa = saved[1 + n + n_given + i];
            out.push_back(gmaa.select(0, i).view(maa.sizes()).to(maa.scalar_type()));
        }
        for (size_t i = 0; i < n_given; ++i) out.push_back(gms[i].to(static_cast<at::ScalarType>(dtypes[i])));
        out.resize(out.size() + 16);     // the arguments that are no tensors
        return out;
    }
};

// ---- normalise and gate ----------------------------------------------------------------------------
struct NormGate : torch::autograd::Function<NormGate> {
    static Tensor forward(AutogradContext* ctx, const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, int64_t group,
                          double eps, int64_t act) {
        const Tensor xf = f32(x), gt = is_bf16(gate) ? gate.contiguous() : f32(gate), wf = f32(weight), bf = f32(bias);
        const int64_t C = x.size(-1), rows = C ? x.numel() / C : 0;
        TORCH_CHECK(gt.sizes() == xf.sizes() && wf.numel() == C && bf.numel() == C,
                    "gate must have the shape of x; gamma and beta must hold C values");
        for (const Tensor* t : {&gt, &wf, &bf}) TORCH_CHECK(t->device() == xf.device(), "tensors are on different devices");
        Tensor out = at::empty_like(xf);
        const int64_t n_groups = group > 0 && C % group == 0 ? C / group : 1;
        Tensor stats = at::empty({2, rows, n_groups}, xf.options());
        if (xf.numel() != 0)
            check(vrwkv_normgate_forward_f32(rows, C, group, static_cast<float>(eps), fp(xf), gt.data_ptr(), is_bf16(gt), act, fp(wf), fp(bf),
                                             fp(out), fp(stats), fp(stats) + rows * n_groups, stream_of(xf)),
                  "vrwkv_normgate_forward_f32");
        ctx->save_for_backward({xf, gt, wf, bf, stats});
        ctx->saved_data["group"] = group;
        ctx->saved_data["act"] = act;
        ctx->saved_data["dtypes"] = std::vector<int64_t>{static_cast<int64_t>(x.scalar_type()), static_cast<int64_t>(gate.scalar_type()),
                                                         static_cast<int64_t>(weight.scalar_type()), static_cast<int64_t>(bias.scalar_type())};
        return out;
    }
    static variable_list backward(AutogradContext* ctx, variable_list gouts) {
        const auto saved = ctx->get_saved_variables();
        const Tensor &x = saved[0], &gate = saved[1], &weight = saved[2], &bias = saved[3], &stats = saved[4];
        const auto dt = ctx->saved_data["dtypes"].toIntVector();
        const int64_t group = ctx->saved_data["group"].toInt(), C = x.size(-1), rows = C ? x.numel() / C : 0;
        const c10::cuda::CUDAGuard guard(x.device());
        const at::NoGradGuard no_grad;
        const Tensor gout = f32(gouts[0]);
        Tensor gx = at::empty_like(x), ggate = at::empty_like(gate), gpar = at::empty({2, C}, x.options());
        if (x.numel() == 0) {
            gpar.zero_();
        } else {
            Tensor ws = workspace(vrwkv_normgate_backward_workspace_bytes(rows, C, group), x);
            check(vrwkv_normgate_backward_f32(rows, C, group, fp(gout), fp(x), gate.data_ptr(), is_bf16(gate), ctx->saved_data["act"].toInt(),
                                              fp(weight), fp(bias), fp(stats), fp(stats) + stats.numel() / 2, fp(gx), ggate.data_ptr(), fp(gpar),
                                              ws.data_ptr(), ws.numel(), stream_of(x)),
                  "vrwkv_normgate_backward_f32");
        }
        const auto as = [&](int i) { return static_cast<at::ScalarType>(dt[i]); };
        return {gx.to(as(0)), ggate.to(as(1)), gpar.select(0, 0).to(as(2)), gpar.select(0, 1).to(as(3)), Tensor(), Tensor(), Tensor()};
    }
};

}  // namespace

std::vector<Tensor> qshift_mix(const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group, bool per_head) {
    TORCH_CHECK(mixes.size() >= 1 && mixes.size() <= 3, "between one and three mix vectors");
    grid_of(x, H, W);
    check_vectors(mixes, x);
    const c10::cuda::CUDAGuard guard(x.device());
    return QShiftMix::apply(x, at::TensorList(mixes), H, W, shift, group, per_head);
}

std::vector<Tensor> qshift_mix_half(const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group,
                                    bool per_head) {
    TORCH_CHECK(mixes.size() >= 1 && mixes.size() <= 3, "between one and three mix vectors");
    grid_of(x, H, W);
    check_vectors(mixes, x);
    refuse_tangents({&x});
    refuse_tangents(mixes);
    const c10::cuda::CUDAGuard guard(x.device());
    return qshift_forward(f32(x), flat_f32(mixes), QShiftArgs{H, W, shift, group, per_head}, true);
}

std::vector<Tensor> qshift_ddlerp_half(const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H,
                                       int64_t W, int64_t shift, int64_t head_dim) {
    TORCH_CHECK(maas.size() >= 1 && maas.size() <= kMost && offsets.size() == maas.size(),
                "between one and five mix vectors, and as many offsets (None for no offset)");
    TORCH_CHECK(head_dim > 0 && head_dim % 16 == 0 && x.size(-1) % head_dim == 0, "head_dim=", head_dim,
                " must be a multiple of 16 that divides C=", x.size(-1));
    const Grid g = grid_of(x, H, W);
    check_vectors(maas, x);
    refuse_tangents({&x});
    refuse_tangents(maas);
    const c10::cuda::CUDAGuard guard(x.device());
    const Tensor xf = f32(x);
    const std::vector<Tensor> flat = flat_f32(maas);
    bool half = true, any = false;
    for (const auto& m : offsets)
        if (m.has_value()) {
            TORCH_CHECK(m->sizes() == x.sizes() && m->device() == x.device(), "offsets must have the shape of x and be on its device");
            refuse_tangents({&*m});
            any = true;
            half = half && is_bf16(*m);
        }
    half = half && any;
    std::vector<Tensor> outs, kept;
    Pointers<const float*> pa;
    Pointers<const void*> pm;
    Pointers<uint16_t*> po;
    for (size_t i = 0; i < maas.size(); ++i) {
        outs.push_back(at::empty_like(xf, xf.options().dtype(at::kBFloat16)));
        pa.set(i, flat[i]);
        po.set(i, outs[i]);
        if (offsets[i].has_value()) {
            kept.push_back(half ? offsets[i]->contiguous() : f32(*offsets[i]));
            pm.set(i, kept.back());
        }
    }
    if (xf.numel() == 0) return outs;
    check(vrwkv_qshift_ddlerp_forward_bf16out(g.B, g.H, g.W, g.C, head_dim, shift, maas.size(), fp(xf), pa.at, pm.at, half, po.at, stream_of(xf)),
          "vrwkv_qshift_ddlerp_forward_bf16out");
    return outs;
}

std::vector<Tensor> qshift_ddlerp(const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H, int64_t W,
                                  int64_t shift, int64_t head_dim) {
    TORCH_CHECK(maas.size() >= 1 && maas.size() <= kMost && offsets.size() == maas.size(),
                "between one and five mix vectors, and as many offsets (None for no offset)");
    TORCH_CHECK(head_dim > 0 && head_dim % 16 == 0 && x.size(-1) % head_dim == 0, "head_dim=", head_dim,
                " must be a multiple of 16 that divides C=", x.size(-1));
    grid_of(x, H, W);
    check_vectors(maas, x);
    const c10::cuda::CUDAGuard guard(x.device());
    std::vector<Tensor> rest = maas;
    std::vector<int64_t> present;
    for (const auto& m : offsets) {
        present.push_back(m.has_value() ? 1 : 0);
        if (m.has_value()) rest.push_back(*m);
    }
    return QShiftDdlerp::apply(x, at::TensorList(rest), present, H, W, shift, head_dim);
}

Tensor norm_gate(const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, int64_t group, double eps, int64_t act) {
    TORCH_CHECK(x.is_cuda(), "x must be a CUDA tensor");
    const c10::cuda::CUDAGuard guard(x.device());
    return NormGate::apply(x, gate, weight, bias, group, eps, act);
}

}  // namespace vrwkv
