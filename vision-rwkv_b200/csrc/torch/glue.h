#pragma once
#include <optional>
#include "native.h"

namespace vrwkv {
std::vector<Tensor> qshift_mix(const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group, bool per_head);
std::vector<Tensor> qshift_ddlerp(const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H, int64_t W,
                                  int64_t shift, int64_t head_dim);
// bfloat16 results, no autograd node
std::vector<Tensor> qshift_mix_half(const Tensor& x, std::vector<Tensor> mixes, int64_t H, int64_t W, int64_t shift, int64_t group,
                                    bool per_head);
std::vector<Tensor> qshift_ddlerp_half(const Tensor& x, std::vector<Tensor> maas, std::vector<std::optional<Tensor>> offsets, int64_t H,
                                       int64_t W, int64_t shift, int64_t head_dim);
Tensor norm_gate(const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, int64_t group, double eps, int64_t act);
// epilogue.cpp
Tensor sigmoid_gate(const Tensor& r, const Tensor& y, bool wide);      // wide: bfloat16 r, y to a float32 result
Tensor relu_square(const Tensor& x, bool wide);      // wide: bfloat16 x to a float32 result
// relu(x weight^T)^2 in bfloat16, as autocast computes it for a linear layer that rounds it; called under bfloat16 autocast
Tensor linear_relu_square(const Tensor& x, const Tensor& weight);
// the same, by one kernel or by torch's product and the pass behind it, whichever takes less time
Tensor key_layer(const Tensor& x, const Tensor& weight);
// up to four linear layers of one shape without a bias on bfloat16 rows, as autocast computes them, in one launch where that is faster
std::vector<Tensor> linear_batch(std::vector<Tensor> xs, std::vector<Tensor> weights);
// what autocast makes of t for a bfloat16 product, from its cache where it has it
Tensor autocast_copy(const Tensor& t);
// bfloat16 copies of float32 weights in one launch; empty where forward-mode differentiation wants the casts themselves
std::vector<Tensor> narrow(std::vector<Tensor> weights);
Tensor add_rows(const Tensor& table, const Tensor& a);
Tensor patch_rows(const Tensor& img, int64_t patch);
Tensor widen(const Tensor& a);
Tensor layer_norm(const Tensor& x, const Tensor& weight, const Tensor& bias, double eps);
Tensor norm_residual(const Tensor& x, const Tensor& a, const std::optional<Tensor>& weight, const std::optional<Tensor>& bias,
                     const std::optional<Tensor>& gamma, double eps);
Tensor gated_norm_residual(const Tensor& x, const Tensor& r, const Tensor& y, const std::optional<Tensor>& weight,
                           const std::optional<Tensor>& bias, const std::optional<Tensor>& gamma, double eps);
Tensor head_norm_gate_half(const Tensor& x, const Tensor& gate, const Tensor& weight, const Tensor& bias, double eps, int64_t act);
}  // namespace vrwkv
