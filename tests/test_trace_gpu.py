"""`torch.jit.trace` records the operators and the steps around them: a traced function computes on new inputs what the function
itself does, with gradients and without."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def rnd(*shape, seed):
    return torch.randn(*shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))


B, H, W, C = 2, 5, 6, 128
T = H * W


def run_biwkv(x):
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    return RUN_CUDA(x[0, 0].abs(), x[0, 1], x, x * 0.5)


def run_biwkv_mae(x):
    from vision_rwkv_b200.mae_vrwkv import RUN_CUDA
    return RUN_CUDA(B, T, C, x[0, 0].abs(), x[0, 1], x, x * 0.5)


def run_wkv6(x):
    from vision_rwkv_b200.vrwkv6 import RUN_CUDA_RWKV6
    return RUN_CUDA_RWKV6(B, T, C, C // 64, x, x * 0.5, x + 1, x * 0.3, x[0, 0].view(C // 64, 64))


def run_wkv6_bf16(x):
    from vision_rwkv_b200.vrwkv6 import inference_rwkv6
    h = x.bfloat16()
    return inference_rwkv6(B, T, C, C // 64, h, h * 0.5, h + 1, x * 0.3, x[0, 0].view(C // 64, 64))


def run_qshift(x):
    from vision_rwkv_b200.qshift import qshift_mix
    return torch.cat(qshift_mix(x, [x[0, 0], x[0, 1]], (H, W)))


def run_qshift_heads(x):
    from vision_rwkv_b200.qshift import qshift_mix
    return torch.cat(qshift_mix(x, [x[0, 0], x[0, 1]], (H, W), head_dim=64))


def run_ddlerp(x):
    from vision_rwkv_b200.qshift import qshift_ddlerp
    return torch.cat(qshift_ddlerp(x, [x[0, 0], x[0, 1]], [None, x * 0.5], (H, W)))


def run_norm_gate(x):
    from vision_rwkv_b200.normgate import norm_gate
    return norm_gate(x, x * 0.5, x[0, 0], x[0, 1], 64, act="silu")


def run_epilogue(x):
    from vision_rwkv_b200 import epilogue
    y = epilogue.sigmoid_gate(epilogue.relu_square(x), x)
    return epilogue.add_rows(x[:1], epilogue.residual(x, y, x[0, 0]).bfloat16())


@pytest.mark.parametrize("fn", [run_biwkv, run_biwkv_mae, run_wkv6, run_wkv6_bf16, run_qshift, run_qshift_heads, run_ddlerp, run_norm_gate,
                                run_epilogue])
@pytest.mark.parametrize("grad", [True, False])
def test_a_traced_call_computes(cuda_device, fn, grad):
    example, x = rnd(B, T, C, seed=1), rnd(B, T, C, seed=2)
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(fn, example, check_trace=False)
        if not grad:
            assert (traced(x) - fn(x)).norm() <= 1e-2 * fn(x).norm()
            return
        a, b = x.clone().requires_grad_(True), x.clone().requires_grad_(True)
        got, want, gout = traced(a), fn(b), rnd(*fn(x).shape, seed=3)
        assert (got - want).norm() <= 1e-2 * want.norm()
        got.backward(gout.to(got.dtype))
        want.backward(gout.to(want.dtype))
        assert (a.grad - b.grad).norm() <= 1e-2 * b.grad.norm()
