"""The per-channel vectors w, u may start at any float: cut out of a larger parameter buffer they are 4-byte aligned, and every
kernel gives the bits it gives for an aligned copy."""
import pytest
import torch

from oracle import biwkv_oracle, wkv6_oracle

pytestmark = pytest.mark.gpu


def shifted(x, by):
    """x at an offset of `by` floats in a larger buffer."""
    flat = torch.empty(x.numel() + by, device=x.device, dtype=x.dtype)[by:]
    flat.copy_(x.reshape(-1))
    assert flat.data_ptr() % 16 == 4 * by % 16
    return flat.view(x.shape)


def results(fn, leaves, gy):
    leaves = [x.detach().requires_grad_(True) for x in leaves]
    y = fn(*leaves)
    return (y.detach(), *torch.autograd.grad(y, leaves, gy))


@pytest.mark.parametrize("by", [1, 2, 3])
@pytest.mark.parametrize("B,T,C,dtype,k_scale", [(2, 70, 40, torch.float32, 1.0), (1, 4200, 32, torch.float32, 1.0),
                                                 (2, 196, 64, torch.float32, 40.0), (2, 196, 64, torch.bfloat16, 1.0),
                                                 (2, 33, 36, torch.float32, 1.0), (2, 33, 35, torch.float32, 1.0)])
def test_biwkv(cuda_device, B, T, C, dtype, k_scale, by):
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    w, u, k, v, gy = (x.to(cuda_device) for x in biwkv_oracle.make_inputs(B, T, C, dtype=torch.float32, seed=T))
    k, v = (k * k_scale).to(dtype), v.to(dtype)
    want = results(RUN_CUDA, (w, u, k, v), gy)
    got = results(RUN_CUDA, (shifted(w, by), shifted(u, by), k, v), gy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("by", [1, 2, 3])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_wkv6(cuda_device, dtype, by):
    from vision_rwkv_b200.vrwkv6 import RUN_CUDA_RWKV6, inference_rwkv6
    B, T, H = 2, 70, 3
    r, k, v, w, u, gy = (x.float().to(cuda_device) for x in wkv6_oracle.make_inputs(B, T, 64 * H, H, seed=1))
    r, k, v = (x.to(dtype) for x in (r, k, v))
    run = lambda *xs: RUN_CUDA_RWKV6(B, T, 64 * H, H, *xs)
    want, got = results(run, (r, k, v, w, u), gy), results(run, (r, k, v, w, shifted(u, by)), gy)
    assert all(torch.equal(a, b) for a, b in zip(got, want))
    with torch.no_grad():
        assert torch.equal(inference_rwkv6(B, T, 64 * H, H, r, k, v, w, shifted(u, by)), inference_rwkv6(B, T, 64 * H, H, r, k, v, w, u))
