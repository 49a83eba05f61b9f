"""Kernels that are launched before the one in front of them has been flushed wait for it by themselves: chains of them, behind a long kernel
that writes their inputs, give bit for bit what the same calls give with a synchronisation after each."""
import pytest
import torch

from vision_rwkv_b200 import epilogue, qshift, vrwkv6

pytestmark = pytest.mark.gpu


def elementwise(x):
    norm = torch.nn.LayerNorm(x.shape[-1], device=x.device)
    r = x.bfloat16()
    yield epilogue.sigmoid_gate(r, r)
    yield epilogue.relu_square(r)
    yield epilogue.layer_norm(norm, x)
    yield epilogue.norm_residual(x, epilogue.sigmoid_gate(r, r), norm, None)


def layers(x):
    stack = [torch.nn.Linear(x.shape[-1], x.shape[-1], bias=False, device=x.device) for _ in range(3)]
    key = torch.nn.Linear(x.shape[-1], 4 * x.shape[-1], bias=False, device=x.device)
    value = torch.nn.Linear(4 * x.shape[-1], x.shape[-1], bias=False, device=x.device)
    for p in stack + [key, value]:
        torch.nn.init.normal_(p.weight, std=0.05, generator=torch.Generator(x.device).manual_seed(1))
    outs = epilogue.linears(stack, [x.bfloat16()] * 3)
    yield from outs
    yield epilogue.linear_relu_square(key, epilogue.sigmoid_gate(outs[0], outs[1]), value)


def shift(x):
    mixes = [torch.full((1, 1, x.shape[-1]), 0.25, device=x.device).requires_grad_() for _ in range(3)]
    side = int(x.shape[1] ** 0.5)
    with torch.enable_grad():
        leaf = x.detach().requires_grad_()
        outs = qshift.qshift_mix(leaf, mixes, (side, side))
        yield from outs
        yield from torch.autograd.grad([o.sum() for o in outs], [leaf, *mixes])


def wkv6(x):
    B, T, C = x.shape
    with torch.enable_grad():
        r, k, v = (x.detach().bfloat16().requires_grad_() for _ in range(3))
        w = x.detach().clone().requires_grad_()
        u = torch.full((C // 64, 64), 0.1, device=x.device).requires_grad_()
        y = vrwkv6.RUN_CUDA_RWKV6(B, T, C, C // 64, r, k, v, w, u)
        yield y
        yield from torch.autograd.grad(y.float().sum(), [r, k, v, w, u])


@pytest.mark.parametrize("chain", [elementwise, layers, shift, wkv6])
def test_behind_a_long_kernel(cuda_device, chain):
    a = torch.randn(4096, 4096, device=cuda_device)
    source = torch.randn(16, 144, 192, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = []
        for out in chain(source):
            torch.cuda.synchronize()
            want.append(out.clone())
        for _ in range(3):
            x = torch.zeros_like(source)
            torch.cuda.synchronize()
            late = (a @ a)[:16, :144].sum() * 0                  # the inputs are written at the end of this
            x.copy_(source + late)
            got = list(chain(x))
            assert all(torch.equal(p, q) for p, q in zip(got, want))
