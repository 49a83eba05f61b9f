"""Kernels that are launched before the one in front of them has been flushed wait for it by themselves: chains of them, behind a long kernel
that writes their inputs, give bit for bit what the same calls give with a synchronisation after each.  Bi-WKV's strips let the kernel behind them
start while they still store, so what takes their results shows a wait that is missing; behind other kernels a launch starts
when their blocks are gone, and what is left to see is that it finds their stores."""
import pytest
import torch

from vision_rwkv_b200 import _lib, epilogue, qshift, vrwkv, vrwkv6

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


def biwkv(x, half):
    """Behind Bi-WKV: the gate, the layers, the passes that take its float32 or bfloat16 result, one call of it behind another"""
    C = x.shape[-1]
    stack = [torch.nn.Linear(C, C, bias=False, device=x.device) for _ in range(3)]
    for layer in stack:
        torch.nn.init.normal_(layer.weight, std=0.05, generator=torch.Generator(x.device).manual_seed(1))
    norm, gate = torch.nn.LayerNorm(C, device=x.device), torch.full_like(x, 0.25, dtype=torch.bfloat16 if half else torch.float32)
    k, w, u = x.to(gate.dtype), torch.full((C,), -0.01, device=x.device), torch.full((C,), -0.005, device=x.device)
    run = vrwkv.inference_biwkv if half else vrwkv.RUN_CUDA
    yield epilogue.sigmoid_gate(gate, run(w, u, k, k))
    yield run(w, u, run(w, u, k, k).to(gate.dtype), k)
    if half:
        yield from epilogue.linears(stack, [run(w, u, k, k)] * 3)
        yield epilogue.relu_square(run(w, u, k, k), stack[0])
        yield epilogue.widened(norm, run(w, u, k, k))
    else:
        yield epilogue.layer_norm(norm, run(w, u, k, k))
        yield epilogue.norm_residual(x, run(w, u, k, k), norm, None)
        yield qshift.qshift_mix(run(w, u, k, k), [w, u], (x.shape[1], 1))[0]
        yield vrwkv6.RUN_CUDA_RWKV6(*x.shape, C // 64, *[run(w, u, k, k)] * 3, x, u.view(-1, 64))


def biwkv_one_cta(x):
    yield from biwkv(x, False)


def biwkv_clusters(x):
    yield from biwkv(x.reshape(1, -1, x.shape[-1]), False)


def biwkv_one_cta_half(x):
    yield from biwkv(x, True)


def biwkv_clusters_half(x):
    yield from biwkv(x.reshape(1, -1, x.shape[-1]), True)


def wkv6_float(x):
    """the float32 sweeps, whole sequences and in segments, with their gradients"""
    for part in (x, x.reshape(1, -1, x.shape[-1])):
        B, T, C = part.shape
        with torch.enable_grad(), torch.autocast("cuda", enabled=False):
            r, k, v, w = (part.detach().clone().requires_grad_() for _ in range(4))
            u = torch.full((C // 64, 64), 0.1, device=x.device).requires_grad_()
            y = vrwkv6.RUN_CUDA_RWKV6(B, T, C, C // 64, r, k, v, w, u)
            yield y
            yield from torch.autograd.grad(y.sum(), [r, k, v, w, u])


def matrix_state(x):
    """what an inference of the matrix-state network is made of: shift with offsets, walk, norm and gate of heads, table, patches, casts"""
    B, T, C = x.shape
    native, side = _lib.native(), int(T ** 0.5)
    half = x.bfloat16()
    for offsets in ([None] * 5, [half] * 5):
        yield from native.qshift_ddlerp_half(x, [x[0, 0]] * 5, offsets, side, side, 1, 64)
    y = native.wkv6_walk(half, half, half, epilogue.add_rows(x[:1, :1], half), x[0, 0].view(-1, 64))
    yield y
    norm, out = torch.nn.GroupNorm(C // 64, C, device=x.device), torch.nn.Linear(C, C, bias=False, device=x.device)
    yield epilogue.head_norm_gate(y, half, norm, 64, out, "silu")
    yield native.patch_rows(x.reshape(16, 3, 96, 96), 16)
    yield from native.narrow([native.widen(half), y])


@pytest.mark.parametrize("chain", [elementwise, layers, shift, wkv6, biwkv_one_cta, biwkv_clusters, biwkv_one_cta_half, biwkv_clusters_half, wkv6_float,
                                   matrix_state])
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
