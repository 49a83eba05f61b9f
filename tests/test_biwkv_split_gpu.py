"""Bi-WKV on sequences longer than one cluster holds (T > 4096) where there are enough of them for separate launches (from 512
CTAs of 256 tokens on): against the float64 oracle, through the tensor-level calls (a backward that rebuilds everything) and
through autograd (a backward that starts from what the forward kept).  Tolerances as in test_biwkv_gpu.py: 1e-5, above 8192
tokens 2e-5, 5e-5 for huge exponent ranges; bfloat16 tensors 1e-2, their float32 gw and gu 1e-5."""
import pytest
import torch

from conftest import rel_err
from oracle import biwkv_oracle as O

pytestmark = pytest.mark.gpu
NAMES = ("y", "gw", "gu", "gk", "gv")


def errors(dev, B, T, C, half, k_scale=1.0, w_scale=None):
    from vision_rwkv_b200 import _lib, ops
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    lib = _lib.load()
    w, u, k, v, gy = O.make_inputs(B, T, C, dtype=torch.float32, seed=T + C)
    k = k * k_scale
    if w_scale is not None:
        w = w * w_scale
    if half:
        k, v, gy = k.bfloat16(), v.bfloat16(), gy.bfloat16()
    d = [x.to(dev).contiguous() for x in (w, u, k, v, gy)]
    before = lib.vrwkv_launch_count()
    plain = (ops.biwkv_forward(*d[:4]), *ops.biwkv_backward(*d))
    between = lib.vrwkv_launch_count()
    xs = [x.clone().requires_grad_(True) for x in d[:4]]
    y = RUN_CUDA(*xs)
    kept = (y.detach(), *torch.autograd.grad(y, xs, d[4].to(y.dtype)))
    ops.raise_if_failed()
    launches = between - before, lib.vrwkv_launch_count() - between
    f = [x.double() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    return launches, [{n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref)} for got in (plain, kept)], plain, kept


# one token, one sub-chunk and one CTA more or less than full CTAs; a strip of 8 channels behind a full one; more CTAs (81) than the
# chain takes in one batch
@pytest.mark.parametrize("B,T,C", [(16, 4097, 40), (16, 4112, 32), (16, 4113, 40), (8, 4352, 128), (4, 4607, 256), (4, 8192, 128),
                                   (8, 20500, 32)])
@pytest.mark.parametrize("half", [False, True])
def test_against_the_oracle(cuda_device, B, T, C, half):
    B = max(B, -(-512 // (-(-C // 32) * -(-T // 256))))
    launches, errs, plain, kept = errors(cuda_device, B, T, C, half)
    # sums, chain, spread and what stands by; the backward all of these twice, and three sums of gw, gu; less one pair when kept
    assert launches == (4 + 8, 4 + 6)
    for e in errs:
        for name, x in e.items():
            assert x <= (1e-2 if half and name in ("y", "gk", "gv") else 2e-5 if T > 8192 else 1e-5), (name, errs)
    assert torch.equal(plain[0].float(), kept[0].float())


@pytest.mark.parametrize("k_scale,w_scale", [(30.0, None), (1.0, -50.0)])
@pytest.mark.parametrize("half", [False, True])
def test_outside_the_plain_float_range(cuda_device, k_scale, w_scale, half):
    """The separate launches decline and the chunked kernels that stand by produce the result, with and without kept states."""
    _, errs, _, _ = errors(cuda_device, 16, 4200, 64, half, k_scale, w_scale)
    assert all(x <= (1e-2 if half and name in ("y", "gk", "gv") else 5e-5) for e in errs for name, x in e.items()), errs


def test_few_tokens_take_one_launch(cuda_device):
    """Below 512 CTAs the linked clusters serve the call, and nothing is kept."""
    from vision_rwkv_b200 import _lib
    lib = _lib.load()
    assert lib.vrwkv_biwkv_kept_bytes(1, 4200, 64) == 0 and lib.vrwkv_biwkv_kept_bytes(64, 4096, 768) == 0
    assert lib.vrwkv_biwkv_kept_bytes(16, 4200, 768) > 0
    launches, errs, _, _ = errors(cuda_device, 1, 4200, 64, False)
    assert launches == (2 + 4, 2 + 4)
    assert all(x <= 1e-5 for e in errs for x in e.values()), errs


def test_a_backward_the_kept_states_cannot_serve(cuda_device):
    """gy that is not 16-byte aligned: the entry point refuses before launching."""
    from vision_rwkv_b200 import _lib
    lib = _lib.load()
    B, T, C = 16, 4200, 64
    w, u, k, v, gy = [x.float().to(cuda_device).contiguous() for x in O.make_inputs(B, T, C, seed=3)]
    odd = torch.empty(gy.numel() + 1, device=cuda_device)[1:].view_as(gy).copy_(gy)
    y, gk, gv, gwgu = torch.empty_like(k), torch.empty_like(k), torch.empty_like(k), torch.empty(2, C, device=cuda_device)
    kept = torch.empty(lib.vrwkv_biwkv_kept_bytes(B, T, C), dtype=torch.uint8, device=cuda_device)
    ws = torch.empty(lib.vrwkv_biwkv_backward_workspace_bytes(B, T, C), dtype=torch.uint8, device=cuda_device)
    s = torch.cuda.current_stream().cuda_stream
    p = lambda t: t.data_ptr()
    forward = lambda size: lib.vrwkv_biwkv_forward_keep(B, T, C, p(w), p(u), p(k), p(v), p(y), 0, p(kept), size, p(ws), ws.numel(), s)
    backward = lambda g, t: lib.vrwkv_biwkv_backward_kept(B, T, C, p(w), p(u), p(k), p(v), p(g), p(gwgu), p(gk), p(gv), t, p(kept),
                                                          kept.numel(), p(ws), ws.numel(), s)
    assert forward(kept.numel() - 1) == 3 and forward(kept.numel()) == 0
    before = lib.vrwkv_launch_count()
    assert backward(odd, 0) == 8 and backward(gy, 2) == 8 and backward(gy, 3) == 8 and lib.vrwkv_launch_count() == before
    assert backward(gy, 0) == 0
    ref = O.biwkv_scan_backward(*[x.double().cpu() for x in (w, u, k, v, gy)])
    assert all(rel_err(g, r) <= 1e-5 for g, r in zip((gwgu[0], gwgu[1], gk, gv), ref))
