"""Float32 WKV6 walks at the edges of their 8-token batches, whole and in segments, and the backward without gv, against the
float64 oracle (1e-5 of the maximum per tensor, as in test_wkv6_gpu.py) and against each other."""
import pytest
import torch

from conftest import rel_err
from oracle import wkv6_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T", [1, 7, 8, 9, 15, 16, 17, 47, 95, 96, 103, 105])
def test_batch_edges_and_a_call_without_gv(cuda_device, T):
    from vision_rwkv_b200 import _lib, ops
    lib = _lib.load()
    B, H = 2, 3
    C = 64 * H
    args = O.make_inputs(B, T, C, H, seed=100 + T)
    f = [x.float().contiguous().to(cuda_device) for x in args]
    got = (ops.wkv6_forward(*f[:5], H), *ops.wkv6_backward(*f, H))
    d = [x.float().double() for x in args]
    ref = (O.wkv6_forward(*d[:5], H), *O.wkv6_backward(*d, H))
    scale = max(float(r.abs().max()) for r in ref)
    for name, g, r in zip(("y", "gr", "gk", "gv", "gw", "gu"), got, ref):
        # gw of one or two tokens is a difference of equal sums
        assert (g.reshape(r.shape).double().cpu() - r).abs().max() <= 1e-5 * (scale if T <= 2 else float(r.abs().max())), name
    gr, gk, gw = (torch.full_like(f[0], float("nan")) for _ in range(3))
    gu = torch.empty_like(f[4])
    ws = torch.empty(lib.vrwkv_wkv6_backward_workspace_bytes(B, T, C, H), dtype=torch.uint8, device=cuda_device)
    r, k, v, w, u, gy = [x.data_ptr() for x in f]
    assert lib.vrwkv_wkv6_backward_f32(B, T, C, H, r, k, v, w, u, gy, gr.data_ptr(), gk.data_ptr(), None, gw.data_ptr(), gu.data_ptr(),
                                       ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
    for a, b in zip((gr, gk, gw, gu.view(-1)), (got[1], got[2], got[4], got[5].reshape(-1))):
        assert torch.equal(a, b)


def test_many_sequences_are_those_of_one(cuda_device):
    """More blocks than fit the device at once, against single sequences walked as a whole."""
    from vision_rwkv_b200 import _lib, ops
    lib = _lib.load()
    B, T, H = 130, 21, 6
    f = [x.float().contiguous().to(cuda_device) for x in O.make_inputs(B, T, 64 * H, H, seed=9)]
    y, gr, gk, gv, gw, _ = (ops.wkv6_forward(*f[:5], H), *ops.wkv6_backward(*f, H))
    for b in (0, 71, 129):
        one = [x[b:b + 1].contiguous() for x in f[:4]] + [f[4], f[5][b:b + 1].contiguous()]
        parts = (ops.wkv6_forward(*one[:5], H), *ops.wkv6_backward(*one, H))
        for whole, part in zip((y, gr, gk, gv, gw), parts):
            assert torch.equal(whole[b:b + 1], part)
