"""The chunked WKV6 backward where the last 64-token chunk is short: warps without tokens of their own leave their work out, and what they would have
written is not read.  Operands rounded to bfloat16 leave 1e-2 of the largest value; the oracle sees the same rounded inputs."""
import pytest
import torch

from conftest import rel_err
from oracle import wkv6_oracle as O

pytestmark = pytest.mark.gpu


# one token to a whole chunk behind the last full one, at the edges of the warps' 16 and 32 tokens
@pytest.mark.parametrize("last", [1, 15, 16, 17, 31, 32, 33, 47, 48, 49, 63, 64])
@pytest.mark.parametrize("chunks,dtype", [(0, torch.bfloat16), (1, torch.bfloat16), (1, torch.float32)])
def test_short_last_chunk(cuda_device, chunks, dtype, last):
    from vision_rwkv_b200 import ops
    B, T, H = 2, 64 * chunks + last, 1
    r, k, v, w, u, gy = O.make_inputs(B, T, 64 * H, H, seed=T, round_to=torch.bfloat16)
    gy = gy.bfloat16().float()
    ref = O.wkv6_backward(*[x.float().double() for x in (r, k, v, w, u, gy)], H)
    r, k, v, gy = (x.to(dtype).contiguous().to(cuda_device) for x in (r, k, v, gy))
    w, u = (x.float().contiguous().to(cuda_device) for x in (w, u))
    got = ops.wkv6_backward(r, k, v, w, u, gy, H, tensor_cores=True)
    for name, g, want in zip(("gr", "gk", "gv", "gw", "gu"), got, ref):
        assert rel_err(g.reshape(want.shape), want) <= 1e-2, name
