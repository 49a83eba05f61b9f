"""The bounded waits of WKV6 on the tensor cores.  Path 3: every barrier that tiles arrive at waits for 16 bytes more than are copied.
The waits run out, nothing is fetched into a place whose copy is missing, the call returns and is reported, and the next one is right."""
import pytest
import torch

from vision_rwkv_b200 import _lib, ops

pytestmark = pytest.mark.gpu


def inputs(dev, B, T, H, dtype):
    g = torch.Generator(device=dev).manual_seed(T)
    r, k, v, gy = (torch.randn(B, T, 64 * H, device=dev, generator=g).to(dtype) for _ in range(4))
    return r, k, v, torch.randn(B, T, 64 * H, device=dev, generator=g) * 0.5 - 0.6, torch.randn(H, 64, device=dev, generator=g) * 0.1, gy


def check(run, what):
    lib = _lib.load()
    ops.raise_if_failed()
    want = run()
    try:
        assert lib.vrwkv_set_path(3) == 0
        with pytest.raises(_lib.VrwkvError, match=f"earlier launch, {what}:"):
            run()
            ops.raise_if_failed()
    finally:
        lib.vrwkv_set_path(0)
        torch.cuda.synchronize()
        lib.vrwkv_take_failures(torch.cuda.current_device())
    assert all(torch.equal(a, b) for a, b in zip(run(), want))
    ops.raise_if_failed()


# the second kernel alone; one, two and three steps of the walk over chunks (fewer and more than the two sets of tiles); many
@pytest.mark.parametrize("T", [1, 64, 65, 129, 200, 256, 1000])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_chunks(cuda_device, T, dtype):
    B, H = 3, 2
    r, k, v, w, u, gy = inputs(cuda_device, B, T, H, dtype)
    if dtype == torch.float32 and T <= 64:
        return      # float32 tensors come by TMA in the walk over chunks only
    check(lambda: [ops.wkv6_forward(r, k, v, w, u, H, tensor_cores=True)], "WKV6 forward")
    check(lambda: ops.wkv6_backward(r, k, v, w, u, gy, H, tensor_cores=True), "WKV6 backward")


# one to three steps of 16 tokens (fewer and more than the staging slots), a ragged last one, many
@pytest.mark.parametrize("T", [1, 16, 17, 33, 48, 200])
def test_walk(cuda_device, T):
    r, k, v, w, u, _ = inputs(cuda_device, 3, T, 2, torch.bfloat16)
    check(lambda: [_lib.native().wkv6_walk(r, k, v, w, u)], "WKV6 forward")
