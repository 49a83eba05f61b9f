"""Bi-WKV at the sequence lengths where the split over CTAs, warps and clusters changes, against the float64 oracle.
Tolerances as in test_biwkv_gpu.py (1e-5; 2e-5 above 8192 tokens; 5e-5 for huge exponent ranges) and, for bfloat16
tensors, 1e-2 as in test_biwkv_bf16_gpu.py."""
import pytest
import torch

from conftest import rel_err
from oracle import biwkv_oracle as O

pytestmark = pytest.mark.gpu
NAMES = ("y", "gw", "gu", "gk", "gv")


def run(dev, T, C, half, k_scale=1.0):
    from vision_rwkv_b200 import _lib, ops
    lib = _lib.load()
    w, u, k, v, gy = O.make_inputs(2, T, C, dtype=torch.float32, seed=T)
    k = k * k_scale
    if half:
        k, v, gy = k.bfloat16(), v.bfloat16(), gy.bfloat16()
    d = [x.to(dev).contiguous() for x in (w, u, k, v, gy)]
    before = lib.vrwkv_launch_count()
    got = (ops.biwkv_forward(*d[:4]), *ops.biwkv_backward(*d))
    launches = lib.vrwkv_launch_count() - before
    f = [x.double() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    return launches, {n: rel_err(g.float(), r) for n, g, r in zip(NAMES, got, ref)}


# 2 to 16 CTAs, full and by one token too few or too many; three CTAs against four (512 to 768); lengths for which powers of
# two would leave CTAs without tokens (1100, 2100, 2304, 3136)
@pytest.mark.parametrize("T", [257, 512, 513, 576, 577, 640, 641, 768, 769, 1025, 1100, 1280, 1281, 1793, 2049, 2100, 2304, 2305, 2817, 3136, 3329,
                               3840, 3841, 4096])
@pytest.mark.parametrize("half", [False, True])
def test_one_cluster(cuda_device, T, half):
    launches, errs = run(cuda_device, T, 40, half)
    assert launches == 5                     # the cluster-resident kernels: fast and exact, twice, and the reduction
    assert all(e <= (1e-2 if half else 1e-5) for e in errs.values()), errs


# two to eight clusters, around the lengths where one more is taken
@pytest.mark.parametrize("T", [4097, 4608, 4609, 5119, 5120, 7168, 9217, 15360])
@pytest.mark.parametrize("half", [False, True])
def test_several_clusters(cuda_device, T, half):
    _, errs = run(cuda_device, T, 40, half)
    assert all(e <= (1e-2 if half else 1e-5 if T <= 8192 else 2e-5) for e in errs.values()), errs


# inputs outside the plain-float range: the exact kernel takes the same split
@pytest.mark.parametrize("T", [700, 1100, 2305, 3136])
def test_one_cluster_wide_exponent_range(cuda_device, T):
    launches, errs = run(cuda_device, T, 40, False, k_scale=30.0)
    assert launches == 5
    assert all(e <= 5e-5 for e in errs.values()), errs
