"""Which kernel takes the linear layers (csrc/linear_routes.h): by size, and by what the device can run."""
import ctypes
import os
import subprocess

import pytest

from conftest import ROOT

NONE, SLABS, TILES = range(3)


@pytest.fixture(scope="module")
def routes(tmp_path_factory):
    out = tmp_path_factory.mktemp("host") / "linear_routes_host.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(ROOT, "vision-rwkv_b200", "csrc"),
                    os.path.join(ROOT, "tests", "host_harness", "linear_routes_host.cpp"), "-o", str(out)], check=True)
    lib = ctypes.CDLL(str(out))
    lib.batch_route.argtypes = [ctypes.c_int, ctypes.c_longlong] + [ctypes.c_int] * 4
    lib.square_by_slabs.argtypes = [ctypes.c_longlong] + [ctypes.c_int] * 3
    return lib


def test_without_a_device_no_layer_is_taken():
    """The library's own answer on this machine, where it has no device; `-m gpu` tests run where it has one."""
    import torch
    from vision_rwkv_b200 import _lib
    if torch.cuda.is_available():
        pytest.skip("this machine has a device")
    lib = _lib.load()
    for K, N in ((384, 384), (192, 1536), (512, 512), (1024, 1024)):
        assert lib.vrwkv_linear_batch_pays(3, 1000, K, N) == 0


# four layers of 1536 columns are 32 slabs, the key layer's 768 columns 4
@pytest.mark.parametrize("sms,want", [(148, SLABS), (32, SLABS), (31, TILES), (8, TILES), (1, TILES)])
def test_a_device_with_few_multiprocessors_takes_tiles(routes, sms, want):
    assert routes.batch_route(4, 300, 384, 1536, sms, sms) == want
    assert routes.batch_route(4, 300, 384, 1536, 0, sms) == TILES          # the slab kernel cannot be had
    assert routes.batch_route(4, 300, 384, 1536, 0, 0) == NONE
    assert routes.batch_route(4, 300, 384, 192, min(sms, 3), sms) == NONE      # columns that are no whole tiles
    assert routes.square_by_slabs(300, 192, 768, sms) == (sms >= 4)


@pytest.mark.parametrize("rows,K,N,want", [(1, 64, 192, SLABS), (1 << 24, 384, 384, SLABS), ((1 << 24) + 1, 384, 768, NONE), (5, 96, 192, NONE), (5, 64, 200, NONE),
                                           (5, 448, 192, NONE), (5, 448, 256, TILES), (5, 1024, 768, TILES), (5, 1088, 768, NONE), (5, 64, 256, TILES),
                                           (5, 384, 1728, NONE), (5, 384, 2304, TILES), (0, 64, 192, NONE), (5, 0, 192, NONE), (5, 64, 0, NONE)])
def test_by_size(routes, rows, K, N, want):
    assert routes.batch_route(3, rows, K, N, 148, 148) == want
