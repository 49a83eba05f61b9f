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
    lib.batch_pays.argtypes = lib.batch_route.argtypes
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


# measured in a chain of kernels, time with the library's products over time in one launch
@pytest.mark.parametrize("count,rows,C,ratio", [
    (3, 196, 192, 1.296), (3, 100352, 192, 1.128), (3, 200704, 192, 1.003), (4, 200704, 384, 1.048), (3, 200704, 256, 1.026), (4, 100352, 512, 1.025),
    (3, 6400, 512, 1.092), (3, 1536, 1024, 1.330), (3, 1664, 1024, 0.965), (3, 1792, 1024, 1.060), (4, 1664, 1024, 1.184), (3, 3328, 1024, 0.982),
    (3, 3584, 1024, 1.091), (3, 4864, 1024, 1.181), (3, 2304, 768, 0.996), (3, 2432, 768, 1.179), (3, 25600, 768, 1.006), (4, 51200, 768, 1.013),
    (3, 100352, 768, 0.986), (4, 100352, 768, 0.979)])
def test_a_batch_pays_where_it_was_measured_to(routes, count, rows, C, ratio):
    assert routes.batch_pays(count, rows, C, C, 148, 148) == (ratio > 1)
    assert not routes.batch_pays(2, rows, C, C, 148, 148)
