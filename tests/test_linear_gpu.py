"""relu(x W^T)^2 as one matrix product: against the product in float64, rounded where autocast rounds.  A float32 sum p that lies near
the middle of two bfloat16 numbers may go to the other one, an ulp (2^-7 |p| at most) away, and sums of up to 1024 products of size 1
are off by 1e-5: the square differs by 2^-6 p^2 + 2e-5 |p| from that, and by its own rounding, 2^-8 p^2.  Few sums do: 1e-2 in the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around a tile's 128, fewer and more tiles than SMs (several per CTA, both accumulators); K of one slice, of fewer and more than the four stages
@pytest.mark.parametrize("rows,K,N", [(1, 64, 256), (127, 192, 256), (128, 256, 512), (129, 320, 256), (1000, 384, 1536), (19008, 192, 768),
                                      (5000, 1024, 4096), (40001, 64, 256)])
def test_against_float64(cuda_device, rows, K, N):
    from vision_rwkv_b200 import _lib
    g = torch.Generator(device=cuda_device).manual_seed(rows + K)
    x = torch.randn(rows, K, device=cuda_device, generator=g).bfloat16()
    w = (torch.randn(N, K, device=cuda_device, generator=g) / K ** 0.5).bfloat16()
    with torch.autocast("cuda", torch.bfloat16):
        out = _lib.native().linear_relu_square(x, w)
    ref = (x.double() @ w.double().T).bfloat16().double().relu().square()
    assert out.shape == (rows, N) and out.dtype == torch.bfloat16
    assert ((out.double() - ref).norm() / ref.norm()).item() <= 1e-2
    assert ((out.double() - ref).abs() <= (2.0 ** -6 + 2.0 ** -8) * 1.02 * ref + 2e-5 * ref.sqrt() + 1e-9).all()


def test_not_a_number_stays(cuda_device):
    from vision_rwkv_b200 import _lib
    x = torch.ones(130, 64, device=cuda_device).bfloat16()
    x[129, 3] = float("nan")
    x[5, 1] = float("inf")
    with torch.autocast("cuda", torch.bfloat16):
        out = _lib.native().linear_relu_square(x, torch.ones(256, 64, device=cuda_device))
    assert out[129].isnan().all() and out[5].isinf().all() and (out[6] == 4096).all()


def test_layers_that_are_watched_or_replaced_keep_their_call(cuda_device):
    from vision_rwkv_b200 import epilogue
    key, value = torch.nn.Linear(192, 768, bias=False, device=cuda_device), torch.nn.Linear(768, 192, bias=False, device=cuda_device)
    x = torch.randn(20000, 192, device=cuda_device).bfloat16()
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = epilogue.relu_square(key(x), value)
        got = epilogue.linear_relu_square(key, x, value)
        seen = []
        hook = key.register_forward_hook(lambda *a: seen.append(1))
        again = epilogue.linear_relu_square(key, x, value)
        hook.remove()
    assert seen == [1] and torch.equal(again, want)
    assert ((got.float() - want.float()).norm() / want.float().norm()).item() <= 5e-3      # sums in another order: some roundings differ


@pytest.mark.parametrize("rows,C", [(1, 192), (196, 384), (196, 1024), (1568, 768), (40, 2048), (25000, 192), (12544, 768)])
def test_the_key_layer_takes_one_kernel_only_where_it_is_faster(cuda_device, rows, C):
    """By the measured rule: from four rounds of 128 x 256 tiles over the SMs on, before that where a round's SMs are four fifths busy, up to
    1024 channels; of calls that are not captured the small ones too.  Elsewhere the product is torch's."""
    from vision_rwkv_b200 import _lib, epilogue
    lib = _lib.load()
    key, value = torch.nn.Linear(C, 4 * C, bias=False, device=cuda_device), torch.nn.Linear(4 * C, C, bias=False, device=cuda_device)
    x = torch.randn(rows, C, device=cuda_device).bfloat16()
    sms, tiles = torch.cuda.get_device_properties(cuda_device).multi_processor_count, -(-rows // 128) * 4 * C // 256
    rounds = -(-tiles // sms)
    pays = C <= 1024 and (rounds >= 4 or tiles >= 0.8 * rounds * sms)
    assert bool(lib.vrwkv_linear_relu_square_pays(rows, C, 4 * C)) == pays

    def run():
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            before = lib.vrwkv_launch_count()
            out = epilogue.linear_relu_square(key, x, value)
            assert lib.vrwkv_launch_count() == before + 1
            return out

    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        by_torch, by_one = epilogue.relu_square(key(x), value), _lib.native().linear_relu_square(x, key.weight)
    assert torch.equal(run(), by_one if pays or (C <= 1024 and rows * 4 * C <= 128 * 128 * 256) else by_torch)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = run()
    graph.replay()
    assert torch.equal(captured, by_one if pays else by_torch)


def withheld_inputs(dev):
    """Three tiles to a CTA, so that an epilogue's missing arrival is waited for too; K of more slices than stages."""
    g = torch.Generator(device=dev).manual_seed(1)
    rows = 128 * torch.cuda.get_device_properties(dev).multi_processor_count
    return torch.randn(rows, 384, device=dev, generator=g).bfloat16(), torch.randn(768, 384, device=dev, generator=g).bfloat16() / 20


def test_bounded_waits_run_out_and_report(cuda_device):
    """Path 3: in every third CTA the loader, in every third the issuer, in every third the epilogue leaves out what the others wait for."""
    from vision_rwkv_b200 import _lib, epilogue, ops
    lib, native = _lib.load(), _lib.native()
    x, w = withheld_inputs(cuda_device)
    key, value = torch.nn.Linear(384, 768, bias=False, device=cuda_device), torch.nn.Linear(768, 384, bias=False, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = native.linear_relu_square(x, w)
        try:
            assert lib.vrwkv_set_path(3) == 0
            native.linear_relu_square(x, w)
            with pytest.raises(_lib.VrwkvError, match="earlier launch, linear:"):
                ops.raise_if_failed()
            native.linear_relu_square(x, w)
            torch.cuda.synchronize()
            with pytest.raises(_lib.VrwkvError, match="earlier launch, linear:"):
                native.linear_relu_square(x, w)
            torch.cuda.synchronize()
            lib.vrwkv_take_failures(torch.cuda.current_device())
            ops.CHECK_STATUS = True
            with pytest.raises(_lib.VrwkvError, match="linear:"):
                epilogue.linear_relu_square(key, x, value)
        finally:
            ops.CHECK_STATUS = False
            lib.vrwkv_set_path(0)
        ops.raise_if_failed()
        # the context is intact and the next call is right again
        assert torch.equal(native.linear_relu_square(x, w), want)
        ops.raise_if_failed()


def test_a_process_that_calls_nothing_else_hears_of_it(cuda_device):
    import os
    import subprocess
    import sys
    # the library as a C program has it: vrwkv_take_failures (which _lib.load calls) comes after the launch
    code = ("import ctypes, torch, tests.test_linear_gpu as t\nfrom vision_rwkv_b200 import _lib\nlib = ctypes.CDLL(_lib.LIB_PATH)\n"
            "for n in ('vrwkv_set_path', 'vrwkv_linear_relu_square', 'vrwkv_take_failures'):\n    getattr(lib, n).restype, getattr(lib, n).argtypes = _lib.SIGNATURES[n]\n"
            "x, w = t.withheld_inputs(torch.device('cuda'))\nout = torch.empty(x.shape[0], w.shape[0], device='cuda', dtype=torch.bfloat16)\n"
            "lib.vrwkv_set_path(3)\n"
            "assert lib.vrwkv_linear_relu_square(x.shape[0], 384, 768, x.data_ptr(), w.data_ptr(), out.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0\n"
            "torch.cuda.synchronize()\nassert lib.vrwkv_take_failures(0) == 1 | 1 << 12\nassert lib.vrwkv_take_failures(0) == 0\n")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    subprocess.run([sys.executable, "-c", code], check=True, cwd=root, timeout=300)
