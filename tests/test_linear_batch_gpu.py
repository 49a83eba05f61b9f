"""Several linear layers in one launch (and the key layer of the same kernel): against the products in float64, rounded where autocast
rounds.  A float32 sum of up to 384 products of size 1 is off by 1e-5 and may round to the neighbouring bfloat16 number, 2^-7 of it at most
(with its own rounding 2^-8 of that); few do, so 1e-2 in the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# rows around a tile's 128, fewer and more tiles than CTAs to a slab; depths of one slice, of both kinds of stages, of the most; one to eight slabs
@pytest.mark.parametrize("count,rows,K,N", [(3, 1, 64, 192), (4, 127, 192, 192), (3, 128, 256, 384), (4, 129, 320, 192), (3, 19008, 384, 384), (4, 6272, 384, 384),
                                            (3, 40001, 192, 192), (3, 777, 384, 1536), (4, 300, 128, 960),
                                            # by tiles of 128 x 256: deeper, or columns that are no slabs
                                            (3, 1, 448, 256), (4, 129, 768, 768), (3, 12544, 768, 768), (4, 128, 1024, 512), (3, 300, 64, 256)])
def test_against_float64(cuda_device, count, rows, K, N):
    from vision_rwkv_b200 import _lib
    lib = _lib.load()
    g = torch.Generator(device=cuda_device).manual_seed(rows + K)
    xs = [torch.randn(rows, K, device=cuda_device, generator=g).bfloat16() for _ in range(count)]
    ws = [(torch.randn(N, K, device=cuda_device, generator=g) / K ** 0.5).bfloat16() for _ in range(count)]
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        before = lib.vrwkv_launch_count()
        outs = _lib.native().linear_batch(xs, ws)
        assert lib.vrwkv_launch_count() == before + 1
    for x, w, out in zip(xs, ws, outs):
        ref = x.double() @ w.double().T
        assert out.shape == (rows, N) and out.dtype == torch.bfloat16
        assert ((out.double() - ref.bfloat16().double()).norm() / ref.norm()).item() <= 1e-2
        assert ((out.double() - ref).abs() <= (2.0 ** -7 + 2.0 ** -8) * ref.abs() + 1e-5).all()


def test_layers_of_one_shape_give_the_products_of_each(cuda_device):
    """Through `epilogue.linears`: one launch for three or four layers on bfloat16 rows; else each layer's own call."""
    from vision_rwkv_b200 import epilogue, launch_count
    layers = [torch.nn.Linear(384, 384, bias=False, device=cuda_device) for _ in range(4)]
    xs = [torch.randn(2, 500, 384, device=cuda_device).bfloat16() for _ in range(4)]
    odd = torch.empty(384000 + 1, device=cuda_device, dtype=torch.bfloat16)[1:].view(2, 500, 384).copy_(xs[1])      # 2-byte aligned
    biased = torch.nn.Linear(384, 384, device=cuda_device)
    wide = torch.nn.Linear(384, 768, bias=False, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = [layer(x) for layer, x in zip(layers, xs)]
        for n, launches in ((4, 1), (3, 1), (2, 0), (1, 0)):
            before = launch_count()
            got = epilogue.linears(layers[:n], xs[:n])
            assert launch_count() == before + launches
            for a, b in zip(got, want):
                assert ((a.float() - b.float()).norm() / b.float().norm()).item() <= 5e-3      # sums in another order: some roundings differ
        assert torch.equal(epilogue.linears(layers, [xs[0], odd, *xs[2:]])[1], epilogue.linears(layers, xs)[1])
        for others, inputs in (([*layers[:2], biased], xs[:3]), ([*layers[:2], wide], xs[:3]), (layers[:3], [xs[0].float(), *xs[1:3]]),
                               (layers[:3], [xs[0], xs[1], xs[2][:, :100]])):
            before = launch_count()
            got = epilogue.linears(others, inputs)
            assert launch_count() == before and all(torch.equal(a, layer(x)) for a, layer, x in zip(got, others, inputs))
        seen = []
        hook = layers[2].register_forward_hook(lambda *a: seen.append(1))
        before = launch_count()
        epilogue.linears(layers, xs)
        assert seen == [1] and launch_count() == before
        hook.remove()
    with torch.autocast("cuda", torch.bfloat16):      # gradients are wanted: the layers' own graph
        assert all(y.requires_grad for y in epilogue.linears(layers, xs))


def test_not_a_number_stays(cuda_device):
    from vision_rwkv_b200 import _lib
    x = torch.ones(130, 64, device=cuda_device).bfloat16()
    x[129, 3] = float("nan")
    x[5, 1] = float("inf")
    w = torch.ones(192, 64, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        for out in _lib.native().linear_batch([x] * 3, [w] * 3):
            assert out[129].isnan().all() and out[5].isinf().all() and (out[6] == 64).all()


@pytest.mark.parametrize("K,N", [(384, 192), (512, 256), (192, 192)])
def test_bounded_waits_run_out_and_report(cuda_device, K, N):
    """Path 3: in every third CTA the loader, in every third the issuer, in every third the epilogue leaves out what the others wait for."""
    from vision_rwkv_b200 import _lib, ops
    lib, native = _lib.load(), _lib.native()
    rows = 128 * torch.cuda.get_device_properties(cuda_device).multi_processor_count      # three tiles to a CTA
    x = torch.randn(rows, K, device=cuda_device).bfloat16()
    w = torch.randn(N, K, device=cuda_device).bfloat16() / 20
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = native.linear_batch([x] * 3, [w] * 3)
        try:
            assert lib.vrwkv_set_path(3) == 0
            native.linear_batch([x] * 3, [w] * 3)
            with pytest.raises(_lib.VrwkvError, match="earlier launch, linear:"):
                ops.raise_if_failed()
        finally:
            lib.vrwkv_set_path(0)
        ops.raise_if_failed()
        assert all(torch.equal(a, b) for a, b in zip(native.linear_batch([x] * 3, [w] * 3), want))
        ops.raise_if_failed()


@pytest.mark.parametrize("K,N", [(64, 768), (192, 768), (256, 768)])
def test_bounded_waits_of_the_key_layer_by_slabs(cuda_device, K, N):
    """The same with the squared ReLU, four tiles to a CTA."""
    from vision_rwkv_b200 import _lib, ops
    lib, native = _lib.load(), _lib.native()
    x = torch.randn(128 * torch.cuda.get_device_properties(cuda_device).multi_processor_count, K, device=cuda_device).bfloat16()
    w = torch.randn(N, K, device=cuda_device).bfloat16() / 20
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        want = native.linear_relu_square(x, w)
        try:
            assert lib.vrwkv_set_path(3) == 0
            native.linear_relu_square(x, w)
            with pytest.raises(_lib.VrwkvError, match="earlier launch, linear:"):
                ops.raise_if_failed()
        finally:
            lib.vrwkv_set_path(0)
        ops.raise_if_failed()
        assert torch.equal(native.linear_relu_square(x, w), want)
        ops.raise_if_failed()
