"""The weights of a mixer cast to bfloat16 in one launch: the bits of the casts that autocast makes, and the calls that are left to autocast."""
import pytest
import torch

from vision_rwkv_b200 import _lib, backbone, backbone6, epilogue

pytestmark = pytest.mark.gpu


# one block of the kernel takes 8192 values: around it, and arrays that are not 16-byte aligned
@pytest.mark.parametrize("sizes,offset", [((1,), 0), ((8192,), 0), ((8191, 8193), 0), ((7, 24576, 100000), 0), ((8192, 16384), 1), ((4096,) * 16, 0)])
def test_rounds_as_torch_does(cuda_device, sizes, offset):
    g = torch.Generator(device=cuda_device).manual_seed(len(sizes))
    arrays = []
    for n in sizes:
        bits = torch.randint(-2 ** 31, 2 ** 31, (n + offset,), device=cuda_device, generator=g).int()      # NaN, infinities, subnormals among them
        arrays.append(bits.view(torch.float32)[offset:])
    got = _lib.native().narrow(arrays)
    for a, b in zip(arrays, got):
        want = a.bfloat16()
        assert torch.equal(b.isnan(), want.isnan())
        assert torch.equal(b.nan_to_num().view(torch.int16), want.nan_to_num().view(torch.int16))


def networks(device):
    torch.manual_seed(0)
    for build, mod in ((lambda: backbone.VRWKV(img_size=64, embed_dims=192, depth=2, init_values=1.0, post_norm=True), backbone),
                       (lambda: backbone.VRWKV(img_size=64, embed_dims=64, depth=2, key_norm=True), backbone),
                       (lambda: backbone6.VRWKV6(img_size=64, embed_dims=128, num_heads=2, depth=2), backbone6)):
        yield build().to(device).eval()


@pytest.fixture
def casts(monkeypatch):
    """how often weights were cast together"""
    count, own = [0], epilogue.weights_for

    def counting(*args):
        got = own(*args)
        count[0] += got is not None
        return got
    monkeypatch.setattr(epilogue, "weights_for", counting)
    return count


def test_networks_keep_their_bits(cuda_device, casts, monkeypatch):
    img = torch.randn(2, 3, 64, 64, device=cuda_device)
    for model in networks(cuda_device):
        def run():
            return model(img)[0]
        with monkeypatch.context() as m, torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            m.setattr(epilogue, "weights_for", lambda *args: None)
            want = run()
        casts[0] = 0
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            for calls in (4, 4, 4):          # a context that is held: the second call has autocast cast, the third finds the copies
                assert torch.equal(run(), want) and casts[0] == calls
        for n in (8, 12):                    # each context on its own
            with torch.inference_mode(n == 12), torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
                assert torch.equal(run(), want) and casts[0] == n
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16, cache_enabled=False):
            for n in (16, 20):
                assert torch.equal(run(), want) and casts[0] == n
        model.requires_grad_(False)
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            for n in (24, 28):
                assert torch.equal(run(), want) and casts[0] == n
        model.requires_grad_(True)
        with torch.no_grad():                # changed weights are seen by the next context
            model.layers[0].att.key.weight.mul_(1.5)
        with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
            assert not torch.equal(run(), want)


def test_calls_that_somebody_would_see_are_left_alone(cuda_device, casts):
    model, img, seen = next(networks(cuda_device)), torch.randn(1, 3, 64, 64, device=cuda_device), []
    model.layers[0].att.output.register_forward_hook(lambda *args: seen.append(1))
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        model(img)
    assert seen == [1] and casts[0] == 3     # the other mixers'
    with torch.no_grad():
        model(img)
    assert casts[0] == 3                     # float32
    with torch.autocast("cuda", torch.bfloat16):
        model(img)[0].float().sum().backward()
    assert casts[0] == 3 and model.layers[1].ffn.key.weight.grad is not None


@pytest.mark.parametrize("warm", [1, 3])
def test_captured_in_a_held_context(cuda_device, warm):
    """A captured call's casts run with the replays alone; eager calls before and after it have their own."""
    model, img = next(networks(cuda_device)), torch.randn(2, 3, 64, 64, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        for _ in range(warm):
            want = model(img)[0].clone()
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=side):
                out = model(img)[0]
        torch.cuda.current_stream().wait_stream(side)
        assert torch.equal(model(img)[0], want)
        graph.replay()
        assert torch.equal(out, want) and torch.equal(model(img)[0], want)


def mixer(device):
    """four layers and an input for `weights_for`"""
    return [torch.nn.Linear(64, 64, bias=False, device=device, dtype=torch.float32) for _ in range(4)], torch.randn(2, 8, 64, device=device, dtype=torch.float32)


@pytest.mark.parametrize("default", [torch.float64, torch.bfloat16, torch.float16])
def test_the_count_ends_with_autocasts_copies_whatever_the_default_type_is(cuda_device, monkeypatch, default):
    layers, x = mixer(cuda_device)
    monkeypatch.setattr(epilogue, "_NOTHING", {})      # as at a process's first call
    before = torch.get_default_dtype()
    try:
        torch.set_default_dtype(default)
        for _ in range(4):
            with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
                assert epilogue.weights_for(layers[0], x, *layers) is not None
    finally:
        torch.set_default_dtype(before)


def test_the_count_is_of_the_owner_and_not_of_its_address(cuda_device):
    class Owner:
        pass
    layers, x = mixer(cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        owner = Owner()
        for cast in (True, False, False):
            assert (epilogue.weights_for(owner, x, *layers) is not None) == cast
        address = id(owner)
        del owner
        others = [Owner() for _ in range(1000)]
        again = [o for o in others if id(o) == address]
        assert again and epilogue.weights_for(again[0], x, *layers) is not None


def test_a_mode_sees_the_operations_of_layers_only(cuda_device):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.extend(a for a in args if isinstance(a, torch.Tensor) and a.numel() == 0)
            return func(*args, **(kwargs or {}))
    layers, x = mixer(cuda_device)
    seen = []
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16), Watch():
        assert epilogue.weights_for(layers[0], x, *layers) is None
        [layer(x) for layer in layers]
    assert not seen
    casts = []
    with pytest.MonkeyPatch.context() as m, torch.no_grad(), torch.autocast("cuda", torch.float16):
        native = _lib.native()

        class Native:
            def __getattr__(self, name):
                casts.append(name)
                return getattr(native, name)
        m.setattr(_lib, "native", Native)
        assert epilogue.weights_for(layers[0], x, *layers) is None
    assert not casts
