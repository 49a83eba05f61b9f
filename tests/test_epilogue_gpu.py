"""The inference steps between a block's matrix products (epilogue.py) against the tensor operations they stand for, which
run under autograd (`torch.enable_grad`) in the same functions."""
import pytest
import torch
import torch.nn as nn
import torch.utils._python_dispatch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def normal(dev, *shape, dtype=torch.float32, seed=0):
    return torch.randn(*shape, generator=torch.Generator().manual_seed(seed)).to(dev, dtype)


def both(fn):
    """fn through the kernel and through the tensor operations"""
    from vision_rwkv_b200 import _lib
    lib = _lib.load()
    with torch.no_grad():
        before = lib.vrwkv_launch_count()
        fast = fn()
        assert lib.vrwkv_launch_count() > before
    with torch.enable_grad():
        return fast, fn()


# one element, fewer than a thread's eight, one block (2048) and one over, and a ragged tail
@pytest.mark.parametrize("n", [1, 7, 2048, 2049, 40003])
@pytest.mark.parametrize("r_type,y_type", [(torch.float32, torch.float32), (torch.bfloat16, torch.float32), (torch.bfloat16, torch.bfloat16)])
def test_elementwise_steps(cuda_device, n, r_type, y_type):
    from vision_rwkv_b200 import epilogue
    r, y = normal(cuda_device, n, dtype=r_type, seed=n) * 4, normal(cuda_device, n, dtype=y_type, seed=n + 1)
    a, b = both(lambda: epilogue.sigmoid_gate(r, y))
    # the same roundings; the two compilations of the sigmoid may differ in a last float32 bit
    assert a.dtype == r_type and a.isfinite().all()
    assert rel_err(a.float(), b.double()) < (1e-2 if r_type == torch.bfloat16 else 1e-6)
    if r_type == torch.bfloat16:
        assert (a != b).float().mean().item() < 1e-3 + 1.0 / n
    for special in (float("nan"), float("inf"), -float("inf")):
        r[n // 2] = special
        a, b = both(lambda: epilogue.relu_square(r))
        assert a.dtype == r_type and torch.equal(a.isnan(), b.isnan()) and torch.equal(a.nan_to_num(), b.nan_to_num())


@pytest.mark.parametrize("n", [1, 7, 2048, 2049])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("autocast", [torch.bfloat16, torch.float16])
def test_squares_under_autocast_have_the_chains_type(cuda_device, n, dtype, autocast):
    """torch squares in float32 there; only a linear layer that would round to bfloat16 first may be given bfloat16."""
    from vision_rwkv_b200 import epilogue
    x, layer = normal(cuda_device, n, dtype=dtype, seed=n) * 4, nn.Linear(4, 4)
    with torch.autocast("cuda", autocast):
        a, b = both(lambda: epilogue.relu_square(x))
        assert a.dtype == b.dtype == torch.float32 and torch.equal(a, b)
        a, b = both(lambda: epilogue.relu_square(x, layer))
        assert torch.equal(a.to(autocast), b.to(autocast))
        assert a.dtype == (torch.bfloat16 if dtype == autocast == torch.bfloat16 else torch.float32)
        layer.register_forward_pre_hook(lambda *args: None)
        assert both(lambda: epilogue.relu_square(x, layer))[0].dtype == torch.float32


@pytest.mark.parametrize("version", [4, 6])
def test_a_norm_behind_the_square_takes_it_in_float32(cuda_device, version):
    from vision_rwkv_b200 import backbone, backbone6
    mix = (backbone6.ChannelMixV6 if version == 6 else backbone.ChannelMix)(128, 2, 0, key_norm=True).to(cuda_device)
    for p in mix.parameters():
        torch.nn.init.normal_(p, std=0.1)
    seen, x = [], normal(cuda_device, 2, 16, 128)
    mix.key_norm.register_forward_pre_hook(lambda m, args: seen.append(args[0]))
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        mix(x, (4, 4))
    with torch.autocast("cuda", torch.bfloat16):
        mix(x, (4, 4))
    assert seen[0].dtype == seen[1].dtype == torch.float32 and torch.equal(seen[0], seen[1])


# a row in one lane, a row that fills 128 channels, one vector more, the model widths, the widest
@pytest.mark.parametrize("rows,C", [(1, 4), (9, 128), (17, 132), (200, 192), (33, 768), (8, 1024)])
@pytest.mark.parametrize("a_type", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("scaled", [True, False])
def test_residual_steps(cuda_device, rows, C, a_type, scaled):
    from vision_rwkv_b200 import epilogue
    x, a = normal(cuda_device, rows, C, seed=C), normal(cuda_device, rows, C, dtype=a_type, seed=rows) * 3 + 1
    gamma = normal(cuda_device, C, seed=3) if scaled else None
    norm = nn.LayerNorm(C).to(cuda_device)
    norm.weight.data.copy_(normal(cuda_device, C, seed=4))
    norm.bias.data.copy_(normal(cuda_device, C, seed=5))
    fast, chain = both(lambda: epilogue.residual(x, a, gamma))
    assert torch.equal(fast, chain)
    with torch.autocast("cuda", torch.bfloat16):
        fast, chain = both(lambda: epilogue.norm_residual(x, a, norm, gamma))
    assert fast.dtype == chain.dtype == torch.float32
    want = nn.functional.layer_norm(a.double(), (C,), norm.weight.double(), norm.bias.double(), norm.eps)
    want = x.double() + (want if gamma is None else gamma.double() * want)
    assert rel_err(fast, want.detach()) < 1e-6 and rel_err(chain.detach(), want.detach()) < 1e-6


def test_layers_that_are_not_stock_keep_their_calls(cuda_device):
    from vision_rwkv_b200 import epilogue
    x, a, seen = normal(cuda_device, 4, 64), normal(cuda_device, 4, 64, seed=1), []
    norm = nn.LayerNorm(64).to(cuda_device)
    norm.register_forward_hook(lambda *args: seen.append(1))
    with torch.no_grad():
        epilogue.norm_residual(x, a, norm, None)
        epilogue.norm_residual(x.half(), a.half(), nn.LayerNorm(64).to(cuda_device).half(), None)
        wide = normal(cuda_device, 3, 1028)
        epilogue.norm_residual(wide, wide, nn.LayerNorm(1028).to(cuda_device), None)
    assert seen == [1]


def all_modules_hook(fn):
    return nn.modules.module.register_module_forward_hook(lambda *args: fn())


def all_modules_pre_hook(fn):
    return nn.modules.module.register_module_forward_pre_hook(lambda *args: fn())


def own_forward(fn):
    def watch(module):
        plain = module.forward
        module.forward = lambda *args: (fn(), plain(*args))[1]
    return watch


@pytest.mark.parametrize("watch", [all_modules_hook, all_modules_pre_hook, own_forward])
def test_watched_layers_keep_their_calls(cuda_device, watch):
    """Hooks for all modules and a replaced forward see the call of every layer whose work a kernel can take over."""
    from vision_rwkv_b200 import epilogue
    from vision_rwkv_b200.qshift import feeds_autocast_linears
    x, a, img = normal(cuda_device, 4, 64), normal(cuda_device, 4, 64, seed=1), normal(cuda_device, 1, 3, 32, 32)
    norm, conv, layer = nn.LayerNorm(64).to(cuda_device), nn.Conv2d(3, 64, 16, stride=16).to(cuda_device), nn.Linear(64, 64).to(cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        assert epilogue.patch_embedding(img, conv) is not None and feeds_autocast_linears(x, layer)
        seen, handle = [], None
        if watch is own_forward:
            for m in (norm, conv, layer):
                own_forward(lambda: seen.append(1))(m)
        else:
            handle = watch(lambda: seen.append(1))
        try:
            epilogue.norm_residual(x, a, norm, None)
            assert seen == [1]
            assert epilogue.patch_embedding(img, conv) is None and not feeds_autocast_linears(x, layer)
        finally:
            if handle is not None:
                handle.remove()


# a part of one block, exactly one block (64 heads), one head more, odd numbers of heads per row
@pytest.mark.parametrize("rows,C", [(1, 64), (64, 64), (65, 64), (7, 192), (196, 768)])
@pytest.mark.parametrize("gate_type", [torch.float32, torch.bfloat16])
def test_head_norm_gate_is_the_float32_result_rounded(cuda_device, rows, C, gate_type):
    from vision_rwkv_b200 import epilogue
    x, gate = normal(cuda_device, 1, rows, C, seed=C) * 2 + 0.5, normal(cuda_device, 1, rows, C, dtype=gate_type, seed=rows)
    norm, layer = nn.GroupNorm(C // 64, C).to(cuda_device), nn.Linear(C, 8).to(cuda_device)
    norm.weight.data.copy_(normal(cuda_device, C, seed=4))
    norm.bias.data.copy_(normal(cuda_device, C, seed=5))
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        half = epilogue.head_norm_gate(x, gate, norm, 64, layer, "silu")
    with torch.no_grad():
        wide = epilogue.head_norm_gate(x, gate, norm, 64, layer, "silu")
    assert half.dtype == torch.bfloat16 and wide.dtype == torch.float32
    assert torch.equal(half, wide.bfloat16())


# one vector, one block of vectors (2048 elements) and more, tables of one row and of several
@pytest.mark.parametrize("shape,table", [((1, 1, 8), (1, 1, 8)), ((2, 128, 8), (1, 1, 8)), ((3, 50, 192), (1, 1, 192)), ((5, 49, 40), (1, 49, 40)),
                                         ((2, 9, 12), (1, 1, 12)), ((1, 7, 64), (1, 1, 64))])
def test_add_rows(cuda_device, shape, table):
    from vision_rwkv_b200 import epilogue
    t, a = normal(cuda_device, *table, seed=1), normal(cuda_device, *shape, dtype=torch.bfloat16, seed=2)
    with torch.no_grad():
        out = epilogue.add_rows(t, a)
    assert out.dtype == torch.float32 and torch.equal(out, t + a)
    with pytest.raises(RuntimeError):
        epilogue.add_rows(t[..., :-1], a)


# a single patch, patches of 8 pixels, sides that leave pixels over, widths that only the convolution takes
@pytest.mark.parametrize("B,channels,H,W,patch", [(1, 3, 16, 16, 16), (2, 3, 40, 72, 16), (3, 1, 24, 20, 8), (2, 3, 35, 47, 16), (1, 3, 224, 224, 16)])
def test_patch_embedding(cuda_device, B, channels, H, W, patch):
    from vision_rwkv_b200 import epilogue
    img, conv = normal(cuda_device, B, channels, H, W, seed=H), nn.Conv2d(channels, 24, patch, stride=patch).to(cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        tokens = epilogue.patch_embedding(img, conv)
        by_conv = conv(img)
    if W % 4:
        assert tokens is None
        return
    want = nn.functional.conv2d(img.bfloat16().double(), conv.weight.bfloat16().double(), conv.bias.bfloat16().double(), stride=patch)
    want = want.flatten(2).transpose(1, 2).detach()
    assert tokens.dtype == torch.bfloat16 and tokens.shape == want.shape
    # a rounding to bfloat16 moves an element by up to 2^-8 of it; both round before and behind the bias (which may make
    # the first of the two a little larger than the result)
    bound = 2 * 2.0 ** -8 * 1.25
    assert rel_err(tokens.double(), want) < bound and rel_err(by_conv.flatten(2).transpose(1, 2).double(), want) < bound
    with torch.no_grad():
        assert epilogue.patch_embedding(img, conv) is None                       # float32 networks keep the convolution


class Seen(torch.overrides.TorchFunctionMode):
    def __init__(self):
        self.names = []

    def __torch_function__(self, func, types, args=(), kwargs=None):
        self.names.append(getattr(func, "__name__", ""))
        return func(*args, **(kwargs or {}))


class Dispatched(torch.utils._python_dispatch.TorchDispatchMode):
    def __init__(self):
        super().__init__()
        self.products = []

    def __torch_dispatch__(self, func, types, args=(), kwargs=None):
        if "mm" in func.__name__:
            a, b = args[-2:]
            self.products.append((a.shape[0], a.shape[1], b.shape[1]))
        return func(*args, **(kwargs or {}))


class Wrapped(torch.Tensor):
    pass


def test_layers_are_called_where_a_mode_or_a_tensor_subclass_would_see_it(cuda_device):
    """What a dispatch mode (a FLOP counter that knows no modules, say), a function mode or a tensor subclass sees are the layers' own
    operations: key, value and receptance of a channel mix, its norms."""
    from vision_rwkv_b200 import backbone, epilogue, launch_count
    C, rows = 192, 20000
    mix = backbone.ChannelMix(C, 4, 0).to(cuda_device).eval()
    norm = nn.LayerNorm(C, device=cuda_device)
    x = torch.randn(1, rows, C, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        with Dispatched() as counter:
            watched = mix(x, (125, 160))
        assert sorted(counter.products) == sorted([(rows, C, 4 * C), (rows, 4 * C, C), (rows, C, C)])
        with Seen() as seen:
            normed = epilogue.layer_norm(norm, x)
            widened = epilogue.widened(norm, x.bfloat16())
            mix(x, (125, 160))
        assert seen.names.count("linear") == 3 and "layer_norm" in seen.names and widened.dtype == torch.bfloat16
        assert type(epilogue.layer_norm(norm, x.as_subclass(Wrapped))) is Wrapped
        norm.weight = nn.Parameter(norm.weight.detach().as_subclass(Wrapped))
        before = launch_count()
        epilogue.layer_norm(norm, x)
        assert launch_count() == before
        norm.weight = nn.Parameter(torch.ones(C, device=cuda_device))
        with torch.device(cuda_device):      # a default device is a mode that watches nothing
            assert torch.equal(epilogue.layer_norm(norm, x), epilogue.layer_norm(norm, x)) and launch_count() == before + 2
        assert ((epilogue.layer_norm(norm, x) - normed).norm() / normed.norm()).item() <= 1e-6
        assert ((mix(x, (125, 160)).float() - watched.float()).norm() / watched.float().norm()).item() <= 1e-2


def test_the_gate_rounds_every_bfloat16_sigmoid_as_its_float64_value(cuda_device):
    """All 65536 bfloat16 r: the result is within half a unit of the last place of the float64 sigmoid, but for the approximation's 2^-20
    (and absolutely below bfloat16's smallest normal number)."""
    from vision_rwkv_b200 import _lib
    r = torch.arange(65536, device=cuda_device, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    got = _lib.native().sigmoid_gate(r, torch.ones_like(r), False).double()
    want = torch.sigmoid(r.double())
    assert torch.equal(got.isnan(), r.isnan())
    ok = ~r.isnan()
    unit = torch.exp2(torch.floor(torch.log2(want[ok].clamp_min(2.0 ** -126))) - 7)
    # below e^-88.7 the exponential is infinite in float32 and the sigmoid zero
    assert ((got[ok] - want[ok]).abs() <= 0.5 * unit + 2.0 ** -20 * want[ok] + 2.0 ** -127).all()


@pytest.mark.parametrize("wide", [False, True])
def test_the_gate_has_the_bits_of_the_float32_sigmoid(cuda_device, wide):
    """All 65536 bfloat16 r: the approximate exponential and reciprocal round to what 1 / (1 + exp(-r)) in float32 rounds to."""
    from vision_rwkv_b200 import _lib
    r = torch.arange(65536, device=cuda_device, dtype=torch.int32).to(torch.int16).view(torch.bfloat16)
    want = (1 / (1 + torch.exp(-r.float()))).bfloat16()
    got = _lib.native().sigmoid_gate(r, torch.ones_like(r), wide).bfloat16()      # widened bfloat16: exact
    assert torch.equal(got.isnan(), want.isnan())
    assert torch.equal(got.nan_to_num().view(torch.int16), want.nan_to_num().view(torch.int16))
    norm_in = torch.zeros(64, 1024, device=cuda_device)
    gated = _lib.native().gated_norm_residual(norm_in, r.view(64, 1024), torch.ones_like(r).view(64, 1024), None, None, None, 0.0).view(-1)
    assert torch.equal(gated.nan_to_num(), want.float().nan_to_num())
