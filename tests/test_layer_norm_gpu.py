"""The plain LayerNorm of the networks in inference, against float64: float32 sums over up to 1024 channels, 1e-6 in the 2-norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,C", [(1, 4), (7, 128), (9, 132), (1000, 384), (33, 1024)])
def test_against_float64(cuda_device, rows, C):
    from vision_rwkv_b200 import epilogue, launch_count
    norm = torch.nn.LayerNorm(C, device=cuda_device)
    torch.nn.init.normal_(norm.weight)
    torch.nn.init.normal_(norm.bias)
    x = torch.randn(rows, C, device=cuda_device) * 3 + 5
    with torch.no_grad():
        before = launch_count()
        got = epilogue.layer_norm(norm, x)
        assert launch_count() == before + 1
        ref = torch.nn.functional.layer_norm(x.double(), (C,), norm.weight.double(), norm.bias.double(), norm.eps)
        assert ((got - ref).norm() / ref.norm()).item() <= 1e-6
        # a hook, another type and gradients keep the layer's call
        seen = []
        hook = norm.register_forward_hook(lambda *a: seen.append(1))
        epilogue.layer_norm(norm, x)
        hook.remove()
        assert seen == [1] and launch_count() == before + 1
    assert epilogue.layer_norm(norm, x).requires_grad


@pytest.mark.parametrize("n", [8, 2048, 2056, 12544 * 768])
def test_a_widened_input_is_torchs_cast(cuda_device, n):
    from vision_rwkv_b200 import epilogue, launch_count
    norm = torch.nn.LayerNorm(8, device=cuda_device)
    a = torch.randn(n // 8, 8, device=cuda_device).bfloat16()
    a.view(-1)[:3] = torch.tensor([float("nan"), float("-inf"), -0.0])
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        before = launch_count()
        got = epilogue.widened(norm, a)
        assert launch_count() == before + 1 and got.dtype == torch.float32
        assert torch.equal(got.view(torch.int32), a.float().view(torch.int32))
        assert epilogue.widened(norm, a[:, :5]).dtype == torch.bfloat16
        assert epilogue.widened(torch.nn.GroupNorm(8, 8), a) is a
    assert epilogue.widened(norm, a) is a       # no autocast: the layer refuses or takes it as it is


@pytest.mark.parametrize("C", [192, 384, 768, 1024])
@pytest.mark.parametrize("mean", [3.0, 100.0])
def test_rows_with_a_mean_are_no_further_from_float64_than_torchs_layer(cuda_device, C, mean):
    """4096 rows: the two errors, each an average over millions of roundings, repeat to a few percent; a tenth covers that."""
    from vision_rwkv_b200 import epilogue
    norm = torch.nn.LayerNorm(C, device=cuda_device)
    x = torch.randn(4096, C, device=cuda_device, generator=torch.Generator(device=cuda_device).manual_seed(C)) + mean
    with torch.no_grad():
        ref = torch.nn.functional.layer_norm(x.double(), (C,), eps=norm.eps)
        error = [((y - ref).norm() / ref.norm()).item() for y in (epilogue.layer_norm(norm, x), norm(x))]
    assert error[0] <= 1.1 * error[1], error
