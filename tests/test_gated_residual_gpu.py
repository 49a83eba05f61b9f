"""Inference: the channel mix's gate taken together with the residual (and its norm), or leaving in float32 for a norm, gives the
bits of the separate steps."""
import pytest
import torch
import torch.nn as nn

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,C", [(1, 4), (3, 128), (33, 132), (7, 384), (9, 1020), (5, 1024)])
@pytest.mark.parametrize("normed", [False, True])
@pytest.mark.parametrize("scaled", [False, True])
def test_same_bits_as_gate_then_residual(cuda_device, rows, C, normed, scaled):
    from vision_rwkv_b200 import epilogue, launch_count
    g = torch.Generator(device=cuda_device).manual_seed(rows * C)
    x = torch.randn(1, rows, C, device=cuda_device, generator=g)
    r, y = (torch.randn(1, rows, C, device=cuda_device, generator=g).bfloat16() * 3 for _ in range(2))
    r[0, 0, :2] = torch.tensor([float("-inf"), 90.0], device=cuda_device)
    gamma = torch.randn(C, device=cuda_device, generator=g) if scaled else None
    norm = None
    if normed:
        norm = nn.LayerNorm(C, device=cuda_device)
        nn.init.normal_(norm.weight)
        nn.init.normal_(norm.bias)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        a = epilogue.sigmoid_gate(r, y)
        want = epilogue.norm_residual(x, a, norm, gamma) if normed else epilogue.residual(x, a, gamma)
        before = launch_count()
        got = epilogue.gated_residual(x, r, y, norm, gamma)
        assert launch_count() == before + 1
        assert torch.equal(got, want)
        if normed:
            wide = epilogue.sigmoid_gate(r, y, norm=norm)
            assert wide.dtype == torch.float32 and torch.equal(wide, a.float()) and torch.equal(norm(wide), norm(a))
        odd = torch.empty(x.numel() + 1, device=cuda_device, dtype=torch.bfloat16)[1:].view_as(r).copy_(r)      # 2-byte aligned
        assert torch.equal(epilogue.gated_residual(x, odd, y, norm, gamma), want)


@pytest.mark.parametrize("name,overrides", [("vrwkv_t", {}), ("vrwkv_t", dict(post_norm=False)), ("vrwkv6_t", {}),
                                            ("vrwkv6_t", dict(post_norm=True, init_values=1.0))])
def test_networks_keep_their_bits_and_their_hooks(cuda_device, monkeypatch, name, overrides):
    from vision_rwkv_b200 import backbone, backbone6, epilogue, launch_count
    torch.manual_seed(3)
    build = backbone6.build_v6 if "6" in name else backbone.build
    model = build(name, img_size=64, depth=2, **overrides).to(cuda_device).eval()
    img = torch.randn(2, 3, 64, 64, device=cuda_device)
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        gates, gate = [], epilogue.sigmoid_gate
        monkeypatch.setattr(epilogue, "sigmoid_gate", lambda r, y, norm=None: (gates.append(norm), gate(r, y, norm))[1])
        before = launch_count()
        fused = model(img)[0]
        launches, widened, seen = launch_count() - before, [g for g in gates if g is not None], []
        handles = [layer.ffn.register_forward_hook(lambda m, i, o: seen.append(o.dtype)) for layer in model.layers]
        before = launch_count()
        stepwise = model(img)[0]
        assert seen == [torch.bfloat16] * 2 and torch.equal(fused, stepwise)
        # the fused pass took the gate with the residual, one launch less per layer, or (matrix-state, post-norm) widened it for the norm
        if "6" in name and overrides.get("post_norm"):
            assert widened == [layer.ln2 for layer in model.layers] and launch_count() - before == launches
        else:
            assert not widened and launch_count() - before == launches + 2
        for h in handles:
            h.remove()
