"""Inference takes over the work of a layer only while calling that layer would run the forward it was written with: one that is
replaced on its class, or compiled in place, is called."""
import pytest
import torch
import torch.nn as nn

from vision_rwkv_b200 import backbone, backbone6
from vision_rwkv_b200.qshift import stock


class Skip(nn.Module):
    def forward(self, x, resolution):
        return torch.zeros_like(x)


def layers():
    return [(nn.Linear, nn.Linear(8, 8)), (nn.LayerNorm, nn.LayerNorm(8)), (nn.Conv2d, nn.Conv2d(3, 8, 8, stride=8)),
            (backbone.ChannelMix, backbone.ChannelMix(64, 2, 0)), (backbone6.ChannelMixV6, backbone6.ChannelMixV6(64, 2, 0))]


@pytest.mark.parametrize("i", range(5))
def test_stock_sees_what_a_call_would_run(monkeypatch, i):
    cls, module = layers()[i]
    assert stock(module, cls)
    with monkeypatch.context() as m:
        m.setattr(cls, "forward", lambda self, *args: args[0])
        assert not stock(module, cls)
    assert stock(module, cls)
    module.compile(backend="eager")
    assert not stock(module, cls)


@pytest.mark.parametrize("post_norm", [False, True])
@pytest.mark.parametrize("how", ["class", "compiled"])
@pytest.mark.parametrize("v6", [False, True])
def test_a_block_calls_a_replaced_channel_mix(monkeypatch, v6, how, post_norm):
    if v6:
        cls, block = backbone6.ChannelMixV6, backbone6.BlockV6(64, 1, 2, 1, post_norm=post_norm)
    else:
        cls, block = backbone.ChannelMix, backbone.Block(64, 2, 1, post_norm=post_norm)
    block.att = Skip()
    mine = lambda self, x, resolution: x * 2
    if how == "class":
        monkeypatch.setattr(cls, "forward", mine)
    else:
        block.ffn._compiled_call_impl = lambda x, resolution: mine(block.ffn, x, resolution)      # what ffn.compile() sets
    x = torch.randn(2, 4, 64)
    with torch.no_grad():
        got = block(x, (2, 2))
        want = x + block.ln1(torch.zeros_like(x)) if post_norm else x
        want = want + block.ln2(want * 2) if post_norm else want + block.ln2(want) * 2
    assert torch.equal(got, want)


def test_a_trace_keeps_the_channel_mix_as_a_call():
    block = backbone.Block(64, 2, 1, shift_pixel=0)
    block.att = Skip()

    class Net(nn.Module):
        def __init__(self):
            super().__init__()
            self.block = block

        def forward(self, x):
            return self.block(x, (2, 2))

    x = torch.randn(2, 4, 64)
    with torch.no_grad():
        traced = torch.jit.trace(Net(), x)
        assert "(ffn).forward(" in traced.block.code
        assert torch.equal(traced(x), block(x, (2, 2)))
