"""Autograd wrapper of the fused Q-Shift + token-mix kernel.

`qshift_mix(x, (mix_k, mix_v, mix_r), patch_resolution)` returns what
`VRWKV_SpatialMix.jit_func` computes before its linear layers
(classification/mmcls_custom/models/backbones/vrwkv.py:156-164):
`xx = q_shift(x, shift_pixel, channel_gamma, patch_resolution)` followed by
`x * mix + xx * (1 - mix)` per mix vector; with two vectors it serves `VRWKV_ChannelMix`
(:247-250).  Mix parameters may have the reference's (1, 1, C) shape.
"""
from __future__ import annotations

import torch
import torch.nn as nn

from . import _lib, ops, traced


_FORWARDS = {}      # what `forward` of a class was when its work was taken over by kernels


def taken_over(cls):
    """Class decorator: kernels may do the work of `cls.forward` as it stands (torch's own, if it is torch's class)."""
    f = cls.forward
    if f.__module__ == cls.__module__ and f.__qualname__ == f"{cls.__qualname__}.forward":
        _FORWARDS[cls] = f
    return cls


for _cls in (nn.Linear, nn.LayerNorm, nn.Conv2d):
    taken_over(_cls)


def stock(module, cls):
    """Whether calling `module` runs the `cls.forward` that was `taken_over` and nothing else: no subclass, no forward put in its
    place (on the class or the instance), not compiled in place, no hooks (its own or those registered for all modules)."""
    return (type(module) is cls and _FORWARDS.get(cls) is cls.forward and "forward" not in module.__dict__
            and module._compiled_call_impl is None and not module._forward_hooks and not module._forward_pre_hooks
            and not nn.modules.module._global_forward_hooks and not nn.modules.module._global_forward_pre_hooks)


def autocast_linears(*layers):
    """True when `layers` round what they are given to bfloat16 first: inference (training keeps the float32 graph) under
    bfloat16 autocast, and every layer is a stock `nn.Linear`."""
    return (not torch.is_grad_enabled() and torch.is_autocast_enabled("cuda") and torch.get_autocast_dtype("cuda") == torch.bfloat16
            and not traced.tracing() and all(stock(m, nn.Linear) for m in layers))


def feeds_autocast_linears(x, *layers):
    """True when results of float32 x may leave in bfloat16 because the layers that take them round them to it."""
    return x.is_cuda and x.dtype == torch.float32 and autocast_linears(*layers)


def qshift_mix(x, mixes, patch_resolution, shift_pixel=1, channel_gamma=0.25, head_dim=None):
    """head_dim=None: `q_shift` with `channel_gamma` (VRWKV).  head_dim=n: `q_shift_multihead` of VRWKV6
    (classification/mmcls_custom/models/backbones/vrwkv6.py:75-101), the shift its ChannelMix uses."""
    if traced.tracing():
        return traced.QShiftMix.apply(x, patch_resolution, shift_pixel, channel_gamma, head_dim, *mixes)
    H, W = patch_resolution
    group = ops.qshift_group(x.shape[-1], channel_gamma, head_dim)
    return tuple(_lib.native().qshift_mix(x, list(mixes), H, W, shift_pixel, group, head_dim is not None))


def qshift_mix_to(layers, x, mixes, patch_resolution, shift_pixel=1, channel_gamma=0.25, head_dim=None):
    """`qshift_mix` for the linear layers `layers`: in bfloat16 where those would round to it first anyway (the same bits
    reach the matrix product, for 2 instead of 4 + 4 + 2 bytes per element and output)."""
    if not feeds_autocast_linears(x, *layers):
        return qshift_mix(x, mixes, patch_resolution, shift_pixel, channel_gamma, head_dim)
    H, W = patch_resolution
    group = ops.qshift_group(x.shape[-1], channel_gamma, head_dim)
    return tuple(_lib.native().qshift_mix_half(x, list(mixes), H, W, shift_pixel, group, head_dim is not None))


def qshift_ddlerp(x, maas, offsets, patch_resolution, shift_pixel=1, head_dim=64):
    """`[x + xx * (maa + m) for maa, m in zip(maas, offsets)]` with `xx = q_shift_multihead(x) - x`: the mixing steps of
    VRWKV6's spatial mix (classification/mmcls_custom/models/backbones/vrwkv6.py:180-193) in one pass.  `offsets`
    entries may be None (`xxx = x + xx * time_maa_x`).  Results are float32, as the reference's promotion makes them;
    float32 or bfloat16 offsets are read as they are."""
    if traced.tracing():
        return traced.QShiftDdlerp.apply(x, patch_resolution, shift_pixel, head_dim, len(maas), *maas, *offsets)
    H, W = patch_resolution
    return tuple(_lib.native().qshift_ddlerp(x, list(maas), list(offsets), H, W, shift_pixel, head_dim))


def qshift_ddlerp_to(layers, x, maas, offsets, patch_resolution, shift_pixel=1, head_dim=64):
    """`qshift_ddlerp` for the linear layers `layers` and plain matrix products, as `qshift_mix_to`."""
    if not feeds_autocast_linears(x, *layers):
        return qshift_ddlerp(x, maas, offsets, patch_resolution, shift_pixel, head_dim)
    H, W = patch_resolution
    return tuple(_lib.native().qshift_ddlerp_half(x, list(maas), list(offsets), H, W, shift_pixel, head_dim))
