"""Autograd wrapper of the fused Q-Shift + token-mix kernel.

`qshift_mix(x, (mix_k, mix_v, mix_r), patch_resolution)` returns what
`VRWKV_SpatialMix.jit_func` computes before its linear layers
(classification/mmcls_custom/models/backbones/vrwkv.py:156-164):
`xx = q_shift(x, shift_pixel, channel_gamma, patch_resolution)` followed by
`x * mix + xx * (1 - mix)` per mix vector; with two vectors it serves `VRWKV_ChannelMix`
(:247-250).  Mix parameters may have the reference's (1, 1, C) shape.
"""
from __future__ import annotations

from . import _lib, ops


def qshift_mix(x, mixes, patch_resolution, shift_pixel=1, channel_gamma=0.25, head_dim=None):
    """head_dim=None: `q_shift` with `channel_gamma` (VRWKV).  head_dim=n: `q_shift_multihead` of VRWKV6
    (classification/mmcls_custom/models/backbones/vrwkv6.py:75-101), the shift its ChannelMix uses."""
    H, W = patch_resolution
    group = ops.qshift_group(x.shape[-1], channel_gamma, head_dim)
    return tuple(_lib.native().qshift_mix(x, list(mixes), H, W, shift_pixel, group, head_dim is not None))


def qshift_ddlerp(x, maas, offsets, patch_resolution, shift_pixel=1, head_dim=64):
    """`[x + xx * (maa + m) for maa, m in zip(maas, offsets)]` with `xx = q_shift_multihead(x) - x`: the mixing steps of
    VRWKV6's spatial mix (classification/mmcls_custom/models/backbones/vrwkv6.py:180-193) in one pass.  `offsets`
    entries may be None (`xxx = x + xx * time_maa_x`).  Results are float32, as the reference's promotion makes them;
    float32 or bfloat16 offsets are read as they are."""
    H, W = patch_resolution
    return tuple(_lib.native().qshift_ddlerp(x, list(maas), list(offsets), H, W, shift_pixel, head_dim))
