"""Autograd wrapper of the fused normalise-and-gate epilogue.

`norm_gate(x, gate, weight, bias, group, eps)` returns `(normalise(x) * weight + bias) * gate`:

* `group = C`: what `VRWKV_SpatialMix.forward` computes after the operator when `key_norm` is on,
  `sr * self.key_norm(x)` (classification/mmcls_custom/models/backbones/vrwkv.py:184-186);
* `group = 64`: `self.ln_x(x.view(B * T, C)).view(B, T, C) * g` of VRWKV6's `jit_func_2`
  (classification/mmcls_custom/models/backbones/vrwkv6.py:133, 205-212; GroupNorm with one group per head).

`gate` is the activated gate (`sr`, `g`), or with `act="sigmoid"` / `act="silu"` the projection it is the
activation of (`self.receptance(xr)`, `self.gate(xg)`): float32 or bfloat16.  The result is float32, as torch's type
promotion makes the reference's product.  Shapes the kernel does not cover (group not a multiple of 64 or
above 1024) are refused by the library; `supported(C, group)` tells beforehand.
"""
from __future__ import annotations

from . import _lib, ops, traced


def supported(C: int, group: int) -> bool:
    return group > 0 and group % 64 == 0 and group <= 1024 and C % group == 0


def norm_gate(x, gate, weight, bias, group=None, eps=1e-5, act=None):
    """x, gate: (..., C); weight, bias: (C,); group: channels per normalisation group (default C); act: None when
    `gate` is the gate itself, "sigmoid" / "silu" when it is the projection the gate is that activation of (the
    activation and its derivative then run inside the same pass)."""
    group = x.shape[-1] if group is None else group
    if traced.tracing():
        return traced.NormGate.apply(x, gate, weight, bias, group, eps, act)
    return _lib.native().norm_gate(x, gate, weight, bias, group, eps, ops.GATE_ACTIVATIONS[act])
