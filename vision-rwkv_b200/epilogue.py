"""The steps between a block's matrix products, for the networks of `backbone` and `backbone6`.

Each function is the reference's expression; when a network is only being run (no gradients wanted) on CUDA tensors in
float32 or bfloat16 it is one kernel of csrc/mixer_epilogue.cu instead of a chain of tensor operations.  Training keeps the
tensor operations and their graph.  A layer whose work a kernel takes over must be one whose call is torch's own
(`qshift.stock`).
"""
from __future__ import annotations

import weakref

import torch
import torch.nn as nn
from torch.utils._device import DeviceContext

from . import _lib, normgate, ops, traced
from .qshift import autocast_linears, feeds_autocast_linears, stock

KERNEL_DTYPES = (torch.float32, torch.bfloat16)
DEEPEST_BATCH = 1024            # of vrwkv_linear_batch_pays: deeper layers are not worth the questions
MOST_NORM_CHANNELS = 1024       # a row of norm_residual lives in one warp's registers


def _inference(*tensors):
    return not torch.is_grad_enabled() and not traced.tracing() and all(t.is_cuda and t.dtype in KERNEL_DTYPES for t in tensors)


_dispatch_modes, _function_modes, _PLAIN = torch._C._len_torch_dispatch_stack, torch._C._len_torch_function_stack, (nn.Parameter, torch.Tensor)


def _unwatched(x, *parameters):
    """Whether nobody would see a layer's own call on x: it and the parameters are plain tensors, and no mode that watches or replaces
    tensor operations is active (a default device is not one)."""
    if type(x) is not torch.Tensor or _dispatch_modes() or (
            _function_modes() and any(type(m) is not DeviceContext for m in torch.overrides._get_current_function_mode_stack())):
        return False
    for p in parameters:
        if type(p) not in _PLAIN:
            return False
    return True


_NOTHING = {}       # by device: an empty parameter.  Autocast keeps its copy of it, which takes no launch, as long as its copies of others.


def _left_to_autocast(owner, device):
    """Whether `owner` has been called before while autocast keeps what it casts (it forgets that when its outermost context ends, or at once
    where it is not to keep anything).  The calls are counted on autocast's own copy of an empty parameter, so the count goes where the
    copies go.  A captured call leaves no copies behind that an eager one could use: it counts for nothing, and takes autocast's only where
    an earlier call has made them."""
    nothing = _NOTHING.get(device)
    if nothing is None:
        with torch.inference_mode(False):
            nothing = _NOTHING[device] = nn.Parameter(torch.empty(0, device=device, dtype=torch.float32))      # what autocast copies
    calls = _lib.native().autocast_copy(nothing).__dict__.setdefault("calls", {})
    before = calls.get(key := weakref.ref(owner), 0)        # equal to another owner's never, also not to that of a gone one at its address
    if before > 1:
        return True
    if torch.cuda.is_current_stream_capturing():
        return False
    calls[key] = before + 1
    return before > 0


def weights_for(owner, x, *sources):
    """The weights of `sources` (linear layers, matrices) as bfloat16 autocast makes them for the products of one call of `owner` on x, cast
    in one launch instead of one each; None where each is left to its own product.  That is wherever somebody would see the cast or
    the layer's call, and from the second call of `owner` on in an autocast context that is held: autocast keeps what it casts by itself, and
    after that second call has no more to cast."""
    if (not x.is_cuda or torch.is_grad_enabled() or not torch.is_autocast_enabled("cuda") or torch.get_autocast_dtype("cuda") != torch.bfloat16
            or traced.tracing() or x.dtype not in KERNEL_DTYPES or not _unwatched(x)):
        return None
    if _left_to_autocast(owner, x.device) and (type(sources[0]) is not nn.Linear or sources[0].weight.requires_grad):
        return None                                  # (autocast keeps no others)
    layers = [s for s in sources if isinstance(s, nn.Module)]
    if not autocast_linears(*layers) or any(layer.bias is not None for layer in layers):
        return None
    weights = [s.weight if isinstance(s, nn.Module) else s for s in sources]
    for w in weights:
        if type(w) is not nn.Parameter or w.dtype != torch.float32 or w.device != x.device or not w.is_contiguous() or w.numel() == 0:
            return None
    return _lib.native().narrow(weights) or None


def linear(layer, x, weight=None):
    """layer(x), with the layer's weight as `weights_for` gave it"""
    return layer(x) if weight is None else nn.functional.linear(x, weight)


def relu_square(x, layer=None):
    """relu(x)^2 (classification/mmcls_custom/models/backbones/vrwkv.py:251).  Under autocast torch squares bfloat16 x in float32;
    the result leaves in bfloat16 only for a linear layer `layer` that rounds it to that first anyway."""
    if not _inference(x):
        return torch.square(torch.relu(x))
    wide = x.dtype == torch.bfloat16 and torch.is_autocast_enabled("cuda") and not (layer is not None and autocast_linears(layer))
    return _lib.native().relu_square(x, wide)


def linear_relu_square(key, x, layer=None, weight=None):
    """relu_square(linear(key, x, weight), layer), the linear layer and what follows it in one call where `layer` rounds the result to bfloat16 anyway (in
    one kernel where that is faster: vrwkv_linear_relu_square_pays)."""
    if layer is not None and x.dtype == torch.bfloat16 and _inference(x) and autocast_linears(key, layer) and key.bias is None:
        w = key.weight if weight is None else weight
        if (_unwatched(x, w) and w.dtype in KERNEL_DTYPES and w.device == x.device and w.dim() == 2 and w.shape[1] == x.shape[-1]
                and w.shape[1] % 64 == 0 and w.shape[1] > 0 and w.shape[0] % 256 == 0 and w.shape[0] > 0):
            out = _lib.native().key_layer(x, w)
            if ops.CHECK_STATUS:
                ops.raise_if_failed(x.device)
            return out
    return relu_square(linear(key, x, weight), layer)


def linears(layers, xs, weights=None):
    """[linear(layer, x, weight) for ...] of up to four layers, in one launch where they are of one shape and that is faster
    (vrwkv_linear_batch_pays)."""
    x, w = xs[0], layers[0].weight if type(layers[0]) is nn.Linear else None
    if (w is not None and len(layers) <= 4 and x.shape[-1] <= DEEPEST_BATCH and x.dtype == torch.bfloat16 and _inference(*xs) and autocast_linears(*layers)
            and all(layer.bias is None and _unwatched(t, layer.weight) and t.dtype == x.dtype and t.shape == x.shape and t.device == x.device
                    and layer.weight.dtype in KERNEL_DTYPES and layer.weight.shape == w.shape and layer.weight.device == x.device
                    for layer, t in zip(layers, xs))
            and w.dim() == 2 and w.shape[1] == x.shape[-1]):
        outs = _lib.native().linear_batch(list(xs), weights or [layer.weight for layer in layers])
        if ops.CHECK_STATUS:
            ops.raise_if_failed(x.device)
        return outs
    return [linear(layer, t, weight) for layer, t, weight in zip(layers, xs, weights or [None] * len(layers))]


def sigmoid_gate(r, y, norm=None):
    """sigmoid(r) * y in the dtype of r (vrwkv.py:182-187, 253-257).  For a LayerNorm `norm` that takes it under autocast, where torch
    widens a bfloat16 result to float32 first, it leaves widened."""
    if _inference(r, y) and r.shape == y.shape and (y.dtype == torch.float32 or r.dtype == torch.bfloat16):
        wide = norm is not None and r.dtype == y.dtype == torch.bfloat16 and torch.is_autocast_enabled("cuda") and stock(norm, nn.LayerNorm)
        return _lib.native().sigmoid_gate(r, y, wide)
    return torch.sigmoid(r) * y.to(r.dtype)


def _residual_kernel(x, a, gamma):
    return (_inference(x, a) and x.dtype == torch.float32 and x.shape == a.shape and x.shape[-1] % 4 == 0
            and x.shape[-1] <= MOST_NORM_CHANNELS and (gamma is None or gamma.dtype == torch.float32))


def residual(x, a, gamma):
    """x + gamma * a (gamma None: x + a)."""
    if _residual_kernel(x, a, gamma):
        return _lib.native().norm_residual(x, a, None, None, gamma, 0.0)
    return x + (a if gamma is None else gamma * a)


def _norm_kernel(a, norm, C):
    return (stock(norm, nn.LayerNorm) and norm.normalized_shape == (C,) and norm.bias is not None
            and norm.weight.dtype == norm.bias.dtype == torch.float32 and (a.dtype == torch.float32 or torch.is_autocast_enabled("cuda")))


def layer_norm(norm, x):
    """norm(x) for a LayerNorm `norm` over the channels"""
    C = x.shape[-1]
    if (_inference(x) and x.dtype == torch.float32 and C % 4 == 0 and 0 < C <= MOST_NORM_CHANNELS and x.numel() // C < 2 ** 31
            and _norm_kernel(x, norm, C) and _unwatched(x, norm.weight, norm.bias)):
        return _lib.native().layer_norm(x, norm.weight, norm.bias, norm.eps)
    return norm(x)


def widened(norm, a):
    """a as a LayerNorm `norm` takes it under autocast: torch widens a bfloat16 input to float32 first."""
    if (a.dtype == torch.bfloat16 and _inference(a) and a.is_contiguous() and a.numel() % 8 == 0 and a.numel() < 2 ** 33
            and torch.is_autocast_enabled("cuda") and stock(norm, nn.LayerNorm) and _unwatched(a)):
        return _lib.native().widen(a)
    return a


def norm_residual(x, a, norm, gamma):
    """x + gamma * norm(a) for a LayerNorm `norm` (post-norm blocks).  Under autocast torch computes that norm in float32."""
    if _residual_kernel(x, a, gamma) and _norm_kernel(a, norm, x.shape[-1]):
        return _lib.native().norm_residual(x, a, norm.weight, norm.bias, gamma, norm.eps)
    return residual(x, norm(a), gamma)


def takes_gate_of(mix, cls):
    """Whether a block may take the gate's operands from its channel mix `mix` instead of calling it: when it is only being run, and
    the call would do nothing else.  (A trace keeps the call, and with it the module in its graph.)"""
    return not torch.is_grad_enabled() and not traced.tracing() and stock(mix, cls)


def gated_residual(x, r, y, norm, gamma):
    """norm_residual(x, sigmoid_gate(r, y), norm, gamma), or residual(x, sigmoid_gate(r, y), gamma) where norm is None: what a block
    does with its channel mix, in one pass where all of it is kernels."""
    if (_residual_kernel(x, y, gamma) and _inference(r) and r.dtype == y.dtype == torch.bfloat16 and r.shape == y.shape
            and (norm is None or _norm_kernel(y, norm, x.shape[-1]))):
        if norm is None:
            return _lib.native().gated_norm_residual(x, r, y, None, None, gamma, 0.0)
        return _lib.native().gated_norm_residual(x, r, y, norm.weight, norm.bias, gamma, norm.eps)
    a = sigmoid_gate(r, y)
    return residual(x, a, gamma) if norm is None else norm_residual(x, a, norm, gamma)


def head_norm_gate(x, gate, norm, head_size, layer, act):
    """Per-head GroupNorm `norm` of x times the activated gate (vrwkv6.py:205-212), for the linear layer `layer`: in
    bfloat16 where that layer would round to it first anyway."""
    if head_size == 64 and feeds_autocast_linears(x, layer) and _inference(gate):
        return _lib.native().head_norm_gate_half(x, gate, norm.weight, norm.bias, norm.eps, ops.GATE_ACTIVATIONS[act])
    return normgate.norm_gate(x, gate, norm.weight, norm.bias, head_size, norm.eps, act=act)


def add_rows(table, a):
    """table + a, the table (leading sizes 1) repeated over the rows of a: the decay of vrwkv6.py:200, the positions of
    vrwkv.py:392."""
    sizes = list(table.shape)
    while sizes and sizes[0] == 1:
        sizes.pop(0)
    if (_inference(table, a) and a.dtype == torch.bfloat16 and table.dtype == torch.float32 and a.is_contiguous()
            and table.numel() % 8 == 0 and 0 < table.numel() and a.numel() < 2 ** 33 and table.dim() <= a.dim()
            and list(a.shape[a.dim() - len(sizes):]) == sizes):
        return _lib.native().add_rows(table, a)
    return table + a


def patch_embedding(img, conv):
    """The tokens (B, h * w, C) of a patch embedding `conv` (kernel = stride; vrwkv.py:357) as one matrix product over the
    patches, or None where the convolution itself has to run (training, other data types, other convolutions)."""
    p = conv.kernel_size[0]
    if not (feeds_autocast_linears(img) and stock(conv, nn.Conv2d) and conv.kernel_size == conv.stride == (p, p)
            and conv.padding == (0, 0) and conv.dilation == (1, 1) and conv.groups == 1
            and img.dim() == 4 and img.shape[1] == conv.in_channels and img.is_contiguous() and p % 8 == 0
            and img.shape[2] >= p and img.shape[3] >= p and img.shape[3] % 4 == 0 and img.numel() < 2 ** 33):
        return None
    tokens = nn.functional.linear(_lib.native().patch_rows(img, p), conv.weight.flatten(1))
    # the convolution rounds to bfloat16 before its bias too
    return tokens if conv.bias is None else tokens + conv.bias.to(tokens.dtype)
