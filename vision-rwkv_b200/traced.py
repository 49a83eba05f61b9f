"""Python autograd nodes of the steps around the operators, for `torch.jit.trace`.

The tracer records a Python autograd Function as a call; of a C++ function that writes through raw pointers it would record
only the allocation of the results.  So while a trace is taken, `qshift`, `normgate`, `vrwkv`, `vrwkv6` and `mae_vrwkv` go
through Python nodes (the operators keep theirs in their own modules), and the inference kernels of `epilogue` stay out.
"""
from __future__ import annotations

import torch

from . import ops


tracing = torch._C._is_tracing        # torch.jit.is_tracing without its test for scripting, 0.1 us that small calls would pay each time


class QShiftMix(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, resolution, shift_pixel, gamma, head_dim, *mixes):
        ctx.args = tuple(resolution), shift_pixel, gamma, head_dim
        ctx.x_dtype, ctx.mix_shapes = x.dtype, [m.shape for m in mixes]
        xf = x.float().contiguous()
        flat = [m.float().reshape(-1).contiguous() for m in mixes]
        ctx.save_for_backward(xf, *flat)
        return tuple(o.to(x.dtype) for o in ops.qshift_mix_forward(xf, flat, *ctx.args))

    @staticmethod
    def backward(ctx, *gouts):
        xf, *flat = ctx.saved_tensors
        gx, gmix = ops.qshift_mix_backward(xf, flat, [g.float().contiguous() for g in gouts], *ctx.args)
        return (gx.to(ctx.x_dtype), None, None, None, None, *[g.reshape(shape) for g, shape in zip(gmix, ctx.mix_shapes)])


class QShiftDdlerp(torch.autograd.Function):
    """The first n of `rest` are the vectors, then come the offsets (or None), one per vector."""

    @staticmethod
    def forward(ctx, x, resolution, shift_pixel, head_dim, n, *rest):
        maas, offsets = rest[:n], rest[n:]
        ctx.args, ctx.n = (tuple(resolution), shift_pixel, head_dim), n
        ctx.x_dtype, ctx.maa_types = x.dtype, [(a.shape, a.dtype) for a in maas]
        ctx.offset_dtypes = [None if m is None else m.dtype for m in offsets]
        xf = x.float().contiguous()
        flat = [a.float().reshape(-1).contiguous() for a in maas]
        given = [m for m in offsets if m is not None]
        half = bool(given) and all(m.dtype == torch.bfloat16 for m in given)
        offsets = [None if m is None else (m.contiguous() if half else m.float().contiguous()) for m in offsets]
        ctx.save_for_backward(xf, *flat, *[m for m in offsets if m is not None])
        return tuple(ops.qshift_ddlerp_forward(xf, flat, offsets, *ctx.args))

    @staticmethod
    def backward(ctx, *gouts):
        xf, *kept = ctx.saved_tensors
        flat, given = kept[:ctx.n], iter(kept[ctx.n:])
        offsets = [None if t is None else next(given) for t in ctx.offset_dtypes]
        gx, goffsets, gmaas = ops.qshift_ddlerp_backward(xf, flat, offsets, [g.float().contiguous() for g in gouts], *ctx.args)
        return (gx.to(ctx.x_dtype), None, None, None, None,
                *[g.reshape(shape).to(dtype) for g, (shape, dtype) in zip(gmaas, ctx.maa_types)],
                *[None if g is None else g.to(dtype) for g, dtype in zip(goffsets, ctx.offset_dtypes)])


class NormGate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, gate, weight, bias, group, eps, act):
        xf, wf, bf = x.float().contiguous(), weight.float().contiguous(), bias.float().contiguous()
        gt = gate.contiguous() if gate.dtype in (torch.float32, torch.bfloat16) else gate.float().contiguous()
        out, mean, rstd = ops.normgate_forward(xf, gt, wf, bf, group, eps, act)
        ctx.save_for_backward(xf, gt, wf, bf, mean, rstd)
        ctx.group, ctx.act, ctx.dtypes = group, act, (x.dtype, gate.dtype, weight.dtype, bias.dtype)
        return out

    @staticmethod
    def backward(ctx, gout):
        xf, gt, wf, bf, mean, rstd = ctx.saved_tensors
        grads = ops.normgate_backward(gout.float().contiguous(), xf, gt, wf, bf, mean, rstd, ctx.group, ctx.act)
        return (*[g.to(dtype) for g, dtype in zip(grads, ctx.dtypes)], None, None, None)
