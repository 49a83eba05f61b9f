"""Bi-WKV in narrow strips at the edges of its split: a walker's tokens (15 or 17), a warp's span (60, 68, 120, 136), a CTA's (480, 544, 960,
1088) and those of clusters, one token less or more; strips past the last channel.  Against the float64 oracle with the tolerances
of test_biwkv_gpu.py (1e-5) and test_biwkv_bf16_gpu.py (1e-2 for bfloat16 results; gw, gu are float32)."""
import pytest
import torch

from conftest import rel_err
from oracle import biwkv_oracle as O

pytestmark = pytest.mark.gpu
NAMES = ("y", "gw", "gu", "gk", "gv")


def errors(dev, B, T, C, types, w_range=None, k_scale=1.0):
    from vision_rwkv_b200 import ops
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    w, u, k, v, gy = O.make_inputs(B, T, C, dtype=torch.float32, seed=7 * T + C)
    k = k * k_scale
    if w_range is not None:
        w = torch.linspace(*w_range, C) / T
    if types != "f32":
        k, v, gy = k.bfloat16(), v.bfloat16(), gy.bfloat16()
    if types == "bf16":
        w, u = w.bfloat16(), u.bfloat16()
    if types == "wide":
        gy = gy.float()      # the kernels round it; its rounding is not what is checked here
    xs = [x.to(dev).contiguous().requires_grad_(True) for x in (w, u, k, v)]
    y = RUN_CUDA(*xs)
    got = (y.detach(), *torch.autograd.grad(y, xs, gy.to(dev)))
    ops.raise_if_failed()
    f = [x.double() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    return {n: rel_err(g.float(), r) if r.abs().max() > 0 else g.abs().max().item() for n, g, r in zip(NAMES, got, ref)}


def check(errs, types):
    for name, e in errs.items():
        assert e <= (1e-5 if types == "f32" or (types == "wide" and name in ("gw", "gu")) else 1e-2), (name, errs)


EDGES = [1, 2, 15, 16, 17, 18, 34, 35, 60, 61, 68, 69, 120, 121, 136, 137, 300, 301, 480, 481, 544, 545, 600, 601, 680, 681, 960, 961, 1088, 1089, 1632, 1633,
         2176, 2177, 3264, 3265, 3808, 3809]


@pytest.mark.parametrize("T", EDGES)
@pytest.mark.parametrize("C,types", [(44, "f32"), (40, "wide"), (24, "bf16")])
def test_edges(cuda_device, T, C, types):
    check(errors(cuda_device, 2, T, C, types), types)


@pytest.mark.parametrize("T", [1, 2, 3, 5, 16, 49, 61, 200])
@pytest.mark.parametrize("w_range", [(-30.0, -1.0), (1.0, 30.0), (-5.0, 3.0)])
def test_steep_weights(cuda_device, T, w_range):
    """Weights that grow or fall by orders of magnitude within the sequence: past its end they would overflow, or leave a denominator of
    zero, and nothing of that may reach a valid token.  The shortest sequences are outside the plain-float range where weights grow most, the others
    inside (both kinds in one call: test_units_inside_and_outside_the_plain_float_range).
    Tolerance: 5e-5, that of test_biwkv_gpu.py for extreme exponents."""
    for types, tol in (("f32", 5e-5), ("wide", 1e-2)):
        errs = errors(cuda_device, 3, T, 48, types, w_range)
        assert all(e <= tol for e in errs.values()), errs


# enough sequences of more than 4096 tokens: clusters of 4 to 16 CTAs, the longest that a cluster holds; one token more goes back to separate launches
@pytest.mark.parametrize("B,T", [(23, 4200), (12, 8704), (12, 8705), (6, 17408), (6, 17409)])
@pytest.mark.parametrize("types", ["f32", "wide", "bf16"])
def test_long_sequences(cuda_device, B, T, types):
    from vision_rwkv_b200 import _lib
    C, lib = 64, _lib.load()
    before = lib.vrwkv_launch_count()
    errs = errors(cuda_device, B, T, C, types)
    one_pass = lib.vrwkv_biwkv_one_pass(B, T, C, ("f32", "bf16", "wide").index(types))
    assert one_pass == (T <= (8704 if types == "bf16" else 17408))
    assert (lib.vrwkv_launch_count() - before == 5) == bool(one_pass)
    for name, e in errs.items():
        assert e <= (1e-2 if types == "bf16" or (types == "wide" and name not in ("gw", "gu")) else 1e-5 if T <= 8192 else 2e-5), (name, errs)


@pytest.mark.parametrize("T", [4200, 9000])
def test_long_sequences_outside_the_plain_float_range(cuda_device, T):
    errs = errors(cuda_device, 24, T, 64, "f32", k_scale=30.0)
    assert all(e <= 5e-5 for e in errs.values()), errs


def test_nothing_is_kept_where_one_pass_serves(cuda_device):
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    w, u, k, v, _ = [x.float().to(cuda_device) for x in O.make_inputs(23, 4200, 64, seed=1)]
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.dtype), t)[1], lambda t: t):
        RUN_CUDA(w, u, k.requires_grad_(True), v)
    assert torch.uint8 not in seen


@pytest.mark.parametrize("T,k_scale", [(100, 1.0), (100, 30.0), (1200, 1.0), (1200, 30.0)])      # 30: left to the exact kernel
@pytest.mark.parametrize("fill", [0x00, 0xFF])
def test_a_workspace_needs_no_clearing(cuda_device, T, k_scale, fill):
    from vision_rwkv_b200 import _lib
    import ctypes
    B, C, lib = 2, 40, _lib.load()
    w, u, k, v, gy = [x.float().to(cuda_device).contiguous() for x in O.make_inputs(B, T, C, seed=T)]
    k = k * k_scale
    y, gk, gv, gwgu = torch.empty_like(k), torch.empty_like(k), torch.empty_like(k), torch.empty(2, C, device=cuda_device)
    ws = [torch.full((f(B, T, C),), fill, dtype=torch.uint8, device=cuda_device) for f in (lib.vrwkv_biwkv_forward_workspace_bytes, lib.vrwkv_biwkv_backward_workspace_bytes)]
    s, p = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    assert lib.vrwkv_biwkv_forward_f32(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws[0]), ws[0].numel(), s) == 0
    assert lib.vrwkv_biwkv_backward_f32(B, T, C, p(w), p(u), p(k), p(v), p(gy), p(gwgu), p(gk), p(gv), p(ws[1]), ws[1].numel(), s) == 0
    for x in ws:
        status = ctypes.c_uint(9)
        assert lib.vrwkv_workspace_status(p(x), s, ctypes.byref(status)) == 0 and status.value == 0
    f = [x.double().cpu() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    for a, b in zip((y, gwgu[0], gwgu[1], gk, gv), ref):
        assert rel_err(a, b) <= (1e-5 if k_scale == 1.0 else 5e-5)


# Clusters of 2 to 16 CTAs, and (last two) several clusters to a sequence, csrc/biwkv_resident.cu.  `late`: the tokens of the CTA that sends nothing are outside the plain-float range, so that it leaves the unit to the
# exact kernel while the others do not hear of it.
@pytest.mark.parametrize("B,T", [(1, 1000), (1, 2000), (3, 4096), (24, 8704), (1, 4200), (1, 20000)])
@pytest.mark.parametrize("types", ["f32", "wide", "bf16"])
@pytest.mark.parametrize("late", [False, True])
def test_a_call_returns_when_a_cta_sends_nothing(cuda_device, B, T, types, late):
    from vision_rwkv_b200 import _lib
    import ctypes
    C, lib = 64, _lib.load()
    one_pass = lib.vrwkv_biwkv_one_pass(B, T, C, ("f32", "bf16", "wide").index(types))
    assert one_pass == (T <= 4096 or B > 1)
    if not one_pass and types == "wide":
        pytest.skip("no such kernels")
    w, u, k, v, gy = [x.float().to(cuda_device) for x in O.make_inputs(B, T, C, seed=T)]
    dt = torch.float32 if types == "f32" else torch.bfloat16
    clean = k.to(dt, copy=True)
    if late:
        at = 544 if one_pass else 300      # of the second CTA, where a CTA holds 544 (256) tokens or fewer
        k[:, at:at + 12] = 100.0
    k, v, gy = k.to(dt), v.to(dt), gy.to(dt)
    if types == "wide":
        gy = gy.float()      # the kernels round it; its rounding is not what is checked here
    y, gk, gv, gwgu = torch.empty_like(gy), torch.empty_like(k), torch.empty_like(k), torch.empty(2, C, device=cuda_device)
    name = {"f32": "f32", "bf16": "bf16", "wide": "bf16_wide"}[types]
    forward, backward = getattr(lib, "vrwkv_biwkv_forward_" + name), getattr(lib, "vrwkv_biwkv_backward_" + name)
    s, p = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()

    def calls(k):
        ws = [torch.empty(f(B, T, C), dtype=torch.uint8, device=cuda_device) for f in (lib.vrwkv_biwkv_forward_workspace_bytes, lib.vrwkv_biwkv_backward_workspace_bytes)]
        assert forward(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws[0]), ws[0].numel(), s) == 0
        assert backward(B, T, C, p(w), p(u), p(k), p(v), p(gy), p(gwgu), p(gk), p(gv), p(ws[1]), ws[1].numel(), s) == 0
        found = []
        for x in ws:
            status = ctypes.c_uint(0)
            assert lib.vrwkv_workspace_status(p(x), s, ctypes.byref(status)) == 0
            found.append(status.value & 1)
        return found

    try:
        assert lib.vrwkv_set_path(3) == 0
        for _ in range(3):
            assert calls(k) == [1, 1]
    finally:
        lib.vrwkv_set_path(0)
        lib.vrwkv_take_failures(torch.cuda.current_device())
    assert calls(clean) == [0, 0]      # the context is intact
    f = [x.double().cpu() for x in (w, u, clean, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    for a, b, n in zip((y, gwgu[0], gwgu[1], gk, gv), ref, NAMES):
        assert rel_err(a.float(), b) <= (2e-5 if types == "f32" or n in ("gw", "gu") else 1e-2), n


# weights that grow by e^5 to e^45 over the sequence, so that 2 max|k| + |u| + |w| + max(-w, 0) T is below 60 by what 14 to 16 rows past T may cost
@pytest.mark.parametrize("T,growth", [(1, 5.0), (1, 100.0), (2, 7.0), (4, 11.0), (7, 18.0), (12, 30.0), (17, 28.0), (20, 33.0), (31, 34.0), (49, 45.0), (61, 42.0), (200, 45.0)])
@pytest.mark.parametrize("types", ["f32", "wide"])
def test_short_sequences_with_steep_weights_need_no_exact_kernel(cuda_device, T, growth, types):
    """Rows past T fill up a walker's 15 or 17 tokens; the first e^8 that weights grow over them is free, and a single token knows no weights.  The words of the CTAs (256 bytes into a
    workspace) say whether a unit was left to the exact kernel.  Tolerance: 5e-5, that of test_biwkv_gpu.py for extreme exponents."""
    from vision_rwkv_b200 import _lib
    B, C, lib = 3, 48, _lib.load()
    w, u, k, v, gy = [x.float().to(cuda_device) for x in O.make_inputs(B, T, C, seed=T)]
    w = torch.linspace(-growth, -growth / 2, C, device=cuda_device) / T
    k = k.clamp(-1, 1)
    dt = torch.float32 if types == "f32" else torch.bfloat16
    k, v, gy = k.to(dt), v.to(dt), gy.to(dt).float()
    y, gk, gv, gwgu = torch.empty_like(gy), torch.empty_like(k), torch.empty_like(k), torch.empty(2, C, device=cuda_device)
    name = "f32" if types == "f32" else "bf16_wide"
    ws = [torch.zeros(f(B, T, C), dtype=torch.uint8, device=cuda_device) for f in (lib.vrwkv_biwkv_forward_workspace_bytes, lib.vrwkv_biwkv_backward_workspace_bytes)]
    s, p = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    assert getattr(lib, "vrwkv_biwkv_forward_" + name)(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws[0]), ws[0].numel(), s) == 0
    assert getattr(lib, "vrwkv_biwkv_backward_" + name)(B, T, C, p(w), p(u), p(k), p(v), p(gy), p(gwgu), p(gk), p(gv), p(ws[1]), ws[1].numel(), s) == 0
    for x in ws:
        assert not (x[256:256 + 4 * B * 3].view(torch.int32) & 1).any()
    f = [x.double().cpu() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    for a, b, n in zip((y, gwgu[0], gwgu[1], gk, gv), ref, NAMES):
        if T > 1 or n in ("y", "gv"):      # one token: no gradient but gv = gy
            assert rel_err(a.float(), b) <= (5e-5 if types == "f32" or n in ("gw", "gu") else 1e-2), n
        else:
            assert a.float().abs().max() <= 1e-5 * max(1.0, gy.abs().max().item())


@pytest.mark.parametrize("B,T", [(2, 196), (1, 2000), (24, 4200)])
@pytest.mark.parametrize("types", ["f32", "wide", "bf16"])
def test_scratch_memory(cuda_device, B, T, types):
    """Calls that the one-pass kernels serve need a word per CTA and the partial sums of gw and gu, less than a byte per element here, where the
    entry points' own queries give 1.5 and 8.1; that is what a training step allocates.  Tensors that those kernels cannot take need all of it."""
    from vision_rwkv_b200 import _lib
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    C, lib, n, which = 64, _lib.load(), B * T * 64, ("f32", "bf16", "wide").index(types)
    small = [lib.vrwkv_biwkv_one_pass_workspace_bytes(B, T, C, which, d) for d in (0, 1)]
    full = [lib.vrwkv_biwkv_forward_workspace_bytes(B, T, C), lib.vrwkv_biwkv_backward_workspace_bytes(B, T, C)]
    assert 0 < small[0] <= small[1] <= full[1] and small[0] <= full[0] and small[1] < 0.25 * n + 4096
    w, u, k, v, gy = [x.float().to(cuda_device) for x in O.make_inputs(B, T, C, seed=T)]
    dt = torch.float32 if types == "f32" else torch.bfloat16
    k, v, gy = k.to(dt), v.to(dt), gy.to(dt if types == "bf16" else torch.float32)
    name = "bf16_wide" if types == "wide" else types
    forward = getattr(lib, "vrwkv_biwkv_forward_" + name)
    s, p = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    y, ws = torch.empty_like(gy), torch.empty(full[1], dtype=torch.uint8, device=cuda_device)
    assert forward(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws), small[0], s) == 0
    assert forward(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws), small[0] - 1, s) == 3
    odd = torch.empty(n + 8, dtype=dt, device=cuda_device)[2:n + 2].view(B, T, C).copy_(k)      # off a 16-byte boundary
    assert forward(B, T, C, p(w), p(u), p(odd), p(v), p(y), p(ws), small[0], s) == 3
    ref = O.biwkv_scan_forward(*[x.double().cpu() for x in (w, u, k, v)])
    tol = 1e-5 if types == "f32" else 1e-2
    assert rel_err(y.float(), ref) <= tol
    assert rel_err(RUN_CUDA(w, u, odd, v).float(), ref) <= tol

    if types == "bf16":
        w, u = w.bfloat16(), u.bfloat16()
    xs = [x.requires_grad_(True) for x in (w, u, k, v)]
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = RUN_CUDA(*xs)
    grads = torch.autograd.grad(out, xs, gy.to(out.dtype))
    kept = out.numel() * out.element_size() + sum(g.numel() * g.element_size() for g in grads)
    assert torch.cuda.max_memory_allocated() - before - kept < 0.25 * n + (1 << 20)


@pytest.mark.parametrize("T", [50, 200, 1000, 2000, 4096])
@pytest.mark.parametrize("types", ["f32", "wide"])
def test_units_inside_and_outside_the_plain_float_range(cuda_device, T, types):
    """Weights that grow by e^10 to e^100 over the sequence, from channel to channel, and large k in one strip of one sequence: the exact kernel
    serves some units of a call and skips the others, in single CTAs and in clusters.  Tolerance: 5e-5, that of test_biwkv_gpu.py for extreme exponents."""
    from vision_rwkv_b200 import _lib
    B, C, lib = 3, 80, _lib.load()
    w, u, k, v, gy = [x.float().to(cuda_device) for x in O.make_inputs(B, T, C, seed=T)]
    w = torch.linspace(-100, -10, C, device=cuda_device) / T
    k = k.clamp(-1, 1)
    k[1, ::7, 70] *= 60
    dt = torch.float32 if types == "f32" else torch.bfloat16
    k, v, gy = k.to(dt), v.to(dt), gy.to(dt).float()
    y, gk, gv, gwgu = torch.empty_like(gy), torch.empty_like(k), torch.empty_like(k), torch.empty(2, C, device=cuda_device)
    name, which = ("f32", 0) if types == "f32" else ("bf16_wide", 2)
    ws = [torch.full((lib.vrwkv_biwkv_one_pass_workspace_bytes(B, T, C, which, d),), 0xFF, dtype=torch.uint8, device=cuda_device) for d in (0, 1)]
    s, p = torch.cuda.current_stream().cuda_stream, lambda t: t.data_ptr()
    assert getattr(lib, "vrwkv_biwkv_forward_" + name)(B, T, C, p(w), p(u), p(k), p(v), p(y), p(ws[0]), ws[0].numel(), s) == 0
    assert getattr(lib, "vrwkv_biwkv_backward_" + name)(B, T, C, p(w), p(u), p(k), p(v), p(gy), p(gwgu), p(gk), p(gv), p(ws[1]), ws[1].numel(), s) == 0
    words = ws[0][256:-768].view(torch.int32)      # of the forward's CTAs: 1 for a unit left to the exact kernel, 0 for one that was not
    words = words[words >= 0]
    assert set(words.tolist()) == {0, 1}
    # strips of 8 or 16 channels: the last 32 channels are inside the range, but for one strip of the sequence with large k
    per_sequence = words.view(B, -1).sum(1)
    assert per_sequence[0] == per_sequence[2] < per_sequence[1] < words.numel() // B
    f = [x.double().cpu() for x in (w, u, k, v, gy)]
    ref = (O.biwkv_scan_forward(*f[:4]), *O.biwkv_scan_backward(*f))
    for a, b, n in zip((y, gwgu[0], gwgu[1], gk, gv), ref, NAMES):
        assert rel_err(a.float(), b) <= (5e-5 if types == "f32" or n in ("gw", "gu") else 1e-2), n
