"""What a forward under autograd keeps for its backward on sequences above 4096 tokens, as autograd's users meet it: saved-tensor
hooks, a graph used twice, memory.  The bits are those of the pair that keeps nothing (see test_biwkv_split_gpu.py for both against
the oracle), which takes two launches more."""
import pytest
import torch

from oracle import biwkv_oracle as O

pytestmark = pytest.mark.gpu
SHAPE = (16, 4200, 64)      # 544 CTAs of 256 tokens, the last of a sequence holding 104


def leaves(dev, half=False):
    w, u, k, v, gy = [x.to(dev) for x in O.make_inputs(*SHAPE, dtype=torch.float32, seed=11)]
    if half:
        k, v = k.bfloat16(), v.bfloat16()
    return [x.contiguous().requires_grad_(True) for x in (w, u, k, v)], gy.contiguous()


def gradients(dev, pack=lambda t: t, unpack=lambda t: t):
    """The gradients and the number of launches of the backward."""
    from vision_rwkv_b200 import launch_count
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    xs, gy = leaves(dev)
    seen = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: (seen.append(t.dtype), pack(t))[1], unpack):
        y = RUN_CUDA(*xs)
    before = launch_count()
    grads = torch.autograd.grad(y, xs, gy)
    assert seen.count(torch.uint8) == 1      # the kept states
    return grads, launch_count() - before


def rebuilt(dev):
    from vision_rwkv_b200 import launch_count, ops
    xs, gy = leaves(dev)
    before = launch_count()
    return ops.biwkv_backward(*[x.detach() for x in xs], gy), launch_count() - before


def shifted(t, by):
    if t.dtype != torch.uint8:
        return t
    return torch.empty(t.numel() + by, dtype=torch.uint8, device=t.device)[by:].copy_(t)


@pytest.mark.parametrize("hook", ["host memory", "off by 1", "off by 16", "floats", "shorter", "dropped", "folded"])
def test_saved_tensor_hooks(cuda_device, hook):
    """Hooks that hand the bytes back, wherever they lie, keep the short backward; after others the states are rebuilt."""
    pack, unpack, short = {
        "host memory": (lambda t: t.cpu(), lambda t: t.to(cuda_device), True),
        "off by 1": (lambda t: shifted(t, 1), lambda t: t, True),
        "off by 16": (lambda t: shifted(t, 16), lambda t: t, True),
        "floats": (lambda t: t.float(), lambda t: t, False),
        "shorter": (lambda t: t[:-1] if t.dtype == torch.uint8 else t, lambda t: t, False),
        "dropped": (lambda t: t[:0] if t.dtype == torch.uint8 else t, lambda t: t, False),
        "folded": (lambda t: t.view(2, -1) if t.dtype == torch.uint8 else t, lambda t: t, False),
    }[hook]
    want, most = rebuilt(cuda_device)
    got, launches = gradients(cuda_device, pack, unpack)
    assert launches == (most - 2 if short else most)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def allocated(f):
    """What f() returns, the bytes it allocates in all and the most it holds at once."""
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    total, held = torch.cuda.memory_stats()["allocated_bytes.all.allocated"], torch.cuda.memory_allocated()
    out = f()
    return out, torch.cuda.memory_stats()["allocated_bytes.all.allocated"] - total, torch.cuda.max_memory_allocated() - held


@pytest.mark.parametrize("half", [False, True])
def test_nothing_is_allocated_twice(cuda_device, half):
    """bfloat16 k, v with float32 w, as under autocast, have no kernels for a float32 y or gy at this size (vrwkv_biwkv_one_pass): y is widened and gy
    narrowed around the bfloat16 ones, and nothing else is set up first."""
    from vision_rwkv_b200 import _lib
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    lib = _lib.load()
    xs, gy = leaves(cuda_device, half)
    n, size = gy.numel(), 2 if half else 4
    slack = 5 << 20      # five tensors at most, and the allocator leaves up to 1 MiB of a block in place
    y, total, _ = allocated(lambda: RUN_CUDA(*xs))
    states, scratch = lib.vrwkv_biwkv_kept_bytes(*SHAPE), lib.vrwkv_biwkv_forward_workspace_bytes(*SHAPE)
    assert 0 < states and total <= n * (size + (4 if half else 0)) + states + scratch + slack
    _, total, most = allocated(lambda: torch.autograd.grad(y, xs, gy, retain_graph=True))
    scratch = lib.vrwkv_biwkv_backward_workspace_bytes(*SHAPE)
    assert total <= n * (2 * size + (2 if half else 0)) + scratch + slack
    assert most <= n * (2 * size + (2 if half else 0)) + scratch + slack


def test_kept_states_are_not_in_the_workspace_too(cuda_device):
    """The workspace of a call with kept states is smaller by them, and enough: memory behind it is not touched."""
    from vision_rwkv_b200 import _lib, ops
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    lib = _lib.load()
    B, T, C = SHAPE
    states = lib.vrwkv_biwkv_kept_bytes(B, T, C)
    sizes = [lib.vrwkv_biwkv_kept_workspace_bytes(B, T, C, backward) for backward in (0, 1)]
    assert 0 < sizes[0] <= lib.vrwkv_biwkv_forward_workspace_bytes(B, T, C) - 2 * states // 3      # it would not hold the moments
    assert 0 < sizes[1] <= lib.vrwkv_biwkv_backward_workspace_bytes(B, T, C) - states
    assert lib.vrwkv_biwkv_kept_workspace_bytes(B, 4096, C, 0) == 0
    xs, gy = leaves(cuda_device)
    w, u, k, v = [x.detach() for x in xs]
    y, gk, gv = (torch.empty_like(k) for _ in range(3))
    gwgu, kept = torch.empty(2, C, device=cuda_device), torch.empty(states, dtype=torch.uint8, device=cuda_device)
    buffers = [torch.full((size + 4096,), 0xA5, dtype=torch.uint8, device=cuda_device) for size in sizes]
    s = torch.cuda.current_stream().cuda_stream
    p = lambda t: t.data_ptr()
    forward = lambda size: lib.vrwkv_biwkv_forward_keep(B, T, C, p(w), p(u), p(k), p(v), p(y), 0, p(kept), states, p(buffers[0]), size, s)
    backward = lambda size: lib.vrwkv_biwkv_backward_kept(B, T, C, p(w), p(u), p(k), p(v), p(gy), p(gwgu), p(gk), p(gv), 0, p(kept), states,
                                                          p(buffers[1]), size, s)
    assert forward(sizes[0] - 1) == 3 and forward(sizes[0]) == 0 and backward(sizes[1] - 1) == 3 and backward(sizes[1]) == 0
    for buffer, size in zip(buffers, sizes):
        assert bool((buffer[size:] == 0xA5).all())
    want = (ops.biwkv_forward(w, u, k, v), *ops.biwkv_backward(w, u, k, v, gy))
    for got, ref in zip((y, gwgu[0], gwgu[1], gk, gv), want):
        assert torch.equal(got, ref)
    # and the autograd node allocates no more than that
    _, total, _ = allocated(lambda: RUN_CUDA(*xs))
    assert total <= y.numel() * 4 + states + sizes[0] + (3 << 20)      # three tensors, as above


@pytest.mark.parametrize("k_scale", [1.0, 30.0])      # 30: outside the plain-float range, the kept word for that switches the kernels
def test_a_second_backward_finds_the_states_unchanged(cuda_device, k_scale):
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    xs, gy = leaves(cuda_device)
    xs[2] = (xs[2].detach() * k_scale).requires_grad_(True)
    y = RUN_CUDA(*xs)
    first = torch.autograd.grad(y, xs, gy, retain_graph=True)
    again = torch.autograd.grad(y, xs, gy)
    for a, b in zip(first, again):
        assert torch.equal(a, b) and bool(a.isfinite().all())


def test_vectors_that_start_at_an_odd_float(cuda_device):
    """w and u go through a copy in the workspace, for the chain of the CTAs' sums as for the other launches."""
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    xs, gy = leaves(cuda_device)
    odd = [torch.empty(x.numel() + 1, device=cuda_device)[1:].copy_(x.detach()).requires_grad_(True) for x in xs[:2]]
    assert all(x.data_ptr() % 8 == 4 for x in odd)
    y, y_odd = RUN_CUDA(*xs), RUN_CUDA(*odd, *xs[2:])
    assert torch.equal(y, y_odd)
    for a, b in zip(torch.autograd.grad(y, xs, gy), torch.autograd.grad(y_odd, [*odd, *xs[2:]], gy)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("half", [False, True])
def test_a_captured_step_replays_on_new_inputs(cuda_device, half):
    from vision_rwkv_b200.vrwkv import RUN_CUDA
    xs, gy = leaves(cuda_device, half)

    def step():
        y = RUN_CUDA(*xs)
        return (y.detach(), *torch.autograd.grad(y, xs, gy))

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    with torch.no_grad():
        for k_scale in (0.5, 40.0, 0.025):      # in the plain-float range, outside it, inside again
            xs[2].mul_(k_scale)
            graph.replay()
            torch.cuda.synchronize()
            with torch.enable_grad():
                want = step()
            for a, b in zip(captured, want):
                assert torch.equal(a, b)
