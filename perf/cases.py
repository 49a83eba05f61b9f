"""Workloads of this package, as a program that uses it runs them.

Four kinds, each through the entry points a model calls:

  biwkv     `vrwkv.RUN_CUDA(w, u, k, v)`, forward alone (inference) or with its gradients (training)
  wkv6      `vrwkv6.RUN_CUDA_RWKV6(B, T, C, H, r, k, v, w, u)`, the same two ways
  qshift    `qshift.qshift_mix(x, mixes, resolution)`, the token shift in front of both mixers, with its gradients
  backbone  the VRWKV / VRWKV6 networks of `backbone.build` / `backbone6.build_v6`, inference under bfloat16 autocast

Sizes are those of the shipped models (widths 192 to 1024, 16-pixel patches) on images from 224 pixels to
dense-prediction and long-sequence resolutions.
"""
import math

import torch

from vision_rwkv_b200 import backbone, backbone6
from vision_rwkv_b200.qshift import qshift_mix
from vision_rwkv_b200.vrwkv import RUN_CUDA
from vision_rwkv_b200.vrwkv6 import RUN_CUDA_RWKV6

WIDTHS = (192, 256, 384, 768, 1024)
PATCH = 16
BACKBONES = ("vrwkv_t", "vrwkv_s", "vrwkv_b", "vrwkv_l", "vrwkv6_t", "vrwkv6_s", "vrwkv6_b")

# The largest calls, in elements of one (B, T, C) tensor, and the largest backbone pass, in flops.
MOST_BIWKV = 64 * 4096 * 768
MOST_WKV6 = {"bf16": 32 * 4096 * 768, "fp32": 32 * 1024 * 768}
MOST_QSHIFT = 64 * 576 * 1024
MOST_BACKBONE_FLOPS = 2.4e12


def listed():
    return [
        # One 224-pixel image in the narrowest model: a single operator call, all latency.
        dict(name="biwkv_one_image", kind="biwkv", B=1, T=196, C=192, dtype="fp32", train=False),
        # Batch inference at 224 pixels under autocast: many short sequences.
        dict(name="biwkv_batch_224_bf16", kind="biwkv", B=256, T=196, C=384, dtype="bf16", train=False),
        # One layer of the large model's training step at 384 pixels under autocast.
        dict(name="biwkv_train_384_bf16", kind="biwkv", B=64, T=576, C=1024, dtype="bf16", train=True),
        # Dense prediction on 1344 x 800 images (84 x 50 tokens, no multiple of a tile), float32.
        dict(name="biwkv_train_dense", kind="biwkv", B=16, T=4200, C=768, dtype="fp32", train=True),
        # The largest operator call: 64 sequences of 4096 tokens, float32.
        dict(name="biwkv_train_4096", kind="biwkv", B=64, T=4096, C=768, dtype="fp32", train=True),
        # Few, very long sequences: 2048-pixel images.
        dict(name="biwkv_train_16384", kind="biwkv", B=8, T=16384, C=768, dtype="fp32", train=True),
        # One layer of the matrix-state model's training step at 224 pixels, under autocast and in float32.
        dict(name="wkv6_train_224_bf16", kind="wkv6", B=32, T=196, H=12, dtype="bf16", train=True),
        dict(name="wkv6_train_224_fp32", kind="wkv6", B=32, T=196, H=12, dtype="fp32", train=True),
        # The same layer on 1024-pixel images.
        dict(name="wkv6_train_4096_bf16", kind="wkv6", B=32, T=4096, H=12, dtype="bf16", train=True),
        # Token shift and its three interpolations in the large model's training step.
        dict(name="qshift_train_384", kind="qshift", B=64, grid_h=24, grid_w=24, C=1024, outputs=3),
        # Whole networks: the small model on 256 images, the matrix-state model on 64.
        dict(name="vrwkv_s_infer_256", kind="backbone", model="vrwkv_s", B=256, grid_h=14, grid_w=14),
        dict(name="vrwkv6_b_infer_64", kind="backbone", model="vrwkv6_b", B=64, grid_h=14, grid_w=14),
    ]


def _between(rng, lo, hi):
    """A whole number from lo to hi, even over its logarithm."""
    return min(hi, max(lo, round(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def _batch(rng, elements_each, most, limit=256):
    return _between(rng, 1, max(1, min(limit, most // elements_each)))


def draw(rng):
    kind = rng.choices(("biwkv", "wkv6", "qshift", "backbone"), (6, 3, 1, 2))[0]
    if kind == "biwkv":
        C, T = rng.choice(WIDTHS), _between(rng, 49, 16384)
        return dict(kind=kind, B=_batch(rng, T * C, MOST_BIWKV), T=T, C=C, dtype=rng.choice(("fp32", "bf16")),
                    train=rng.random() < 0.6)
    if kind == "wkv6":
        dtype = rng.choice(("bf16", "bf16", "fp32"))
        H, T = rng.choice((3, 6, 12)), _between(rng, 49, 4096 if dtype == "bf16" else 1024)
        return dict(kind=kind, B=_batch(rng, T * H * 64, MOST_WKV6[dtype]), T=T, H=H, dtype=dtype, train=rng.random() < 0.6)
    if kind == "qshift":
        C, h, w = rng.choice(WIDTHS), _between(rng, 7, 64), _between(rng, 7, 64)
        return dict(kind=kind, B=_batch(rng, h * w * C, MOST_QSHIFT), grid_h=h, grid_w=w, C=C, outputs=rng.choice((2, 3)))
    model, h, w = rng.choice(BACKBONES), rng.randint(10, 32), rng.randint(10, 32)
    case = dict(kind=kind, model=model, B=1, grid_h=h, grid_w=w)
    case["B"] = _batch(rng, 1, int(MOST_BACKBONE_FLOPS / work(case)["flops"]))
    return case


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _normal(g, *shape, dtype=torch.float32):
    return torch.randn(*shape, device="cuda", generator=g).to(dtype)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, device="cuda", generator=g) * (hi - lo) + lo


DTYPES = {"fp32": torch.float32, "bf16": torch.bfloat16}


def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    if kind == "biwkv":
        B, T, C, train = case["B"], case["T"], case["C"], case["train"]
        # spatial_decay / T over the range the models initialise it to, spatial_first / T around its log(0.3)
        w = _uniform(g, -5.0, 3.0, C) / T
        u = (math.log(0.3) + _uniform(g, -0.5, 0.5, C)) / T
        k, v = (_normal(g, B, T, C, dtype=DTYPES[case["dtype"]]) for _ in range(2))
        gy = _normal(g, B, T, C) if train else None        # the operator's result is float32 while w is
        return dict(case=case, leaves=[x.requires_grad_(train) for x in (w, u, k, v)], gout=gy)
    if kind == "wkv6":
        B, T, H, train = case["B"], case["T"], case["H"], case["train"]
        C = 64 * H
        r, k, v = (_normal(g, B, T, C, dtype=DTYPES[case["dtype"]]) for _ in range(3))
        w = _normal(g, B, T, C) * 0.5 - 0.6                # data-dependent decay exp(-exp(w))
        u = _normal(g, H, 64) * 0.1
        gy = _normal(g, B, T, C) if train else None
        return dict(case=case, leaves=[x.requires_grad_(train) for x in (r, k, v, w, u)], gout=gy)
    if kind == "qshift":
        B, T, C = case["B"], case["grid_h"] * case["grid_w"], case["C"]
        x = _normal(g, B, T, C).requires_grad_(True)
        mixes = [_uniform(g, 0.0, 1.0, 1, 1, C).requires_grad_(True) for _ in range(case["outputs"])]
        return dict(case=case, leaves=[x, *mixes], gout=[_normal(g, B, T, C) for _ in mixes])
    size = (case["grid_h"] * PATCH, case["grid_w"] * PATCH)
    with torch.random.fork_rng(devices=[torch.cuda.current_device()]), torch.device("cuda"):
        torch.manual_seed(seed)
        build = backbone6.build_v6 if case["model"].startswith("vrwkv6") else backbone.build
        # layer scale at one: at its initial 1e-5 an untrained network would be close to the identity
        model = build(case["model"], img_size=size, init_values=1.0).eval()
        torch.nn.init.normal_(model.pos_embed, std=0.02)
    return dict(case=case, model=model, img=_normal(g, case["B"], 3, *size))


def _grads(outs, state):
    return torch.autograd.grad(outs, state["leaves"], state["gout"])


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "biwkv":
        if not case["train"]:
            with torch.no_grad():
                return RUN_CUDA(*state["leaves"])
        y = RUN_CUDA(*state["leaves"])
        return (y.detach(), *_grads(y, state))
    if kind == "wkv6":
        B, T, H = case["B"], case["T"], case["H"]
        if not case["train"]:
            with torch.no_grad():
                return RUN_CUDA_RWKV6(B, T, 64 * H, H, *state["leaves"])
        y = RUN_CUDA_RWKV6(B, T, 64 * H, H, *state["leaves"])
        return (y.detach(), *_grads(y, state))
    if kind == "qshift":
        x, *mixes = state["leaves"]
        outs = qshift_mix(x, mixes, (case["grid_h"], case["grid_w"]))
        return (*[o.detach() for o in outs], *_grads(outs, state))
    with torch.no_grad(), torch.autocast("cuda", torch.bfloat16):
        return state["model"](state["img"])


def work(case):
    kind = case["kind"]
    if kind == "biwkv":
        n, size = case["B"] * case["T"] * case["C"], 2 if case["dtype"] == "bf16" else 4
        # k, v -> y (float32); training: k, v, gy (float32) -> gk, gv in the dtype of k, v
        nbytes = n * (2 * size + 4) + (n * (4 * size + 4) if case["train"] else 0)
        return {"bytes": nbytes, "flops": n * (10 if not case["train"] else 40)}
    if kind == "wkv6":
        n, size = case["B"] * case["T"] * case["H"] * 64, 2 if case["dtype"] == "bf16" else 4
        # r, k, v, w (float32) -> y (float32); training: those and gy -> gr, gk, gv like r, k, v, and gw (float32)
        nbytes = n * (3 * size + 8) + (n * (6 * size + 12) if case["train"] else 0)
        # two directions; state update and read-out of a 64-wide state, and four such pairs for the gradients
        return {"bytes": nbytes, "flops": n * 2 * 64 * 4 * (5 if case["train"] else 1)}
    if kind == "qshift":
        n = case["B"] * case["grid_h"] * case["grid_w"] * case["C"]
        return {"bytes": n * 4 * (2 * (1 + case["outputs"]) + 1), "flops": n * 10 * case["outputs"]}
    v6 = case["model"].startswith("vrwkv6")
    cfg = (backbone6.PRESETS_V6 if v6 else backbone.PRESETS)[case["model"]]
    C, depth, tokens = cfg["embed_dims"], cfg["depth"], case["B"] * case["grid_h"] * case["grid_w"]
    weights = 14 * C * C + 2 * (5 * 2 * 32 + 2 * 64) * C if v6 else 13 * C * C
    flops = tokens * (2 * 3 * PATCH * PATCH * C + depth * 2 * weights + (depth * C * 2 * 64 * 4 if v6 else 0))
    return {"bytes": 4 * (depth * weights + 3 * PATCH * PATCH * (C + tokens) + tokens * C), "flops": flops}


def tolerance(case):
    if case["kind"] == "backbone":
        return {"rel": 2e-2}                   # bfloat16 linear layers through 12 or 24 blocks
    if case["kind"] == "wkv6" and case["dtype"] == "bf16":
        return {"rel": 1e-2}                   # bfloat16 operands of the matrix products
    if case["kind"] == "biwkv" and case["dtype"] == "bf16":
        return {"rel": 4e-3}                   # one rounding of results and of gy to bfloat16
    return {"rel": 2e-5}                       # float32 sums, the parameter gradients over B * T terms
