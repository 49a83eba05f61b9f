"""Kernels that may be started while the one before them in the stream still runs (csrc/launch.h), read from their source.  What they find
in global memory may change until they have waited, so each waits before it does anything else, and none tells the compiler that an input never
changes (`__ldg`, `ld.global.nc`, a `const` pointer that is `__restrict__`): such a load needs no order with the wait, wherever it is written."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vision-rwkv_b200", "csrc")
WAIT = "wait_for_launch_before();"


def source(name):
    with open(os.path.join(CSRC, name)) as f:
        text = f.read()
    return re.sub(r"//[^\n]*", "", text)


def included(name, seen):
    """`name` and the files of this folder that it includes"""
    if name not in seen:
        seen[name] = source(name)
        for other in re.findall(r'#include "([^"]+)"', seen[name]):
            if os.path.exists(os.path.join(CSRC, other)):
                included(other, seen)
    return seen


FILES = sorted(f for f in os.listdir(CSRC) if f.endswith(".cu") and "launch.h" in included(f, {}))


def kernels(text):
    """(name, parameters, body up to its end) of every kernel"""
    for head in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\([^)]*\)\s*)?(\w+)\s*\(", text):
        at, depth = head.end(), 1
        while depth:
            depth += {"(": 1, ")": -1}.get(text[at], 0)
            at += 1
        if text[at:].lstrip().startswith("{"):
            yield head.group(1), text[head.end():at - 1], text[text.index("{", at) + 1:]


def test_the_files_are_found():
    assert {"mixer_epilogue.cu", "linear_batch.cu", "linear_tc.cu", "qshift_mix.cu", "qshift_ddlerp.cu", "wkv6_chunk.cu", "wkv6_sweeps.cu", "wkv6_tc.cu",
            "biwkv_strips.cu"} <= set(FILES)
    assert sum(len(list(kernels(source(f)))) for f in FILES) >= 30


@pytest.mark.parametrize("name", FILES)
def test_kernels_launched_early_wait_first(name):
    text = source(name)
    for kernel, _, body in kernels(text):
        before = body.split(WAIT)[0]
        if WAIT in body and re.fullmatch(r"(\s*((extern\s+)?__shared__[^;]*|launch_dependents\(\));)*\s*", before):
            continue
        uses = [m for m in re.finditer(rf"\b{kernel}\b", text) if not re.search(r"(void|__launch_bounds__\([^)]*\))\s*$", text[:m.start()])]
        assert uses
        for use in uses:      # launched in full only
            assert re.match(r"\s*(<[^;<>]*>)?\s*<<<", text[use.end():]), f"{kernel} is launched early and does not wait first"


@pytest.mark.parametrize("name", FILES)
def test_kernels_launched_early_let_their_inputs_change(name):
    for file, text in included(name, {}).items():
        assert "__ldg(" not in text and "ld.global.nc" not in text and "ld.global.L1" not in text, file
        for kernel, parameters, _ in kernels(text):
            for parameter in parameters.split(","):
                assert not ("const" in parameter and "__restrict__" in parameter), f"{file}: {kernel}: {parameter.strip()}"
