"""What the kernels that start under the one before them may do, read from their source: no loads that are defined only for memory
which nothing writes meanwhile, and the next kernel let go only after the wait."""
import glob
import os
import re

import pytest

from helpers import ROOT

CSRC = os.path.join(ROOT, "sparse_mla_sm120_b200", "csrc")


def _code(path):
    with open(path) as f:
        return re.sub(r"//[^\n]*", "", f.read())


SOURCES = {os.path.basename(p): _code(p) for p in sorted(glob.glob(os.path.join(CSRC, "*.cu*")))}


def _launched():
    """kernel -> file, of every kernel that a launch_dependent() names (directly, or through a variable `kernel`)."""
    got = {}
    for name, text in SOURCES.items():
        for args in re.findall(r"launch_dependent\((?!void)(.*?);", text, re.S):
            kernels = re.findall(r"\b(\w+_kernel)\b", args) or re.findall(r"\bkernel = .*?\b(\w+_kernel)\b", text)
            assert kernels, (name, args)
            got.update((k, name) for k in kernels)
    return got


def _body(text, kernel):
    """(parameters, body) of a __global__ function."""
    m = re.search(r"__global__[^;{]*?\b" + kernel + r"\s*\(([^{]*?)\)\s*\{", text, re.S)
    assert m, kernel
    depth, i = 1, m.end()
    while depth:
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        i += 1
    return m.group(1), text[m.end():i]


def test_the_kernels_are_found():
    assert {"attn_duo_kernel", "attn_tile_kernel", "attn_pair_kernel", "attn_exact_kernel", "combine_kernel", "sched_meta_kernel", "pack_kv_kernel",
            "mqa_logits_tc_kernel", "topk_select_kernel", "topk_cluster_kernel"} <= set(_launched())


@pytest.mark.parametrize("kernel,name", sorted(_launched().items()))
def test_loads_and_order(kernel, name):
    params, body = _body(SOURCES[name], kernel)
    assert "__restrict__" not in params
    for load in ("__ldg", "__ldca", "__ldcg", "__ldcs", "__ldlu", "__ldcv", ".nc."):
        assert load not in body, load
    wait, launch = body.index("grid_dep_wait()"), body.index("grid_dep_launch()")
    assert wait < launch and "return;" not in body[:wait]


@pytest.mark.parametrize("name", sorted(n for n in SOURCES if n.endswith(".cuh")))
def test_shared_helpers_load_coherently(name):
    assert not re.search(r"__ld(g|ca|cg|cs|lu|cv)\b|ld\.global\.nc|__restrict__", SOURCES[name])


@pytest.mark.parametrize("name", sorted({n for n in _launched().values()}))
def test_helpers_beside_the_kernels_load_coherently(name):
    """What is left of a file without the kernels that are launched the ordinary way."""
    text = SOURCES[name]
    for kernel in re.findall(r"__global__[^;{]*?\b(\w+_kernel)\s*\(", text):
        if kernel not in _launched():
            params, body = _body(text, kernel)
            text = text.replace(params, "").replace(body, "")
    assert not re.search(r"__ld(g|ca|cg|cs|lu|cv)\b|ld\.global\.nc|__restrict__", text)
