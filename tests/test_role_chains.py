"""The warp roles of a kernel, read from its source: a chain of branches names each role once (a second branch of the same condition
is never entered)."""
import glob
import os
import re

import pytest

from helpers import ROOT

FILES = sorted(glob.glob(os.path.join(ROOT, "sparse_mla_sm120_b200", "csrc", "*.cu")))


@pytest.mark.parametrize("path", FILES, ids=[os.path.basename(p) for p in FILES])
def test_every_role_once(path):
    with open(path) as f:
        kernels = f.read().split("__global__")[1:]
    for text in kernels:
        later = re.findall(r"^    \} else if \((warp [^{]*?)\) \{$", text, re.M)
        assert len(later) == len(set(later)), later
