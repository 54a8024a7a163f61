"""The cut of the indexer's key tiles into runs, compiled from its header for the host: within its bounds, and no longest share of a
CTA longer than that of the shortest runs."""
import ctypes
import os
import subprocess

import pytest

from helpers import ROOT

SMS = 148


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    d = tmp_path_factory.mktemp("runs")
    with open(d / "runs.cpp", "w") as f:
        f.write('#include "logits_runs.cuh"\nextern "C" int runs(int g, int t, int s) { return smla::logits_runs(g, t, s); }\n')
    subprocess.run(["g++", "-std=c++17", "-O2", "-shared", "-fPIC", "-I" + os.path.join(ROOT, "sparse_mla_sm120_b200", "csrc"), "-o", str(d / "runs.so"),
                    str(d / "runs.cpp")], check=True)
    return ctypes.CDLL(str(d / "runs.so")).runs


def _share(groups, tiles, c):
    return -(-groups * c // SMS) * (-(-tiles // c) + 5)


def test_bounds_and_shares(runs):
    for groups in (1, 2, 3, 4, 8, 37, 75, 148, 149, 256, 500, 625, 750, 1024, 1183, 1184, 5000):
        for tiles in (1, 7, 8, 9, 32, 40, 71, 157, 512, 1024, 8192):
            c = runs(groups, tiles, SMS)
            shortest = max(min(-(-8 * SMS // groups), -(-tiles // 8)), 1)
            assert 1 <= c <= shortest
            assert _share(groups, tiles, c) <= _share(groups, tiles, shortest)


def test_two_sides_of_the_lines(runs):
    assert runs(4, 1024, SMS) == 37                       # one run per CTA
    assert runs(750, 512, SMS) == 2                       # 3000 tokens: whole groups would take a sixth round that is nearly empty
    assert runs(625, 157, SMS) == 2
    assert runs(750, 40, SMS) == 1                        # short lists: a second item costs more than the round
    assert runs(1024, 512, SMS) == 2 and runs(1024, 128, SMS) == 1
    assert runs(1184, 512, SMS) == 1                      # eight items per SM
