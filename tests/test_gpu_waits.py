"""The bounded wait of the attention kernels when it runs out: it ends, and the first code stays on record."""
import ctypes
import os
import subprocess

import pytest
import torch

from helpers import ROOT

pytestmark = pytest.mark.gpu


def test_a_wait_that_runs_out(tmp_path):
    lib_path = str(tmp_path / "wait_giveup.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-shared", "-Xcompiler", "-fPIC",
                    "-I" + os.path.join(ROOT, "sparse_mla_sm120_b200", "csrc"), "-o", lib_path, os.path.join(ROOT, "tests", "wait_giveup.cu")], check=True)
    lib = ctypes.CDLL(lib_path)
    result, cycles = torch.full((4,), -1, dtype=torch.int32, device="cuda:0"), torch.zeros(3, dtype=torch.int64, device="cuda:0")
    assert lib.run_waits(ctypes.c_void_p(result.data_ptr()), ctypes.c_void_p(cycles.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert result.tolist() == [1, 0, 0, 71]
    done, first, second = cycles.tolist()
    assert 0 < done < first                       # 4097 polls each
    print("cycles of a poll:", first / 4097, second / 4097)
