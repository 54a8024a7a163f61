"""The merge of partial records at numbers of splits where its read-ahead and the weights that it passes between lanes can go wrong."""
import ctypes

import pytest
import torch

from helpers import make_case, oracle_attn
from test_gpu_attention import TC, _check_hard

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("splits", [1, 2, 3, 4, 5, 31, 32, 33, 40, 65])
def test_fp32_records_of_any_number_of_splits(splits):
    """Against the formula in 64 bits; bf16 results, so half a step of the value and of the sum's largest term."""
    from sparse_mla_sm120_b200 import _lib
    g = torch.Generator().manual_seed(splits)
    t, h = 3, 5
    o = torch.randn(splits, t, h, 512, generator=g)
    lse = 4 * torch.randn(splits, t, h, generator=g)
    lse[0, 1, 2], o[0, 1, 2] = -1e30, 0                    # a split without an entry
    w = torch.exp2(lse.double() - lse.double().amax(0))
    ref = (w.unsqueeze(-1) * o.double()).sum(0) / w.sum(0).unsqueeze(-1)
    ref_lse = lse.double().amax(0) + torch.log2(w.sum(0))
    dev = torch.device("cuda:0")
    od, ld = o.to(dev), lse.to(dev)
    out, out_lse = torch.empty(t, h, 512, dtype=torch.bfloat16, device=dev), torch.empty(t, h, device=dev)
    lib = _lib.load()
    assert lib.smla_combine_parts(od.data_ptr(), ld.data_ptr(), out.data_ptr(), out_lse.data_ptr(), splits, t, h, None,
                                  torch.cuda.current_stream().cuda_stream) == 0
    d = (out.cpu().double() - ref).abs()
    live = ref_lse > -1e20
    assert bool((d <= 2.0 ** -8 * ref.abs() + 1e-5).all())
    assert float((out_lse.cpu().double() - ref_lse)[live].abs().max()) <= 1e-4


@pytest.mark.parametrize("k", [2, 4, 8, 16])
def test_fp16_records_of_equal_partitions(k):
    from sparse_mla_sm120_b200 import _lib, _runtime
    t, h, topk = 2, 128, 2048
    case = make_case(23, t, h, topk, 40, invalid_tail=0.0)
    ref_out, ref_lse = oracle_attn(case)
    dev = torch.device("cuda:0")
    q, kv, idx = case["q"].to(dev), case["packed"].to(dev), case["indices"].to(dev)
    o = torch.empty(k * t, h, 512, dtype=torch.half, device=dev)
    l = torch.empty(k * t, h, device=dev)
    out, lse = torch.empty(t, h, 512, dtype=torch.bfloat16, device=dev), torch.empty(t, h, device=dev)
    lib = _lib.load()
    assert lib.smla_decode_uniform(q.data_ptr(), kv.data_ptr(), idx.data_ptr(), o.data_ptr(), l.data_ptr(), out.data_ptr(), lse.data_ptr(), t, h, topk,
                                   ctypes.c_float(case["sm_scale"]), 64, 64 * 656, k, None, TC, _runtime.status_pointer(0),
                                   torch.cuda.current_stream().cuda_stream) == 0
    _check_hard(out.cpu(), lse.cpu(), ref_out, ref_lse, TC, case)
