"""Rows of the cache that were never written (all bytes zero, scales included) on the FP8-class kernels: a zero row has logit 0
and value 0, like any other row."""
import pytest
import torch

import helpers as H
from helpers import make_case, oracle_attn, orc
from test_gpu_attention import TC, _check, _check_hard, _decode, _prefill
from test_gpu_model1 import _compare, _m1_case, _oracle
from test_gpu_model1 import _decode as _decode_m1

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [16, 64, 128])
@pytest.mark.parametrize("zeros", ["first", "all", "scattered"])
def test_zero_rows(heads, zeros):
    """A first tile of zero rows before real ones (the running maximum starts from them), nothing but zero rows, and groups of
    eight entries that mix zero rows with entries without a row; whole requests and split ones."""
    case = make_case(23, 3, heads, 512, 16, invalid_tail=0.0)
    rows = case["packed"].view(-1, 656)
    empty = torch.arange(rows.shape[0] - 200, rows.shape[0])
    if zeros == "all":
        rows.zero_()
    else:
        rows[empty] = 0
        for t in range(3):
            idx = case["indices"][t]
            idx[idx >= int(empty[0])] = 5
            if zeros == "first":
                idx[:130] = empty[:130].int()
            else:
                idx[::3] = empty[:171].int()
    case["indices"][:, 3::16] = -1
    case["indices"][1, 77:] = -1
    ref_out, ref_lse = oracle_attn(case)
    out, mx, lse = _prefill(case, TC)
    results = [(out, lse)] + [_decode(case, TC, num_sm_parts=parts) for parts in (None, 2, 7)]
    for out, lse in results:
        if zeros == "all":
            assert not out.any()
            _check(out, lse, ref_out, ref_lse, TC)
        else:       # request 1 averages few real rows: the bound is what the roundings cost on these inputs
            _check_hard(out, lse, ref_out, ref_lse, TC, case)


@pytest.mark.parametrize("parts", [None, 3])
def test_zero_rows_of_the_584_byte_layout(parts):
    c = _m1_case(31, 3, 64, 256, nblk=16)
    pages = c["packed"].view(16, -1)
    pages[:8] = 0
    c["indices"][:, 0, :130] = torch.arange(130, dtype=torch.int32)
    c["indices"][2] %= 512
    c["deq"] = orc.dequantize_kv_model1(c["packed"])
    ref_out, ref_lse = _oracle(c)
    out, lse = _decode_m1(c, num_sm_parts=parts, impl=TC)
    H.compare_out(out.cpu(), ref_out, H.TC_ABS, H.TC_REL, H.TC_COS)
    _compare(out, lse, ref_out, ref_lse, impl=TC)
