"""attn_tile_kernel (up to 64 heads over one linear array of 656-byte rows) at the sizes where its tiles, head halves,
partitions and weights can go wrong, against the oracle."""
import pytest
import torch

from helpers import make_case, oracle_attn
from test_gpu_attention import TC, _check_hard, _decode, _prefill

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [1, 16, 32, 33, 64])
@pytest.mark.parametrize("topk", [1, 64, 129, 1024])
def test_edges_of_tiles_and_heads(heads, topk):
    """A tile is two 64-token blocks of a request; partitions that hold whole requests, straddle two or are smaller than a
    tile; a request without entries; lengths and a negative softmax scale."""
    case = make_case(3, 5, heads, topk, 16, invalid_tail=0.2)
    case["indices"][3] = -1
    tl = torch.tensor([topk, 1, max(topk // 2, 1), topk, topk], dtype=torch.int32)
    for scale in (case["sm_scale"], -case["sm_scale"]):
        case["sm_scale"] = scale
        ref_out, ref_lse = oracle_attn(case, topk_length=tl)
        out, mx, lse = _prefill(case, TC, topk_length=tl)
        _check_hard(out, lse, ref_out, ref_lse, TC, case, topk_length=tl)
        for parts in (None, 2, 3, 16):
            out, lse = _decode(case, TC, num_sm_parts=parts, topk_length=tl)
            _check_hard(out, lse, ref_out, ref_lse, TC, case, topk_length=tl)


@pytest.mark.parametrize("tokens,topk", [(1, 2048), (24, 512), (320, 192)])
def test_equal_requests_and_several_per_cta(tokens, topk):
    """Equal partitions (no scheduler), and more requests than CTAs; the four blocks of a row have scales far apart, so that
    every block of dims needs weights of its own."""
    case = make_case(11, tokens, 64, topk, 32, invalid_tail=0.0)
    scales = case["packed"].view(-1, 656)[:, 512:528].view(torch.float32)
    scales[:, 1] *= 2.0 ** -4
    scales[::2, 3] *= 2.0 ** -7
    ref_out, ref_lse = oracle_attn(case)
    out, lse = _decode(case, TC)
    _check_hard(out, lse, ref_out, ref_lse, TC, case)
