"""attn_duo_kernel (65 to 128 heads over one linear array of 656-byte rows) at the sizes where its tiles, head halves,
partitions and shifted pieces of V can go wrong, against the oracle."""
import pytest
import torch

import helpers as H
from helpers import make_case, oracle_attn
from test_gpu_attention import TC, _check_hard, _decode, _prefill
from test_gpu_tile import _prefill_padded

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("heads", [65, 97, 127, 128])
@pytest.mark.parametrize("topk", [1, 64, 129, 1024])
def test_edges_of_tiles_and_heads(heads, topk):
    """A tile is two 64-token blocks of a request, one gathered by each CTA; partitions that hold whole requests, straddle two or
    are smaller than a tile; a request without entries; lengths and a negative softmax scale."""
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


@pytest.mark.parametrize("tokens,topk", [(1, 2048), (24, 512), (160, 192)])
def test_equal_requests_and_several_per_pair(tokens, topk):
    """Equal partitions (no scheduler), and more requests than pairs; the four blocks of a row have scales far apart, so that
    most pieces of V are shifted, some by more powers of two than e4m3 has."""
    case = make_case(11, tokens, 128, topk, 32, invalid_tail=0.0)
    scales = case["packed"].view(-1, 656)[:, 512:528].view(torch.float32)
    scales[:, 1] *= 2.0 ** -4
    scales[::2, 3] *= 2.0 ** -7
    scales[5::8, 2] *= 2.0 ** -20
    ref_out, ref_lse = oracle_attn(case)
    out, lse = _decode(case, TC)
    _check_hard(out, lse, ref_out, ref_lse, TC, case)


@pytest.mark.parametrize("heads,tokens", [(72, 80), (128, 33), (40, 60)])
def test_weights_are_rounded_as_by_the_pair_kernel(heads, tokens):
    """The same whole requests over pages with and without padding (the pair kernel and attn_duo_kernel): the same groups, maxima and
    weights, so the outputs differ by sums in another order and by values below 2^-6 that the pair kernel cuts from K when it
    moves it to its group's scale, not by another realisation of the roundings (3e-3 of the rms)."""
    case = make_case(19, tokens, heads, 1024, 20, invalid_tail=0.1)
    a, mx_a, lse_a = _prefill(case, TC)
    b, mx_b, lse_b = _prefill_padded(case)
    d = (a.float() - b.float()).pow(2).mean().sqrt() / b.float().pow(2).mean().sqrt()
    assert float(d) <= 5e-4, float(d)
    assert float((lse_a - lse_b).abs().max()) <= 1e-4 and float((mx_a - mx_b).abs().max()) <= 1e-4


def test_entries_without_a_row_leave_no_trace():
    """A -1 is a row outside the tensor map: poisoning the row that it would be clamped to with NaN must not change a bit."""
    case = make_case(13, 80, 128, 256, 8, invalid_tail=0.25)
    case["indices"][case["indices"] == 0] = 1

    def run(c):
        out, mx, lse = _prefill(c, TC)
        out2, lse2 = _decode(c, TC, num_sm_parts=60)
        return [t.view(torch.int16) if t.dtype == torch.bfloat16 else t for t in (out, mx, lse, out2, lse2)]
    base = run(case)
    poisoned = case["packed"].clone()
    poisoned.view(-1, 656)[0, :512] = 0x7F
    poisoned.view(-1, 656)[0, 528:] = torch.tensor([0xC0, 0x7F] * 64, dtype=torch.uint8)
    for a, b in zip(run(dict(case, packed=poisoned)), base):
        assert torch.equal(a, b)
    ref_out, ref_lse = oracle_attn(case)
    moved = dict(case, indices=torch.cat([case["indices"][:, 192:], case["indices"][:, :192]], dim=1).contiguous())
    out, mx, lse = _prefill(moved, TC)              # whole tiles' halves without an entry lead
    _check_hard(out, lse, ref_out, ref_lse, TC, moved)


@pytest.mark.parametrize("heads", [65, 97, 127])
@pytest.mark.parametrize("k", [2, 8])
def test_head_halves_of_equal_partitions(heads, k):
    """A CTA has heads without a query and the second fewer than the first; partitions of whole tiles and of two blocks."""
    import ctypes
    from sparse_mla_sm120_b200 import _lib, _runtime
    t, topk = 3, 1024
    case = make_case(29, t, heads, topk, 40, invalid_tail=0.1)
    ref_out, ref_lse = oracle_attn(case)
    dev = torch.device("cuda:0")
    q, kv, idx = case["q"].to(dev), case["packed"].to(dev), case["indices"].to(dev)
    o, l = torch.empty(k * t, heads, 512, dtype=torch.half, device=dev), torch.empty(k * t, heads, device=dev)
    out, lse = torch.empty(t, heads, 512, dtype=torch.bfloat16, device=dev), torch.empty(t, heads, device=dev)
    assert _lib.load().smla_decode_uniform(q.data_ptr(), kv.data_ptr(), idx.data_ptr(), o.data_ptr(), l.data_ptr(), out.data_ptr(), lse.data_ptr(), t, heads,
                                           topk, ctypes.c_float(case["sm_scale"]), 64, 64 * 656, k, None, TC, _runtime.status_pointer(0),
                                           torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    _runtime.check_status(dev)
    _check_hard(out.cpu(), lse.cpu(), ref_out, ref_lse, TC, case)


@pytest.mark.parametrize("heads", [65, 97, 127])
def test_head_halves_of_several_requests_per_pair(heads):
    """More requests than pairs of SMs, of one to three tiles: the next request's q goes through tensor memory."""
    case = make_case(37, 170, heads, 320, 24, invalid_tail=0.0)
    g = torch.Generator().manual_seed(heads)
    tl = torch.randint(0, 321, (170,), generator=g, dtype=torch.int32)
    ref_out, ref_lse = oracle_attn(case, topk_length=tl)
    out, mx, lse = _prefill(case, TC, topk_length=tl)
    _check_hard(out, lse, ref_out, ref_lse, TC, case, topk_length=tl)
