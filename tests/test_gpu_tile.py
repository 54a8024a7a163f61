"""attn_tile_kernel (up to 64 heads over one linear array of 656-byte rows) at the sizes where its tiles, head halves,
partitions and weights can go wrong, against the oracle."""
import pytest
import torch

import helpers as H
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


@pytest.mark.parametrize("heads", [16, 64])
@pytest.mark.parametrize("pattern", ["steady", "late", "mixed"])
def test_small_blocks_keep_their_precision(heads, pattern):
    """Blocks whose scales lie far below the row's largest, with logits of about +-6: every block of dims against its own
    magnitude, held to the emulation's error on the same inputs as test_scale_spread_rows does (there at 128 heads, which
    run on the pair kernel).  steady: small in every row; late: rows of a later tile are the first with a large block, so
    what was accumulated for it has to come down; mixed: small in two rows of three."""
    case = make_case(17, 80, heads, 640, 32, q_std=2.0, invalid_tail=0.0)     # (fewer whole requests run on attn_duo_kernel)
    scales = case["packed"].view(-1, 656)[:, 512:528].view(torch.float32)
    if pattern == "steady":
        scales[:, 1] *= 2.0 ** -6
        scales[:, 2] *= 2.0 ** -9
    elif pattern == "late":
        case["indices"] = torch.sort(case["indices"], dim=1).values.contiguous()
        scales[:500, 1] *= 2.0 ** -9
        scales[500:1000, 2] *= 2.0 ** -5
        scales[:, 3] *= 2.0 ** -11
        scales[1000:, 3] *= 2.0 ** 3
    else:
        scales[0::3, 1] *= 2.0 ** -9
        scales[1::3, 1] *= 2.0 ** -4
        scales[1:, 2] *= 2.0 ** -8
    ref_out, ref_lse = oracle_attn(case)
    emu_out, _ = H.orc.emulate_fp8_attention(case["q"], case["packed"], case["indices"], case["sm_scale"])
    results = [_prefill(case, TC)[0]] + [_decode(case, TC, num_sm_parts=parts)[0] for parts in (None, 2, 90)]
    for out in results:
        for b in range(4):
            sl = slice(128 * b, 128 * b + 128)
            ref = ref_out.float()[..., sl]
            e_k = float((out.cpu().float()[..., sl] - ref).pow(2).mean().sqrt())
            e_e = float((emu_out.float()[..., sl] - ref).pow(2).mean().sqrt())
            rms = float(ref.pow(2).mean().sqrt())
            assert e_k <= H.EMU_MARGIN * e_e + 2.0 ** -8 * rms, (b, e_k / rms, e_e / rms)


def _prefill_padded(case):
    """The call over pages with padding between them: the pair kernel's."""
    from sparse_mla_sm120_b200 import flash_ops
    dev = torch.device("cuda:0")
    nb, stride = case["packed"].shape[0], 64 * 656 + 256
    kv = torch.as_strided(torch.zeros(nb * stride, dtype=torch.uint8, device=dev), (nb, 64, 1, 656), (stride, 656, 656, 1))
    kv.copy_(case["packed"].to(dev))
    out = flash_ops.sparse_mla_prefill_fwd(case["q"].to(dev), kv, case["indices"].to(dev), case["sm_scale"], 512, impl=TC)
    return [t.cpu() for t in out]


@pytest.mark.parametrize("heads", [16, 64])
def test_weights_are_rounded_as_by_the_pair_kernel(heads):
    """The same whole requests over pages with and without padding (the pair kernel and attn_tile_kernel): the same maxima and
    the same rounded weights, so the outputs differ by sums in another order and by values below 2^-6 that the pair
    kernel cuts when it moves them to its group's scale, not by another realisation of the roundings (3e-3 of the rms)."""
    case = make_case(19, 80, heads, 512, 16, invalid_tail=0.1)
    a, mx_a, lse_a = _prefill(case, TC)
    b, mx_b, lse_b = _prefill_padded(case)
    d = (a.float() - b.float()).pow(2).mean().sqrt() / b.float().pow(2).mean().sqrt()
    assert float(d) <= 5e-4, float(d)
    assert float((lse_a - lse_b).abs().max()) <= 1e-4 and float((mx_a - mx_b).abs().max()) <= 1e-4


@pytest.mark.parametrize("heads,topk,tokens", [(33, 448, 74), (33, 449, 74), (33, 704, 74), (33, 705, 74), (33, 705, 75), (32, 960, 74), (32, 961, 74),
                                               (64, 1024, 1), (64, 1024, 76)])
def test_whole_requests_on_either_side_of_the_line_to_the_pair_kernel(heads, topk, tokens):
    """Lists and numbers of requests at which whole requests go to the other kernel, with and without maximum logits."""
    case = make_case(31, tokens, heads, topk, 20, invalid_tail=0.1)
    ref_out, ref_lse = oracle_attn(case)
    out, mx, lse = _prefill(case, TC)
    _check_hard(out, lse, ref_out, ref_lse, TC, case)
    out2, lse2 = _decode(case, TC, num_sm_parts=tokens)
    _check_hard(out2, lse2, ref_out, ref_lse, TC, case)
    d = (out.float() - out2.float()).pow(2).mean().sqrt() / out.float().pow(2).mean().sqrt()
    assert float(d) <= 5e-4 and float((lse - lse2).abs().max()) <= 1e-4      # the same roundings on both (see above)
