"""attn_exact_kernel (exact numerics over the 584-byte layout) at the sizes where its tiles, head halves and number
conversions can go wrong, against the oracle."""
import pytest
import torch

import helpers as H
from helpers import orc
from test_gpu_model1 import FP32, _compare, _decode, _m1_case, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h", [1, 32, 33, 64, 65, 128])
@pytest.mark.parametrize("topk,extra", [(1, 0), (64, 1), (129, 65), (190, 0)])
def test_edges_of_tiles_and_heads(h, topk, extra):
    """A tile is two 64-token blocks of a request, a CTA 64 heads; requests shorter than a tile, ragged ends, a second
    cache that starts in the middle of a tile; whole requests, straddling partitions and more partitions than blocks."""
    c = _m1_case(7, 3, h, topk, extra_topk=extra, nblk=8)
    c["indices"] = torch.randint(0, 8 * 64, (3, 1, topk), generator=torch.Generator().manual_seed(1), dtype=torch.int32)
    c["indices"][1, 0, ::3] = -1
    ref_out, ref_lse = _oracle(c)
    for parts in (None, 2, 3, 16):
        out, lse = _decode(c, num_sm_parts=parts, impl=FP32)
        _compare(out, lse, ref_out, ref_lse, impl=FP32)


def test_every_byte_and_scale():
    """Subnormal values, scales beyond 2^7 (which a bf16 power of two cannot hold together with the 2^120 of the
    conversion) and the smallest scale."""
    c = _m1_case(9, 2, 64, 256, nblk=8)
    g = torch.Generator().manual_seed(2)
    page = c["packed"].reshape(8, 64 * 584)
    data, foot = page[:, :64 * 576].view(8, 64, 576), page[:, 64 * 576:].view(8, 64, 8)
    sign = torch.randint(0, 2, (8, 64, 128), generator=g, dtype=torch.uint8) * 128
    data[:, :, :128] = torch.randint(0, 8, (8, 64, 128), generator=g, dtype=torch.uint8) + sign      # subnormal: m x 2^-9
    foot[:, :, 0] = torch.randint(128, 136, (8, 64), generator=g, dtype=torch.uint8)
    foot[:, :, 1] = 0
    c["q"][..., :64] *= 0.02                                                                          # moderate logits all the same
    c["deq"] = orc.dequantize_kv_model1(c["packed"])
    ref_out, ref_lse = _oracle(c)
    out, lse = _decode(c, impl=FP32)
    H.compare_out(out.cpu(), ref_out, 1e-4, H.SCALAR_REL)
    _compare(out[..., 128:], lse, ref_out[..., 128:], ref_lse, impl=FP32)


@pytest.mark.parametrize("byte", [0x7F, 0xFF])
@pytest.mark.parametrize("at", [0, 15, 16, 250, 447])
def test_a_byte_that_is_no_number_stays_none(byte, at):
    """A NaN in a row that a request selects makes all of that request's outputs NaN, and nobody else's; as the fp32 kernel has it,
    which serves the same call over caches that are only 4-byte aligned."""
    c = _m1_case(12, 3, 64, 200, nblk=8)
    c["indices"][:, 0, 190:] = -1
    c["indices"][c["indices"] == 77] = 78
    c["indices"][1, 0, 131] = 77
    base_out, base_lse = _decode(c, num_sm_parts=3, impl=FP32)
    c["packed"].view(8, -1)[1, 13 * 576 + at] = byte           # row 77: token 13 of page 1
    out, lse = _decode(c, num_sm_parts=3, impl=FP32)
    assert torch.isnan(out[1].float()).all()
    for r in (0, 2):
        assert torch.equal(out[r], base_out[r]) and torch.equal(lse[r], base_lse[r])
    buf = torch.zeros(c["packed"].numel() + 64, dtype=torch.uint8, device="cuda:0")
    moved = buf[4:4 + c["packed"].numel()].view(c["packed"].shape)
    moved.copy_(c["packed"])
    slow, slow_lse = _decode(dict(c, packed=moved), num_sm_parts=3, impl=FP32)
    assert torch.equal(torch.isnan(slow.float()), torch.isnan(out.float())) and torch.equal(slow_lse[1], lse[1])


def test_a_scale_byte_of_255():
    """No number in UE8M0: infinity times the block's values in both kernels."""
    c = _m1_case(13, 2, 8, 64, nblk=8)
    c["indices"][c["indices"] == 5] = 6
    c["indices"][0, 0, 3] = 5
    c["packed"].view(8, -1)[0, 64 * 576 + 5 * 8 + 2] = 255
    out, lse = _decode(c, num_sm_parts=2, impl=FP32)
    assert not torch.isfinite(out[0].float()).any() and torch.isfinite(out[1].float()).all()
