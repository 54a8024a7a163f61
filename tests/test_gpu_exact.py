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
