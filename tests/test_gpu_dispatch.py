"""Which kernels a call launches, read from the nodes of a captured graph: both sides of every line of the dispatch of the
FP8-class attention over 656-byte rows."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
KERNELS = ("attn_tile_kernel", "attn_duo_kernel", "attn_pair_kernel", "attn_exact_kernel", "attn_scalar_kernel", "combine_kernel", "sched_meta_kernel")


def _launches(call, tmp_path):
    call()                                       # scratch, attributes of the first call
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    path = str(tmp_path / "graph.dot")
    cudart = ctypes.CDLL("libcudart.so.12")      # torch's
    cudart.cudaGraphDebugDotPrint.argtypes = [ctypes.c_void_p, ctypes.c_char_p, ctypes.c_uint]
    assert cudart.cudaGraphDebugDotPrint(graph.raw_cuda_graph(), path.encode(), 1) == 0
    with open(path) as f:
        text = f.read()
    return {k for k in KERNELS if k in text}


def _call(kind, heads, tokens, topk, parts=None, lengths=False, pad=0):
    from sparse_mla_sm120_b200 import flash_ops
    g = torch.Generator(device=DEV).manual_seed(1)
    pages = 64
    cache = torch.zeros(pages, 64 * 656 + pad, dtype=torch.uint8, device=DEV).as_strided((pages, 64, 1, 656), (64 * 656 + pad, 656, 656, 1))
    q = torch.randn(tokens, heads, 576, device=DEV, generator=g).to(torch.bfloat16)
    idx = torch.randint(0, pages * 64, (tokens, topk), device=DEV, generator=g, dtype=torch.int32)
    length = torch.full((tokens,), topk, device=DEV, dtype=torch.int32) if lengths else None
    if kind == "prefill":
        return lambda: flash_ops.sparse_mla_prefill_fwd(q, cache, idx, 576 ** -0.5, topk_length=length)
    return lambda: flash_ops.sparse_mla_decode_fwd(q, cache, idx, 576 ** -0.5, topk_length=length, num_sm_parts=parts)


@pytest.mark.parametrize("want,call", [
    ({"attn_duo_kernel"}, ("decode", 128, 64, 2048)),
    ({"attn_duo_kernel", "combine_kernel"}, ("decode", 128, 1, 2048)),             # equal partitions
    ({"attn_duo_kernel", "combine_kernel"}, ("decode", 65, 37, 2048)),
    ({"sched_meta_kernel", "attn_pair_kernel", "combine_kernel"}, ("decode", 128, 13, 2048, None, True)),
    ({"attn_duo_kernel"}, ("decode", 128, 16, 2048, None, True)),                  # ragged, half as many as a list has blocks
    ({"attn_duo_kernel"}, ("decode", 128, 1, 1024, None, True)),                   # ragged, short lists
    ({"sched_meta_kernel", "attn_pair_kernel", "combine_kernel"}, ("decode", 128, 3, 512, 7)),
    ({"attn_pair_kernel"}, ("decode", 128, 64, 2048, None, False, 656)),           # pages with padding between them
    ({"attn_duo_kernel"}, ("prefill", 128, 296, 960)),                             # four requests per pair of SMs
    ({"attn_pair_kernel"}, ("prefill", 128, 297, 960)),
    ({"attn_duo_kernel"}, ("prefill", 128, 297, 961)),
    ({"attn_duo_kernel"}, ("prefill", 65, 74, 64)),
    ({"attn_tile_kernel"}, ("prefill", 64, 75, 2048)),
    ({"attn_duo_kernel"}, ("prefill", 64, 74, 2048)),
    ({"attn_tile_kernel"}, ("prefill", 64, 74, 448)),
    ({"attn_duo_kernel"}, ("prefill", 64, 74, 512)),
    ({"attn_tile_kernel"}, ("prefill", 32, 74, 960)),
    ({"attn_duo_kernel"}, ("prefill", 32, 74, 1024)),
    ({"attn_tile_kernel", "combine_kernel"}, ("decode", 16, 48, 2048)),
])
def test_kernels_of_a_call(want, call, tmp_path):
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("the lines are those of 148 SMs")
    assert _launches(_call(*call), tmp_path) == want
