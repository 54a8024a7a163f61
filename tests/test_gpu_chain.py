"""Kernels that start their prologue before the one in front of them has ended: calls back to back give what calls one at a time give."""
import pytest
import torch

from helpers import make_case

pytestmark = pytest.mark.gpu

DEV = "cuda:0"

# heads, tokens, topk, partitions: one CTA per request, pairs with and without cuts, the scheduler's partitions
FORMS = [(16, 2, 512, None), (16, 70, 2048, None), (128, 1, 2048, None), (128, 90, 512, None), (128, 3, 512, 7), (48, 5, 64, None), (8, 1, 192, 5)]


def _cases(heads, tokens, topk):
    got = []
    for seed in range(6):
        case = make_case(31 + seed, tokens, heads, topk, 48, invalid_tail=0.3 if seed & 1 else 0.0)
        got.append({k: v.to(DEV) if torch.is_tensor(v) else v for k, v in case.items()})
    return got


def _step(case, parts, q=None):
    from sparse_mla_sm120_b200 import flash_ops
    return flash_ops.sparse_mla_decode_fwd(case["q"] if q is None else q, case["packed"], case["indices"], case["sm_scale"], num_sm_parts=parts)


@pytest.mark.parametrize("heads,tokens,topk,parts", FORMS)
def test_calls_back_to_back(heads, tokens, topk, parts):
    """The scratch of a call is that of the one before it, and q is overwritten between them on the stream."""
    cases = _cases(heads, tokens, topk)
    want = []
    for c in cases:
        torch.cuda.synchronize()
        want.append([t.clone() for t in _step(c, parts)])
    torch.cuda.synchronize()
    q = torch.empty_like(cases[0]["q"])
    for _ in range(8):
        got = []
        for c in cases:
            got.append(_step(c, parts))
        for c in cases:
            q.copy_(c["q"])
            got.append(_step(c, parts, q))
        torch.cuda.synchronize()
        for (o, l), (wo, wl) in zip(got, want + want):
            assert torch.equal(o, wo) and torch.equal(l, wl)


@pytest.mark.parametrize("heads,tokens,topk,parts", FORMS)
def test_a_capture_that_joins_two_streams_before_the_call(heads, tokens, topk, parts):
    cases = _cases(heads, tokens, topk)[:2]
    side, other = torch.cuda.Stream(), torch.cuda.Stream()
    q, staged = torch.zeros_like(cases[0]["q"]), torch.empty_like(cases[0]["q"])
    with torch.cuda.stream(side):
        want = [[t.clone() for t in _step(c, parts)] for c in cases]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            other.wait_stream(side)
            with torch.cuda.stream(other):
                q.copy_(staged)
            first = _step(cases[1], parts)
            side.wait_stream(other)
            second = _step(cases[0], parts, q)
    staged.copy_(cases[0]["q"])
    torch.cuda.synchronize()
    for _ in range(5):
        q.zero_()
        torch.cuda.synchronize()
        graph.replay()
        torch.cuda.synchronize()
        for got, w in ((first, want[1]), (second, want[0])):
            assert torch.equal(got[0], w[0]) and torch.equal(got[1], w[1])


@pytest.mark.parametrize("heads", [16, 128])
@pytest.mark.parametrize("tokens", [2, 90])
def test_selection_packing_and_attention_over_the_same_buffers(tokens, heads):
    """Every input of the attention written by library kernels right in front of it: lengths (two places back), indices by the selection,
    cache rows by the packing, in buffers that every round overwrites."""
    from sparse_mla_sm120_b200 import _lib, flash_ops
    lib, topk, rows, rounds = _lib.load(), 512, 4096, 6
    g = torch.Generator(device=DEV).manual_seed(tokens + heads)
    latents = [torch.randn(rows, 576, device=DEV, generator=g).to(torch.bfloat16) for _ in range(rounds)]
    logits = [torch.randn(tokens, rows, device=DEV, generator=g) for _ in range(rounds)]
    lens = [torch.randint(1, topk + 1, (tokens,), device=DEV, generator=g, dtype=torch.int32) for _ in range(rounds)]
    q = (0.5 * torch.randn(tokens, heads, 576, device=DEV, generator=g)).to(torch.bfloat16)
    cache = torch.zeros(rows // 64, 64, 1, 656, dtype=torch.uint8, device=DEV)
    idx = torch.zeros(tokens, topk, dtype=torch.int32, device=DEV)
    length = torch.ones(tokens, dtype=torch.int32, device=DEV)

    def one(i, wait):
        stream = torch.cuda.current_stream().cuda_stream
        length.copy_(lens[i])
        wait()
        assert lib.smla_topk(logits[i].data_ptr(), None, None, idx.data_ptr(), tokens, rows, rows, topk, stream) == 0
        wait()
        assert lib.smla_pack_kv(latents[i].data_ptr(), cache.data_ptr(), rows, stream) == 0
        wait()
        got = flash_ops.sparse_mla_decode_fwd(q, cache, idx, 576 ** -0.5, topk_length=length)
        wait()
        return [t.clone() for t in got] if wait is torch.cuda.synchronize else got
    want = [one(i, torch.cuda.synchronize) for i in range(rounds)]
    for _ in range(6):
        got = [one(i, lambda: None) for i in range(rounds)]
        torch.cuda.synchronize()
        for (o, l), (wo, wl) in zip(got, want):
            assert torch.equal(o, wo) and torch.equal(l, wl)
