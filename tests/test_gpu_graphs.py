"""Captured decode steps beside each other and beside eager ones: nothing that a call needs for itself is shared with a graph."""
import pytest
import torch

from helpers import make_case

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def _step(case, parts):
    from sparse_mla_sm120_b200 import flash_ops
    return flash_ops.sparse_mla_decode_fwd(case["q"], case["packed"], case["indices"], case["sm_scale"], num_sm_parts=parts)


def _on_gpu(seed, topk=512):
    case = make_case(seed, 3, 128, topk, 32, invalid_tail=0.0)
    return {k: v.to(DEV) if torch.is_tensor(v) else v for k, v in case.items()}


@pytest.mark.parametrize("parts", [None, 7])
def test_a_capture_allocates_its_scratch(parts):
    """What the capture asks the allocator for holds the partial records too, although an eager call of the same shape ran on the
    stream before (None: equal partitions with 16-bit records, k of them per request; 7: the scheduler's 32-bit ones)."""
    case = _on_gpu(1, topk=2048)
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        _step(case, parts)
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["requested_bytes.all.allocated"]
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out, lse = _step(case, parts)
    asked = torch.cuda.memory_stats()["requested_bytes.all.allocated"] - before
    records = (3 + 7) * 128 * 512 * 4 if parts else 2 * 3 * 128 * 512 * 2
    assert asked >= out.nbytes + lse.nbytes + records, (asked, out.nbytes, lse.nbytes, records)


def test_graphs_of_one_stream_replayed_side_by_side():
    """Two graphs captured on one stream, replayed on two others at a time, and eager steps on the stream of the capture: every
    result is that of the step alone."""
    cases = [_on_gpu(s) for s in (1, 2, 3)]
    side, streams = torch.cuda.Stream(), [torch.cuda.Stream(), torch.cuda.Stream()]
    with torch.cuda.stream(side):
        want = [[t.clone() for t in _step(c, 7)] for c in cases]
        graphs, got = [], []
        for c in cases[:2]:
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=side):
                got.append(_step(c, 7))
            graphs.append(g)
    torch.cuda.synchronize()
    for _ in range(100):
        for g, s in zip(graphs, streams):
            with torch.cuda.stream(s):
                g.replay()
        with torch.cuda.stream(side):
            eager = _step(cases[2], 7)
        torch.cuda.synchronize()
        for (o, l), (wo, wl) in zip(got + [eager], want):
            assert torch.equal(o, wo) and torch.equal(l, wl)
