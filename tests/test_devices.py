"""Calls whose tensors lie on several GPUs are refused, and a call on another GPU than the current one runs there."""
import pytest
import torch

DEV = "cuda:0"


def _calls(q, kv, idx, other):
    """Every op with one of its tensors replaced by ``other(shape, dtype)``, one at a time."""
    from sparse_mla_sm120_b200 import flash_ops, indexer
    f32, i32, u8, e4 = torch.float32, torch.int32, torch.uint8, torch.float8_e4m3fn
    for op in (flash_ops.sparse_mla_decode_fwd, flash_ops.sparse_mla_prefill_fwd):
        yield lambda op=op: op(q, other((4, 64, 1, 656), u8), idx, 1.0)
        yield lambda op=op: op(q, kv, other((1, 64), i32), 1.0)
        yield lambda op=op: op(q, kv, idx, 1.0, attn_sink=other((128,), f32))
        yield lambda op=op: op(q, kv, idx, 1.0, topk_length=other((1,), i32))
        yield lambda op=op: op(q, kv, idx, 1.0, out=other((1, 128, 512), torch.bfloat16))
        yield lambda op=op: op(q, kv, idx, 1.0, extra_k_cache=other((4, 64, 1, 656), u8), extra_indices=idx, extra_topk=64)
    make = lambda shape, dt: torch.empty(shape, dtype=dt, device=DEV)
    shapes = [((2, 64, 128), e4), ((9, 128), e4), ((9,), f32), ((2, 64), f32), ((2,), i32), ((2,), i32)]
    for i in range(1, 6):
        yield lambda i=i: indexer.fp8_mqa_logits(*[other(*s) if j == i else make(*s) for j, s in enumerate(shapes)])
    yield lambda: indexer.topk_indices(make((2, 9), f32), other((2,), i32), make((2,), i32), 3)
    yield lambda: indexer.topk_indices(make((2, 9), f32), make((2,), i32), other((2,), i32), 3)


def test_tensors_of_several_devices_are_refused():
    """With tensors that have a device but no memory (no GPU needed: the refusal comes before anything is launched)."""
    from torch._subclasses.fake_tensor import FakeTensorMode
    with FakeTensorMode():
        q = torch.empty(1, 128, 576, dtype=torch.bfloat16, device=DEV)
        kv = torch.empty(4, 64, 1, 656, dtype=torch.uint8, device=DEV)
        idx = torch.empty(1, 64, dtype=torch.int32, device=DEV)
        calls = list(_calls(q, kv, idx, lambda shape, dt: torch.empty(shape, dtype=dt, device="cuda:1")))
        for call in calls:
            with pytest.raises(ValueError, match="different devices"):
                call()


@pytest.mark.gpu
@pytest.mark.skipif(torch.cuda.device_count() < 2, reason="needs two GPUs")
def test_a_call_runs_on_its_tensors_device():
    """The default stream of cuda:1 while cuda:0 is current."""
    from helpers import make_case
    from sparse_mla_sm120_b200 import flash_ops
    from sparse_mla_sm120_b200._lib import native
    case = make_case(1, 3, 64, 256, 8)
    want = [t.cpu() for t in flash_ops.sparse_mla_decode_fwd(case["q"].to(DEV), case["packed"].to(DEV), case["indices"].to(DEV), case["sm_scale"])]
    with torch.cuda.device(0):
        q, kv, idx = (case[k].to("cuda:1") for k in ("q", "packed", "indices"))
        got = flash_ops.sparse_mla_decode_fwd(q, kv, idx, case["sm_scale"])
        copy = torch.zeros_like(q)
        native().copy_into((copy,), (q,))
        torch.cuda.synchronize(1)
        assert torch.cuda.current_device() == 0
    assert all(torch.equal(a.cpu(), b) for a, b in zip(got, want)) and torch.equal(copy, q)
