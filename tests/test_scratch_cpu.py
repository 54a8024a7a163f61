"""Who shares the scratch of the split steps: never a graph with anybody, never two streams with each other."""
import torch

from sparse_mla_sm120_b200 import _runtime


class _Stream:
    def __init__(self, handle):
        self.cuda_stream = handle


def test_a_capture_gets_buffers_of_its_own(monkeypatch):
    state = {"stream": 1, "capturing": False}
    monkeypatch.setattr(_runtime, "_scratch", {})
    monkeypatch.setattr(torch.cuda, "current_stream", lambda device=None: _Stream(state["stream"]))
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: state["capturing"])
    dev = torch.device("cpu")

    def address(tokens=2):
        ws = _runtime.scratch(dev, tokens + 3, 4, tokens, 3)
        return ws, {k: t.data_ptr() for k, t in ws.items() if torch.is_tensor(t)}

    warm, at_warm = address()
    state["capturing"] = True
    first, at_first = address()
    second, at_second = address()
    state["capturing"] = False
    again, at_again = address()
    assert at_again == at_warm                       # eager calls of a stream share theirs
    for k in at_warm:
        assert len({at_warm[k], at_first[k], at_second[k]}) == 3, k
    state["stream"] = 2
    _, at_other = address()
    assert all(at_other[k] != at_warm[k] for k in at_warm)
    kept = [address(t)[0] for t in range(4, 4 + 2 * _runtime._SCRATCH_LIMIT)]
    assert len(_runtime._scratch) <= _runtime._SCRATCH_LIMIT and kept[-1] is list(_runtime._scratch.values())[-1]
