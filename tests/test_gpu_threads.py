"""Several threads, each with a stream of its own."""
import threading
import time

import pytest
import torch

from helpers import make_case

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def test_a_launch_that_waits_does_not_stop_other_threads():
    """A stream whose queue is full makes the next launch wait; another thread's Python code runs on meanwhile."""
    from sparse_mla_sm120_b200 import indexer
    kv = torch.randn(4, 576, device=DEV).to(torch.bfloat16)
    indexer.pack_kv_cache(kv)
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def clock():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now
    other = threading.Thread(target=clock)
    other.start()
    time.sleep(0.05)
    torch.cuda._sleep(2_000_000_000)              # about a second
    t0 = time.perf_counter()
    while time.perf_counter() - t0 < 0.2:         # until a call takes long: the queue was full
        indexer.pack_kv_cache(kv)
    waited = time.perf_counter() - t0
    torch.cuda.synchronize()
    stop.set()
    other.join()
    assert waited > 0.4, f"no launch waited ({waited:.2f} s)"
    assert max(gaps) < 0.25, f"the other thread stood still for {max(gaps):.2f} s while one launch waited {waited:.2f} s"


def test_threads_with_streams_of_their_own():
    from sparse_mla_sm120_b200 import flash_ops
    cases = [{k: v.to(DEV) if torch.is_tensor(v) else v for k, v in make_case(40 + i, 2 + i, heads, 512, 16).items()}
             for i, heads in enumerate((16, 64, 128, 128))]
    parts = (None, 7, None, 9)

    def step(i):
        c = cases[i]
        return flash_ops.sparse_mla_decode_fwd(c["q"], c["packed"], c["indices"], c["sm_scale"], num_sm_parts=parts[i])
    want = [step(i) for i in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(100):
                out, lse = step(i)
                torch.cuda.current_stream().synchronize()
                if not (torch.equal(out, want[i][0]) and torch.equal(lse, want[i][1])):
                    wrong.append(i)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
