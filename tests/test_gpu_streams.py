"""Handles on a stream that the caller owns and uses from another thread too: what that
thread enqueues runs once, in its order, also while the library records its graphs
(at creation and, for graphs of several cycles, in the middle of a run)."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(sgh, p, st, stream):
    with sgh.SGHSolver(p, stream=stream) as s:
        s.set_state(st)
        for n in (20, 40, 20):  # past the mark where larger graphs are made
            s.run(n)
        return s.get_state(), s.time()


def test_foreign_work_on_the_callers_stream(lib_built):
    import torch

    from fierro_gb300 import problems, sgh
    p = problems.noh(6, jitter=0.1, seed=2, permute=True, cycles=100)
    st = sgh.setup(p)
    want, wt = _run(sgh, p, st, None)
    stream = torch.cuda.Stream()
    count = torch.zeros(1, dtype=torch.int64, device="cuda")
    count.add_(1)  # the kernel is loaded before the thread starts
    torch.cuda.synchronize()
    done, added, errors = threading.Event(), [1], []

    def foreign():
        try:
            with torch.cuda.stream(stream):
                while not done.is_set() and added[0] < 2_000_000:
                    count.add_(1)
                    added[0] += 1
        except Exception as exc:  # reported by the main thread
            errors.append(exc)

    t = threading.Thread(target=foreign)
    t.start()
    try:
        runs = []
        while len(runs) < 12 or (added[0] < 1000 and len(runs) < 200 and not errors):
            runs.append(_run(sgh, p, st, stream.cuda_stream))
    finally:
        done.set()
        t.join()
    stream.synchronize()
    assert not errors, errors
    assert added[0] > 1000
    assert int(count.item()) == added[0]
    for got, gt in runs:
        assert gt == wt
        for k in want:
            assert np.array_equal(got[k], want[k]), k


@pytest.mark.parametrize("before", [0, 20, 30])
def test_cycles_enqueued_while_the_caller_captures_another_stream(lib_built, before):
    """Enqueueing makes the larger graphs on the way; the caller's open capture goes on."""
    import torch

    from fierro_gb300 import problems, sgh
    p = problems.noh(6, jitter=0.1, seed=2, permute=True, cycles=100)
    st = sgh.setup(p)
    with sgh.SGHSolver(p) as s:
        s.set_state(st)
        s.run_stages(2 * (before + 40))
        want, wt = s.get_state(), s.time()
    stream, x, g = torch.cuda.Stream(), torch.zeros(4, device="cuda"), torch.cuda.CUDAGraph()
    with sgh.SGHSolver(p) as s:
        s.set_state(st)
        s.run(before)
        torch.cuda.synchronize()
        with torch.cuda.graph(g, stream=stream):
            x.add_(1.0)
            s.enqueue(40)
        s.synchronize()
        got, gt = s.get_state(), s.time()
    g.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [1.0] * 4 and gt == wt
    for k in want:
        assert np.array_equal(got[k], want[k]), k
