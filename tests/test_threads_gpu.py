"""Two threads, each with a workspace and a stream of its own, calling at the
same time with sizes whose launches of one kernel need different amounts of
shared memory: every call succeeds and gives what it gives alone."""
import threading

import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu

PAIRS = {
    "chains": (cases._lvl("a", 640, 480, 16, cases.CENSUS, True), cases._lvl("b", 320, 180, 16, cases.CENSUS, True)),
    "columns": (cases._ss("a", 400, 300, 96, cases.CENSUS), cases._ss("b", 1280, 121, 96, cases.CENSUS)),
    "strips": (cases._ss("a", 200, 60, 64, cases.BT), cases._ss("b", 200, 60, 16, cases.BT)),
    "boxes": (cases._ss("a", 200, 60, 32, cases.BT, bs=25), cases._ss("b", 200, 60, 32, cases.BT, bs=29)),
}


def _caller(case):
    """A call of the case on a stream of its own -> (return code, its outputs)."""
    import torch
    import pyrsgm_gb300 as pg
    left, right, parent = _runners.inputs(case)
    left, right = _runners._dev(left), _runners._dev(right)
    parent = [_runners._dev(p) if p is not None else None for p in parent]
    h, w = left.shape
    out = [torch.zeros((h, w), dtype=t, device="cuda") for t in (torch.int16, torch.float32, torch.float32)]
    ws, stream = pg.Workspace(), torch.cuda.Stream()
    common = dict(num_disparities=case["D"], block_size=case["bs"], p1=case["P1"], p2=case["P2"], cost_mode=case["cost"],
                  stream=stream)
    torch.cuda.synchronize()

    def call():
        if case["kind"] == "ss":
            return pg.compute_single_scale(ws, left, right, *out, **common)
        return pg.compute_level(ws, left, right, *parent, *out, max_disparity=case["maxD"], refine=case["refine"],
                                **common)
    return call, stream, out


@pytest.mark.parametrize("kind", sorted(PAIRS))
def test_two_threads_do_not_fail_each_other(kind):
    callers = [_caller(c) for c in PAIRS[kind]]
    alone = []
    for call, stream, out in callers:
        assert call() == 0
        stream.synchronize()
        alone.append([t.clone() for t in out])
    wrong = [[], []]

    def work(i):
        call, stream, out = callers[i]
        for n in range(6000):
            if call() != 0:
                wrong[i].append(n)
            if n % 1000 == 999:
                stream.synchronize()
                if not all(bool((a == b).all()) for a, b in zip(out, alone[i])):
                    wrong[i].append(-n)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert wrong == [[], []]
