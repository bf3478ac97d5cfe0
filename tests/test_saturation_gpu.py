"""Penalties on both sides of the point where an active chain's best may reach
SHRT_MAX (k_paths_seg.cuh: load_penalties, highest cost + 2 P2), fixed and
through the adaptive table, against the oracle: coarse and refinement levels,
every chain shape and a label count that keeps one path volume, the lowest and
the highest costs."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu

# (cost, block size, highest cost of a label)
COSTS = [(cases.CENSUS, 3, 24), (cases.BT, 1, 255), (cases.BT, 11, 255 * 121)]


def _check(case):
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, _runners.device_lut(case)))
    assert not bad, bad


@pytest.mark.parametrize("D", [16, 32, 64, 96])
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("cost,bs,top", COSTS)
@pytest.mark.parametrize("step", [0, 1, 4000])
@pytest.mark.parametrize("adaptive", [False, True])
def test_penalties_around_the_saturation_bound_match_the_oracle(D, refine, cost, bs, top, step, adaptive):
    P2 = (32767 - top) // 2 + step
    if adaptive:
        P2 = int(P2 / 1.77)          # the table's highest entry is 1.77 P2
    _check(cases._lvl("sat", 260, 47, D, cost, refine, bs=bs, P1=P2 // 3, P2=P2, adaptive=adaptive, minConf=0.0,
                      maxD=min(259, 2 * D), seed=D + step))
