"""Penalties below zero (k_paths_signed.cu), which the C entry points take as
the reference does, against the oracle: label counts of every number of labels
a lane, each path count, both costs, adaptive penalties."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu

PENALTIES = [(-5, 900), (200, -20), (-7, -30)]


def _check(case):
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, _runners.device_lut(case)))
    assert not bad, bad


@pytest.mark.parametrize("P1,P2", PENALTIES)
@pytest.mark.parametrize("D,w,h", [(16, 121, 30), (48, 144, 41), (96, 230, 30), (272, 400, 12), (1024, 1100, 5)])
@pytest.mark.parametrize("cost,paths,minD", [(cases.BT, 3, 0), (cases.CENSUS, 2, -6), (cases.CENSUS, 1, 4),
                                             (cases.CENSUS, 3, 0)])
def test_single_scale_negative_penalties_match_the_oracle(P1, P2, D, w, h, cost, paths, minD):
    _check(cases._ss("neg", w, h, D, cost, P1=P1, P2=P2, paths=paths, minD=minD, adaptive=paths == 3,
                     post=cases.LRC | (cases.MED if paths == 2 else 0)))


@pytest.mark.parametrize("P1,P2", PENALTIES)
@pytest.mark.parametrize("D,w,h", [(16, 121, 30), (64, 150, 41), (112, 230, 30), (256, 300, 12)])
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("cost,paths", [(cases.BT, 3), (cases.CENSUS, 2), (cases.CENSUS, 1)])
def test_level_negative_penalties_match_the_oracle(P1, P2, D, w, h, refine, cost, paths):
    _check(cases._lvl("neg", w, h, D, cost, refine, P1=P1, P2=P2, paths=paths, adaptive=paths == 3, minConf=0.0,
                      maxD=min(w - 1, 2 * D)))
