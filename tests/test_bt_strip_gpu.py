"""Birchfield-Tomasi cost of fixed disparities in strips (k_cost_bt_strip)
against the oracle's cost volume: label blocks of every width, column and
strip remainders, windows of 3 to 9 pixels (9 takes the general kernel)."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(31, 9), (64, 28), (65, 29), (131, 61), (259, 13)])
@pytest.mark.parametrize("D", [16, 32, 48, 64, 80, 112, 128])
@pytest.mark.parametrize("bs", [3, 5, 7, 9])
def test_single_scale_cost_matches_the_oracle(w, h, D, bs):
    case = cases._ss("strip", w, h, D, cases.BT, bs=bs, minD=-3 if bs == 5 else 2 if bs == 3 else 0, seed=w + D)
    mine = _runners.run_mine(case)
    bad = _runners.compare(mine, _runners.run_oracle(case, None))
    assert not bad, bad


@pytest.mark.parametrize("w,h,D,bs", [(240, 135, 32, 3), (133, 70, 16, 5), (97, 200, 64, 7)])
def test_coarse_level_cost_matches_the_oracle(w, h, D, bs):
    case = cases._lvl("strip", w, h, D, cases.BT, False, bs=bs)
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad
