"""Birchfield-Tomasi cost of refinement levels (k_cost_bt_tiled) against the
oracle's cost volume: sizes with ragged tiles and halves of one, parents that
need several clusters a tile, label counts of more than one pass, windows of
1 to 7 pixels (7 takes the direct sums)."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(40, 17), (157, 61), (209, 100), (320, 64)])
@pytest.mark.parametrize("D", [16, 32, 48])
@pytest.mark.parametrize("bs", [1, 3, 5, 7])
def test_refinement_cost_matches_the_oracle(w, h, D, bs):
    case = cases._lvl("tiled", w, h, D, cases.BT, True, bs=bs, seed=w + D + bs)
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad
