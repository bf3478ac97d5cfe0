"""Block sizes below 1, which the C entry points take: a negative one has
empty windows, so that every valid Birchfield-Tomasi cost is 0; 0 and -1 are
windows of one pixel."""
import numpy as np
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bs", [0, -1, -2, -3, -5, -41])
@pytest.mark.parametrize("D", [16, 48])
def test_refinement_block_sizes_match_the_oracle(bs, D):
    case = cases._lvl("bs", 163, 61, D, cases.BT, True, bs=bs)
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad


@pytest.mark.parametrize("bs", [-2, -5, -41])
@pytest.mark.parametrize("level", [False, True])
def test_fixed_disparities_empty_windows_cost_nothing(bs, level):
    case = cases._lvl("bs", 163, 61, 32, cases.BT, False, bs=bs) if level else cases._ss("bs", 163, 61, 32, cases.BT, bs=bs)
    assert not np.any(_runners.run_mine(case)["cost"])
