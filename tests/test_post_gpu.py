"""LR check and median (k_post) against the oracle: tile remainders, widths
that are no multiple of four, every way the check decides (no winner counting
or not, limits from 0 to wider than the image)."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu

SIZES = [(128, 8), (131, 17), (260, 33), (97, 7)]


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("maxdiff", [0, 2, 4000, 65500, 70000])
@pytest.mark.parametrize("minD", [0, 5, -4])
def test_single_scale_check_matches_the_oracle(w, h, maxdiff, minD):
    case = cases._ss("post", w, h, 32, cases.CENSUS, minD=minD, maxdiff=maxdiff, uniq=0, post=cases.LRC | cases.MED,
                     seed=w)
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("maxdiff", [0, 2, 4000, 65500, 70000])
@pytest.mark.parametrize("refine", [False, True])
def test_level_check_matches_the_oracle(w, h, maxdiff, refine):
    case = cases._lvl("post", w, h, 16, cases.CENSUS, refine, maxdiff=maxdiff, uniq=0, post=cases.LRC | cases.MED,
                      seed=w)
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad
