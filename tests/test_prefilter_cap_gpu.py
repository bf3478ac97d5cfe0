"""Birchfield-Tomasi costs with gradient caps of every size against the
oracle, whose gradients are bytes as the reference's: the last cap whose
offset gradient fits a byte, the first whose does not, caps above every
gradient and above 16 bits; the strip, the general and the refinement kernel."""
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu

CAPS = [127, 128, 200, 1020, 1023, 31747, 31749, 32767, 40000, 65537, 2**31 - 1]


def _check(case):
    bad = _runners.compare(_runners.run_mine(case), _runners.run_oracle(case, None))
    assert not bad, bad


@pytest.mark.parametrize("cap", CAPS)
@pytest.mark.parametrize("D,bs", [(32, 5), (48, 9)])
def test_single_scale_caps_match_the_oracle(cap, D, bs):
    _check(cases._ss("cap", 163, 41, D, cases.BT, bs=bs, pfc=cap))


@pytest.mark.parametrize("cap", CAPS)
@pytest.mark.parametrize("bs", [1, 3, 5])
def test_refinement_caps_match_the_oracle(cap, bs):
    _check(cases._lvl("cap", 163, 41, 16, cases.BT, True, bs=bs, pfc=cap))
