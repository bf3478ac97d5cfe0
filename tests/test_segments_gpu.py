"""Path chains cut into segments (k_paths_seg.cuh) against the oracle.

Sizes leave remainders at the segment, chunk and chain-group edges; the
images are the ones on which a chain forgets its start slowly or never
(flat, a flat band between textures, stripes), so that segments are walked
again, several times over and across their ends.
"""
import numpy as np
import pytest

from . import _runners, cases

pytestmark = pytest.mark.gpu


def _images(kind, w, h, seed=5):
    rng = np.random.default_rng(seed)
    tex = rng.integers(0, 256, (h, w + 64)).astype(np.uint8)
    shift = 7
    if kind == "flat":
        left = np.full((h, w), 90, np.uint8)
        right = left.copy()
    elif kind == "band":                    # texture, a wide flat band, texture
        left, right = tex[:, 32:32 + w].copy(), tex[:, 32 + shift:32 + shift + w].copy()
        for im in (left, right):
            im[:, w // 4:3 * w // 4] = 120
            im[h // 4:3 * h // 4, :] = 120
    elif kind == "stripes":                 # ambiguous matches
        x = np.arange(w + 64)
        row = np.where((x // 4) % 2 == 0, 200, 40).astype(np.uint8)
        img = np.repeat(row[None, :], h, 0)
        left, right = img[:, 32:32 + w], img[:, 32 + shift:32 + shift + w]
    else:
        left, right = tex[:, 32:32 + w], tex[:, 32 + shift:32 + shift + w]
    return np.ascontiguousarray(left), np.ascontiguousarray(right)


SIZES = [(400, 121), (163, 242), (1281, 41)]


def _check(case):
    mine = _runners.run_mine(case)
    bad = _runners.compare(mine, _runners.run_oracle(case, _runners.device_lut(case)))
    assert not bad, bad


@pytest.mark.parametrize("kind", ["flat", "band", "stripes", "texture"])
@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("D,cost,adaptive", [(16, cases.CENSUS, True), (32, cases.BT, False), (64, cases.CENSUS, True),
                                             (64, cases.BT, False)])
def test_single_scale_segments_match_the_oracle(kind, w, h, D, cost, adaptive):
    case = cases._ss("seg", w, h, D, cost, adaptive=adaptive)
    case["pair"] = _images(kind, w, h)
    _check(case)


@pytest.mark.parametrize("kind", ["flat", "band", "stripes", "texture"])
@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("paths", [1, 2, 3])
@pytest.mark.parametrize("D,cost", [(16, cases.BT), (32, cases.CENSUS), (64, cases.BT)])
def test_coarse_level_segments_match_the_oracle(kind, w, h, D, cost, paths):
    case = cases._lvl("seg", w, h, D, cost, False, paths=paths, adaptive=paths == 3)
    case["pair"] = _images(kind, w, h)
    _check(case)


@pytest.mark.parametrize("w,h", SIZES)
@pytest.mark.parametrize("D,cost,P2", [(16, cases.BT, None), (16, cases.CENSUS, None), (32, cases.CENSUS, None),
                                       (64, cases.BT, None), (16, cases.BT, 20000)])
def test_refinement_segments_match_the_oracle(w, h, D, cost, P2):
    _check(cases._lvl("seg", w, h, D, cost, True, P2=P2, adaptive=P2 is None, seed=w))
