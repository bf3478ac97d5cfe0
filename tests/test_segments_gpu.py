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


# Label counts that keep one path volume (k_paths_sum.cuh): the middle of a
# row, where the two directions meet, at even and odd widths.
@pytest.mark.parametrize("kind", ["band", "texture"])
@pytest.mark.parametrize("w,h", [(301, 43), (190, 66)])
@pytest.mark.parametrize("paths,minD", [(1, 0), (2, 0), (3, 0), (3, -9), (3, 5)])
@pytest.mark.parametrize("D,cost", [(48, cases.CENSUS), (96, cases.BT), (128, cases.BT), (160, cases.CENSUS)])
def test_one_volume_single_scale_matches_the_oracle(kind, w, h, paths, minD, D, cost):
    case = cases._ss("sum", w, h, D, cost, paths=paths, minD=minD, adaptive=paths == 3)
    case["pair"] = _images(kind, w, h)
    _check(case)


@pytest.mark.parametrize("w,h,D", [(700, 19, 272), (1100, 17, 512), (1100, 9, 1008), (1500, 130, 1024)])
def test_one_volume_large_label_counts_match_the_oracle(w, h, D):
    case = cases._ss("sum", w, h, D, cases.CENSUS)
    case["pair"] = _images("texture", w, h)
    _check(case)
    case = cases._lvl("sum", w, h, D, cases.CENSUS, False, paths=3)
    case["pair"] = _images("band", w, h)
    _check(case)


@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("paths", [1, 2, 3])
@pytest.mark.parametrize("w,h,D", [(301, 131, 48), (202, 57, 112), (330, 40, 256)])
def test_one_volume_pyramid_levels_match_the_oracle(refine, paths, w, h, D):
    _check(cases._lvl("sum", w, h, D, cases.BT if D == 48 else cases.CENSUS, refine, paths=paths, adaptive=paths != 2,
                      maxD=min(w - 1, 2 * D), seed=w))


# ... and walks of a few steps, whose parts are less than a chunk.
@pytest.mark.parametrize("extra", [1, 2, 3, 4, 5, 7, 9, 14])
@pytest.mark.parametrize("D", [48, 80, 128, 144])
@pytest.mark.parametrize("paths,minD", [(1, 0), (2, 0), (3, 0), (3, -3), (2, 4)])
def test_one_volume_short_rows_match_the_oracle(extra, D, paths, minD):
    _check(cases._ss("sum", D + max(minD, 0) + extra, 19, D, cases.CENSUS, paths=paths, minD=minD, adaptive=extra % 2 == 1))


@pytest.mark.parametrize("w", [49, 50, 51, 52, 55])
@pytest.mark.parametrize("refine", [False, True])
@pytest.mark.parametrize("paths", [1, 2, 3])
def test_one_volume_narrow_levels_match_the_oracle(w, refine, paths):
    _check(cases._lvl("sum", w, 23, 48, cases.BT, refine, paths=paths, adaptive=paths != 2, seed=w))
