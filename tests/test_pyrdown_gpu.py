"""pyrDown (k_pyrdown) against the oracle: widths of every alignment, images
smaller than a tile, tiles at every border."""
import numpy as np
import pytest

from . import _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [4, 37, 258, 259, 513, 514, 515, 516])
@pytest.mark.parametrize("h", [3, 32, 67, 70])
@pytest.mark.parametrize("pad", [0, 3, 4])
def test_pyrdown_matches_the_oracle(w, h, pad):
    import torch
    import pyrsgm_gb300 as pg
    src = np.random.default_rng(w * 100 + h).integers(0, 256, (h, w)).astype(np.uint8)
    src[: h // 2, : w // 2] = 255
    buf = torch.zeros((h, w + pad), dtype=torch.uint8, device="cuda")
    view = buf[:, :w]
    view.copy_(torch.from_numpy(src))
    out = torch.zeros(((h + 1) // 2, (w + 1) // 2), dtype=torch.uint8, device="cuda")
    pg.pyrdown(view, out)
    assert np.array_equal(out.cpu().numpy(), _oracle.orc_pyrdown(src))
