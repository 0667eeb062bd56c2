"""The score of a frame with more rows of tiles than a grid's y dimension takes,
against the C restatement of the reference."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import cref

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,nan", [(65535 * 64, False), (65535 * 64 + 70, True)])
def test_tall_frames(h, nan):
    w = 3
    rng = np.random.default_rng(h)
    img = rng.standard_normal((h, w), dtype=np.float32)
    var = rng.uniform(0.5, 2.0, (h, w)).astype(np.float32)
    if nan:
        img[h - 40, 1] = np.nan
    psf = rng.uniform(0.0, 1.0, (3, 3)).astype(np.float32)
    np.testing.assert_array_equal(_core.matched_filter(img, psf, var), cref.matched_filter(img, psf, var))
