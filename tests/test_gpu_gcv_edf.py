"""The edf part of the stamp-GCV gradient at the edges of its tiling, against
the FP64 oracle.

grad_gcv - alpha grad_rss = beta dedf (alpha = n / (n - edf)^2) holds only the
effective-degrees-of-freedom part, a smooth sum of positive weights without the
residual's cancellation: the device's float32 stamp convolutions (relative
error about 1e-7 each, entering twice) leave it within 1e-5 of the FP64 value,
and the bound is ten times that.
"""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core, validation
from oracle import grad_ref
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


# Component pairs below, at and above one tile of 48 and of 96; 9, 16 and 25
# knots (design pairs 45, 136 and 325: a remainder of the 16-pair chunk each);
# rows that are not a multiple of 128, masked rows and clipped stamps among them.
@pytest.mark.parametrize("n_max,side,sr", [(0, 3, 5), (1, 4, 6), (2, 3, 8), (3, 4, 7), (4, 3, 6), (5, 4, 6), (6, 5, 7)])
def test_edf_gradient_matches_fp64_oracle(n_max, side, sr):
    w, h = 210, 190
    p = validation.synthetic_pair(w, h, 60, 20 + n_max, mask_fraction=0.02)
    rng = np.random.default_rng(n_max)
    sx = np.concatenate([[3, w - 4], rng.integers(10, w - 10, 13)]).astype(np.int32)
    sy = np.concatenate([[5, h - 2], rng.integers(10, h - 10, 13)]).astype(np.int32)
    knots = nr.grid_knots(0, 0, w - 1, h - 1, side, side)
    x = (np.log(3.0), 0.11, -0.17, 1.03)
    got = _core.stamp_gcv(p.science, p.reference, knots, sx, sy, sr, 1.6, n_max, *x, science_var=p.science_var,
                          reference_var=p.reference_var, science_mask=p.science_mask, reference_mask=p.reference_mask)
    want = grad_ref.StampGCV(p.science, p.reference, p.science_var, p.reference_var, p.science_mask, p.reference_mask,
                             knots, sx, sy, sr, 1.6, n_max).grad(*x)

    def edf_part(r):
        n = got["n_pixels"]
        return (np.asarray(r["grad_gcv"]) - n / (n - r["effective_dof"]) ** 2 * np.asarray(r["grad_rss"]))[1:]

    a, b = edf_part(got), edf_part(want)
    np.testing.assert_allclose(a, b, rtol=0, atol=1e-4 * np.abs(b).max())
