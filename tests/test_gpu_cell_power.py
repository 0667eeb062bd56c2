"""Decorrelation on both sides of the rule that sends the kernel powers through one
launch, against the FP64 oracle."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


# Kernels of up to half a block take one launch (63 of 128 columns; 65 do not), while
# their rows fit in shared memory (81 of 256; 129 do not); blocks of 64 never do. One
# cell, several, and more than the CTAs that share a cell's columns.
@pytest.mark.parametrize("h,w,block,cells,n_max,radius", [
    (200, 190, 128, 0, 3, 31), (200, 190, 128, 0, 3, 32), (90, 100, 128, 1, 0, 0), (300, 310, 256, 1, 3, 40),
    (300, 310, 256, 1, 3, 64), (300, 310, 256, 0, 9, 0), (1000, 900, 128, 1, 2, 0), (100, 110, 64, 1, 2, 5)])
def test_kernel_power_rule(h, w, block, cells, n_max, radius):
    rng = np.random.default_rng(h + w + radius)
    beta, nk = 1.3, 4
    knots = nr.grid_knots(0, 0, w - 1, h - 1, nk, nk)
    nc, k = (n_max + 1) * (n_max + 2) // 2, nk * nk
    theta = 0.02 * rng.standard_normal((nc + 1) * k)
    theta[k - 3] = 1.0
    diff = (rng.standard_normal((h, w)) * 10.0).astype(np.float32)
    vs = rng.uniform(80.0, 120.0, (h, w)).astype(np.float32)
    vr = rng.uniform(40.0, 60.0, (h, w)).astype(np.float32)
    args = (diff, knots, theta, beta, n_max, vs, vr)
    got = _core.decorrelate(*args, block=block, radius=radius, kernel_cell_blocks=cells)
    want = nr.decorrelate(*args, block=block, radius=radius, kernel_cell_blocks=cells)
    np.testing.assert_allclose(got["variance"], want["variance"], rtol=2e-6)
    assert np.max(np.abs(got["difference"] - want["difference"]) / np.sqrt(want["variance"])) < 1e-4
