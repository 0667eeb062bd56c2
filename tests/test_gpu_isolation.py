"""Brightest-first isolation on both sides of the rule that resolves a chunk a kept
stamp at a time where a frame has room for few, against NumPy (positions: equal)."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_select_sizes import _greedy, _image

from delta_b200 import _core

pytestmark = pytest.mark.gpu


# At 1024 x 1024 the rule turns between radius 59 and 60. One candidate, a full chunk,
# one more, several chunks and more than one CTA sorts; one stamp, a few, all there is
# room for; a radius larger than the frame.
@pytest.mark.parametrize("count", [1, 1024, 1025, 3000, 16385])
@pytest.mark.parametrize("iso,most", [(59, 8192), (60, 1), (60, 200), (61, 8192), (200, 3), (200, 5000), (3000, 200)])
def test_isolation_of_few_stamps(count, iso, most):
    size, margin = 1024, 30
    rng = np.random.default_rng(count + iso)
    grid = np.arange(margin, size - margin, 5)
    at = rng.choice(len(grid) ** 2, count, replace=False)
    xs, ys = grid[at % len(grid)], grid[at // len(grid)]
    values = (200.0 + rng.integers(0, 500, count)).astype(np.float32)
    got = _core.detect_stamps(_image(xs, ys, values, size), stamp_radius=6, threshold_sigma=60.0, max_stamps=most,
                              isolation_radius=iso)
    kx, ky = _greedy(xs, ys, values, size, iso, most)
    np.testing.assert_array_equal(got["x"], kx)
    np.testing.assert_array_equal(got["y"], ky)
