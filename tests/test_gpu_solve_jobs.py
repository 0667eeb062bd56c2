"""The batched solver's job ring at the edges of its job counts and at each of its
cluster sizes: against the FP64 oracle, and the same bits whatever the number of CTAs."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _problem(nc, nk, n):
    rng = np.random.default_rng(100 * nc + nk)
    knots = nr.grid_knots(0, 0, 499, 399, nk, nk)
    pts = np.column_stack([rng.uniform(0, 500, n), rng.uniform(0, 400, n)])
    bn = rng.standard_normal((n, nc)) * rng.uniform(0.5, 5.0, nc)
    f = nr.ThinPlate(knots).design(pts) @ (rng.standard_normal((nc + 1, knots.shape[0])).T * 0.3)
    target = f[:, nc] + np.sum(f[:, :nc] * bn, axis=1) + 0.05 * rng.standard_normal(n)
    return knots, pts, target, rng.uniform(0.5, 2.0, n), bn


# Unknowns: 8 and 32 (one tile: no trailing job), 36 (two), 99 and 175 (ragged), 725.
# Grid points: clusters of 8 (1, 18), 4 (40), 2 (100) CTAs and single ones (160).
@pytest.mark.parametrize("nc,nk,grids", [(1, 2, (1, 18, 40, 100, 160)), (1, 4, (1, 160)), (3, 3, (1, 18, 40, 100, 160)),
                                         (10, 3, (1, 18, 40, 100, 160)), (6, 5, (1, 40, 100, 160)),
                                         (28, 5, (1, 18, 40, 100, 160))])
def test_every_cluster_size_matches_the_oracle(nc, nk, grids):
    args = _problem(nc, nk, 4000 if nc < 20 else 12000)
    lam = 10.0 ** -1.5
    one = _core.solve_gls(*args, lam)
    want = nr.solve_gls(*args, lam)
    np.testing.assert_allclose(one["theta"], want["theta"], rtol=1e-6, atol=1e-8)
    np.testing.assert_allclose(one["effective_dof"], want["effective_dof"], rtol=1e-7)
    for size in grids:
        # the point itself, and all others far above it: they cannot win
        grid = np.r_[lam, np.logspace(7, 9, size)[: size - 1]]
        got = _core.solve_gls_gcv(*args, grid)
        assert got["lambda"] == lam
        np.testing.assert_array_equal(got["theta"], one["theta"])
        np.testing.assert_allclose(got["effective_dof"], one["effective_dof"], rtol=1e-12)
