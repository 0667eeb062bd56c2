"""FP64 normal equations at the edges of their tiling, against NumPy.

theta of a fixed-lambda solve is compared with the dense FP64 solution of the
same rows. Both accumulate X^T W X over n rows (relative error at most n eps
of the products' magnitude, in practice sqrt(n) eps) and solve a system of
condition number c, so they agree to about sqrt(n) eps c; the bound is ten
times that.
"""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _dense(knots, pts, t, w, bn, lam):
    tp = nr.ThinPlate(knots)
    d = tp.design(pts)
    b = np.column_stack([bn, np.ones(len(t))])
    x = (b[:, :, None] * d[:, None, :]).reshape(len(t), -1)
    a = x.T @ (x * w[:, None]) + lam * np.kron(np.eye(b.shape[1]), tp.penalty)
    return np.linalg.solve(a, x.T @ (w * t)), np.linalg.cond(a)


# (components, knots per side, rows): one product pair in all, a tile row of
# each height (1 to 7 groups of 32 pairs, exact and with a remainder), one and
# several tiles of 48 design pairs, rows below a chunk, at its edge and past
# it, and the widest rows a fit accepts.
@pytest.mark.parametrize("nc,side,n", [
    (0, 3, 40), (1, 3, 31), (1, 3, 32), (1, 3, 33), (2, 4, 64), (6, 3, 500), (9, 3, 1025), (13, 3, 2048), (15, 3, 1999),
    (18, 4, 3001), (20, 3, 1023), (21, 5, 4096), (28, 4, 4097), (28, 5, 6001), (40, 4, 5000), (66, 3, 4003),
    (1, 14, 3000),
])
def test_fp64_normal_equations_at_tile_edges(nc, side, n):
    rng = np.random.default_rng(1000 * nc + 10 * side + n)
    knots = nr.grid_knots(0, 0, 100, 80, side, side)
    pts = np.column_stack([rng.uniform(0, 100, n), rng.uniform(0, 80, n)])
    bn = rng.normal(size=(n, nc))
    w = rng.uniform(0.2, 2.0, n)
    t = bn.sum(1) + 0.5 + rng.normal(size=n)
    got = _core.solve_gls(knots, pts, t, w, bn, 1e-2)["theta"]
    want, cond = _dense(knots, pts, t, w, bn, 1e-2)
    tol = 10 * np.sqrt(n) * np.finfo(float).eps * cond
    assert np.linalg.norm(got - want) <= tol * np.linalg.norm(want)



# Unknowns below, at and past the 32-column panels of the LDL^T, up to 23
# panels. One component is zero at every row, so the Cholesky fails and the
# system goes through the fallback; its zero pivots are the diagonal's ties.
# The other unknowns are well determined (the bound of the fallback's own test).
@pytest.mark.parametrize("nc,side,n", [(3, 3, 900), (6, 3, 1500), (7, 4, 2500), (12, 5, 4000), (28, 5, 6000)])
def test_ldlt_fallback_at_panel_edges(nc, side, n):
    rng = np.random.default_rng(nc)
    knots = nr.grid_knots(0, 0, 100, 80, side, side)
    pts = np.column_stack([rng.uniform(0, 100, n), rng.uniform(0, 80, n)])
    bn = rng.normal(size=(n, nc))
    bn[:, 2] = 0.0
    w = rng.uniform(0.5, 2.0, n)
    t = bn.sum(1) + 0.5 + 0.1 * rng.normal(size=n)
    got = _core.solve_gls(knots, pts, t, w, bn, 0.1)
    want = nr.solve_gls(knots, pts, t, w, bn, 0.1)
    assert got["used_ldlt"]
    np.testing.assert_allclose(got["theta"], want["theta"], rtol=1e-7, atol=1e-9)
    np.testing.assert_allclose(got["effective_dof"], want["effective_dof"], rtol=1e-8)
