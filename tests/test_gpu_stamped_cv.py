"""The stamped cross-validation (per-stamp moments and their fold sums on the FP64
tensor cores, fold systems without the degrees-of-freedom rows) at the edges of its
tiles, against the NumPy fit. Both sides form the same float32 B_n and FP64 sums in
another order, so a solution is known to 2^-53 times its system's condition; held-out
errors are compared to 1e-6 or, where that is larger, to 8 times this."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu

GRID = np.logspace(-4, 6, 21)


def _frame(n_stamps, sr, side=420, seed=0):
    rng = np.random.default_rng(seed + n_stamps)
    ref = rng.normal(100.0, 1.0, (side, side))
    ys, xs = np.mgrid[0:side, 0:side]
    px, py = rng.integers(sr + 2, side - sr - 2, (2, n_stamps))
    for x, y, f in zip(px, py, rng.uniform(300.0, 3000.0, n_stamps)):
        near = (slice(max(0, y - 9), y + 10), slice(max(0, x - 9), x + 10))
        ref[near] += f * np.exp(-((xs[near] - x) ** 2 + (ys[near] - y) ** 2) / 4.0)
    sci = nr.convolve_y(nr.convolve_x(ref, np.array([0.1, 0.25, 0.4, 0.2, 0.05])), np.array([0.2, 0.5, 0.3]))
    sci += rng.normal(0.0, 1.0, ref.shape)
    mask = (rng.random(ref.shape) < 0.03).astype(np.uint8)
    return sci.astype(np.float32), ref.astype(np.float32), mask, px.astype(np.int32), py.astype(np.int32)


def _compare(sci, ref, mask, px, py, sr, n_max, nk, folds, monkeypatch, beta=1.1):
    monkeypatch.setenv("DELTA_STAMP_APPROX", "1")
    side = sci.shape[0]
    knots = nr.grid_knots(0, 0, side - 1, side - 1, nk, nk)
    var = np.full_like(sci, 1.3)
    kw = dict(clip_sigma=0.0, clip_iterations=0, min_stamps=1, cv_folds=folds, science_var=var, science_mask=mask)
    args = (sci, ref, knots, px, py, sr, beta, n_max, GRID)
    got = _core.fit_kernel(*args, **kw)
    cond, finish = [], nr.cv_finish

    def spy(mf, rf, ysq, groups, penalty, n, nc, k, grid, warm):
        out = finish(mf, rf, ysq, groups, penalty, n, nc, k, grid, warm)
        p0 = np.kron(np.eye(nc + 1), penalty)
        for lam, err in zip(grid, out["gcv_curve"]):
            eig = [np.abs(np.linalg.eigvalsh(sum(mf) - m + lam * p0)) for m in mf] if np.isfinite(err) else [np.ones(1)]
            cond.append(max(e.max() / max(e.min(), 1e-300) for e in eig))
        return out

    monkeypatch.setattr(nr, "cv_finish", spy)
    want = nr.fit_kernel(*args, **kw)
    monkeypatch.setattr(nr, "cv_finish", finish)
    assert got["n_pixels"] == want["n_pixels"] and got["lambda"] == want["lambda"]
    fin = np.isfinite(want["gcv_curve"])
    assert fin.any() and np.array_equal(np.isfinite(got["gcv_curve"]), fin)
    off = np.abs(got["gcv_curve"][fin] / want["gcv_curve"][fin] - 1.0)
    bound = np.maximum(1e-6, 8 * 2.0**-53 * np.array(cond)[fin]) if not got["used_ldlt"] else 1e-6
    assert np.all(off <= bound), (off, bound)
    np.testing.assert_allclose(got["theta"], want["theta"], rtol=1e-6, atol=1e-7 * np.abs(want["theta"]).max())
    return got


# Fields and one more: 3, 8 (whole tiles of eight), 12, 17, 30, and 68 (81 tiles, two
# passes over a stamp's rows); stamps of 9 rows, of 49 and 169 (not multiples of 64).
@pytest.mark.parametrize("n_max,sr,nk", [(0, 1, 3), (2, 3, 3), (3, 6, 4), (4, 3, 3), (6, 4, 5), (10, 3, 3)])
def test_moments_of_every_field_count(n_max, sr, nk, monkeypatch):
    _compare(*_frame(90 if n_max == 10 else 40, sr), sr, n_max, nk, 4, monkeypatch)


# Folds without stamps, of one stamp, and of more stamps than are staged at a time (64).
@pytest.mark.parametrize("stamps,folds", [(12, 20), (30, 30), (150, 2)])
def test_folds_of_every_size(stamps, folds, monkeypatch):
    _compare(*_frame(stamps, 4), 4, 1, 3, folds, monkeypatch)


def test_stamps_without_active_rows(monkeypatch):
    sci, ref, mask, px, py = _frame(40, 4, seed=3)
    for i in (0, 5, 39):
        mask[py[i] - 4:py[i] + 5, px[i] - 4:px[i] + 5] = 1
    mask[py[7] - 4:py[7] + 5, px[7] - 4:px[7] + 5] = 1
    mask[py[7], px[7]] = 0  # one row left
    _compare(sci, ref, mask, px, py, 4, 2, 3, 3, monkeypatch)


def test_singular_folds_fall_back(monkeypatch):
    """A reference of zeros: every B_n row is exactly zero, and each fold's system is
    solved by the pivoted LDL^T without its degrees of freedom."""
    sci, ref, mask, px, py = _frame(30, 4, seed=5)
    got = _compare(sci, np.zeros_like(ref), mask, px, py, 4, 1, 3, 3, monkeypatch)
    assert got["used_ldlt"]
    np.testing.assert_allclose(got["theta"][:3 * 9], 0.0, atol=1e-12)
