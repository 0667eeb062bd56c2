"""The catalog on both sides of the number of components that get a warp each for
their finish, against NumPy (flux: the same FP64 additions in raster order, equal)."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 148 * 32, 148 * 32 + 1])
@pytest.mark.parametrize("radius", [0, 3, 40])
def test_catalog_of_many_components(count, radius):
    side, step = 700, 9
    rng = np.random.default_rng(count + radius)
    score = np.zeros((side, side), np.float32)
    per = side // step
    at = np.sort(rng.choice(per * per, count, replace=False))
    y0, x0 = (at // per) * step + 3, (at % per) * step + 3
    for dy, dx in ((0, 0), (0, 1), (1, 1)):  # one to three pixels, the first always there
        on = np.ones(count, bool) if (dy, dx) == (0, 0) else rng.random(count) < 0.5
        score[y0[on] + dy, x0[on] + dx] = rng.uniform(6.0, 20.0, on.sum()).astype(np.float32)
    diff = rng.normal(0.0, 5.0, score.shape).astype(np.float32)
    diff[rng.random(score.shape) < 0.01] = np.nan
    diff[rng.random(score.shape) < 0.01] = 0.0
    got = _core.build_catalog(score, diff, expected_fwhm=3.0, aperture_radius=radius)
    assert len(got["x"]) == count
    r = radius if radius > 0 else 4  # round(3 sigma) of the expected width
    for c in range(count) if count < 100 else rng.choice(count, 60, replace=False):
        ys, xs = (v + o for v, o in zip(np.nonzero(score[y0[c]:y0[c] + 2, x0[c]:x0[c] + 2]), (y0[c], x0[c])))
        wt = score[ys, xs].astype(np.float64)
        cx, cy = (wt * xs).sum() / wt.sum(), (wt * ys).sum() / wt.sum()
        np.testing.assert_allclose([got["x"][c], got["y"][c]], [cx, cy], rtol=1e-14)
        assert got["n_pix"][c] == len(xs) and got["peak_snr"][c] == wt.max()
        px, py = (int(np.floor(got[k][c] + 0.5)) for k in ("x", "y"))
        total = 0.0
        for yy in range(max(0, py - r), min(side, py + r + 1)):
            for xx in range(max(0, px - r), min(side, px + r + 1)):
                if (xx - px) ** 2 + (yy - py) ** 2 <= r * r and np.isfinite(diff[yy, xx]):
                    total += float(diff[yy, xx])
        assert got["flux"][c] == total
