"""Medians and stamp isolation at the edges of their sizes, against NumPy (order
statistics and positions: equal)."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _data(kind, n, rng):
    v = rng.normal(100.0, 3.0, n).astype(np.float32)
    mask = (rng.random(n) < 0.05).astype(np.uint8)
    if kind == "constant":
        v[:] = -2.5
    elif kind == "ties":
        v = np.round(v / 4.0).astype(np.float32)
    elif kind == "wide":  # both signs, all magnitudes, values that are not finite
        v = (rng.normal(size=n) * 10.0 ** rng.integers(-30, 30, n)).astype(np.float32)
        v[rng.random(n) < 0.02] = np.nan
        v[rng.random(n) < 0.02] = -np.inf
    elif kind == "masked":
        mask[:] = 1
    return v, mask


KINDS = ["plain", "constant", "ties", "wide", "masked"]


# One element, a sample in shared memory below and above 2^16 elements, and the
# two sides of the sampling step at 2^18 (the sample is largest just below 2^19).
@pytest.mark.parametrize("n", [1, 2, 255, 1 << 16, (1 << 16) + 1, 1 << 18, (1 << 18) + 1, (1 << 19) - 1, 1 << 19, 3000001])
@pytest.mark.parametrize("kind", KINDS)
def test_background_medians(n, kind):
    v, mask = _data(kind, n, np.random.default_rng(n % 1009))
    got = _core.estimate_background(v.reshape(1, n), mask.reshape(1, n))
    step = max(n // (1 << 18), 1)
    ok = (mask[::step] == 0) & np.isfinite(v[::step])
    s = v[::step][ok]
    med = nr.upper_median(s)
    want = (0.0, 0.0) if med is None else (float(med), 1.4826 * float(nr.upper_median(np.abs(s - med))))
    assert got == want


# A zero model leaves the science image as the difference, and a masked pixel
# takes the median of every seventh good one: samples of at most 2^16, at most
# 2^19 and more than 2^19 elements.
@pytest.mark.parametrize("h,w", [(9, 11), (448, 1024), (449, 1024), (1792, 2048), (1793, 2048), (2048, 2401), (1911, 2309)])
@pytest.mark.parametrize("kind", KINDS[:4])
def test_difference_fill_median(h, w, kind):
    rng = np.random.default_rng(h + w)
    v, mask = _data(kind, h * w, rng)
    if kind == "wide":
        v[~np.isfinite(v)] = 0.0
    sci, mask = v.reshape(h, w), mask.reshape(h, w)
    mask[4, 5] = 1
    knots = nr.grid_knots(0.0, 0.0, w - 1.0, h - 1.0, 2, 2)
    theta = np.zeros(2 * len(knots))
    ref = np.ones((h, w), np.float32)
    got = _core.subtract(sci, ref, knots, theta, 1.0, 0, 1, 0.0, None, None, mask, None)
    fixed = mask != 0
    good = got["mask"].ravel()[::7] == 0
    want = sci.copy()
    want[fixed] = nr.upper_median(sci.ravel()[::7][good])
    np.testing.assert_array_equal(got["difference"], want)


def _greedy(x, y, value, w, iso, most):
    kx, ky = [], []
    for i in np.lexsort((y * w + x, -value)):
        if len(kx) == most:
            break
        d = (np.array(kx, np.int64) - x[i]) ** 2 + (np.array(ky, np.int64) - y[i]) ** 2
        if not (d < iso * iso).any():
            kx.append(x[i])
            ky.append(y[i])
    return np.array(kx), np.array(ky)


def _image(xs, ys, values, size):
    img = np.random.default_rng(1).normal(0.0, 1.0, (size, size)).astype(np.float32)
    img[ys, xs] = values
    return img


# One candidate, the sort at each of its sizes, and past the 16384 that one CTA
# sorts; few and many kept stamps (9000: more than the one CTA keeps); equal values.
@pytest.mark.parametrize("count", [1, 1023, 1024, 1025, 2049, 4097, 8193, 16384, 16385, 30000])
@pytest.mark.parametrize("iso,most", [(1, 200), (9, 9000), (60, 8192)])
def test_isolation_is_brightest_first(count, iso, most):
    size, margin = 1024, 30
    rng = np.random.default_rng(count)
    grid = np.arange(margin, size - margin, 5)
    at = rng.choice(len(grid) ** 2, count, replace=False)
    xs, ys = grid[at % len(grid)], grid[at // len(grid)]
    values = (200.0 + rng.integers(0, 500, count)).astype(np.float32)
    img = _image(xs, ys, values, size)
    got = _core.detect_stamps(img, stamp_radius=6, threshold_sigma=60.0, max_stamps=most, isolation_radius=iso)
    kx, ky = _greedy(xs, ys, values, size, iso, most)
    np.testing.assert_array_equal(got["x"], kx)
    np.testing.assert_array_equal(got["y"], ky)


def test_isolation_along_a_chain():
    """Every candidate waits for the one before it, over several chunks of 1024."""
    size = 1024
    ys, xs = np.mgrid[30:990:12, 30:990:5]
    order = np.where((np.arange(ys.shape[0]) % 2)[:, None] == 0, np.arange(xs.shape[1]), np.arange(xs.shape[1])[::-1])
    values = (20000.0 - (np.arange(ys.shape[0])[:, None] * xs.shape[1] + order)).astype(np.float32)
    xs, ys, values = xs.ravel(), ys.ravel(), values.ravel()
    got = _core.detect_stamps(_image(xs, ys, values, size), stamp_radius=6, threshold_sigma=60.0, max_stamps=8192,
                              isolation_radius=9)
    kx, ky = _greedy(xs, ys, values, size, 9, 8192)
    np.testing.assert_array_equal(got["x"], kx)
    np.testing.assert_array_equal(got["y"], ky)


def test_pair_equals_its_images():
    """Both images share their launches; one image of the pair past one CTA's sort."""
    size = 1024
    rng = np.random.default_rng(3)
    grid = np.arange(30, size - 30, 5)
    xs, ys = (g.ravel() for g in np.meshgrid(grid, grid))
    many = _image(xs, ys, (200.0 + rng.integers(0, 500, xs.size)).astype(np.float32), size)
    few = _image(xs[::50], ys[::50], (300.0 + rng.random(xs[::50].size)).astype(np.float32), size)
    kw = dict(stamp_radius=6, threshold_sigma=60.0, max_stamps=400, isolation_radius=12)
    for sci, ref in ((many, few), (few, many)):
        a, b = (_core.detect_stamps(i, **kw) for i in (sci, ref))
        near = (np.abs(a["x"][:, None] - b["x"]) <= 2) & (np.abs(a["y"][:, None] - b["y"]) <= 2)
        got = _core.select_stamps(sci, ref, match_radius=2, **kw)
        keep = near.any(axis=1)
        assert set(zip(got["x"], got["y"])) <= set(zip(a["x"][keep], a["y"][keep]))
        assert len(got["x"]) > 0 or not keep.any()


def test_too_many_stamps_are_refused():
    img = _image(np.array([100]), np.array([100]), np.float32(500.0), 256)
    with pytest.raises((ValueError, RuntimeError)):
        _core.detect_stamps(img, stamp_radius=6, max_stamps=20481)
