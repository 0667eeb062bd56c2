"""Brightest-first isolation on both sides of the rule that resolves a chunk a kept
stamp at a time where a frame has room for few, against NumPy (positions: equal)."""

from __future__ import annotations

import numpy as np
import pytest
from test_gpu_select_sizes import _greedy, _image

from delta_b200 import _core, _lib

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


def _matched(a, b, radius, most):
    """The pair's stamps from those of its images: each of the reference (in order) with
    the nearest of the science image, the first of them on a tie."""
    rows = []
    for x, y, f in zip(b["x"], b["y"], b["fwhm"]):
        d2 = (x - a["x"].astype(np.int64)) ** 2 + (y - a["y"].astype(np.int64)) ** 2
        if len(d2) and d2.min() <= radius * radius:
            rows.append((x, y, a["fwhm"][int(np.argmin(d2))], f))
    return rows[:most]


# Both images in one CTA's sort, one of them past it, one without candidates, and more
# stamps than the one CTA keeps.
@pytest.mark.parametrize("left,right,most", [(40, 30, 400), (1, 50, 400), (1, 1, 400), (7, 0, 400), (3, 4, 5000)])
def test_pair_lists_are_those_of_its_images(left, right, most):
    size, radius = 1024, 2
    rng = np.random.default_rng(10 * left + right)
    grid = np.arange(30, size - 30, 5)
    xs, ys = (g.ravel() for g in np.meshgrid(grid, grid))

    def image(step, jitter):
        if step == 0:
            return _image(np.zeros(0, int), np.zeros(0, int), np.zeros(0, np.float32), size)
        x, y = xs[::step] + jitter, ys[::step]
        return _image(x, y, (200.0 + rng.integers(0, 500, x.size)).astype(np.float32), size)

    for sci, ref in ((image(left, 0), image(right, 1)), (image(right, 1), image(left, 0))):
        kw = dict(stamp_radius=6, threshold_sigma=60.0, max_stamps=most, isolation_radius=12)
        a, b = (_core.detect_stamps(i, **kw) for i in (sci, ref))
        want = _matched(a, b, radius, len(b["x"]))
        got = _core.select_stamps(sci, ref, match_radius=radius, **kw)
        rows = list(zip(got["x"], got["y"], got["fwhm_science"], got["fwhm_reference"]))
        assert len(rows) == len(want)
        np.testing.assert_array_equal(np.array(rows, float).reshape(-1, 4), np.array(want, float).reshape(-1, 4))
        assert left == 0 or right == 0 or len(rows) > 0


@pytest.mark.parametrize("most", [20480, 20481, 2**31 - 1])
def test_workspace_does_not_follow_the_most_stamps(most):
    """A bound on the stamps far above what can be kept costs no memory; it is refused
    only where there is a candidate."""
    torch = pytest.importorskip("torch")
    import ctypes

    size = 256
    ctx = _lib.context()
    params = _core._detect_params(6, 60.0, most, 0.0, 0, 0, 0, 2)
    out = [np.zeros(4, np.int32), np.zeros(4, np.int32), np.zeros(4), np.zeros(4), np.zeros(4)]
    n = ctypes.c_int(-1)

    def detect(img):
        return _lib.lib().dgpu_detect_stamps(ctx.handle, _lib.MEM_HOST, ctypes.c_int64(size), ctypes.c_int64(size),
                                             _lib.ptr(img), None, ctypes.byref(params), 4,
                                             *[_lib.ptr(a) for a in out], ctypes.byref(n))

    _core.detect_stamps(np.zeros((size, size), np.float32))
    free = torch.cuda.mem_get_info()[0]
    assert detect(np.zeros((size, size), np.float32)) == _lib.DGPU_OK and n.value == 0
    assert free - torch.cuda.mem_get_info()[0] < 1 << 28
    rc = detect(_image(np.array([100]), np.array([90]), np.float32(500.0), size))
    if most > 20480:
        assert rc == _lib.DGPU_ERR_INVALID
    else:
        assert rc == _lib.DGPU_OK and n.value == 1 and (out[0][0], out[1][0]) == (100, 90)
