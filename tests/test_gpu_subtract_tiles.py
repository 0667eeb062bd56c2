"""Mask, variance and model of the subtraction at the edges of their tiles, words and
tap counts, against the oracle."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import cref
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _case(h, w, n_max, radius, var_range, rng):
    knots = nr.grid_knots(0, 0, w - 1, h - 1, 3, 3)
    nc = (n_max + 1) * (n_max + 2) // 2
    theta = 0.03 * rng.standard_normal((nc + 1) * 9)
    theta[6] = 1.0
    sci, ref = (rng.normal(100.0, 5.0, (h, w)).astype(np.float32) for _ in range(2))
    vs, vr = (rng.uniform(*var_range, (h, w)).astype(np.float32) for _ in range(2))
    sm, rm = ((rng.random((h, w)) < 0.01) * rng.integers(1, 8, (h, w)) for _ in range(2))
    ref[rng.random((h, w)) < 0.002] = np.nan
    sci[rng.random((h, w)) < 0.002] = np.inf
    return sci, ref, knots, theta, vs, vr, sm.astype(np.uint8), rm.astype(np.uint8)


# Frames below, at and past a tile of 32 and 64, rows of whole words and not, large
# enough for tiles of 64 (1216 x 1024); radii whose window is and is not a whole number
# of words, whose tap count leaves one or three taps after the fours, one without a
# neighbour and one larger than the frame; flat and varying variance windows.
@pytest.mark.parametrize("h,w", [(31, 33), (32, 32), (33, 64), (64, 65), (65, 130), (1216, 1024), (1217, 1023)])
@pytest.mark.parametrize("n_max,radius,var_range", [(2, 4, (1.0, 9.0)), (3, 7, (1.0, 9.0)), (2, 5, (4.0, 4.001)),
                                                    (0, 1, (1.0, 9.0)), (4, 19, (1.0, 9.0))])
def test_subtract_at_tile_edges(h, w, n_max, radius, var_range):
    rng = np.random.default_rng(h * 7 + w + radius)
    sci, ref, knots, theta, vs, vr, sm, rm = _case(h, w, n_max, radius, var_range, rng)
    args = (sci, ref, knots, theta, 1.1, n_max, radius, 118.0, vs, vr, sm, rm)
    got, want = _core.subtract(*args), cref.subtract(*args)
    np.testing.assert_array_equal(got["mask"], want["mask"])
    np.testing.assert_allclose(got["difference"], want["difference"], rtol=1e-5, atol=1e-3)
    np.testing.assert_allclose(got["variance"], want["variance"], rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_zero_taps_skip_what_is_not_finite(bad):
    """A window with infinities or NaN keeps the reference's skip of zero taps."""
    rng = np.random.default_rng(2)
    sci, ref, knots, theta, vs, vr, sm, rm = _case(80, 90, 0, 5, (1.0, 9.0), rng)
    vr[20, 30] = bad
    args = (sci, ref, knots, theta, 0.4, 0, 5, 0.0, vs, vr, None, None)
    got, want = _core.subtract(*args), cref.subtract(*args)
    np.testing.assert_allclose(got["variance"], want["variance"], rtol=1e-5, atol=1e-5)


def test_device_frames_at_any_element_alignment():
    """Device layers that start off a 16-byte (images) or 4-byte (masks) boundary."""
    torch = pytest.importorskip("torch")
    from types import SimpleNamespace

    from delta_b200 import _device

    sci, ref, knots, theta, vs, vr, sm, rm = _case(96, 128, 2, 4, (1.0, 9.0), np.random.default_rng(9))
    sol = SimpleNamespace(knots=knots, theta=theta, beta=1.1, n_max=2, radius=4)

    def up(a, offset):
        t = torch.empty(a.size + offset, dtype=torch.float32 if a.dtype == np.float32 else torch.uint8, device="cuda")
        v = t[offset:].view(a.shape)
        v.copy_(torch.from_numpy(a))
        return v

    outs = [[t.cpu().numpy() for t in _device.subtract(*(up(a, o) for a in (sci, ref, vs, vr, sm, rm)), sol, 118.0)]
            for o in (0, 1, 3)]
    for o in outs[1:]:
        for a, b in zip(o, outs[0]):
            np.testing.assert_array_equal(a, b)
