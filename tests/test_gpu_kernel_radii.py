"""Decorrelation and the whitened PSF with the largest kernels that their shared
memory takes, against the FP64 oracle."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _case(radius, nk):
    h, w, n_max = 260, 270, 2
    rng = np.random.default_rng(radius)
    knots = nr.grid_knots(0, 0, w - 1, h - 1, nk, nk)
    k = nk * nk
    theta = 0.02 * rng.standard_normal(7 * k)
    theta[k - 3] = 1.0
    vs = rng.uniform(80.0, 120.0, (h, w)).astype(np.float32)
    vr = rng.uniform(40.0, 60.0, (h, w)).astype(np.float32)
    return rng, knots, theta, 1.3, n_max, vs, vr


# 229 x 229 (the most that fitted beside 1024 knots' scratch), past it, and 239 x 239,
# the most that 227 KB holds, with few knots and with 64.
@pytest.mark.parametrize("radius,nk", [(114, 3), (115, 3), (119, 3), (119, 8)])
def test_largest_kernels(radius, nk):
    rng, knots, theta, beta, n_max, vs, vr = _case(radius, nk)
    diff = (rng.standard_normal(vs.shape) * 10.0).astype(np.float32)
    args = (diff, knots, theta, beta, n_max, vs, vr)
    got = _core.decorrelate(*args, block=256, radius=radius)
    want = nr.decorrelate(*args, block=256, radius=radius)
    np.testing.assert_allclose(got["variance"], want["variance"], rtol=2e-6)
    assert np.max(np.abs(got["difference"] - want["difference"]) / np.sqrt(want["variance"])) < 1e-4
    u = np.arange(-5, 6)
    psf = np.exp(-(u[:, None] ** 2 + u[None, :] ** 2) / 8.0).astype(np.float32)
    psf /= psf.sum()
    out = _core.whiten_score_psf(psf, knots, theta, beta, n_max, vs, vr, 256, radius)
    np.testing.assert_allclose(out, nr.whiten_score_psf(psf, knots, theta, beta, n_max, vs, vr, 256, radius),
                               atol=2e-6)


def test_larger_kernels_are_refused():
    rng, knots, theta, beta, n_max, vs, vr = _case(125, 3)
    with pytest.raises((ValueError, RuntimeError)):
        _core.decorrelate(vs, knots, theta, beta, n_max, vs, vr, block=256, radius=125)
