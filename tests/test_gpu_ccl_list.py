"""Labels and per-component flags of the seed-list catalog at the edges of its
blocks, against NumPy (whole numbers and flags: equal)."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import numpy_ref as nr

pytestmark = pytest.mark.gpu


def _expected(score, mask, bit_pos):
    pos, neg = nr.seed_mask(score, 5.0, +1, mask, True), nr.seed_mask(score, 3.0, -1, mask, True)
    seed, other = (pos, neg) if bit_pos else (neg, pos)
    labels, n = nr.label_components(seed)
    pad = lambda a: np.pad(a, 1)  # noqa: E731
    flags, dip = np.zeros(n, np.uint8), np.zeros(n, bool)
    lp, op, mp = pad(labels), pad(np.asarray(other, bool)), pad(mask)
    h, w = score.shape
    for dy in range(3):
        for dx in range(3):
            near_o, near_m = op[dy:dy + h, dx:dx + w], mp[dy:dy + h, dx:dx + w]
            ring = lp[dy:dy + h, dx:dx + w] != labels
            for i in np.flatnonzero(labels):
                c = labels.flat[i] - 1
                dip[c] |= near_o.flat[i]
                if ring.flat[i] or (dy == 1 and dx == 1):
                    flags[c] |= near_m.flat[i]
    return labels, n, np.bincount(labels.ravel(), minlength=n + 1)[1:], flags, dip


# One pixel, one row and column, rows that are not whole bitmap words, frames
# below, at and past one block of 8192 pixels and several blocks; no seed, every
# pixel a seed, and sparse and dense seeds of both signs.
@pytest.mark.parametrize("h,w", [(1, 1), (1, 77), (77, 1), (31, 33), (64, 128), (91, 91), (128, 129), (130, 257)])
@pytest.mark.parametrize("density", [0.0, 0.01, 0.4, 1.0])
@pytest.mark.parametrize("positive", [True, False])
def test_seed_list_catalog(h, w, density, positive):
    rng = np.random.default_rng(h * 1000 + w + int(100 * density))
    sign = np.where(rng.random((h, w)) < 0.7, 1.0, -1.0) if density < 1 else (1.0 if positive else -1.0)
    score = np.where(rng.random((h, w)) < density, 9.0 * sign, 0.0).astype(np.float32)
    mask = ((rng.random((h, w)) < 0.05) * rng.integers(1, 8, (h, w))).astype(np.uint8)
    got = _core.build_catalog(score, score, mask=mask, expected_fwhm=3.0, return_negative=not positive)
    labels = _core.catalog_labels((h, w))
    want, n, npix, flags, dip = _expected(score, mask, positive)
    assert np.array_equal(labels, want) and len(got["x"]) == n
    np.testing.assert_array_equal(got["n_pix"], npix)
    np.testing.assert_array_equal(got["mask_flags"], flags)
    np.testing.assert_array_equal(got["is_dipole"], dip)


def test_images_at_any_element_alignment():
    """Device images that start off a 16-byte (score) or 4-byte (mask) boundary."""
    torch = pytest.importorskip("torch")
    from delta_b200 import _device

    rng = np.random.default_rng(5)
    h, w = 60, 301
    score = np.where(rng.random((h, w)) < 0.02, 9.0, 0.0).astype(np.float32)
    mask = (rng.random((h, w)) < 0.05).astype(np.uint8)
    psf = np.ones((5, 5), np.float32) / 25
    want = _device.build_catalog(*(torch.from_numpy(a).cuda() for a in (score, score, mask)), psf)
    for off in (1, 2, 3):
        def shifted(a):
            t = torch.zeros(a.size + off, dtype=torch.from_numpy(a).dtype, device="cuda")[off:]
            t.copy_(torch.from_numpy(a.ravel()))
            return t.view(a.shape)
        got = _device.build_catalog(shifted(score), shifted(score), shifted(mask), psf)
        assert np.array_equal(got["peak_x"], want["peak_x"]) and np.array_equal(got["n_pix"], want["n_pix"])
