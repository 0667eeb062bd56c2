"""The oracle's float32 convolution: each multiply-add is rounded once, and the B_n
stack is the reference's bit for bit."""

from __future__ import annotations

from fractions import Fraction

import numpy as np
import pytest
from conftest import load_golden

from oracle import numpy_ref as nr


def test_fma32_rounds_once():
    rng = np.random.default_rng(0)
    a, b, c = ((rng.normal(size=2000) * 10.0 ** rng.integers(-6, 6, 2000)).astype(np.float32) for _ in range(3))
    c[:700] = -(a[:700] * b[:700])  # cancellation down to the product's rounding error
    c[700:1400] = a[700:1400] * b[700:1400] * np.float32(2.0**-24)  # next to the ties
    for x, y, z, got in zip(a, b, c, nr.fma32(a, b, c)):
        exact = Fraction(float(x)) * Fraction(float(y)) + Fraction(float(z))
        off = abs(Fraction(float(got)) - exact)
        for side in (np.float32(-np.inf), np.float32(np.inf)):
            assert off <= abs(Fraction(float(np.nextafter(got, side))) - exact)


def test_basis_convolve_is_the_references_bit_for_bit():
    g = load_golden("basis")
    beta, n_max, r = g["conv_params"]
    np.testing.assert_array_equal(nr.basis_convolve(g["conv_image"], float(beta), int(n_max), int(r)), g["conv_out"])


@pytest.mark.parametrize("shape,beta,n_max,r", [((24, 31), 1.5, 2, 5), ((40, 33), 1.1, 6, 8), ((5, 3), 0.8, 0, 3)])
def test_basis_convolve_is_near_its_float64_sums(shape, beta, n_max, r):
    """A sum of 2 r + 1 terms per direction, each step off by at most 2^-24 of its partial
    sum: together below (2 r + 2) 2^-23 of the sums of absolute values."""
    img = np.random.default_rng(1).standard_normal(shape).astype(np.float32)
    k1 = nr.gauss_hermite_basis1d(beta, n_max, r).astype(np.float32)
    got = nr.basis_convolve(img, beta, n_max, r)
    for c, (nx, ny) in enumerate(nr.basis_orders(n_max)):
        want = nr.convolve_y(nr.convolve_x(img, k1[nx]), k1[ny])
        size = nr.convolve_y(nr.convolve_x(np.abs(img), np.abs(k1[nx])), np.abs(k1[ny]))
        assert np.all(np.abs(got[c] - want) <= (2 * r + 2) * 2.0**-23 * size)
