"""chi^2 and its gradients at the edges of the tiled kernels, against the FP64
CPU adjoint, with the bounds of tests/test_gpu_grad.py (float32 forward, FP64
sums). The value alone takes its own kernel: it must be the gradient call's."""

from __future__ import annotations

import numpy as np
import pytest

from delta_b200 import _core
from oracle import grad_ref
from test_gpu_grad import _frame, _rel

pytestmark = pytest.mark.gpu


# Frames below one tile, at its edge and just past it (32 x 64 and 104 x 32
# tiles); every component count with its own instantiation and the generic
# ones around them (n_max 1, 7); 7 to 43 taps: each tap block count and both
# sides of the limits; 9, 16, 25 and 36 knots (design tiles of 16 and 32).
@pytest.mark.parametrize("w,h,n_max,side,radius", [
    (31, 63, 2, 3, 3), (32, 64, 3, 3, 5), (33, 65, 4, 4, 8), (104, 32, 5, 5, 11), (105, 33, 6, 4, 12),
    (97, 131, 6, 5, 13), (70, 90, 6, 6, 16), (75, 61, 3, 3, 19), (80, 70, 4, 3, 21), (90, 50, 1, 3, 4),
    (64, 48, 7, 4, 9), (300, 200, 6, 3, 11),
])
def test_chi2_tiles_match_fp64_oracle(w, h, n_max, side, radius):
    p, wt, knots, theta, beta = _frame(w, h, 40, w + h, n_max, side, beta=1.1)
    args = dict(dx=-0.2, dy=0.15, scale=0.96, radius=radius, reference_mask=p.reference_mask)
    got = _core.kernel_chi2(p.science, p.reference, wt, knots, theta, beta, n_max, grad=True, grad_reference=True, **args)
    value = _core.kernel_chi2(p.science, p.reference, wt, knots, theta, beta, n_max, grad=False, **args)
    assert value["chi2"] == pytest.approx(got["chi2"], rel=1e-13)  # the same float32 residuals, summed per tile
    m = grad_ref.KernelModel(p.science, p.reference, wt, knots, beta, n_max, radius=radius,
                             reference_mask=p.reference_mask)
    want = m.grad(theta, -0.2, 0.15, 0.96, reference=True)
    assert got["chi2"] == pytest.approx(want["chi2"], rel=1e-5)
    assert _rel(got["grad_shift"], want["grad_shift"]) < 1e-4
    assert got["grad_scale"] == pytest.approx(want["grad_scale"], rel=1e-4)
    assert _rel(got["grad_theta"], want["grad_theta"]) < 1e-4
    assert _rel(got["grad_reference"], want["grad_reference"]) < 1e-4
    assert np.all(got["grad_reference"][m.replaced] == 0.0)
