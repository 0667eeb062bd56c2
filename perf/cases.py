"""Timed cases of the difference-imaging path.

Each case is one call (or one forward + backward) a user's program makes: the
stages of ``Subtractor.subtract`` on layers resident on the device, the kernel
fit, the two differentiable objectives, and whole frames. ``prepare`` makes what
such a program holds before the call (seeded synthetic layers of the benchmark's
distributions, the frozen kernel solution, the stamp list), ``run`` is the call,
``work`` the bytes and operations it cannot do without, and ``exact`` the same
results in 64 bits from plain torch / numpy where they have a closed form.

The layers follow ``delta_b200.validation.synthetic_pair``: sky 500 e-, gain
1.5, read noise 4 e-, fluxes dN/dF ~ F^-2.5 on 1e3..1e6 e-, a Gaussian FWHM 2.5
reference, an elliptical Moffat science PSF (beta 3, q 0.85, PA 30 deg) whose
FWHM grows by half along the diagonal, bad columns over 1% of the pixels and
saturated cores. Science PSFs start at FWHM 2.9: with nearly matching PSFs theta
is not determined by the data, so its digits say nothing.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import delta_b200 as delta
from delta_b200 import _device
from delta_b200.autograd import KernelProblem, StampProblem
from delta_b200.pipeline import Subtractor
from delta_b200.solution import KernelSolution

GAIN, READ_NOISE, SKY, SATURATION_E = 1.5, 4.0, 500.0, 2.0e5
SATURATION = SATURATION_E / GAIN
STARS_PER_PX = 20000 / 4096**2
FWHM_TO_SIGMA = 1.0 / 2.354820045030949
TABLE_ROWS = 4096  # of a program's catalog and stamp tables
KINDS = ("subtract", "decorrelate", "score", "catalog", "select", "fit", "chi2", "gcv", "frame", "call")


def listed():
    return [
        # A cut-out of a larger frame: launches and host work count, not pixels.
        dict(name="subtract 256x320", kind="subtract", height=256, width=320, n_max=4, n_knots=3, fwhm=3.0),
        # The benchmark frame's subtraction: variance, masks, saturation.
        dict(name="subtract 4096x4096", kind="subtract", height=4096, width=4096, n_max=6, n_knots=4, fwhm=3.0),
        # Noise decorrelation of an uneven-batch frame.
        dict(name="decorrelate 2048x4096", kind="decorrelate", height=2048, width=4096, n_max=6, n_knots=4, fwhm=3.0),
        # The score of a mid-size frame with the pipeline's 17 x 17 PSF stamp.
        dict(name="score 2048x2048", kind="score", height=2048, width=2048, psf_radius=8, fwhm=3.5),
        # The catalog of a survey frame: few sources among many empty pixels.
        dict(name="catalog 4096x4096", kind="catalog", height=4096, width=4096, psf_radius=8, fwhm=3.5),
        # Stamp selection on an odd-sized frame, the first stage of every subtraction.
        dict(name="select 1003x1531", kind="select", height=1003, width=1531, n_max=6, n_knots=4, fwhm=3.0),
        # The kernel fit with the public defaults: FP64, 5 x 5 knots, 5-fold cross-validation, up to 200 stamps.
        dict(name="fit fp64 cv 2048x2048", kind="fit", height=2048, width=2048, n_max=6, n_knots=5, fwhm=3.2,
             cv_folds=5, precision="fp64"),
        # One gradient step of the registration refinement: chi^2 and its gradients in every parameter and the image.
        dict(name="chi2 2048x2048", kind="chi2", height=2048, width=2048, n_max=6, n_knots=4, fwhm=3.0),
        # One evaluation of the fit's GCV objective with its gradient.
        dict(name="gcv 2048x2048", kind="gcv", height=2048, width=2048, n_max=6, n_knots=4, fwhm=3.0),
        # The 1024^2 configuration: fixed 21 x 21 kernel, 3 x 3 knots, GCV, score but no decorrelation, FP64.
        dict(name="frame 1024x1024 fp64", kind="frame", height=1024, width=1024, n_max=4, n_knots=3, fwhm=3.0,
             radius=10, cv_folds=0, precision="fp64", decorrelate=False),
        # The benchmark's step: one resident 4096^2 frame through every stage, mixed precision.
        dict(name="frame 4096x4096 mixed", kind="frame", height=4096, width=4096, n_max=6, n_knots=4, fwhm=3.0,
             radius=0, cv_folds=0, precision="mixed", decorrelate=True),
        # delta_b200.subtract() of a small ragged frame from ordinary host arrays, every default kept, all stages on.
        dict(name="call 801x1203", kind="call", height=801, width=1203, n_max=6, n_knots=5, fwhm=3.2),
    ]


def draw(rng: random.Random) -> dict:
    """One more case: any kind, sizes log-uniform over the kind's range (odd ones as likely as even)."""
    kind = rng.choice(KINDS)
    lo, hi = {"subtract": (200, 4096), "decorrelate": (300, 4096), "score": (200, 4096), "catalog": (200, 4096),
              "select": (400, 4096), "fit": (800, 2048), "chi2": (256, 2048), "gcv": (800, 2048),
              "frame": (800, 2400), "call": (700, 1100)}[kind]

    def side():
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    c = dict(kind=kind, height=side(), width=side(), fwhm=round(rng.uniform(2.9, 4.0), 2))
    if kind in ("score", "catalog"):
        c["psf_radius"] = rng.choice((5, 6, 7, 8))
    elif kind == "call":
        c.update(n_max=6, n_knots=5)
    else:
        c.update(n_max=rng.choice((4, 5, 6)), n_knots=rng.choice((3, 4, 5)))
    if kind == "fit":
        c.update(cv_folds=rng.choice((0, 5)), precision="fp64")
    if kind == "frame":
        c.update(radius=0, cv_folds=rng.choice((0, 5)), precision=rng.choice(("fp64", "mixed")),
                 decorrelate=rng.choice((True, False)))
    return c


# ---- inputs ----------------------------------------------------------------------------


def _render(out, xy, flux, fwhm, kind, box):
    """Add stars to `out` (int64, units of 2^-20 e-: the sum does not depend on the order of its terms)."""
    h, w = out.shape
    flat = out.view(-1)
    rad = int(math.ceil(box * float(fwhm.max())))
    off = torch.arange(-rad, rad + 1, device=out.device)
    dy, dx = (v.reshape(-1) for v in torch.meshgrid(off, off, indexing="ij"))
    cpa, spa, q = math.cos(math.radians(30.0)), math.sin(math.radians(30.0)), 0.85
    for s in range(0, xy.shape[0], 1000):
        x, y, f, fw = (v[s:s + 1000, None] for v in (xy[:, 0], xy[:, 1], flux, fwhm))
        ix, iy = x.round().long() + dx, y.round().long() + dy
        ex, ey = ix - x, iy - y
        if kind == "gaussian":
            sig2 = (fw * FWHM_TO_SIGMA) ** 2
            v = f / (2 * math.pi * sig2) * torch.exp(-(ex**2 + ey**2) / (2 * sig2))
        else:
            a = fw / (2.0 * math.sqrt(2.0 ** (1.0 / 3.0) - 1.0))
            u, t = (cpa * ex + spa * ey) / a, (-spa * ex + cpa * ey) / (a * q)
            v = f * 2.0 / (math.pi * a * a * q) * (1.0 + u * u + t * t) ** -3
        ok = (ix >= 0) & (ix < w) & (iy >= 0) & (iy < h)
        flat.index_add_(0, (iy * w + ix)[ok], (v[ok] * 2.0**20).round().long())


def _bad_columns(mask, fraction, g):
    """Bad columns (bit 1) over about `fraction` of the pixels of a mask."""
    h, w = mask.shape
    n = max(1, int(fraction * w / 0.6))
    cols = torch.randint(0, w, (n,), generator=g).tolist()
    for col in cols:
        y0 = int(torch.randint(0, h, (1,), generator=g))
        run = min(h - y0, int(torch.randint(max(16, h // 8), h + 16, (1,), generator=g)))
        mask[y0:y0 + run, col] |= 1


def _layers(case, seed):
    """{science, reference, science_var, reference_var, science_mask, reference_mask} on the device."""
    h, w = case["height"], case["width"]
    dev = torch.device("cuda")
    g = torch.Generator(dev).manual_seed(seed)
    gc = torch.Generator().manual_seed(seed + 7)
    n = max(60, int(STARS_PER_PX * h * w))
    rnd = torch.rand((3, n), generator=g, device=dev, dtype=torch.float64)
    xy = torch.stack([8 + rnd[0] * (w - 17), 8 + rnd[1] * (h - 17)], 1)
    flux = (1e3**-1.5 + rnd[2] * (1e6**-1.5 - 1e3**-1.5)) ** (-1 / 1.5)
    fw = case["fwhm"] * (1.0 + 0.25 * (xy[:, 0] / (w - 1) + xy[:, 1] / (h - 1)))
    images = {}
    for name in ("reference", "science"):
        e = torch.zeros((h, w), dtype=torch.int64, device=dev)
        if name == "reference":
            _render(e, xy, flux, torch.full_like(fw, 2.5), "gaussian", 5.0)
        else:
            _render(e, xy, flux, fw, "moffat", 5.0)
            m = max(3, int(50 * h * w / 4096**2))
            t = torch.rand((3, m), generator=g, device=dev, dtype=torch.float64)
            txy = torch.stack([24 + t[0] * (w - 49), 24 + t[1] * (h - 49)], 1)
            tfw = torch.full((m,), case["fwhm"], dtype=torch.float64, device=dev)
            tf = 5.0 * 10.0 ** t[2] * math.sqrt(SKY + READ_NOISE**2) * math.sqrt(4 * math.pi) * tfw * FWHM_TO_SIGMA
            _render(e, txy, tf, tfw, "moffat", 5.0)
        e = e.double() * 2.0**-20 + SKY
        noise = torch.randn((h, w), generator=g, device=dev, dtype=torch.float64) * READ_NOISE
        adu = (torch.poisson(e, generator=g) + noise) / GAIN
        mask = torch.zeros((h, w), dtype=torch.uint8)
        _bad_columns(mask, 0.005, gc)
        mask = mask.to(dev)
        sat = adu >= SATURATION
        mask[sat] |= 2
        adu[sat] = SATURATION
        images[name] = adu.float().contiguous()
        images[name + "_var"] = ((e + READ_NOISE**2) / GAIN**2).float().contiguous()
        images[name + "_mask"] = mask
    return images


def _beta(case):
    """The pipeline's basis scale for the two median FWHMs."""
    sci = case["fwhm"] * 1.25 * FWHM_TO_SIGMA
    return float(max(0.8 * math.sqrt(max(sci**2 - (2.5 * FWHM_TO_SIGMA) ** 2, 0.0)), 0.5))


def _basis(beta, n_max, r, d=0.0):
    """g_n(u - d) at u = -r..r, FP64, as a differentiable function of the tensor (or number) d."""
    t = (torch.arange(-r, r + 1, dtype=torch.float64, device="cuda") - d) / beta
    e, hm1, hc, out = torch.exp(-0.5 * t * t), torch.zeros_like(t), torch.ones_like(t), []
    for n in range(n_max + 1):
        norm = math.exp(-0.5 * (n * math.log(2.0) + math.lgamma(n + 1.0) + 0.5 * math.log(math.pi) + math.log(beta)))
        out.append(norm * hc * e)
        hm1, hc = hc, 2.0 * t * hc - 2.0 * n * hm1
    return torch.stack(out)


def _orders(n_max):
    return [(total - ny, ny) for total in range(n_max + 1) for ny in range(total + 1)]


def _radius(case):
    return case.get("radius") or max(int(math.ceil(3.0 * _beta(case) * math.sqrt(case["n_max"] + 1))), 3)


def _solution(case, seed):
    """A frozen kernel solution as a fit leaves it: a unit-flux core, smaller higher orders, slow spatial terms."""
    h, w, n_max, kk = case["height"], case["width"], case["n_max"], case["n_knots"]
    rng = np.random.default_rng(seed + 13)
    knots = delta.grid_knots(0.0, 0.0, w - 1.0, h - 1.0, kk, kk)
    k, orders = kk * kk, _orders(n_max)
    sums = _basis(_beta(case), n_max, _radius(case)).sum(1).cpu().numpy()
    theta = np.zeros((len(orders) + 1, k))
    for c, (nx, ny) in enumerate(orders):
        size = 0.12 / (1 + nx + ny) if nx + ny else 1.0 / sums[0] ** 2
        theta[c, k - 3] = size if nx + ny == 0 else size * rng.normal()
        theta[c, k - 2:] = 0.05 * size * rng.normal(size=2)
        theta[c, :k - 3] = 0.02 * size * rng.normal(size=k - 3)
    theta[-1, k - 3] = 5.0
    theta[-1, :k - 3] = 0.3 * rng.normal(size=k - 3)
    return KernelSolution(beta=_beta(case), n_max=n_max, radius=0, knots=knots, theta=theta.ravel(),
                          n_components=len(orders), n_spatial=k, lam=1.0, gcv=1.0, effective_dof=1.0, rss=1.0,
                          component_sums=np.array([sums[a] * sums[b] for a, b in orders]), direction="reference",
                          shape=(h, w))


def _psf(case):
    r = case["psf_radius"]
    u = np.arange(-r, r + 1)
    p = np.exp(-0.5 * (u / (case["fwhm"] * FWHM_TO_SIGMA)) ** 2)
    p = np.outer(p, p * (1 + 0.02 * u / r))
    return (p / p.sum()).astype(np.float32)


def _separable(img, p):
    """img correlated with outer(p, p) by shifted sums (zero outside)."""
    r = p.size // 2
    for axis in (0, 1):
        pad = torch.nn.functional.pad(img, (0, 0, r, r) if axis == 0 else (r, r, 0, 0))
        img = sum(float(v) * pad.narrow(axis, j, img.shape[axis]) for j, v in enumerate(p))
    return img


def _difference(case, seed):
    """A difference image, its variance and mask: noise, point sources of both signs, bad columns."""
    h, w = case["height"], case["width"]
    dev = torch.device("cuda")
    g = torch.Generator(dev).manual_seed(seed)
    gc = torch.Generator().manual_seed(seed + 7)
    yy, xx = (torch.linspace(0, 1, n, device=dev) for n in (h, w))
    var = (450.0 * (1.0 + 0.2 * yy[:, None] + 0.1 * xx[None, :])).float()
    d = torch.randn((h, w), generator=g, device=dev) * var.sqrt()
    m = max(4, int(200 * h * w / 4096**2))
    t = torch.rand((4, m), generator=g, device=dev, dtype=torch.float64)
    e = torch.zeros((h, w), dtype=torch.int64, device=dev)
    xy = torch.stack([t[0] * (w - 1), t[1] * (h - 1)], 1)
    f = torch.where(t[3] < 0.7, 1.0, -1.0) * 400.0 * 60.0 ** t[2]
    _render(e, xy, f, torch.full((m,), case["fwhm"], dtype=torch.float64, device=dev), "gaussian", 4.0)
    d = (d.double() + e.double() * 2.0**-20).float()
    mask = torch.zeros((h, w), dtype=torch.uint8)
    _bad_columns(mask, 0.01, gc)
    return d, var.contiguous(), mask.to(dev)


def _frame(x):
    return _device.DeviceFrame(x["science"], x["reference"], x["science_var"], x["reference_var"], x["science_mask"],
                               x["reference_mask"])


def _subtractor(case):
    return Subtractor(n_max=case["n_max"], n_knots=case["n_knots"], radius=case.get("radius", 0),
                      cv_folds=case.get("cv_folds", 0), precision=case.get("precision", "fp64"),
                      decorrelate=case.get("decorrelate", True), score=True, saturation=SATURATION)


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case, table={})
    if kind in ("score", "catalog"):
        s["diff"], s["var"], s["mask"] = _difference(case, seed)
        s["psf"] = _psf(case)
        if kind == "catalog":
            u = np.arange(-case["psf_radius"], case["psf_radius"] + 1)
            p = np.exp(-0.5 * (u / (case["fwhm"] * FWHM_TO_SIGMA)) ** 2)
            p /= p.sum()
            s["score"] = (_separable(s["diff"], p) / (s["var"] * float((p**2).sum() ** 2)).sqrt()).contiguous()
        return s
    x = _layers(case, seed)
    if kind == "call":  # the user holds ordinary host arrays
        s["layers"] = {k: v.cpu().numpy() for k, v in x.items()}
        return s
    s["x"], s["sub"], s["frame"] = x, _subtractor(case), _frame(x)
    if kind in ("subtract", "decorrelate", "chi2"):
        s["sol"] = _solution(case, seed)
    if kind == "chi2":
        good = (x["science_mask"] == 0) & (x["reference_mask"] == 0)
        weights = torch.where(good, 1.0 / (x["science_var"] + x["reference_var"]), 0.0)
        sol = s["sol"]
        s["problem"] = KernelProblem(x["science"], weights, sol.knots, sol.beta, sol.n_max, sol.radius,
                                     reference_mask=x["reference_mask"])
        rng = np.random.default_rng(seed + 29)
        s["leaves"] = [torch.tensor(v, dtype=torch.float64, requires_grad=True)
                       for v in (sol.theta, rng.uniform(-0.3, 0.3, 2), 1.0 + rng.uniform(-0.05, 0.05))]
        s["leaves"].append(x["reference"].clone().requires_grad_(True))
    if kind in ("fit", "gcv"):
        sel = _device.select_stamps(s["frame"], s["sub"])
        h, w = case["height"], case["width"]
        s["stamps"] = sel["x"], sel["y"]
        s["knots"] = delta.grid_knots(0.0, 0.0, w - 1.0, h - 1.0, case["n_knots"], case["n_knots"])
    if kind == "gcv":
        rng = np.random.default_rng(seed + 29)
        s["problem"] = StampProblem(x["science"], x["reference"], s["knots"], *s["stamps"], 15, _beta(case),
                                    case["n_max"], 0, target_var=x["science_var"], convolved_var=x["reference_var"],
                                    target_mask=x["science_mask"], convolved_mask=x["reference_mask"])
        s["at"] = (torch.tensor(rng.uniform(-3.0, 1.0), dtype=torch.float64),
                   torch.tensor(rng.uniform(-0.2, 0.2, 2), dtype=torch.float64),
                   torch.tensor(1.0 + rng.uniform(-0.05, 0.05), dtype=torch.float64))
    return s


# ---- the calls ---------------------------------------------------------------------------


def _into(table, columns):
    """Lists of this frame's length as the head of the program's fixed-size table (zeros after it), and their length."""
    n = 0
    for name, v in columns:
        if name not in table:
            table[name] = np.zeros(TABLE_ROWS, np.uint8 if v.dtype == np.bool_ else v.dtype)
        n = len(v)
        table[name][:n], table[name][n:] = v, 0
    table["rows"] = n
    return table


def run(s):
    case = s["case"]
    kind = case["kind"]
    x = s.get("x")
    if kind == "subtract":
        d, v, m = _device.subtract(x["science"], x["reference"], x["science_var"], x["reference_var"],
                                   x["science_mask"], x["reference_mask"], s["sol"], SATURATION)
        return {"difference": d, "variance": v, "mask": m}
    if kind == "decorrelate":
        d, v = _device.decorrelate(x["science"], s["sol"], x["science_var"], x["reference_var"], 256)
        return {"difference": d, "variance": v}
    if kind == "score":
        return {"score": _device.matched_filter(s["diff"], s["psf"], s["var"])}
    if kind == "catalog":
        cat = _device.build_catalog(s["score"], s["diff"], s["mask"], s["psf"])
        return _into(s["table"], ((name, cat[name]) for name in cat.dtype.names))
    if kind == "select":
        r = _device.select_stamps(s["frame"], s["sub"])
        lists = ("x", "y", "fwhm_science", "fwhm_reference")
        return {**_into(s["table"], ((k, r[k]) for k in lists)),
                **{k: r[k] for k in ("median_fwhm_science", "median_fwhm_reference")}}
    if kind == "fit":
        r = _device.fit_kernel(x["science"], x["reference"], x["science_var"], x["reference_var"],
                               x["science_mask"], x["reference_mask"], s["knots"], *s["stamps"], s["sub"],
                               _beta(case))
        lists = ("stamp_x", "stamp_y", "stamp_chi2", "stamp_accepted")
        return {**_into(s["table"], ((k, r[k]) for k in lists)),
                **{k: v for k, v in r.items() if k not in lists + ("precision_used", "refine_correction")}}
    if kind == "chi2":
        for t in s["leaves"]:
            t.grad = None
        chi2 = s["problem"].chi2(*s["leaves"])
        chi2.backward()
        return {"chi2": chi2.detach(), **{k: t.grad for k, t in zip(("theta", "shift", "scale", "reference"),
                                                                     s["leaves"])}}
    if kind == "gcv":
        return s["problem"].evaluate(*s["at"], grad=True)
    if kind == "frame":
        r = _device.run(s["sub"], s["frame"])
        # The catalog's columns are compared by the catalog cases, on fixed images.
        return {"theta": r["solution"].theta, **{k: r[k] for k in ("difference", "variance", "mask", "score", "psf")}}
    r = delta.subtract(**s["layers"], saturation=SATURATION, decorrelate=True, score=True)
    return {"theta": r.solution.theta, "difference": r.difference, "variance": r.variance, "mask": r.mask,
            "score": r.score, "psf": r.psf}


# ---- what a call cannot do without ----------------------------------------------------------


def work(case):
    kind, px = case["kind"], case["height"] * case["width"]
    if kind in ("score", "catalog"):
        taps = (2 * case["psf_radius"] + 1) ** 2
        return {"bytes": (12 if kind == "score" else 9) * px, "flops": 2 * taps * px if kind == "score" else 0}
    n_max, k, ks = case["n_max"], case["n_knots"] ** 2, 2 * _radius(case) + 1
    nc = (n_max + 1) * (n_max + 2) // 2
    p = (nc + 1) * k
    model = 2 * ((n_max + 1) * ks + nc * ks + nc)  # separable convolutions and the blend, per pixel
    stamps = max(5, min(200, int(0.4 * STARS_PER_PX * px)))
    rows = stamps * 31 * 31
    normal = rows * p * (p + 1)  # the symmetric X^T W X
    sub = {"bytes": 27 * px, "flops": model * px}
    dec = {"bytes": 20 * px, "flops": 4 * 2 * 2.5 * 16 * px}
    folds = max(1, case.get("cv_folds", 5 if kind == "call" else 0))
    solve = 25 * folds * p**3 / 3
    fit = {"bytes": rows * 17, "flops": normal + solve}
    if kind == "subtract":
        return sub
    if kind == "decorrelate":
        return dec
    if kind == "select":
        return {"bytes": 10 * px, "flops": 0}
    if kind == "fit":
        return fit
    if kind == "chi2":
        return {"bytes": 17 * px + 4 * px, "flops": 3 * model * px + 2 * nc * k * px}
    if kind == "gcv":
        return {"bytes": rows * 17, "flops": normal + p**3 / 3 + 4 * rows * p * (nc + 1) * (k - 3)}
    whole = {"bytes": 18 * px + 13 * px, "flops": fit["flops"] + sub["flops"] + 2 * 289 * px}
    if case.get("decorrelate", True):
        whole["flops"] += dec["flops"]
    return whole


# ---- the same in 64 bits ---------------------------------------------------------------------


class _Spline:
    """The thin-plate regression spline in FP64: design rows, bilinear lattice of the fields."""

    def __init__(self, knots):
        knots = np.asarray(knots, np.float64)
        self.k = len(knots)
        self.c = knots.mean(0)
        self.scale = max(np.abs(knots - self.c).max(), 1e-12)
        self.kn = (knots - self.c) / self.scale
        t = np.column_stack([np.ones(self.k), self.kn])
        self.z = np.linalg.qr(t, mode="complete")[0][:, 3:]
        d = self.kn[:, None] - self.kn[None]
        self.spacing = math.sqrt(min((d[i, j] ** 2).sum() for i in range(self.k) for j in range(i))) * self.scale

    def design(self, xs, ys):
        u = (np.column_stack([xs, ys]) - self.c) / self.scale
        r2 = ((u[:, None] - self.kn[None]) ** 2).sum(2)
        green = 0.5 * r2 * np.log(np.where(r2 > 0, r2, 1.0))
        return np.column_stack([green @ self.z, np.ones(len(u)), u])

    def on_frame(self, h, w):
        """The design functions over the frame (k, h, w), blended from the coarse lattice as the model defines them."""
        stride = min(max(int(self.spacing / 16), 1), 64)
        if stride < 4 or w <= 2 * stride or h <= 2 * stride:
            ys, xs = np.mgrid[0:h, 0:w]
            return torch.from_numpy(self.design(xs.ravel(), ys.ravel()).T.reshape(self.k, h, w).copy()).cuda()
        axes = []
        for n in (h, w):
            g = np.append(np.arange(0, n - 1, stride), n - 1)
            c = np.minimum(np.arange(n) // stride, len(g) - 2)
            f = (np.arange(n) - g[c]) / np.maximum(g[c + 1] - g[c], 1)
            axes.append((g, torch.from_numpy(c).cuda(), torch.from_numpy(f).cuda()))
        (gy, cy, fy), (gx, cx, fx) = axes
        ys, xs = np.meshgrid(gy, gx, indexing="ij")
        lat = torch.from_numpy(self.design(xs.ravel(), ys.ravel()).T.reshape(self.k, len(gy), len(gx)).copy()).cuda()
        rows = torch.lerp(lat[:, cy], lat[:, cy + 1], fy[None, :, None].expand(self.k, -1, len(gx)))
        return torch.lerp(rows[:, :, cx], rows[:, :, cx + 1], fx.expand(self.k, len(cy), -1))


def _upper_median(v):
    return v.sort().values[v.numel() // 2] if v.numel() else torch.zeros((), device="cuda")


def _clean(ref, mask):
    """The reference with masked pixels replaced by the fill value; which were replaced."""
    sample, ok = ref.reshape(-1)[::7], mask.reshape(-1)[::7] == 0
    bad = (mask != 0) | ~torch.isfinite(ref)
    return torch.where(bad, _upper_median(sample[ok & torch.isfinite(sample)]).to(ref.dtype), ref), bad


def _component(clean, gx, gy):
    """One component's convolution, zero outside the frame."""
    r, (h, w) = gx.numel() // 2, clean.shape
    pad = torch.nn.functional.pad(clean, (r, r, 0, 0))
    t = (pad.unfold(1, 2 * r + 1, 1) @ gx.flip(0).unsqueeze(1)).squeeze(-1)
    pad = torch.nn.functional.pad(t, (0, 0, r, r))
    return (pad.unfold(0, 2 * r + 1, 1) @ gy.flip(0).unsqueeze(1)).squeeze(-1)


def _model_parts(case, clean, design, theta, gx, gy):
    """sum_c a_c (K_c * R) and the background, FP64, in row bands so that a 4096^2 frame fits."""
    h, w = clean.shape
    r = gx.shape[1] // 2
    coeff = theta.reshape(-1, design.shape[0])
    kernel = torch.zeros_like(clean)
    for c, (nx, ny) in enumerate(_orders(case["n_max"])):
        a = torch.einsum("j,jyx->yx", coeff[c], design)
        bands = [_component(torch.nn.functional.pad(clean, (0, 0, r, r))[y:y + 512 + 2 * r], gx[nx], gy[ny])[r:-r]
                 for y in range(0, h, 512)]
        kernel = kernel + a * torch.cat(bands)
    return kernel, torch.einsum("j,jyx->yx", coeff[-1], design)


def _exact_subtract(case, s):
    x, sol = s["x"], s["sol"]
    h, w, r = case["height"], case["width"], _radius(case)
    clean, _ = _clean(x["reference"], x["reference_mask"])
    basis = _basis(sol.beta, sol.n_max, r).float().double()  # the taps are float32 values
    kernel, bg = _model_parts(case, clean.double(), _Spline(sol.knots).on_frame(h, w),
                              torch.from_numpy(sol.theta).cuda(), basis, basis)
    d = x["science"].double() - kernel - bg
    grow = x["reference_mask"] | torch.where(x["reference"] >= np.float32(SATURATION), 2, 0).to(torch.uint8)
    direct = x["science_mask"] | torch.where(x["science"] >= np.float32(SATURATION), 2, 0).to(torch.uint8)
    fix = (grow != 0) | (direct != 0)
    wide = torch.nn.functional.max_pool2d((grow != 0).float()[None, None], 2 * r + 1, 1, r)[0, 0] > 0
    bad = wide | (direct != 0)
    bad[:r], bad[h - r:], bad[:, :r], bad[:, w - r:] = True, True, True, True
    fill = _upper_median(d.reshape(-1)[::7][~bad.reshape(-1)[::7]])
    return {"difference": torch.where(fix, fill, d), "variance": None, "mask": None}


def _exact_chi2(case, s):
    x, sol = s["x"], s["sol"]
    theta, shift, scale, ref = (t.detach().cuda().double().requires_grad_(True) for t in s["leaves"])
    clean, bad = _clean(ref.detach(), x["reference_mask"])
    clean = torch.where(bad, clean, ref)
    wt, sci = s["problem"].weights.double(), x["science"].double()
    good = (wt > 0) & torch.isfinite(sci)
    design = _Spline(sol.knots).on_frame(case["height"], case["width"])
    r = _radius(case)
    gx, gy = (_basis(sol.beta, sol.n_max, r, shift[i]) for i in (0, 1))
    coeff = theta.reshape(-1, design.shape[0])
    # The residual first, then the gradients one component at a time: the graph of all 28 would not fit beside it.
    with torch.no_grad():
        kernel, bg = _model_parts(case, clean, design, theta, gx, gy)
        res = torch.where(good, sci - scale * kernel - bg, 0.0)
        chi2 = (wt * res * res).sum()
        rbar = -2.0 * wt * res
        g_bg = torch.einsum("yx,jyx->j", rbar, design)
        g_scale = (rbar * kernel).sum()
    grads = [torch.zeros_like(t) for t in (theta, shift, ref)]
    for c, (nx, ny) in enumerate(_orders(case["n_max"])):
        gx, gy = (_basis(sol.beta, sol.n_max, r, shift[i]) for i in (0, 1))
        clean_c = torch.where(bad, clean.detach(), ref)
        part = torch.einsum("j,jyx->yx", coeff[c], design) * _component(clean_c, gx[nx], gy[ny])
        for g, v in zip(grads, torch.autograd.grad((scale.detach() * rbar * part).sum(), (theta, shift, ref),
                                                   retain_graph=True)):
            g += v
    grads[0].view(coeff.shape)[-1] = g_bg
    return {"chi2": chi2, "theta": grads[0], "shift": grads[1], "scale": g_scale, "reference": grads[2]}


def _exact_decorrelate(case, s):
    """Overlap-add whitening in Hann-weighted 256-pixel blocks at half-block steps, FP64 transforms."""
    x, sol, n = s["x"], s["sol"], 256
    h, w = case["height"], case["width"]
    spline, r = _Spline(sol.knots), _radius(case)
    basis = _basis(sol.beta, sol.n_max, r)
    phi = torch.stack([torch.outer(basis[ny], basis[nx]) for nx, ny in _orders(sol.n_max)])
    coeff = torch.from_numpy(sol.theta).cuda().reshape(-1, spline.k)[:-1]

    def origins(extent):
        o = list(range(0, max(extent - n, 0) + 1, n // 2))
        return o + [extent - n] if o[-1] + n < extent else o

    def mirrored(o, extent):
        v = np.arange(o, o + n)
        v = np.where(v >= extent, 2 * extent - v - 1, v)
        return torch.from_numpy(np.clip(v, 0, extent - 1)).cuda()

    oy, ox = origins(h), origins(w)
    group = max(1, int(math.floor(spline.spacing / 4 / (n // 2) + 0.5)))
    hann = 0.5 * (1.0 - torch.cos(2.0 * math.pi * (torch.arange(n, dtype=torch.float64, device="cuda") + 0.5) / n))
    acc, vacc, wsum = (torch.zeros((h, w), dtype=torch.float64, device="cuda") for _ in range(3))
    cells = {}
    for iy, by in enumerate(oy):
        for ix, bx in enumerate(ox):
            cell = (iy // group, ix // group)
            if cell not in cells:
                cx, cy = (min(max(o[min(q * group + group // 2, len(o) - 1)] + n / 2, 0.0), e - 1.0)
                          for o, q, e in ((ox, cell[1], w), (oy, cell[0], h)))
                a = coeff @ torch.from_numpy(spline.design([cx], [cy])[0]).cuda()
                kern = torch.einsum("c,cyx->yx", a, phi)
                full = torch.zeros((n, n), dtype=torch.float64, device="cuda")
                full[:2 * r + 1, :2 * r + 1] = kern
                cells[cell] = torch.fft.rfft2(full).abs() ** 2, float((kern**2).sum())
            power, k2 = cells[cell]
            med = []
            for name in ("science_var", "reference_var"):
                v = x[name][by:min(by + n, h):4, bx:min(bx + n, w):4].reshape(-1)
                med.append(float(_upper_median(v[torch.isfinite(v) & (v > 0)])))
            num = med[0] + med[1] * k2
            block = x["science"][mirrored(by, h)][:, mirrored(bx, w)].double()
            out = torch.fft.irfft2(torch.fft.rfft2(block) * math.sqrt(num) / torch.sqrt(med[0] + med[1] * power),
                                   s=(n, n))
            ny, nx = min(n, h - by), min(n, w - bx)
            wgt = torch.outer(hann[:ny], hann[:nx])
            acc[by:by + ny, bx:bx + nx] += wgt * out[:ny, :nx]
            vacc[by:by + ny, bx:bx + nx] += wgt * num
            wsum[by:by + ny, bx:bx + nx] += wgt
    return {"difference": acc / wsum, "variance": vacc / wsum}


def _exact_score(case, s):
    r, (h, w) = case["psf_radius"], s["diff"].shape
    pad = torch.nn.functional.pad(s["diff"].double(), (r, r, r, r))
    p = s["psf"].astype(np.float64)
    acc = torch.zeros((h, w), dtype=torch.float64, device="cuda")
    for y in range(2 * r + 1):
        for c in range(2 * r + 1):
            acc += p[y, c] * pad[y:y + h, c:c + w]
    return {"score": acc / torch.sqrt(s["var"].double() * float((p**2).sum()))}


def exact(case, seed):
    """None where the results are lists and counts, or rest on a search (the lambda of a fit, a whole frame)."""
    how = {"subtract": _exact_subtract, "decorrelate": _exact_decorrelate, "score": _exact_score, "chi2": _exact_chi2}
    kind = case["kind"]
    return how[kind](case, prepare(case, seed)) if kind in how else None
