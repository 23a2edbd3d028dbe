"""Noisy single peaks of eta columns, one and eight columns per warp, against bounded least squares in
FP64 from the same start and bounds: centre, height, background and signal to noise."""
from __future__ import annotations

import numpy as np
import pytest
import torch
from scipy.optimize import least_squares

from midas_b200.peakfit import FitPlan
from test_gpu_fit_jobs import _pv

pytestmark = pytest.mark.gpu

STEP, HALF, LOCS = 0.25, 12, (115.0, 140.0, 165.0)
R = 100.0 + STEP * (np.arange(320) + 0.5)


def _fit(x, y, loc):
    """pf_fit_singlet_pv (PeakFit.c:922-1013): centre, height, background, SNR, their standard errors"""
    n, bg0, mx = x.size, max(0.0, 0.5 * (y[0] + y[-1])), y.max()
    lb = [x[0], STEP / 2, (mx - bg0) / 100, 0, 0]
    ub = [x[-1], STEP * n / 2, mx * 1.5, 1, bg0 * 1.5 if bg0 > 0 else mx * 0.5]
    p0 = np.clip([loc, 3 * STEP, mx - bg0, 0.5, bg0], lb, ub)
    r = least_squares(lambda p: _pv(x, p, 1) - y, p0, bounds=(lb, ub), x_scale="jac", xtol=1e-14, ftol=1e-14, gtol=1e-14,
                      max_nfev=20000)
    se = np.sqrt(np.diag(np.linalg.inv(r.jac.T @ r.jac)) * (r.fun ** 2).sum() / (n - 5))
    rms = np.sqrt((r.fun ** 2).sum() / n)
    return r.x[[0, 2, 4]], se[[0, 2, 4]], r.x[2] / rms


# units of one plan against 148 SMs x 16 warps: 90, one a warp; 18,000, eight
@pytest.mark.parametrize("F,E", [(1, 30), (20, 300)])
def test_matches_bounded_least_squares(cuda, F, E):
    rng = np.random.default_rng(E)
    y = np.full((F, R.size, E), 90.0)
    for c in LOCS:
        d2 = (R[None, :, None] - c - rng.uniform(-0.06, 0.06, (F, 1, E))) ** 2 / rng.uniform(1.0, 1.3, (F, 1, E)) ** 2
        mu = rng.uniform(0.4, 0.6, (F, 1, E))
        y += rng.uniform(700, 1200, (F, 1, E)) * (mu / (1 + 4 * d2) + (1 - mu) * np.exp(-4 * np.log(2) * d2))
    y = (y + rng.normal(0, 1.5, y.shape)).astype(np.float32)
    plan = FitPlan(R, LOCS, kind="eta", half_window=HALF, x_bin=STEP, device=cuda)
    out = plan.fit_cake_eta(torch.from_numpy(y).to(cuda)).params.view(F, E, len(LOCS), -1).cpu().numpy()
    for f, e in [(0, k) for k in range(0, E, max(1, E // 12))] + [(F - 1, E - 1)]:
        for k, c in enumerate(LOCS):
            sel = (R >= c - HALF * STEP) & (R <= c + HALF * STEP)
            p, se, snr = _fit(R[sel], y[f, sel, e].astype(np.float64), c)
            # the fit ends when chi^2 falls by less than 1e-9 of itself twice: parameters within
            # sqrt(1e-9 x 20 degrees of freedom) = 1.4e-4 standard errors; FP32 values of the model (6e-8
            # of about 1000 against a noise of 1.5) add as little.  A hundredth holds both
            assert np.all(np.abs(out[f, e, k, [1, 7, 8]] - p) <= 1e-2 * se), (f, e, k)
            # height / rms: the height's hundredth of an error is 1e-5 of it, chi^2's 1e-9 nothing
            assert abs(out[f, e, k, 6] - snr) <= 1e-4 * snr, (f, e, k)
