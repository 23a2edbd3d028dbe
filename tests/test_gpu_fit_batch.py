"""Ring-fit windows at the sizes where the batched fitter's layout changes: one and several
windows per warp, windows longer than a warp, clipped and rejected windows.  A window's fit
does not depend on the windows beside it, and isolated peaks come out as the oracle's fit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from midas_b200 import peakfit

pytestmark = pytest.mark.gpu


def _lineouts(F, n_x, peaks, seed):
    rng = np.random.default_rng(seed)
    x = 10.0 + 0.5 * (np.arange(n_x) + 0.5)
    y = np.full((F, n_x), 50.0)
    for p in peaks:
        a, c = rng.uniform(500, 5000, (F, 1)), p + rng.uniform(-0.3, 0.3, (F, 1))
        w, e = rng.uniform(1.5, 3.0, (F, 1)), rng.uniform(0.2, 0.8, (F, 1))
        q = ((x[None] - c) / (0.5 * w)) ** 2
        y += a * (e / (1 + q) + (1 - e) * np.exp(-np.log(2.0) * q))
    return x, y + rng.standard_normal(y.shape)


# windows F x (n_peaks + 2) against 148 SMs x 16 warps = 2368: 3 and 2360 (one per warp), 2370
# (two per warp), 9480 (five per warp, the last warp partly filled); half_window 15 / 16 / 40: a
# sample per lane, one more than a warp, three rounds
@pytest.mark.parametrize("model", ["pv", "tch"])
@pytest.mark.parametrize("F,n_peaks,half", [(1, 1, 15), (236, 8, 15), (790, 1, 16), (948, 8, 15), (37, 3, 40)])
def test_windows_do_not_depend_on_their_neighbours(cuda, model, F, n_peaks, half):
    peaks = np.linspace(60.0, 460.0, n_peaks) if n_peaks > 1 else np.array([200.0])
    peaks = np.append(peaks, [12.0, 2000.0])   # a window clipped at the start of the axis; no window
    x, y = _lineouts(F, 1000, peaks[:-2], 3)
    xt, pk = torch.from_numpy(x).to(cuda), torch.from_numpy(peaks).to(cuda)
    yt = torch.from_numpy(y).to(cuda)
    r = peakfit.fit_batch(xt, yt, pk, model=model, half_window=half, x_bin=0.5)
    assert torch.all(r.iters[:, -1] == -1) and torch.all(r.params[:, -1] == 0)
    assert torch.all(r.iters[:, :-2] > 0)
    for f in sorted({0, F // 2, F - 1}):
        one = peakfit.fit_batch(xt, yt[f:f + 1], pk, model=model, half_window=half, x_bin=0.5)
        assert torch.equal(one.params[0], r.params[f]) and torch.equal(one.iters[0], r.iters[f])
        for k in range(min(2, n_peaks)):
            ref, _ = oracle.fit(x, y[f], float(peaks[k]), model={"pv": 0, "tch": 1}[model], half_window=half,
                                max_iter=500, x_bin=0.5)
            assert abs(float(r.params[f, k, 1]) - ref[1]) <= 1e-4
