"""Per-eta fits where the units of a warp change: one and several columns per warp, the last warp
partly filled, windows longer than a warp, single peaks beside doublets, skipped columns.  A
column's fits do not depend on the columns fit beside it, and its centres are the peaks'."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200.peakfit import FitPlan

pytestmark = pytest.mark.gpu

X = 10.0 + 0.5 * (np.arange(600) + 0.5)


def _cake(F, E, peaks, seed):
    rng = np.random.default_rng(seed)
    y = np.full((F, X.size, E), 20.0)
    for p in peaks:
        a, w = rng.uniform(400, 900, (F, 1, E)), rng.uniform(1.6, 2.4, (F, 1, E))
        q = ((X[None, :, None] - p) / (0.5 * w)) ** 2
        y += a * (0.5 / (1 + q) + 0.5 * np.exp(-np.log(2.0) * q))
    return y


# singles x columns against 148 SMs x 16 warps: 3 units; 2367 (one per warp), 2370 (two), 21000 (eight,
# the most); half_window 5 / 16 / 40 bins: 11, 33 and 81 samples
@pytest.mark.parametrize("F,E,half", [(1, 1, 5), (1, 789, 5), (2, 395, 16), (7, 1000, 5), (1, 9, 40)])
@pytest.mark.parametrize("doublet", [0.0, 6.0])
def test_columns_do_not_depend_on_their_neighbours(cuda, F, E, half, doublet):
    peaks = [60.0, 64.0, 120.0, 250.0] if doublet else [60.0, 120.0, 250.0]
    y = _cake(F, E, peaks, E)
    if E > 4:
        y[0, :, 3] = 0.0                 # no sample: skipped
        y[0, :, 4] = 0.0
        y[0, 100:105, 4] = 5.0           # five nonzero samples: fit
    cake = torch.from_numpy(y.astype(np.float32)).to(cuda)
    fp = FitPlan(X, peaks, kind="eta", half_window=half, x_bin=0.5, doublet_sep=doublet, device=cuda)
    r = fp.fit_cake_eta(cake)
    it = r.iters.view(F, E, -1)
    if E > 4:
        assert torch.all(it[0, 3] == -3) and torch.all(r.params.view(F, E, -1)[0, 3] == 0)
        assert torch.all(it[0, 4] >= 0)
    for f, e in {(0, 0), (F - 1, E - 1), (F // 2, min(E // 2 + 1, E - 1))}:      # none of the columns above
        one = fp.fit_cake_eta(cake[f:f + 1, :, e:e + 1].contiguous())
        assert torch.equal(one.params[0], r.params[f * E + e]) and torch.equal(one.iters[0], r.iters[f * E + e])
        # noise-free symmetric peaks: the optimum's centre is the peak's; 1e-3 px is a 500th of a bin,
        # far above float resolution of a window and below any misplaced window's error
        c = r.params[f * E + e, -2:, 1].cpu().numpy()
        assert np.all(np.abs(c - np.array(peaks[-2:])) <= 1e-3)
