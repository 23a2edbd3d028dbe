"""Eta columns with few nonzero samples: skipped below five, wherever in the column they are, and a
column without any costs about what one with data does."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200.peakfit import FitPlan

pytestmark = pytest.mark.gpu


# samples read by one step of a block's warps: 128; series of a block: 32
@pytest.mark.parametrize("n_x", [40, 127, 128, 129, 700])
@pytest.mark.parametrize("F,E", [(1, 1), (1, 33), (3, 32), (2, 70)])
@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
def test_five_samples_anywhere(cuda, n_x, F, E, dt):
    rng = np.random.default_rng(n_x + E)
    x = 10.0 + 0.5 * np.arange(n_x)
    y = np.zeros((F, n_x, E))
    n = rng.integers(0, 8, (F, E))
    for f in range(F):
        for e in range(E):
            where = rng.permutation(n_x)[:n[f, e]] if (f + e) % 2 else np.arange(n_x)[n_x - n[f, e]:]
            y[f, where, e] = rng.choice([3.0, -2.0, np.nan], n[f, e])
    plan = FitPlan(x, [x[n_x // 2]], kind="eta", half_window=8, x_bin=0.5, device=cuda)
    r = plan.fit_cake_eta(torch.as_tensor(y, device=cuda).to(dt))
    skipped = r.iters.view(F, E, -1).cpu().numpy()[:, :, 0] == -3
    np.testing.assert_array_equal(skipped, n < 5)
    assert torch.all(r.params.view(F, E, -1)[torch.as_tensor(skipped, device=cuda)] == 0)


def test_columns_without_data_are_not_dear(cuda):
    """3960 rows x 360 columns: read once by a block of warps, not sample by sample"""
    x = 10.0 + 0.25 * np.arange(3960)
    plan = FitPlan(x, [300.0], kind="eta", half_window=12, x_bin=0.25, device=cuda)
    full = torch.full((1, x.size, 360), 100.0, device=cuda)

    def us(cake):
        times = []
        for _ in range(30):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            plan.fit_cake_eta(cake)
            b.record()
            torch.cuda.synchronize()
            times.append(a.elapsed_time(b) * 1e3)
        return float(np.median(times))

    assert us(torch.zeros_like(full)) <= 4.0 * us(full)       # a thread a column: 22 times
