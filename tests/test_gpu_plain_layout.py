"""The one-frame path's record layout at its edges: eta columns and R rows that do not fill a
slice of 32 bins, one to three columns, empty bins, bins of one record; against the oracle."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import oracle
from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["floor", "bilinear", "gradient"])
@pytest.mark.parametrize("n_r,n_eta", [(1, 1), (33, 1), (17, 2), (16, 3), (7, 4), (9, 5), (8, 36), (65, 7)])
def test_bins_that_do_not_fill_a_slice(cuda, mode, n_r, n_eta):
    rng = np.random.default_rng(100 * n_r + n_eta)
    ny, nz, n_bins = 37, 41, n_r * n_eta
    counts = rng.integers(0, 12, n_bins).astype(np.int32)
    counts[rng.random(n_bins) < 0.2] = 0
    counts[0] = 70                                     # far more records than its neighbours
    offsets = (np.cumsum(counts) - counts).astype(np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(0, ny - 1, recs.size), rng.uniform(0, nz - 1, recs.size)
    recs["frac"] = rng.uniform(0.1, 1.0, recs.size)
    recs["areaWeight"] = recs["frac"]
    recs["deltaR"] = rng.uniform(-0.5, 0.5, recs.size)
    raw = rng.integers(100, 3000, (nz, ny)).astype(np.uint16)
    plan = CakePlan(PixelMap(recs, counts, offsets), n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, mode=mode,
                    bc_y=18.2, bc_z=20.7, device=cuda)
    ck, _, _ = plan.integrate_plain(torch.from_numpy(raw).to(cuda))
    ref, _ = oracle.integrate(recs, np.stack([counts, offsets], 1), n_bins, ny, nz, raw.astype(np.float64), mode=mode,
                              semantics="gpustream", bc_y=18.2, bc_z=20.7)
    got = ck.reshape(-1).cpu().numpy()
    assert np.all(got[counts == 0] == 0)
    # FP32 positions and sums of up to 70 terms, as the reference's kernel: the bar of its own test
    scale = np.maximum(np.abs(ref), 1e-3 * np.median(np.abs(ref[counts > 0])))
    assert np.max(np.abs(got - ref) / scale) <= 2e-6
