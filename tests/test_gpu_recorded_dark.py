"""A recorded graph reads the plan's dark as it is when the graph is replayed: a dark set, changed
or cleared after ``capture`` holds for the next ``replay``, for every encoding and frame count."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("enc,frames", [(e, f) for e in ("runs", "csr", "mma") for f in (1, 4, 20, 40)])
def test_replay_follows_the_dark(cuda, enc, frames):
    ny, nz, n_r, n_eta = 61, 53, 30, 7
    rng = np.random.default_rng(frames)
    counts = np.full(n_r * n_eta, 9, np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(0, ny, recs.size), rng.uniform(0, nz, recs.size)
    recs["frac"] = recs["areaWeight"] = rng.uniform(0.1, 1.0, recs.size)
    pm = PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))
    plan = CakePlan(pm, n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, device=cuda, encoding=enc)
    raw = torch.from_numpy(rng.integers(0, 60000, (frames, nz, ny)).astype(np.uint16)).to(cuda)
    out = dict(zip(("cake", "lineout_aw", "lineout_sm"), plan.integrate(raw)))
    graph = plan.capture(raw, out)
    seen = []
    for dark in (rng.normal(100, 5, (nz, ny)), rng.normal(900, 5, (nz, ny)), None):
        plan.set_dark(dark)
        graph.replay()
        torch.cuda.synchronize()
        got = [out[k].clone() for k in ("cake", "lineout_aw", "lineout_sm")]
        for x, y in zip(got, plan.integrate(raw)):
            assert torch.equal(x, y)
        seen.append(got[0])
    assert not torch.equal(seen[0], seen[1]) and not torch.equal(seen[1], seen[2])
    plan.close()
