"""mi_integrate_batch_static on a CSR plan keeps its scratch in the library's array, so it may overlap
mi_integrate_batch on the same plan: both give what they give alone, at the frame counts of the
lane-per-bin kernels and of the batched one."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200 import _lib as L
from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan

pytestmark = pytest.mark.gpu


# bins: 64 x 40 fit the array beside the partial sums of these frames; 1000 x 140 (8 results a bin are
# over 8 MiB) do not, and 16 or fewer frames take the batched kernel
@pytest.mark.parametrize("n_r,n_eta,terms", [(64, 40, 200), (1000, 140, 3)])
@pytest.mark.parametrize("frames", [1, 8, 13, 20])
def test_static_beside_ordinary(cuda, n_r, n_eta, terms, frames):
    ny, nz, reps = 256, 250, 60
    rng = np.random.default_rng(frames)
    counts = np.full(n_r * n_eta, terms, np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(0, ny, recs.size), rng.uniform(0, nz, recs.size)
    recs["frac"] = recs["areaWeight"] = rng.uniform(0.1, 1.0, recs.size)
    pm = PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))
    plan = CakePlan(pm, n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, device=cuda, encoding="csr")
    raw = [torch.from_numpy(rng.integers(0, 60000, (frames, nz, ny)).astype(np.uint16)).to(cuda) for _ in range(2)]
    want = [plan.integrate(f) for f in raw]
    new = lambda like: [torch.zeros((reps, *t.shape), dtype=t.dtype, device=cuda) for t in like]
    got = [new(w) for w in want]
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    flat = raw[1].reshape(frames, -1)

    def static(i, s):
        ck, aw, sm = (g[i] for g in got[1])
        L.check(L.lib().mi_integrate_batch_static(plan._h, flat.data_ptr(), L.DT_U16, frames, flat.stride(0),
                                                  ck.data_ptr(), aw.data_ptr(), sm.data_ptr(), s.cuda_stream),
                "mi_integrate_batch_static")
    static(0, torch.cuda.current_stream())       # looks the array's address up
    torch.cuda.synchronize()
    for i in range(reps):
        plan.integrate(raw[0], out={"cake": got[0][0][i], "lineout_aw": got[0][1][i], "lineout_sm": got[0][2][i]},
                       stream=streams[0])
        static(i, streams[1])
    torch.cuda.synchronize()
    for w, g in zip(want, got):
        for x, y in zip(w, g):
            assert torch.equal(y, x.expand_as(y))
    plan.close()
