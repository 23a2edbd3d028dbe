"""A stream is admitted by an estimate of its device memory: at least what the opened stream holds, for
every encoding, with few and many records a bin."""
from __future__ import annotations

import numpy as np
import pytest

from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.server import DeviceBackend, StreamConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("enc,dt", [("mma", "uint16"), ("csr", "int32"), ("runs", "uint16"), ("mmad", "uint16")])
@pytest.mark.parametrize("mode", ["floor", "gradient"])
@pytest.mark.parametrize("n_r,n_eta,per_bin", [(400, 180, 2), (120, 60, 40)])
def test_estimate_holds_the_stream(cuda, enc, dt, mode, n_r, n_eta, per_bin):
    ny, nz = 500, 480
    rng = np.random.default_rng(per_bin)
    counts = np.full(n_r * n_eta, per_bin, np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    # neighbouring bins on neighbouring pixels, as a detector's
    at = np.repeat(np.arange(n_r * n_eta), per_bin) * (ny * nz / (n_r * n_eta)) + rng.uniform(0, 40, recs.size)
    recs["y"], recs["z"] = at % ny, np.minimum(at // ny, nz - 1)
    recs["frac"] = recs["areaWeight"] = rng.uniform(0.1, 1.0, recs.size)
    pm = PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))
    backend = DeviceBackend(max_batch=4, max_inflight=2, graph_batches=0)
    cfg = StreamConfig("s", pm, n_r, n_eta, ny, nz, mode=mode, bc_y=250.0, bc_z=240.0, frame_dtype=dt, encoding=enc,
                       r_axis=np.arange(n_r, dtype=np.float64), peaks=np.array([20.0, 60.0]), want_cake=True)
    state, held = backend.open(cfg)
    try:
        assert backend.footprint_estimate(cfg) >= held
    finally:
        backend.close(state)
