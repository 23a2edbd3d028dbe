"""Upload of page-locked frames by one kernel: the same bytes as the copies of pageable frames,
and no other byte of the device frames touched, for widths and types whose rows start at every
alignment, for host frames that start off the device frames' alignment, and for many frames."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

from midas_b200 import synth
from midas_b200.kernels import CakePlan
from midas_b200.mapper import build_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [128, 121, 9])
@pytest.mark.parametrize("dt", [np.uint8, np.uint16, np.int32])
@pytest.mark.parametrize("F", [1, 3])
def test_kernel_upload_equals_copies(cuda, ny, dt, F):
    w = synth.scaled(synth.detector_1024(0), 8)
    m = replace(w.mapper, NrPixelsY=ny, RMax=40.0)      # the band's ends and columns leave pixels out
    pm, _ = build_map(m, device=0)
    plan = CakePlan(pm, n_r=m.n_r, n_eta=m.n_eta, n_pixels_y=ny, n_pixels_z=128, device=cuda)
    rng = np.random.default_rng(ny)
    host = torch.from_numpy(rng.integers(1, 200, (F + 1, 128, ny)).astype(dt))
    pinned = host.pin_memory()
    for off in (0, 1):                                  # frame 1 starts ny * 128 * itemsize bytes later
        a = torch.zeros((F, 128, ny), dtype=host.dtype, device=cuda)
        b = torch.zeros_like(a)
        plan.upload(pinned[off:off + F], a)
        plan.upload(host[off:off + F], b)               # pageable: copies
        torch.cuda.synchronize()
        got, want = a.cpu().numpy(), b.cpu().numpy()
        np.testing.assert_array_equal(got, want)
        moved = got != 0                                # the frames hold no zeros
        assert moved.sum() == F * plan.info["upload_pixels"]
        np.testing.assert_array_equal(got[moved], host[off:off + F].numpy()[moved])
