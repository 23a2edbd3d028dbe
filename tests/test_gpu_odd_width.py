"""16-bit frames whose rows start at every alignment (widths and frame strides of every residue
modulo 8, a first frame off the 16-byte grid): the batched caking equals that of the same counts as
8-bit frames, read an element at a time, for both staging layouts and part and full batches."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

from midas_b200 import synth
from midas_b200.kernels import CakePlan
from midas_b200.mapper import build_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [64, 65, 67, 70, 300])
@pytest.mark.parametrize("enc", ["mma", "runs"])
def test_rows_at_every_alignment(cuda, ny, enc):
    w = synth.scaled(synth.detector_1024(0), 8)
    m = replace(w.mapper, NrPixelsY=ny, NrPixelsZ=53, BC_y=ny / 2, BC_z=25.0, RMin=1.0, RMax=160.0)
    pm, _ = build_map(m, device=0)
    plan = CakePlan(pm, n_r=m.n_r, n_eta=m.n_eta, n_pixels_y=ny, n_pixels_z=53, device=cuda, encoding=enc)
    rng = np.random.default_rng(ny)
    raw = rng.integers(0, 256, (129, 53 * ny))
    for pad in (0, 1, 6):                              # pixels between frames: other strides and starts
        wide = torch.zeros((129, 53 * ny + pad), dtype=torch.uint16, device=cuda)
        wide[:, pad:] = torch.from_numpy(raw.astype(np.uint16)).to(cuda)
        a = plan.integrate(wide.as_strided((129, 53, ny), (53 * ny + pad, ny, 1), pad))
        b = plan.integrate(torch.from_numpy(raw.astype(np.uint8).reshape(129, 53, ny)).to(cuda))
        for x, y in zip(a, b):
            np.testing.assert_array_equal(x.cpu().numpy(), y.cpu().numpy())
