"""Panels of different widths, one with rows that hold no referenced pixel, on a virtual detector
whose width is no multiple of 8: the empty rows take no room in the pixel-major buffer."""
from __future__ import annotations

from dataclasses import replace

import numpy as np
import pytest
import torch

from midas_b200 import synth
from midas_b200.kernels import CakePlan, PanelPlan
from midas_b200.mapper import build_map

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("encoding", ["runs", "mma"])
@pytest.mark.parametrize("wide", [124, 126, 128])
def test_narrow_panel_with_empty_rows(cuda, encoding, wide):
    base = synth.scaled(synth.detector_1024(0), 8)                 # 128 x 128
    ws = [replace(base, mapper=replace(base.mapper, NrPixelsY=ny)) for ny in (wide, 74)]
    rows = np.zeros((128, 74), dtype=np.uint8)
    rows[20:29] = 1                                                # a module gap: nine masked rows
    masks = [None, rows]
    maps = [build_map(w.mapper, device=0, mask=k)[0] for w, k in zip(ws, masks)]
    kw = dict(n_r=base.n_r, n_eta=base.n_eta, mode="floor", normalize=False, device=cuda, encoding=encoding)
    shapes = [(w.mapper.NrPixelsY, w.mapper.NrPixelsZ) for w in ws]
    rng = np.random.default_rng(wide)
    frames = [torch.from_numpy(rng.integers(0, 60000, size=(5, 128, ny)).astype(np.uint16)).to(cuda)
              for ny, _ in shapes]
    merged, _, _ = PanelPlan(maps, shapes=shapes, **kw).integrate(frames)
    single = [CakePlan(pm, n_pixels_y=ny, n_pixels_z=nz, **kw).integrate(f)[0].double()
              for pm, (ny, nz), f in zip(maps, shapes, frames)]
    want = single[0] + single[1]
    # sums of like sign: the unit partials and the result are rounded to float on both sides
    assert torch.allclose(merged.double(), want, rtol=5 * 2.0 ** -24, atol=0.0)
