"""Pixels and darks that are not finite: they reach the bins whose terms hold the pixel and no
others, and a frame's cake and lineouts do not depend on how many frames the call has."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan, PanelPlan

pytestmark = pytest.mark.gpu

N_R, N_ETA, NY, NZ = 50, 7, 61, 53
NAN_PX, INF_PX = (20, 20), (30, 31)          # (z, y)
COUNTS = (1, 2, 5, 8, 16, 17, 24, 25, 32, 33, 280)


def _map(ny, nz, seed):
    rng = np.random.default_rng(seed)
    counts = rng.integers(0, 25, N_R * N_ETA).astype(np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.integers(0, ny, recs.size), rng.integers(0, nz, recs.size)
    for k, (z, y) in ((5, NAN_PX), (1900, NAN_PX), (700, INF_PX), (2500, INF_PX)):     # in a few bins each
        recs["z"][k], recs["y"][k] = z, y
    recs["frac"] = recs["areaWeight"] = rng.uniform(0.1, 1.0, recs.size)
    return PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))


def _hit(pm, pixel):
    """bins with a record of the pixel"""
    bins = np.repeat(np.arange(N_R * N_ETA), pm.counts)
    out = np.zeros(N_R * N_ETA, bool)
    out[bins[(pm.pxList["z"] == pixel[0]) & (pm.pxList["y"] == pixel[1])]] = True
    return out


def _check(run, total, nan, inf, counts=COUNTS):
    whole = [x.cpu().numpy() for x in run(total)]
    bins = whole[0].reshape(total, -1)
    for f in (0, total - 1):
        np.testing.assert_array_equal(~np.isfinite(bins[f]), nan | inf)
        assert np.isnan(bins[f][nan]).all()
    for n in counts:
        for x, y in zip(run(n), whole):
            np.testing.assert_array_equal(x.cpu().numpy(), y[:n])


@pytest.mark.parametrize("enc,rows", [("runs", 8), ("runs", 16), ("runs", 32), ("csr", 16), ("mma", 0)])
def test_dark(cuda, enc, rows):
    pm = _map(NY, NZ, 3)
    plan = CakePlan(pm, n_r=N_R, n_eta=N_ETA, n_pixels_y=NY, n_pixels_z=NZ, device=cuda, encoding=enc, tile_rows=rows)
    dark = np.zeros((NZ, NY), np.float32)
    dark[NAN_PX], dark[INF_PX] = np.nan, np.inf
    plan.set_dark(dark)
    raw = np.random.default_rng(1).integers(0, 60000, (280, NZ, NY))
    for dt in (np.uint8, np.uint16):
        frames = torch.from_numpy(raw.astype(dt)).to(cuda)
        _check(lambda n: plan.integrate(frames[:n]), 280, _hit(pm, NAN_PX), _hit(pm, INF_PX))
    plan.close()


@pytest.mark.parametrize("enc,rows", [("runs", 8), ("runs", 16), ("runs", 32), ("csr", 16)])
@pytest.mark.parametrize("dt", [torch.float32, torch.float64])
def test_frames(cuda, enc, rows, dt):
    pm = _map(NY, NZ, 4)
    plan = CakePlan(pm, n_r=N_R, n_eta=N_ETA, n_pixels_y=NY, n_pixels_z=NZ, device=cuda, encoding=enc, tile_rows=rows)
    frames = torch.from_numpy(np.random.default_rng(2).uniform(0, 6e4, (280, NZ, NY))).to(cuda, dt)
    frames[:, NAN_PX[0], NAN_PX[1]] = float("nan")
    frames[:, INF_PX[0], INF_PX[1]] = float("inf")
    _check(lambda n: plan.integrate(frames[:n]), 280, _hit(pm, NAN_PX), _hit(pm, INF_PX))
    plan.close()


def test_panel_dark(cuda):
    shapes = [(61, 53), (44, 70)]
    maps = [_map(ny, nz, 7 + ny) for ny, nz in shapes]
    plan = PanelPlan(maps, shapes=shapes, n_r=N_R, n_eta=N_ETA, device=cuda)
    darks = [np.zeros((nz, ny), np.float32) for ny, nz in shapes]
    darks[0][NAN_PX] = np.nan
    darks[1][INF_PX] = np.inf
    plan.set_dark(darks)
    rng = np.random.default_rng(5)
    frames = [torch.from_numpy(rng.integers(0, 60000, (280, nz, ny)).astype(np.uint16)).to(cuda) for ny, nz in shapes]
    _check(lambda n: plan.integrate([f[:n] for f in frames]), 280, _hit(maps[0], NAN_PX), _hit(maps[1], INF_PX),
           (1, 8, 32, 33))
    plan.close()
