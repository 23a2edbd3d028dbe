"""Frames through the lane-per-bin kernels (few frames, and eight frames of a pixel side by side):
the same bits as the batched kernels give those frames in a large batch, for every encoding, frame
type, strips of 8, 16 and 32 rows, variance weights, OpenMP semantics, grids that do not fill a
slice, counts on both sides of every dispatch limit, and panels of two types."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan, PanelPlan

pytestmark = pytest.mark.gpu


def _map(n_r, n_eta, ny, nz, seed):
    rng = np.random.default_rng(seed)
    counts = rng.integers(0, 25, n_r * n_eta).astype(np.int32)
    counts[rng.random(counts.size) < 0.1] = 0
    counts[0] = 90
    offsets = (np.cumsum(counts) - counts).astype(np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(-1, ny, recs.size), rng.uniform(-1, nz, recs.size)
    recs["frac"] = rng.uniform(0.1, 1.0, recs.size)
    recs["areaWeight"], recs["deltaR"] = recs["frac"], rng.uniform(-0.5, 0.5, recs.size)
    return PixelMap(recs, counts, offsets)


@pytest.mark.parametrize("enc,rows", [("runs", 8), ("runs", 16), ("runs", 32), ("csr", 16)])
@pytest.mark.parametrize("mode,sem,var", [("floor", "py", False), ("gradient", "py", True), ("bilinear", "omp", False)])
@pytest.mark.parametrize("n_r,n_eta", [(1, 1), (35, 2), (50, 7), (24, 40)])
def test_few_frames_equal_the_batch(cuda, enc, rows, mode, sem, var, n_r, n_eta):
    ny, nz, F = 61, 53, 40
    rng = np.random.default_rng(n_eta)
    kw = dict(n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, mode=mode, semantics=sem, variance=var, bc_y=30.1,
              bc_z=26.4, device=cuda, encoding=enc, tile_rows=rows)
    plan = CakePlan(_map(n_r, n_eta, ny, nz, n_r), **kw)
    if sem == "omp":
        plan.set_bin_mask(np.arange(n_r * n_eta) % 9 == 4)
    raw = rng.integers(0, 250, (F, nz, ny))
    for dark in (False, True):
        if dark:
            plan.set_dark(rng.normal(100, 5, (nz, ny)))
        whole = plan.integrate(torch.from_numpy(raw.astype(np.uint16)).to(cuda))     # 40: the batched kernel
        for dt in (np.uint8, np.uint16, np.int32, np.uint32, np.int64, np.float32, np.float64):
            frames = torch.from_numpy(raw.astype(dt)).to(cuda)
            every = ((0, 1), (3, 2), (7, 4), (2, 5), (9, 8), (4, 16), (10, 17), (3, 33), (0, 40))
            for first, n in every if dt in (np.uint16, np.int32) else ((F - 3, 3), (5, 21)):
                part = plan.integrate(frames[first:first + n])
                for x, y in zip(part, whole):
                    np.testing.assert_array_equal(x.cpu().numpy(), y[first:first + n].cpu().numpy())
            only, _, _ = plan.integrate(frames[5:6], lineouts=sem == "omp")
            np.testing.assert_array_equal(only[0].cpu().numpy(), whole[0][5].cpu().numpy())
    assert plan.status() == 0


@pytest.mark.parametrize("mode,sem,var", [("floor", "py", False), ("gradient", "py", True), ("bilinear", "ic", False)])
@pytest.mark.parametrize("n_r,n_eta", [(1, 1), (13, 2), (50, 7), (24, 40)])
def test_few_frames_equal_the_batch_on_the_tensor_cores(cuda, mode, sem, var, n_r, n_eta):
    """MMA plans: few frames by the lane-per-bin kernels, 70 by the tensor cores; the first call
    after a dark is set or cleared follows it."""
    ny, nz, F = 61, 53, 70
    rng = np.random.default_rng(n_eta)
    plan = CakePlan(_map(n_r, n_eta, ny, nz, n_r), n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, mode=mode,
                    semantics=sem, variance=var, bc_y=30.1, bc_z=26.4, device=cuda, encoding="mma")
    for dark in (None, rng.normal(100, 5, (nz, ny)), None):
        plan.set_dark(dark)
        for dt, top in ((np.uint8, 256), (np.uint16, 65536)):
            frames = torch.from_numpy(rng.integers(0, top, (F, nz, ny)).astype(dt)).to(cuda)
            parts = [(f, n, plan.integrate(frames[f:f + n])) for f, n in ((0, 1), (3, 2), (7, 3), (4, 8), (10, 17), (2, 24), (5, 25))]
            whole = plan.integrate(frames)
            for f, n, part in parts:
                for x, y in zip(part, whole):
                    np.testing.assert_array_equal(x.cpu().numpy(), y[f:f + n].cpu().numpy())
    assert plan.status() == 0


def test_panels_of_two_types_equal_one_type(cuda):
    """u16 and int32 panels (fp32 staging, eight frames side by side) against the same counts as
    u16 panels (40 frames: the batched kernel), for counts on both sides of a block of eight."""
    n_r, n_eta, F = 30, 12, 40
    shapes = [(61, 53), (44, 70)]
    rng = np.random.default_rng(4)
    plan = PanelPlan([_map(n_r, n_eta, ny, nz, 7 + ny) for ny, nz in shapes], shapes=shapes, n_r=n_r, n_eta=n_eta,
                     device=cuda)
    plan.set_dark([rng.normal(100, 5, (nz, ny)) for ny, nz in shapes])
    raw = [rng.integers(0, 60000, (F, nz, ny)) for ny, nz in shapes]
    whole = plan.integrate([torch.from_numpy(r.astype(np.uint16)).to(cuda) for r in raw])
    for types in ((np.uint16, np.int32), (np.float32, np.uint16), (np.uint16, np.uint16)):
        for first, n in ((0, 1), (5, 8), (3, 9), (1, 32), (0, 40)):
            part = plan.integrate([torch.from_numpy(r[first:first + n].astype(t)).to(cuda) for r, t in zip(raw, types)])
            for x, y in zip(part, whole):
                np.testing.assert_array_equal(x.cpu().numpy(), y[first:first + n].cpu().numpy())
    assert plan.status() == 0
