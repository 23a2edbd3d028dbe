"""Which kernels cake a call's frames, and that both give the same bits where the rule's sides meet:
grids of few long bins keep the batched kernels, others take a lane per bin up to their frame counts."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from midas_b200 import _lib as L
from midas_b200.bin_io import PixelMap, PXLIST_DTYPE
from midas_b200.kernels import CakePlan, dtype_code

pytestmark = pytest.mark.gpu

BATCHED, LANE, LANE8 = 0, 1, 2


def _map(n_r, n_eta, ny, nz, lo, hi, seed):
    """lo to hi - 1 records a bin, scattered over the detector"""
    rng = np.random.default_rng(seed)
    counts = rng.integers(lo, hi, n_r * n_eta).astype(np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(0, ny, recs.size), rng.uniform(0, nz, recs.size)
    recs["frac"] = rng.uniform(0.1, 1.0, recs.size)
    recs["areaWeight"], recs["deltaR"] = recs["frac"], rng.uniform(-0.5, 0.5, recs.size)
    return PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))


def _plan(cuda, enc, n_r, n_eta, lo, hi, ny=201, nz=190, **kw):
    pm = _map(n_r, n_eta, ny, nz, lo, hi, n_r + hi)
    return CakePlan(pm, n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, bc_y=100.2, bc_z=95.1, device=cuda,
                    encoding=enc, **kw)


def _route(plan, dt, n, lineouts=True):
    return L.lib().mi_test_cake_route(plan._h, dtype_code(dt), n, int(lineouts))


# by the lines of the rule (mi_internal.h): a walk a term and frame count against 12 us and 0.088 ns a
# staged pixel (MMA; the maps stage 100 to 36,000 pixels, at most 3.2 us) or 6 us a tile in sequence (CSR)
@pytest.mark.parametrize("n_r,n_eta,terms,lane", [
    (2, 1, 1700, ()),                            # 64.6 us at one frame
    (2, 3, 450, ()),                             # 17.1
    (10, 4, 200, (1,)),                          # 7.6, 20, 25
    (40, 9, 60, (1, 2, 3, 8, 9, 16, 24)),        # 2.3, 6, 7.5, 9, 10.5
])
def test_mma_plans(cuda, n_r, n_eta, terms, lane):
    plan = _plan(cuda, "mma", n_r, n_eta, terms - 5, terms)
    for n in (1, 2, 3, 8, 9, 16, 24, 25, 128):
        want = BATCHED if n not in lane else LANE if n < 3 else LANE8
        assert _route(plan, torch.uint16, n) == want and _route(plan, torch.uint8, n, False) == want, n
    plan.close()


# one band of rows, so all tiles follow one another: 100 and 300 terms a bin over few tiles, the batched kernel
# for most counts; 30 to 39 terms over tiles of 64 pixels, about 20 in an item of two columns, a lane per bin for all
@pytest.mark.parametrize("n_eta,lo,hi,pixels", [(1, 95, 100, 0), (1, 295, 300, 0), (24, 30, 40, 64)])
def test_csr_plans(cuda, n_eta, lo, hi, pixels):
    plan = _plan(cuda, "csr", 16, n_eta, lo, hi, tile_pixels=pixels, tile_rows=16)
    assert plan.info["n_items"] == 1 or pixels
    tiles = plan.info["n_tiles"] / plan.info["n_items"] if pixels else plan.info["n_tiles"]
    seen = set()
    for dt in (torch.uint16, torch.float32):
        for n in (1, 2, 3, 8, 9, 16, 17, 128):
            walk = {1: 0.02, 2: 0.05, 3: 0.17, 8: 0.17, 9: 0.3, 16: 0.47}.get(n, 0) * (hi - 1)
            want = LANE if n <= 16 and (pixels or walk + 18 <= 6 * tiles) else BATCHED
            seen.add((n, want))
            assert _route(plan, dt, n) == want, (n, tiles)
    assert ((16, BATCHED) in seen) == (not pixels) and (17, BATCHED) in seen
    plan.close()


@pytest.mark.parametrize("n_r,n_eta", [(2, 1), (16, 1)])
def test_run_plans(cuda, n_r, n_eta):
    plan = _plan(cuda, "runs", n_r, n_eta, 95, 100)
    for dt, last in ((torch.uint16, 32), (torch.int32, 256)):
        for n in (1, 4, 5, 32, 33, 256):
            assert _route(plan, dt, n) == (LANE if n < 5 else LANE8 if n <= last else BATCHED), (dt, n)
    plan.close()


@pytest.mark.parametrize("mode,sem,norm,var", [("floor", "py", True, False), ("gradient", "py", False, True),
                                               ("bilinear", "gpustream", False, False), ("gradient", "ic", True, False)])
@pytest.mark.parametrize("n_r,n_eta", [(16, 24), (37, 27)])
def test_csr_lane_equals_batched(cuda, mode, sem, norm, var, n_r, n_eta):
    """small tiles, many in sequence: a lane per bin for up to 16 frames"""
    plan = _plan(cuda, "csr", n_r, n_eta, 30, 40, tile_pixels=64 if mode == "floor" else 256, mode=mode, semantics=sem, normalize=norm, variance=var)
    rng = np.random.default_rng(n_r)
    raw = rng.integers(0, 250, (40, 190, 201))
    for dark in (None, rng.normal(100, 5, (190, 201))):
        plan.set_dark(dark)
        for dt in (np.uint8, np.uint16, np.int32, np.uint32, np.int64, np.float32, np.float64):
            frames = torch.from_numpy(raw.astype(dt)).to(cuda)
            assert _route(plan, frames.dtype, 40) == BATCHED
            whole = plan.integrate(frames)
            for first, n in ((0, 1), (3, 2), (7, 4), (9, 8), (4, 9), (6, 16)):
                assert _route(plan, frames.dtype, n) == LANE
                for x, y in zip(plan.integrate(frames[first:first + n]), whole):
                    assert torch.equal(x, y[first:first + n])
    assert plan.status() == 0
    plan.close()
