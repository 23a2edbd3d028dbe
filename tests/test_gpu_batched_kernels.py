"""The batched kernels (tensor cores, run records, CSR) against the FP64 oracle at frame counts that
reach them: every mode x semantics x normalisation, variance weights, detector-scale maps, fused plans,
frame types, and the fp32 staging that wide frames take where eight frames side by side do not fit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from conftest import KERNEL_CASES, load_fused_case, load_kernels_case, rel_err
from midas_b200 import _lib as L
from midas_b200 import fused, synth
from midas_b200.bin_io import PixelMap, PXLIST_DTYPE, from_arrays
from midas_b200.kernels import CakePlan, PanelPlan, dtype_code
from midas_b200.mapper import build_map
from test_gpu_fused import _apply
from test_gpu_mma import TOL, _check, _oracle

pytestmark = pytest.mark.gpu

F = 40                            # over the lane-per-bin kernels' counts for every encoding (u16)
SAMPLE = [0, 1, 31, 32, 39]


def _batched(plan, dt=torch.uint16, n=F):
    return L.lib().mi_test_cake_route(plan._h, dtype_code(dt), n, 1) == 0


def _plan(g, cuda, enc, **kw):
    return CakePlan(from_arrays(g["records"], g["nmap"]), n_r=g["n_r"], n_eta=g["n_eta"], n_pixels_y=g["ny"],
                    n_pixels_z=g["nz"], bc_y=g["bc_y"], bc_z=g["bc_z"], device=cuda, encoding=enc, **kw)


@pytest.mark.parametrize("enc", ["mma", "runs", "csr"])
@pytest.mark.parametrize("tag", KERNEL_CASES)
@pytest.mark.parametrize("mode,sem", [(m, s) for m in ("floor", "bilinear", "gradient") for s in ("py", "gpustream", "ic")
                                      if (m, s) != ("floor", "ic")])
@pytest.mark.parametrize("norm", [True, False])
def test_oracle(cuda, enc, tag, mode, sem, norm):
    g = load_kernels_case(tag)
    plan = _plan(g, cuda, enc, mode=mode, semantics=sem, normalize=norm)
    rng = np.random.default_rng(21)
    frames = np.clip(np.rint(g["image"][None] * rng.uniform(20, 65, size=(F, 1, 1))), 0, 65535).astype(np.uint16)
    frames[0, 0, :3] = 65535
    assert _batched(plan)
    res = plan.integrate(torch.from_numpy(frames).to(cuda))
    assert plan.status() == 0
    _check([x[SAMPLE] for x in res], _oracle(g, frames[SAMPLE], mode, norm, sem, g["n_r"]))
    plan.close()


@pytest.mark.parametrize("enc", ["mma", "runs", "csr"])
@pytest.mark.parametrize("mode", ["floor", "gradient"])
def test_variance(cuda, enc, mode):
    g = load_kernels_case("d")
    plan = _plan(g, cuda, enc, mode=mode, variance=True)
    var = np.random.default_rng(4).integers(1, 60000, size=(F, g["nz"], g["ny"])).astype(np.uint16)
    assert _batched(plan)
    res = plan.integrate(torch.from_numpy(var).to(cuda))
    _check([x[SAMPLE] for x in res], _oracle(g, var[SAMPLE], mode, True, "py", g["n_r"], var=True))
    plan.close()


@pytest.mark.parametrize("make,mode,sem", [(lambda: synth.scaled(synth.sweep_2880(), 2), "gradient", "py"),
                                           (lambda: synth.scaled(synth.sweep_2880(), 2), "gradient", "ic"),
                                           (synth.powder_2048, "floor", "py"), (synth.powder_2048, "floor", "gpustream")])
@pytest.mark.parametrize("enc", ["mma", "runs"])
def test_detector_scale(cuda, enc, make, mode, sem):
    """1440^2 with the sweep's fine bins (IntegrationCore's weights include negative ones) and 2048^2 powder"""
    w = make()
    m = w.mapper
    pm, _ = build_map(m, device=0)
    g = dict(records=pm.pxList, nmap=pm.nmap_pairs(), n_r=w.n_r, n_eta=w.n_eta, ny=m.NrPixelsY, nz=m.NrPixelsZ,
             bc_y=m.BC_y, bc_z=m.BC_z)
    plan = _plan(g, cuda, enc, mode=mode, semantics=sem)
    dark = w.dark().cpu().numpy()
    plan.set_dark(dark)
    frames = w.frames(0, F)
    assert _batched(plan)
    res = plan.integrate(frames)
    assert plan.status() == 0
    pick = [0, F - 1]
    sub = frames.cpu().numpy()[pick].astype(np.float32) - dark[None]
    _check([x[pick] for x in res], _oracle(g, sub, mode, True, sem, w.n_r))
    plan.close()


@pytest.mark.parametrize("enc", ["mma", "runs", "csr"])
def test_fused(cuda, enc):
    g = load_fused_case()
    kw = dict(n_eta=g["n_eta"], n_pixels_y=g["ny"], n_pixels_z=g["nz"], mode="gradient", bc_y=g["bc_y"], bc_z=g["bc_z"])
    row_ptr, col, w = fused.fused_csr(g["maps"], g["r_axes"], **kw)
    plan = fused.FusedPlan(g["maps"], g["r_axes"], device=cuda, encoding=enc, **kw)
    rng = np.random.default_rng(5)
    frames = np.clip(np.rint(g["image"][None] * rng.uniform(1, 70, size=(F, 1, 1))), 0, 65535).astype(np.uint16)
    assert _batched(plan)
    cake, _, _ = plan.integrate(torch.from_numpy(frames).to(cuda))
    got = cake.cpu().numpy().reshape(F, -1)
    for f in SAMPLE:
        assert rel_err(got[f], _apply(row_ptr, col, w, frames[f]))[0] <= TOL


@pytest.mark.parametrize("dt", [torch.uint8, torch.uint16, torch.int32, torch.uint32, torch.int64, torch.float32,
                                torch.float64])
@pytest.mark.parametrize("enc", ["runs", "csr"])
@pytest.mark.parametrize("rows", [16, 32])
def test_frame_types(cuda, dt, enc, rows):
    """strips of 32 rows have no pixel-major buffer: the run kernel gathers every type itself"""
    g = load_kernels_case("b")
    plan = _plan(g, cuda, enc, mode="bilinear", tile_rows=rows)
    raw = torch.from_numpy(np.random.default_rng(3).integers(0, 250, size=(F, g["nz"], g["ny"])).astype(np.uint8)).to(cuda)
    assert _batched(plan, torch.uint8) and (_batched(plan, dt) or (enc == "runs" and rows == 16 and dt.itemsize > 2))
    for x, y in zip(plan.integrate(raw.to(dt)), plan.integrate(raw)):
        assert torch.equal(x, y)
    plan.close()


def _random_map(n_r, n_eta, ny, z0, z1, seed):
    rng = np.random.default_rng(seed)
    counts = rng.integers(0, 6, n_r * n_eta).astype(np.int32)
    recs = np.zeros(int(counts.sum()), PXLIST_DTYPE)
    recs["y"], recs["z"] = rng.uniform(0, ny, recs.size), rng.uniform(z0, z1, recs.size)
    recs["frac"] = recs["areaWeight"] = rng.uniform(0.1, 1.0, recs.size)
    return PixelMap(recs, counts, (np.cumsum(counts) - counts).astype(np.int32))


@pytest.mark.parametrize("rows", [8, 16])
@pytest.mark.parametrize("dt", [torch.int32, torch.float32, torch.float64])
def test_wide_frames_without_room_for_eight(cuda, rows, dt):
    """a narrow referenced band (the buffer holds 256 B a referenced pixel, eight frames side by side 32 B a
    detector pixel): over 16 wide frames go through the fp32 rows and the run kernel"""
    ny, nz, n_r, n_eta = 150, 140, 40, 9
    pm = _random_map(n_r, n_eta, ny, 60, 64, rows)
    plan = CakePlan(pm, n_r=n_r, n_eta=n_eta, n_pixels_y=ny, n_pixels_z=nz, device=cuda, encoding="runs", tile_rows=rows)
    rng = np.random.default_rng(6)
    plan.set_dark(rng.normal(100, 5, (nz, ny)))
    raw = rng.integers(0, 60000, (70, nz, ny))
    wide = torch.from_numpy(raw).to(cuda, dt)
    u16 = torch.from_numpy(raw.astype(np.uint16)).to(cuda)
    for n in (17, 32, 33, 64, 65, 70):
        assert _batched(plan, dt, n)
        for x, y, z in zip(plan.integrate(wide[:n]), plan.integrate(u16[:n]), plan.integrate(wide[:8])):
            assert torch.equal(x, y) and torch.equal(x[:8], z)
    assert plan.status() == 0
    plan.close()


def test_wide_panels_without_room_for_eight(cuda):
    """over 3.5 bins a referenced pixel: the bin results of eight frames leave them no room"""
    n_r, n_eta, shapes = 60, 24, [(16, 10), (12, 12)]
    maps = [_random_map(n_r, n_eta, ny, 0, nz, ny) for ny, nz in shapes]
    plan = PanelPlan(maps, shapes=shapes, n_r=n_r, n_eta=n_eta, device=cuda)
    assert n_r * n_eta > 3.5 * plan.info["xc_pixels"]
    rng = np.random.default_rng(8)
    plan.set_dark([rng.normal(100, 5, (nz, ny)) for ny, nz in shapes])
    raw = [torch.from_numpy(rng.integers(0, 60000, (70, nz, ny)).astype(np.uint16)).to(cuda) for ny, nz in shapes]
    want = plan.integrate(raw)                                    # 70: the u16 rows
    for n in (1, 8, 33, 64, 70):
        for types in ((torch.int32, torch.float32), (torch.uint16, torch.float32)):
            got = plan.integrate([r[:n].to(t) for r, t in zip(raw, types)])
            for x, y in zip(got, want):
                assert torch.equal(x, y[:n])
    assert plan.status() == 0
    plan.close()


@pytest.mark.parametrize("enc", ["mma", "runs"])
def test_host_threads(cuda, enc):
    g = load_kernels_case("b")
    frames = torch.from_numpy(np.random.default_rng(12).integers(0, 60000, size=(F, g["nz"], g["ny"])).astype(np.uint16)).to(cuda)
    a, b = _plan(g, cuda, enc, mode="gradient", host_threads=2), _plan(g, cuda, enc, mode="gradient")
    assert _batched(a) and _batched(b)
    for x, y in zip(a.integrate(frames), b.integrate(frames)):
        assert torch.equal(x, y)
