"""The device map build where its route changes: a sample that misses every pixel in range, so that
the records outgrow the first buffer; eta edges that do not ascend (no bisection)."""
from __future__ import annotations

import ctypes as C
from dataclasses import replace

import numpy as np
import pytest

from midas_b200 import _lib as L
from midas_b200.bin_io import PXLIST_DTYPE
from midas_b200.mapper import MapperParams, build_map

pytestmark = pytest.mark.gpu


def test_records_that_outgrow_the_estimate(cuda):
    # every 67th pixel (i * 64 + j) is sampled: none of them lies within 4.5 px of (32, 50)
    p = MapperParams(NrPixelsY=64, NrPixelsZ=64, px=200.0, Lsd=1.0e6, BC_y=32.0, BC_z=50.0, RMin=0.5, RMax=4.5,
                     RBinSize=0.01, EtaMin=-180.0, EtaMax=180.0, EtaBinSize=1.0)
    whole, mask = build_map(p, device=0)
    assert whole.n_entries > 100_000                    # the first buffer holds 65,536 here
    parts = [build_map(replace(p, RMin=0.5 + k, RMax=1.5 + k), device=0) for k in range(4)]
    assert max(q.n_entries for q, _ in parts) < 65_536
    # the parts' edges are the whole's up to rounding of RMin + k * RBin: compare what does not depend on it
    assert abs(sum(q.n_entries for q, _ in parts) - whole.n_entries) <= 1e-3 * whole.n_entries
    area = np.concatenate([q.pxList["areaWeight"] for q, _ in parts]).astype(np.float64).sum()
    assert abs(area - whole.pxList["areaWeight"].astype(np.float64).sum()) <= 1e-6 * area
    assert np.array_equal(whole.offsets, np.cumsum(whole.counts) - whole.counts)
    assert not mask.any()


def _build(p, e_lo, e_hi):
    geo = L.MiGeometry()
    geo.ny, geo.nz, geo.px_um, geo.lsd_um = p.NrPixelsY, p.NrPixelsZ, p.px, p.Lsd
    geo.bc_y, geo.bc_z, geo.ty = p.BC_y, p.BC_z, p.ty
    r_lo, r_hi, _, _ = p.edges()
    arrs = [np.ascontiguousarray(a) for a in (r_lo, r_hi, e_lo, e_hi)]
    b = L.MiBinning(r_lo.size, e_lo.size, *[a.ctypes.data for a in arrs])
    h, n, nb = C.c_void_p(), C.c_int64(), C.c_int64()
    L.check(L.lib().mi_map_build(C.byref(geo), C.byref(b), 0, C.byref(h)), "mi_map_build")
    try:
        L.check(L.lib().mi_map_sizes(h, C.byref(n), C.byref(nb)), "mi_map_sizes")
        recs, nmap = np.zeros(n.value, PXLIST_DTYPE), np.zeros((nb.value, 2), np.int32)
        L.check(L.lib().mi_map_copy(h, recs.ctypes.data, nmap.ctypes.data, None), "mi_map_copy")
    finally:
        L.lib().mi_map_destroy(h)
    return recs, nmap


@pytest.mark.parametrize("start,step", [(-180.0, 7.5), (-200.0, 40.0), (-30.0, 3.0)])
def test_eta_edges_in_any_order(cuda, start, step):
    p = MapperParams(NrPixelsY=90, NrPixelsZ=83, px=200.0, Lsd=1.0e6, BC_y=40.3, BC_z=44.7, ty=0.4, RMin=2.0,
                     RMax=40.0, RBinSize=0.7, EtaMin=-180.0, EtaMax=180.0, EtaBinSize=10.0)
    n = int(360 / step) if start < -100 else 20
    lo = start + step * np.arange(n)
    recs, nmap = _build(p, lo, lo + step)
    order = np.random.default_rng(n).permutation(n)
    recs2, nmap2 = _build(p, lo[order], lo[order] + step)
    for r in range(p.n_r):
        for k, e in enumerate(order):
            (c, o), (c2, o2) = nmap[r * n + e], nmap2[r * n + k]
            assert c == c2 and recs[o:o + c].tobytes() == recs2[o2:o2 + c2].tobytes()
