"""The device map build takes memory for the records it finds, whatever grid the pixels in use lie on."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from midas_b200.mapper import MapperParams, build_map

pytestmark = pytest.mark.gpu

USED_HIGH = 8            # cudaMemPoolAttrUsedMemHigh


def _peak(build):
    """bytes of the device's default pool in use at most during build()"""
    rt, pool, n = C.CDLL("libcudart.so.12"), C.c_void_p(), C.c_uint64(0)
    torch.cuda.synchronize()
    assert rt.cudaDeviceGetDefaultMemPool(C.byref(pool), 0) == 0
    assert rt.cudaMemPoolSetAttribute(pool, USED_HIGH, C.byref(n)) == 0      # from here on
    out = build()
    assert rt.cudaMemPoolGetAttribute(pool, USED_HIGH, C.byref(n)) == 0
    return n.value, out


@pytest.mark.parametrize("first", [0, 66])
def test_pixels_in_step_with_the_sample(cuda, first):
    """one pixel of every 67 in use: those a strided sample takes, all of them or none"""
    ny = nz = 1024
    p = MapperParams(NrPixelsY=ny, NrPixelsZ=nz, px=200.0, Lsd=1.0e6, BC_y=512.0, BC_z=511.0, RMin=5.0, RMax=480.0,
                     RBinSize=0.25, EtaMin=-180.0, EtaMax=180.0, EtaBinSize=5.0)
    mask = np.ones((nz, ny), np.uint8)
    t = np.arange(first, ny * nz, 67)
    mask[t % nz, t // nz] = 0
    peak, (pm, _) = _peak(lambda: build_map(p, device=0, mask=mask))
    n_pix, n_bins = ny * nz, p.n_r * p.n_eta
    # per pixel a mask byte, a count and an offset (13 B) and the scan's and the sort's scratch; per bin two
    # counters; per record 72 B; 65,536 entries of 40 B; 8 MB for the scratch and edges
    assert pm.n_entries > 20_000
    assert peak <= 13 * n_pix + 8 * n_bins + 80 * pm.n_entries + 40 * 65_536 + (8 << 20)
