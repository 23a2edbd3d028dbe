"""The upload kernel reads host memory directly, so it runs only where one page-locked range holds
the frames from their first byte to their last.  Decisions only: no frame is read here."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from midas_b200 import _lib as L


def _holds(start, size, first, last):
    fn = L.lib().mi_test_range_holds
    fn.argtypes, fn.restype = [C.c_uint64] * 4, C.c_int
    return bool(fn(start, size, first, last))


@pytest.mark.parametrize("start,size,first,last,want", [
    (4096, 8192, 4096, 12287, True),             # the whole range
    (4096, 8192, 5000, 5000, True),
    (4096, 8192, 4096, 12288, False),            # one byte past it
    (4096, 8192, 4095, 5000, False),             # one byte before it
    (4096, 8192, 4096, 20479, False),            # ends in another range, pageable memory between
    (4096, 0, 4096, 4096, False),
    (4096, 8192, 6000, 5000, False),             # a size that wrapped
    (2 ** 64 - 4096, 4096, 2 ** 64 - 4096, 2 ** 64 - 1, True),
    (2 ** 64 - 4096, 8192, 2 ** 64 - 10, 5, False),
])
def test_range(start, size, first, last, want):
    assert _holds(start, size, first, last) is want


@pytest.mark.gpu
def test_frames_locked_in_pieces_go_by_copies(cuda):
    """Two frames in one buffer: locked as a whole, by the kernel; locked frame by frame (with
    pageable memory between, or none), only partly or not at all: by copies."""
    import torch

    from midas_b200 import synth
    from midas_b200.kernels import CakePlan, dtype_code
    from midas_b200.mapper import build_map

    w = synth.scaled(synth.detector_1024(0), 8)
    m = w.mapper
    plan = CakePlan(build_map(m, device=0)[0], n_r=w.n_r, n_eta=w.n_eta, n_pixels_y=m.NrPixelsY, n_pixels_z=m.NrPixelsZ,
                    device=cuda)
    npx = m.NrPixelsY * m.NrPixelsZ
    gap = 4096                                   # pixels between the frames
    fn = L.lib().mi_test_upload_by_kernel
    fn.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_int64, C.c_void_p, C.c_int64]
    rt = torch.cuda.cudart()
    raw = np.zeros(2 * npx + gap + 8192, np.uint16)
    base = (raw.ctypes.data + 4095) & ~4095
    dev = torch.zeros((2, npx + gap), dtype=torch.uint16, device=cuda)

    def by_kernel(frames, first=base):
        return fn(plan._h, first, dtype_code(torch.uint16), frames, npx + gap, dev.data_ptr(), npx + gap)

    def locked(*pieces):
        for at, n in pieces:
            assert int(rt.cudaHostRegister(at, n, 0)) == 0
        try:
            return by_kernel(1), by_kernel(2)
        finally:
            for at, _ in pieces:
                assert int(rt.cudaHostUnregister(at)) == 0

    second = base + 2 * (npx + gap)
    assert (by_kernel(1), by_kernel(2)) == (0, 0)
    assert locked((base, 2 * (2 * npx + gap))) == (1, 1)
    assert locked((base, 2 * npx), (second, 2 * npx)) == (1, 0)
    assert locked((base, 2 * (npx + gap)), (second, 2 * npx)) == (1, 0)
    assert locked((base, npx)) == (0, 0)
    pinned = torch.zeros((2, npx + gap), dtype=torch.uint16).pin_memory()
    assert (by_kernel(1, pinned.data_ptr()), by_kernel(2, pinned.data_ptr())) == (1, 1)
    plan.close()
