"""Fits of different sizes from several threads at once: each call launches with its own shared
memory, whatever the others ask for, and gives what it gives alone."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest
import torch

from midas_b200 import _lib as L
from midas_b200.peakfit import FitPlan

pytestmark = pytest.mark.gpu

X = 10.0 + 0.25 * (np.arange(1200) + 0.5)
PEAKS = [100.0, 180.0, 250.0]


def _lines(n, seed):
    rng = np.random.default_rng(seed)
    y = np.full((n, X.size), 20.0)
    for p in PEAKS:
        q = ((X - p) / rng.uniform(0.8, 1.2, (n, 1))) ** 2
        y += rng.uniform(400, 900, (n, 1)) * (0.5 / (1 + q) + 0.5 * np.exp(-np.log(2.0) * q))
    return y


def _check(calls, outs, reps):
    """calls: C entry calls on a stream, each with its outputs; every one from its own thread"""
    def run(i, n, stream):
        for k in range(n):
            rc = calls[i](stream.cuda_stream)
            if rc:
                errors.append((i, k, rc, L.lib().mi_last_error()))
            if k % 64 == 63:
                stream.synchronize()
        stream.synchronize()

    errors = []
    streams = [torch.cuda.Stream() for _ in calls]
    for i, s in enumerate(streams):
        run(i, 1, s)
    want = [[t.clone() for t in o] for o in outs]
    torch.cuda.synchronize()
    threads = [threading.Thread(target=run, args=(i, reps, s)) for i, s in enumerate(streams)]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert not errors, (len(errors), errors[:2])
    for w, g in zip(want, outs):
        assert all(torch.equal(x, y) for x, y in zip(w, g))


def _outputs(cuda, *shape):
    return [torch.zeros((*shape, L.FIT_NOUT), dtype=torch.float64, device=cuda),
            torch.zeros(shape, dtype=torch.int32, device=cuda)]


def test_windows_of_three_sizes(cuda):
    """up to 511 bins a side: 50, 58 and 67 KB of shared memory a block"""
    x, pk = torch.as_tensor(X, device=cuda), torch.as_tensor(PEAKS, device=cuda, dtype=torch.float64)
    lines = torch.as_tensor(_lines(1, 1), device=cuda)
    calls, outs = [], []
    for half in (385, 445, 511) * 2:
        opts, o = L.MiFitOpts(L.FIT_PV, half, 1, 0.25, 0.0, 0.0), _outputs(cuda, 1, len(PEAKS))
        calls.append(lambda s, opts=opts, o=o: L.lib().mi_fit_batch(
            x.data_ptr(), lines.data_ptr(), 1, X.size, pk.data_ptr(), len(PEAKS), C.byref(opts), o[0].data_ptr(),
            o[1].data_ptr(), s))
        outs.append(o)
    _check(calls, outs, 6000)


def test_one_eta_plan_at_three_batch_sizes(cuda):
    """units a warp, and so the shared memory, follow the batch"""
    plan = FitPlan(X, PEAKS, kind="eta", half_window=6, max_iter=1, x_bin=0.25, device=cuda)
    calls, outs = [], []
    for n in (1, 1000, 4000, 1, 2000, 1):
        y = torch.as_tensor(_lines(n, 2).astype(np.float32), device=cuda)
        o = _outputs(cuda, n, len(PEAKS))
        calls.append(lambda s, y=y, n=n, o=o: L.lib().mi_fit_plan_run(
            plan._h, y.data_ptr(), L.DT_F32, n, 1, X.size, 0, 1, o[0].data_ptr(), o[1].data_ptr(), s))
        outs.append(o)
    _check(calls, outs, 6000)
