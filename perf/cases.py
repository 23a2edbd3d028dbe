"""Performance cases: the calls a user of this framework makes, with the inputs they meet.

listed() and draw() give cases (dicts of plain values), prepare() what a program holds before
the call, run() one pass through the public entry points, work() the bytes and operations the
pass cannot do without, exact() the outputs in 64 bits by plain torch.

Detectors, binnings, modes and frame models are those of ``midas_b200.synth`` (the sweep, the
powder patterns, the serving mix, the published PILATUS configuration, the panel set), at full
size and scaled down by whole factors.
"""
from __future__ import annotations

import functools
import math
from dataclasses import replace

import numpy as np
import torch

from midas_b200 import kernels, mapper, peakfit, synth

DEV = torch.device("cuda", 0)
KEEP = 1e-9          # bins whose in-bounds area is at or below this are empty

DETECTORS = {
    "sweep_2880": synth.sweep_2880,                        # 3960 x 360 bins, gradient
    "powder_2048": synth.powder_2048,                      # 990 x 72, floor
    "powder_2048_fine": synth.powder_2048_fine,            # 1980 x 180, gradient
    "pilatus_1679": synth.pilatus_1679,                    # 1475 x 1679 int32, module gaps, floor
    "pilatus3_2m": synth.pilatus3_2m_published,            # 1475 x 1679 uint16, 1108 x 72, floor
    "detector_1024": lambda: synth.detector_1024(0),       # 495 x 45, floor
    "detector_1024_fine": lambda: synth.detector_1024(1),  # 990 x 72, bilinear
}


def listed():
    return [
        # an omega sweep caked 128 frames a call: the framework's headline use
        {"name": "sweep_u16_f128", "kind": "batch", "detector": "sweep_2880", "div": 1, "frames": 128,
         "encoding": "mma", "mode": "gradient"},
        # the reference's published detector and binning, a batch that is no multiple of 32
        {"name": "pilatus3_u16_f100", "kind": "batch", "detector": "pilatus3_2m", "div": 1, "frames": 100,
         "encoding": "mma", "mode": "floor"},
        # 32-bit counts of a hybrid pixel detector through the default encoding
        {"name": "pilatus_i32_f50", "kind": "batch", "detector": "pilatus_1679", "div": 1, "frames": 50,
         "encoding": "auto", "mode": "floor"},
        # a serving stream that fell behind: the few frames that queued up go in one call
        {"name": "burst_u16_f4", "kind": "batch", "detector": "powder_2048_fine", "div": 1, "frames": 4,
         "encoding": "mma", "mode": "gradient"},
        # midas_integrate's own calls: one dark-subtracted float frame, then its lineout
        {"name": "frame_f32_gradient", "kind": "frame", "detector": "powder_2048_fine", "div": 1,
         "mode": "gradient"},
        # the same with the variance propagated
        {"name": "variance_f32_bilinear", "kind": "variance", "detector": "detector_1024_fine", "div": 1,
         "mode": "bilinear"},
        # one serving frame: upload, one-frame integration, ring fits (the smallest stream, the
        # one whose calls are all latency, and an ordinary one)
        {"name": "serve_1024", "kind": "serve", "detector": "detector_1024", "div": 1, "mode": "floor"},
        {"name": "serve_2048", "kind": "serve", "detector": "powder_2048_fine", "div": 1, "mode": "gradient"},
        # five uneven panels, u16 and int32, merged into one cake
        {"name": "panels_f40", "kind": "panels", "div": 2, "frames": 40, "q_bin": 0.004, "eta_bin": 2.0},
        # every ring of every frame of a sweep
        {"name": "fits_pv", "kind": "fits", "frames": 1408, "model": "pv", "half": 15},
        # every ring of every eta column of a batch of cakes
        {"name": "fits_eta", "kind": "eta", "frames": 32, "n_eta": 360, "half": 12},
        # a new geometry: the pixel-split map of a masked detector
        {"name": "map_pilatus", "kind": "map", "detector": "pilatus_1679", "div": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["batch", "batch", "batch", "frame", "variance", "serve", "panels", "fits", "eta", "map"])
    if kind == "panels":
        return {"kind": kind, "div": rng.choice([2, 3, 4]), "frames": _log(rng, 1, 80),
                "q_bin": rng.choice([0.004, 0.006, 0.01]), "eta_bin": rng.choice([2.0, 3.0, 5.0])}
    if kind == "fits":
        return {"kind": kind, "frames": _log(rng, 1, 1408), "model": rng.choice(["pv", "tch"]),
                "half": rng.randint(8, 24)}
    if kind == "eta":
        return {"kind": kind, "frames": _log(rng, 1, 40), "n_eta": rng.choice([45, 72, 180, 360]),
                "half": rng.randint(8, 16)}
    small = ["pilatus_1679", "pilatus3_2m", "powder_2048", "detector_1024", "detector_1024_fine"]
    if kind == "map":
        return {"kind": kind, "detector": rng.choice(small), "div": rng.choice([1, 2, 3])}
    det = rng.choice(small + ["powder_2048_fine", "sweep_2880"])
    case = {"kind": kind, "detector": det,
            "div": rng.choice([2, 3, 4]) if det == "sweep_2880" else rng.choice([1, 1, 2, 3]),
            "mode": rng.choice(["floor", "bilinear", "gradient"])}
    if kind == "batch":
        case["frames"] = _log(rng, 1, 128)
        wide = det == "pilatus_1679"
        case["encoding"] = rng.choice(["auto", "csr"] if wide else ["mma", "mma", "auto"])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _workload(case, seed=0):
    w = DETECTORS[case["detector"]]()
    if case["div"] > 1:
        w = synth.scaled(w, case["div"])
    return replace(w, mode=case.get("mode", w.mode), seed=1000 + seed)


@functools.lru_cache(maxsize=8)
def _map_of(detector, div):
    """The detector's pixel map: a file a program reads once (the geometry has no seed)."""
    w = _workload({"detector": detector, "div": div})
    return mapper.build_map(w.mapper, device=0, mask=w.mask())[0]


@functools.lru_cache(maxsize=4)
def _panel_maps(div, q_bin, eta_bin):
    return [mapper.build_map(w.mapper, device=0, mask=w.mask())[0] for w in _panels(div, q_bin, eta_bin, 0)]


def _panels(div, q_bin, eta_bin, seed):
    ws = synth.scaled_panels(synth.panel_set(q_bin=q_bin, eta_bin=eta_bin, mode="floor"), div)
    return [replace(w, seed=w.seed + 1000 * (seed + 1)) for w in ws]


def _frames(w, n):
    """n raw frames (counts with the dark) of the workload, and its dark."""
    dt = {"uint16": torch.uint16, "int32": torch.int32}[w.frame_dtype]
    return w.frames(0, n, device=DEV, dtype=dt), w.dark(device=DEV)


def _plan_args(w):
    m = w.mapper
    return dict(n_r=w.n_r, n_eta=w.n_eta, n_pixels_y=m.NrPixelsY, n_pixels_z=m.NrPixelsZ, bc_y=m.BC_y,
                bc_z=m.BC_z, device=DEV)


def _image(w):
    """One dark-subtracted float frame, as midas_integrate takes it, and its variance."""
    raw, dark = _frames(w, 1)
    raw = raw[0].to(torch.float32)
    return raw - dark, raw


def _rings():
    return torch.as_tensor(synth.ring_peaks(synth.sweep_2880()), device=DEV)


def _profiles(gen, n, r, rings):
    """n noisy powder profiles over r: pseudo-Voigt rings, heights and widths drifting."""
    def u(lo, hi):
        return lo + (hi - lo) * torch.rand((n, rings.numel(), 1), generator=gen, device=DEV, dtype=torch.float64)
    amp = torch.linspace(1.0e3, 2.0e4, rings.numel(), device=DEV, dtype=torch.float64).view(1, -1, 1) * u(0.8, 1.2)
    c, f, e = rings.view(1, -1, 1) + u(-0.3, 0.3), u(1.3, 1.9), u(0.3, 0.7)
    y = torch.full((n, r.numel()), 100.0, device=DEV, dtype=torch.float64)
    for k in range(rings.numel()):
        q = ((r.view(1, -1) - c[:, k]) / (0.5 * f[:, k])) ** 2
        y += amp[:, k] * (e[:, k] / (1 + q) + (1 - e[:, k]) * torch.exp(-math.log(2.0) * q))
    return y


def _noise(gen, y, per):
    """Counting noise of a mean over ``per`` pixels."""
    return y + torch.sqrt(y / per) * torch.randn(y.shape, generator=gen, device=DEV, dtype=torch.float64)


def _sweep_axis():
    return torch.as_tensor(synth.r_centres(synth.sweep_2880()), device=DEV)


def _lineouts(case, seed):
    gen = torch.Generator(DEV).manual_seed(seed)
    r, rings = _sweep_axis(), _rings()
    return r, rings, _noise(gen, _profiles(gen, case["frames"], r, rings), 400.0)


def _eta_cake(case, seed):
    """A [F, n_r, n_eta] float cake: each frame's profile with texture along eta."""
    gen = torch.Generator(DEV).manual_seed(seed)
    r, rings = _sweep_axis(), _rings()
    F, E = case["frames"], case["n_eta"]
    y = _profiles(gen, F, r, rings)
    tex = 0.7 + 0.6 * torch.rand((F, 1, E), generator=gen, device=DEV, dtype=torch.float64)
    out = torch.empty((F, r.numel(), E), device=DEV, dtype=torch.float32)
    for f in range(F):
        out[f] = _noise(gen, y[f].unsqueeze(1) * tex[f], 6.0).to(torch.float32)
    return r, rings, out


def _map_params(case, seed):
    """The detector with the beam line's corrections in the weights; the seed is the beam's
    polarisation (the same pixels meet the same bins, so every seed's map has one size)."""
    w = _workload(case)
    f = float(np.random.default_rng(seed).uniform(0.9, 0.999))
    return replace(w.mapper, SolidAngleCorrection=1, PolarizationCorrection=1, PolarizationFraction=f), w.mask()


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        w = _workload(case, seed)
        s["plan"] = kernels.CakePlan(_map_of(case["detector"], case["div"]), mode=w.mode, encoding=case["encoding"],
                                     **_plan_args(w))
        s["frames"], dark = _frames(w, case["frames"])
        s["plan"].set_dark(dark.cpu().numpy())
    elif kind in ("frame", "variance"):
        w = _workload(case, seed)
        s["geom"] = kernels.build_csr(_map_of(case["detector"], case["div"]), build_modes=(w.mode,),
                                      compute_variance=kind == "variance", **_plan_args(w))
        s["mode"] = w.mode
        s["image"], s["variance"] = _image(w)
        s["geom"].plan(w.mode, True)
        if kind == "variance":
            s["geom"].plan(w.mode, True, True)
    elif kind == "serve":
        w = _workload(case, seed)
        s["plan"] = kernels.CakePlan(_map_of(case["detector"], case["div"]), mode=w.mode, **_plan_args(w),
                                     encoding="mma" if w.frame_dtype == "uint16" else "csr")
        frames, dark = _frames(w, 1)
        s["plan"].set_dark(dark.cpu().numpy())
        s["host"] = frames.cpu().pin_memory()
        s["dev"] = torch.zeros_like(frames)
        s["x"] = torch.as_tensor(synth.r_centres(w), device=DEV)
        s["peaks"] = torch.as_tensor(synth.ring_peaks(w), device=DEV)
        s["x_bin"] = w.mapper.RBinSize
    elif kind == "panels":
        ws = _panels(case["div"], case["q_bin"], case["eta_bin"], seed)
        s["plan"] = kernels.PanelPlan(
            _panel_maps(case["div"], case["q_bin"], case["eta_bin"]), n_r=ws[0].n_r, n_eta=ws[0].n_eta, device=DEV,
            shapes=[(w.mapper.NrPixelsY, w.mapper.NrPixelsZ) for w in ws],
            beam_centres=[(w.mapper.BC_y, w.mapper.BC_z) for w in ws], mode="floor")
        both = [_frames(w, case["frames"]) for w in ws]
        s["frames"] = [f for f, _ in both]
        s["plan"].set_dark([d.cpu().numpy() for _, d in both])
    elif kind == "fits":
        s["x"], s["peaks"], s["lineouts"] = _lineouts(case, seed)
        s["args"] = dict(model=case["model"], half_window=case["half"], x_bin=0.25)
    elif kind == "eta":
        r, rings, s["cake"] = _eta_cake(case, seed)
        s["plan"] = peakfit.FitPlan(r.cpu().numpy(), rings.cpu().numpy(), kind="eta", half_window=case["half"],
                                    x_bin=0.25, device=DEV)
    elif kind == "map":
        s["params"], s["mask"] = _map_params(case, seed)
    return s


def run(s):
    kind = s["kind"]
    if kind == "batch" or kind == "panels":
        cake, aw, sm = s["plan"].integrate(s["frames"])
        return {"cake": cake, "area_weighted": aw, "simple_mean": sm}
    if kind == "frame":
        cake = kernels.integrate(s["image"], s["geom"], mode=s["mode"])
        return {"cake": cake, "profile": kernels.profile_1d(cake, s["geom"])}
    if kind == "variance":
        cake, var = kernels.integrate_with_variance(s["image"], s["geom"], mode=s["mode"],
                                                    variance_image=s["variance"])
        p, pv = kernels.profile_1d_with_variance(cake, var, s["geom"])
        return {"cake": cake, "variance": var, "profile": p, "profile_variance": pv}
    if kind == "serve":
        s["plan"].upload(s["host"], s["dev"])
        cake, aw, sm = s["plan"].integrate_plain(s["dev"])
        fit = peakfit.fit_batch(s["x"], aw, s["peaks"], half_window=15, x_bin=s["x_bin"])
        return {"cake": cake, "area_weighted": aw, "simple_mean": sm, "fits": fit.params, "rejected": fit.iters < 0}
    if kind == "fits":
        fit = peakfit.fit_batch(s["x"], s["lineouts"], s["peaks"], **s["args"])
        return {"fits": fit.params, "rejected": fit.iters < 0}
    if kind == "eta":
        fit = s["plan"].fit_cake_eta(s["cake"])
        return {"fits": fit.params, "rejected": fit.iters < 0}
    pm, bin_mask = mapper.build_map(s["params"], device=0, mask=s["mask"])
    px = pm.pxList
    return {"y": px["y"], "z": px["z"], "frac": px["frac"], "deltaR": px["deltaR"], "areaWeight": px["areaWeight"],
            "counts": pm.counts, "offsets": pm.offsets, "bin_mask": bin_mask}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=16)
def _map_size(detector, div):
    """(records, referenced pixels) of a detector's map."""
    pm = _map_of(detector, div)
    w = _workload({"detector": detector, "div": div})
    ny, nz = w.mapper.NrPixelsY, w.mapper.NrPixelsZ
    hit = np.zeros(ny * nz, dtype=bool)
    iy = np.clip(pm.pxList["y"].astype(np.int64), 0, ny - 1)
    iz = np.clip(pm.pxList["z"].astype(np.int64), 0, nz - 1)
    hit[iz * ny + iy] = True
    return pm.n_entries, int(hit.sum())


def work(case):
    """Weights at 8 B a term (column and weight; a resampled record has about 1.85 coalesced
    terms), referenced pixels and outputs once; 2 operations a term and frame."""
    kind = case["kind"]
    if kind in ("fits", "eta"):
        # an iteration evaluates the model and its Jacobian at every sample of a window (about 60
        # operations and 28 sums of products) twice; windows converge in 10 to 20 iterations
        n_win = case["frames"] * (case.get("n_eta", 1)) * _rings().numel()
        n = 2 * case["half"] + 1
        return {"bytes": n_win * (n * (8 if kind == "fits" else 4) + 92), "flops": n_win * n * 2 * 15 * 110}
    if kind == "panels":
        F, n_rec, n_px, px_b = case["frames"], 0, 0, 0
        maps = _panel_maps(case["div"], case["q_bin"], case["eta_bin"])
        for w, pm in zip(_panels(case["div"], case["q_bin"], case["eta_bin"], 0), maps):
            n_rec += pm.n_entries
            n_px = w.mapper.NrPixelsY * w.mapper.NrPixelsZ
            px_b += n_px * (2 if w.frame_dtype == "uint16" else 4)
        n_bins, n_r = maps[0].n_bins, _panel_rows(case)
        return {"bytes": 8 * n_rec + F * (px_b + 4 * n_bins + 16 * n_r), "flops": 2 * n_rec * F}
    n_rec, n_px = _map_size(case["detector"], case["div"])
    w = _workload(case)
    n_bins, n_r = w.n_r * w.n_eta, w.n_r
    if kind == "map":
        # the records and tables written once; a few hundred operations a record
        return {"bytes": 24 * n_rec + 12 * n_bins, "flops": 400 * n_rec}
    terms = n_rec if w.mode == "floor" else int(1.85 * n_rec)
    if kind == "batch":
        es = 2 if w.frame_dtype == "uint16" else 4
        F = case["frames"]
        return {"bytes": 8 * terms + F * (es * n_px + 4 * n_bins + 16 * n_r), "flops": 2 * terms * F}
    if kind == "serve":
        es = 2 if w.frame_dtype == "uint16" else 4
        return {"bytes": 8 * terms + es * n_px + 8 * n_bins + 16 * n_r, "flops": 2 * terms}
    both = 2 if kind == "variance" else 1
    return {"bytes": both * (8 * terms + 4 * n_px + 4 * n_bins + 4 * n_r), "flops": both * 2 * terms}


def _panel_rows(case):
    return _panels(case["div"], case["q_bin"], case["eta_bin"], 0)[0].n_r


# ---------------------------------------------------------------------------
# the outputs in 64 bits
# ---------------------------------------------------------------------------
def _terms(pm, w):
    """(bin, pixel, weight) of every term of the map under the workload's mode, and the
    in-bounds area of every bin."""
    m = w.mapper
    ny, nz = m.NrPixelsY, m.NrPixelsZ
    px = {k: torch.as_tensor(np.ascontiguousarray(pm.pxList[k]), device=DEV).to(torch.float64)
          for k in ("y", "z", "frac", "deltaR", "areaWeight")}
    counts = torch.as_tensor(pm.counts.astype(np.int64), device=DEV)
    b = torch.repeat_interleave(torch.arange(pm.n_bins, device=DEV), counts)   # records are in bin order
    y, z = px["y"], px["z"]
    iy, iz = y.to(torch.int64), z.to(torch.int64)
    inside = (iy >= 0) & (iy < ny) & (iz >= 0) & (iz < nz)
    area = torch.zeros(pm.n_bins, dtype=torch.float64, device=DEV)
    area.index_add_(0, b[inside], px["areaWeight"][inside])
    if w.mode == "floor":
        return b[inside], (iz * ny + iy)[inside], px["frac"][inside], area
    if w.mode == "gradient":
        dy, dz = y - m.BC_y, z - m.BC_z
        R = torch.sqrt(dy * dy + dz * dz)
        sc = torch.where(R > 1.0, px["deltaR"] / R, torch.zeros_like(R))
        y, z = y - sc * dy, z - sc * dz
    iy, iz = torch.floor(y), torch.floor(z)
    fy, fz = y - iy, z - iz
    for i, f, n in ((iy, fy, ny), (iz, fz, nz)):
        over, under = i >= n - 1, i < 0
        i[over], f[over] = n - 2, 1.0
        i[under], f[under] = 0, 0.0
    base = (iz * ny + iy).to(torch.int64)
    q = px["frac"]
    cols = torch.cat([base, base + 1, base + ny, base + ny + 1])
    wts = torch.cat([(1 - fy) * (1 - fz) * q, fy * (1 - fz) * q, (1 - fy) * fz * q, fy * fz * q])
    return b.repeat(4), cols, wts, area


def _sums(terms, images):
    """Sum of weight x pixel per bin of each image [n, pixels] (float64)."""
    b, cols, wts, area = terms
    out = torch.zeros((images.shape[0], area.numel()), dtype=torch.float64, device=DEV)
    for f in range(images.shape[0]):
        out[f].index_add_(0, b, wts * images[f][cols])
    return out


def _reduced(sums, area, n_r, power=1):
    """Cake and both profiles; power 2: of variances."""
    a = torch.where(area > KEEP, area, torch.zeros_like(area))
    cake = torch.where(a > 0, sums / torch.where(a > 0, a, torch.ones_like(a)) ** power, torch.zeros_like(sums))
    c, g = cake.view(cake.shape[0], n_r, -1), a.view(1, n_r, -1)
    valid = (g > 0).to(torch.float64)
    den, cnt = g.sum(2) ** power, valid.sum(2) ** power
    aw = torch.where(den > 0, (c * g ** power).sum(2) / den.clamp(min=1e-300), torch.zeros_like(den))
    sm = torch.where(cnt > 0, (c * valid).sum(2) / cnt.clamp(min=1), torch.zeros_like(cnt))
    return c, aw, sm


def _exact_cake(case, seed):
    w = _workload(case, seed)
    terms = _terms(_map_of(case["detector"], case["div"]), w)
    frames, dark = _frames(w, case.get("frames", 1))
    frames = frames.reshape(frames.shape[0], -1)
    d = dark.reshape(-1).to(torch.float64)
    sums = torch.cat([_sums(terms, frames[f:f + 1].to(torch.float64) - d) for f in range(frames.shape[0])])
    return _reduced(sums, terms[3], w.n_r)


def _pv(p, x, xn):
    """Pseudo-Voigt windows: value and Jacobian at x [n, samples]."""
    c, h, fw, e, b0, b1 = (p[:, k:k + 1] for k in range(6))
    hw = 0.5 * fw.clamp(min=1e-6)
    u = (x - c) / hw
    u2 = u * u
    lor, gau = 1 / (1 + u2), torch.exp(-math.log(2.0) * u2)
    shape = e * lor + (1 - e) * gau
    d = -e * lor * lor - (1 - e) * math.log(2.0) * gau
    one = torch.ones_like(x)
    return b0 + b1 * xn + h * shape, torch.stack([h * d * (-2 * u / hw), shape, h * d * (-u2 / hw), h * (lor - gau),
                                                  one, xn.expand_as(x)], 2)


def _pv_flat(p, x, xn):
    """Height-normalised pseudo-Voigt with a flat background (centre, FWHM, height, mixing, level)."""
    c, g, i, mu, b = (p[:, k:k + 1] for k in range(5))
    c0 = 4 * math.log(2.0)
    d = x - c
    q = d * d / (g * g)
    lor, gau = 1 / (1 + 4 * q), torch.exp(-c0 * q)
    jc = i * (mu * 8 * d / (g * g) * lor * lor + (1 - mu) * gau * 2 * c0 * d / (g * g))
    jg = i * (mu * 8 * q / g * lor * lor + (1 - mu) * gau * 2 * c0 * q / g)
    shape = mu * lor + (1 - mu) * gau
    return b + i * shape, torch.stack([jc, jg, shape, i * (lor - gau), torch.ones_like(x)], 2)


def _levenberg(model, p, x, xn, y, lo, hi, steps):
    """Least squares over each window from p, steps kept inside [lo, hi]; (p, chi^2)."""
    p = torch.minimum(torch.maximum(p, lo), hi)
    lam = torch.full((p.shape[0],), 1e-3, dtype=torch.float64, device=DEV)

    def normal(q):
        m, J = model(q, x, xn)
        r = y - m
        return J.transpose(1, 2) @ J, (J * r.unsqueeze(2)).sum(1), (r * r).sum(1)
    A, g, chi = normal(p)
    for _ in range(steps):
        diag = torch.diagonal(A, dim1=1, dim2=2).clamp(min=1e-30)
        step, _ = torch.linalg.solve_ex(A + torch.diag_embed(lam.unsqueeze(1) * diag), g)
        q = torch.minimum(torch.maximum(p + torch.nan_to_num(step), lo), hi)
        A2, g2, chi2 = normal(q)
        ok = chi2 <= chi
        lam = torch.where(ok, (lam * 0.1).clamp(min=1e-12), (lam * 10).clamp(max=1e12))
        p, chi = torch.where(ok.unsqueeze(1), q, p), torch.where(ok, chi2, chi)
        A, g = torch.where(ok.view(-1, 1, 1), A2, A), torch.where(ok.unsqueeze(1), g2, g)
    return p, chi


def _walk(y, at, level):
    """Bins between the first samples at or under ``level`` on both sides of ``at``."""
    n = y.shape[1]
    k = torch.arange(n, device=DEV).view(1, -1)
    low = y <= level.unsqueeze(1)
    left = torch.where(low & (k <= at), k, torch.zeros_like(k)).amax(1)
    right = torch.where(low & (k >= at), k, torch.full_like(k, n - 1)).amin(1)
    return (right - left).to(torch.float64)


def _exact_pv(x, lines, peaks, half, x_bin):
    """fit_batch's outputs for pseudo-Voigt windows that lie inside the axis."""
    F, n = lines.shape[0], 2 * half + 1
    at = (x.view(1, -1) - peaks.view(-1, 1)).abs().argmin(1)
    idx = (at.view(-1, 1) + torch.arange(-half, half + 1, device=DEV)).clamp(0, x.numel() - 1)
    y = lines[:, idx].reshape(-1, n)
    ref = x[at].repeat(F)
    xs = x[idx].repeat(F, 1) - ref.unsqueeze(1)
    xn = 2 * (xs - xs[:, :1]) / (xs[:, -1:] - xs[:, :1]) - 1
    ends = max(1, min(5, n // 4))
    bg = (y[:, :ends].sum(1) + y[:, -ends:].sum(1)) / (2 * ends)
    amp = y[:, half] - bg
    amp = torch.where(amp <= 0, y[:, half], amp)
    fw = _walk(y, half, bg + 0.5 * amp)
    fw = torch.where(fw > 1, fw, torch.full_like(fw, 2.0)) * x_bin
    zero, big = torch.zeros_like(bg), torch.full_like(bg, math.inf)
    span = xs.abs().amax(1)
    p = torch.stack([zero, amp, fw, zero + 0.5, bg, zero], 1)
    lo = torch.stack([-span, zero, zero + 0.05 * x_bin, zero, -big, -big], 1)
    hi = torch.stack([span, big, 4 * span, zero + 1, big, big], 1)
    p, chi = _levenberg(_pv, p, xs, xn, y, lo, hi, 60)
    c, h, f, e = ref + p[:, 0], p[:, 1], p[:, 2], p[:, 3]
    area = h * f * (e * math.pi / 2 + (1 - e) * math.sqrt(math.pi / math.log(2.0)) / 2)
    cols = [area, c, zero, zero, f, e, chi / max(n - 6, 1), h, p[:, 4], p[:, 5], zero]
    return torch.stack(cols, 1).view(F, peaks.numel(), 11)


def _exact_eta(case, seed):
    x, peaks, cake = _eta_cake(case, seed)
    F, n_r, E = cake.shape
    out = torch.zeros((F * E, peaks.numel(), 11), dtype=torch.float64, device=DEV)
    pad = case["half"] * 0.25
    for k in range(peaks.numel()):
        sel = torch.nonzero((x >= peaks[k] - pad) & (x <= peaks[k] + pad)).view(-1)
        y = cake[:, sel, :].to(torch.float64).permute(0, 2, 1).reshape(F * E, -1)
        n = sel.numel()
        xs = (x[sel] - peaks[k]).view(1, -1).expand(F * E, n)
        bg = (0.5 * (y[:, 0] + y[:, -1])).clamp(min=0)
        top = y.amax(1)
        one = torch.ones_like(bg)
        p = torch.stack([0 * one, 0.75 * one, top - bg, 0.5 * one, bg], 1)
        lo = torch.stack([xs[:, 0], 0.125 * one, (top - bg) / 100, 0 * one, 0 * one], 1)
        hi = torch.stack([xs[:, -1], 0.125 * n * one, 1.5 * top, one, torch.where(bg > 0, 1.5 * bg, 0.5 * top)], 1)
        p, chi = _levenberg(_pv_flat, p, xs, xs, y, lo, hi, 60)
        snr = p[:, 2] / torch.sqrt(chi / n)
        keep = (snr > 1).to(torch.float64)
        out[:, k, 1], out[:, k, 6] = keep * (peaks[k] + p[:, 0]), keep * snr
        out[:, k, 7], out[:, k, 8] = keep * p[:, 2], keep * p[:, 4]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        cake, aw, sm = _exact_cake(case, seed)
        return {"cake": cake, "area_weighted": aw, "simple_mean": sm}
    if kind in ("frame", "variance"):
        w = _workload(case, seed)
        b, cols, wts, area = terms = _terms(_map_of(case["detector"], case["div"]), w)
        image, var = (t.reshape(1, -1).to(torch.float64) for t in _image(w))
        cake, aw, _ = _reduced(_sums(terms, image), area, w.n_r)
        if kind == "frame":
            return {"cake": cake[0], "profile": aw[0]}
        # the weights of a (bin, pixel) pair are summed before they are squared
        key, back = torch.unique(b * image.shape[1] + cols, return_inverse=True)
        w2 = torch.zeros(key.numel(), dtype=torch.float64, device=DEV).index_add_(0, back, wts) ** 2
        pairs = (key // image.shape[1], key % image.shape[1], w2, area)
        vk, vaw, _ = _reduced(_sums(pairs, var), area, w.n_r, power=2)
        return {"cake": cake[0], "variance": vk[0], "profile": aw[0], "profile_variance": vaw[0]}
    if kind == "serve":
        cake, aw, sm = _exact_cake(case, seed)
        w = _workload(case, seed)
        fits = _exact_pv(torch.as_tensor(synth.r_centres(w), device=DEV), aw,
                         torch.as_tensor(synth.ring_peaks(w), device=DEV), 15, w.mapper.RBinSize)
        return {"cake": cake[0], "area_weighted": aw[0], "simple_mean": sm[0], "fits": fits, "rejected": None}
    if kind == "panels":
        maps = _panel_maps(case["div"], case["q_bin"], case["eta_bin"])
        ws = _panels(case["div"], case["q_bin"], case["eta_bin"], seed)
        sums, area = 0, 0
        for w, pm in zip(ws, maps):
            terms = _terms(pm, w)
            frames, dark = _frames(w, case["frames"])
            frames = frames.reshape(frames.shape[0], -1).to(torch.float64) - dark.reshape(-1).to(torch.float64)
            sums, area = sums + _sums(terms, frames), area + terms[3]
        cake, aw, sm = _reduced(sums, area, ws[0].n_r)
        return {"cake": cake, "area_weighted": aw, "simple_mean": sm}
    if kind == "fits":
        if case["model"] != "pv":
            return None
        x, peaks, lines = _lineouts(case, seed)
        return {"fits": _exact_pv(x, lines, peaks, case["half"], 0.25), "rejected": None}
    if kind == "eta":
        return {"fits": _exact_eta(case, seed), "rejected": None}
    return None                  # the map's records come from a chain of clipping decisions
