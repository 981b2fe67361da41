"""Workloads the framework is timed on: calls of its public entry points at the sizes users run.

``listed()`` names a dozen fixed cases, ``draw(rng)`` gives more of the same ranges.  ``prepare``
makes what a program holds before the call (a request, an uploaded session, a running server),
``run`` is one pass through the entry points, ``work`` the bytes and operations that pass cannot do
without, and ``exact`` the same outputs from plain torch in 64 bits.

The entry points return MATLAB doubles; the engine computes in single precision (FP64 sums in the
detectors), so a program keeps the images, patterns and exit waves in single precision, and so does
``run``.

Specimens are SrTiO3 [001] blocks (SrO and TiO2 planes, 3.905 Angstrom cell) that fill the
potential grid, or ``cells`` x ``cells`` unit cells in its middle; the seed places the block
(a sub-cell offset) and, with ``thermal``, displaces every atom as one frozen-phonon configuration
does.  Probes carry C3 -5 um and a focal spread where there is more than one.
"""
import math

import numpy as np
import torch

from totem_b200 import capi, specimen
from totem_b200.request import HrtemSpec, StemRequest

KV = 300.0
CELL = 3.905                     # Angstrom, cubic SrTiO3
SLICE = CELL / 2                 # one atomic plane per slice
PLANES = (((38, 0.0, 0.0), (8, 0.5, 0.5)),                     # SrO
          ((22, 0.5, 0.5), (8, 0.5, 0.0), (8, 0.0, 0.5)))      # TiO2
RMS = {38: 0.089, 22: 0.075, 8: 0.088}                         # thermal displacement per axis, Angstrom
DETECTORS = ((60.0, 200.0), (0.0, 10.0), (15.0, 40.0))         # ADF, BF, ABF collection angles, mrad

# relativistic wavelength (Angstrom) and interaction constant (1 / (kV Angstrom)) at KV
_H, _E, _M, _C = 6.6255916e-34, 1.602102e-19, 9.1093807e-31, 2.9979251e8
_EV = _E * KV * 1e3
WAVELENGTH = 1e10 * _H * _C / math.sqrt(_EV * (2 * _M * _C * _C + _EV))
SIGMA = 2 * math.pi / (WAVELENGTH * KV) * (_M * _C * _C + _EV) / (2 * _M * _C * _C + _EV)


def _stem(name, window, grid, rows, cols, slices, step=8, sampling=0.0625, param="p", probes=1, mids=0, detectors=2,
          thermal=False, cells=0, kind="stem"):
    return {"name": name, "kind": kind, "window": window, "grid": grid, "rows": rows, "cols": cols, "step": step,
            "slices": slices, "sampling": sampling, "param": param, "probes": probes, "mids": mids,
            "detectors": detectors, "thermal": thermal, "cells": cells}


def listed():
    return [
        # A first look at a thin specimen: a dozen probes, six slices.  Launches and latency.
        _stem("stem_64_first_look", 64, 128, 3, 4, 6, step=5, sampling=0.2, probes=1, mids=2, detectors=3),
        # The ordinary scan of a small field: Lobato rows, three defocus-spread probes, a mid-slice image.
        _stem("stem_256_spread", 256, 512, 16, 16, 40, param="l", probes=3, mids=1, thermal=True),
        # The full STEM-ADF image: 64 x 64 probes of 512^2 on the 8 x 8 cell block, at 40 slices.
        _stem("stem_512_adf", 512, 1024, 64, 64, 40, cells=8),
        # One frozen-phonon configuration at the wide window, a 16 x 16 part of its scan.
        _stem("stem_1024_phonon", 1024, 2048, 16, 16, 20, thermal=True),
        # The largest window and potential grid.
        _stem("stem_2048", 2048, 4096, 4, 8, 8, thermal=True),
        # A window that is no power of two, on a potential grid that is none either; a ragged scan.
        _stem("stem_640_ragged", 640, 1280, 13, 11, 21, step=7, detectors=3),
        # A window edge outside the fused sizes (the program takes any even edge).
        _stem("stem_304_any_edge", 304, 700, 12, 12, 20, sampling=0.09, mids=1),
        # The one-shot call with host buffers in and out, as the MEX entry point is called.
        _stem("oneshot_256", 256, 512, 8, 8, 20, kind="oneshot"),
        # HRTEM: the transmission, a plane wave through it, the image over a focal series.
        {"name": "hrtem_1024", "kind": "hrtem", "grid": 1024, "slices": 20, "sampling": 0.05, "param": "l",
         "probes": 5, "thermal": False, "cells": 0},
        # CBED at one position with a focal spread: few waves, many slices.
        _stem("cbed_512", 512, 1024, 1, 1, 40, probes=7, thermal=True, kind="cbed"),
        # The transmission stack alone (the transmission-only MEX), used on the device afterwards.
        {"name": "transmission_2048", "kind": "transmission", "grid": 2048, "slices": 20, "sampling": 0.0625,
         "param": "p", "thermal": True, "cells": 0},
        # Several users at once: requests of mixed size through the batching server.
        {"name": "server_mixed", "kind": "server", "window": 256, "window2": 512, "requests": 6, "probes": 96,
         "slices": 30, "thermal": False},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    """One more case: a kind of call, then sizes over the whole range of that kind."""
    kind = rng.choice(["stem"] * 5 + ["oneshot", "hrtem", "cbed", "transmission", "server"])
    slices = rng.randint(6, 40)
    param, thermal = rng.choice("pl"), rng.random() < 0.5
    if kind in ("hrtem", "transmission"):
        grid = rng.choice([256, 384, 400, 512, 600, 640, 768, 1000, 1024, 1280] + ([2048] if kind != "hrtem" else []))
        c = {"kind": kind, "grid": grid, "slices": slices, "sampling": rng.choice([0.05, 0.0625, 0.1]),
             "param": param, "thermal": thermal, "cells": 0}
        if kind == "hrtem":
            c["probes"] = rng.choice([1, 3, 5, 11])
        return c
    if kind == "server":
        return {"kind": kind, "window": rng.choice([128, 256, 320]), "window2": rng.choice([400, 512, 768]),
                "requests": rng.randint(3, 8), "probes": int(_log(rng, 12, 200)), "slices": rng.randint(10, 40),
                "thermal": thermal}
    edge = int(_log(rng, 64, 2100))
    window = min([64, 96, 128, 160, 192, 208, 256, 288, 304, 320, 384, 400, 448, 512, 576, 640, 768, 800, 1024, 1152,
                  1280, 1536, 2048], key=lambda n: abs(math.log(n / edge)))
    if kind != "stem":
        window = min(window, 768)
    # probes so that the waves of one pass hold 2^19 .. 2^27 points (32 at most for the largest window)
    items = max(1, min(4096, int(_log(rng, 2 ** 19, 2 ** 27) / window ** 2)))
    probes = 1
    if kind == "cbed":
        rows = cols = 1
        probes = rng.choice([1, 3, 5, 7, 11])
    else:
        if items >= 9 and rng.random() < 0.3:
            probes = 3
        rows = max(1, int(math.sqrt(items / probes) * rng.uniform(0.6, 1.4)))
        cols = max(1, items // probes // rows)
    step = rng.randint(2, 8)
    need = window + (max(rows, cols) - 1) * step
    grid = 1 << (need - 1).bit_length() if rng.random() < 0.6 else need + need % 2
    c = _stem("", window, grid, rows, cols, min(slices, 8) if window > 1024 else slices, step=step,
              sampling=0.2 if window < 128 else rng.choice([0.0625, 0.09]), param=param, probes=probes,
              mids=rng.choice([0, 0, 1, 2]) if kind != "cbed" else 0, detectors=rng.choice([1, 2, 3]),
              thermal=thermal, kind=kind)
    del c["name"]
    return c


# ----------------------------------------------------------------------------------------------
# Inputs
# ----------------------------------------------------------------------------------------------

def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _axis(n, sampling):
    """Centred reciprocal axis, 1/Angstrom."""
    return torch.arange(-(n // 2), n - n // 2, dtype=torch.float64, device=_device()) / (n * sampling)


def _k2(n, sampling):
    a = _axis(n, sampling)
    return a[:, None] ** 2 + a[None, :] ** 2


def _np(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _shift(t):
    return torch.fft.ifftshift(t, dim=(-2, -1))


def _rows(case, rng):
    """Coefficient rows (x, y, occupancy, a1 b1 .. a5 b5[, B]) of every slice and their counts."""
    field = case["grid"] * case["sampling"]
    cells = case["cells"] or max(1, int(field // CELL))
    origin = (field - cells * CELL) / 2 + rng.uniform(-0.5, 0.5, size=2)
    lobato = case["param"] == "l"
    form = {}
    for z in RMS:
        p = specimen.element_params(z, case["param"])
        form[z] = np.concatenate([[1.0], np.stack([p[:5], p[5:]], axis=1).reshape(-1), [0.0] if lobato else []])
    i, j = (v.reshape(-1) for v in np.meshgrid(np.arange(cells), np.arange(cells), indexing="ij"))
    rows, counts = [], []
    for k in range(case["slices"]):
        count = 0
        for z, fx, fy in PLANES[k % 2]:
            xy = np.stack([(i + fx) * CELL + origin[0], (j + fy) * CELL + origin[1]], axis=1)
            if case["thermal"]:
                xy += rng.standard_normal(xy.shape) * RMS[z]
            rows.append(np.concatenate([xy, np.broadcast_to(form[z], (len(xy), len(form[z])))], axis=1))
            count += len(xy)
        counts.append(float(count))
    return np.ascontiguousarray(np.concatenate(rows)), np.array(counts)


def _probes(n, sampling, count):
    """``count`` unit probes of 25 mrad, C3 -5 um, defoci 2 nm apart about zero, and their weights."""
    k2 = _k2(n, sampling)
    defoci = (np.arange(count) - (count - 1) / 2) * 20.0
    w = np.exp(-0.5 * (defoci / 40.0) ** 2)
    out = []
    for d in defoci:
        chi = math.pi * WAVELENGTH * k2 * (d + 0.5 * -5e4 * WAVELENGTH ** 2 * k2)
        spec = torch.polar((k2 <= (25e-3 / WAVELENGTH) ** 2).double(), -chi)
        psi = torch.fft.ifft2(_shift(spec))
        out.append(torch.fft.fftshift(psi) / torch.linalg.vector_norm(psi))
    return _np(torch.stack(out)), w / w.sum()


def _masks(n, sampling, count):
    """0/1 annuli, centred; coarse sampling brings the ADF ring inside the propagator's cut."""
    k2, cut = _k2(n, sampling), 1e3 * WAVELENGTH / (3 * sampling)
    rings = [(min(lo, 0.5 * cut), hi) for lo, hi in DETECTORS[:count]]
    return torch.stack([((k2 >= (lo * 1e-3 / WAVELENGTH) ** 2) & (k2 <= (hi * 1e-3 / WAVELENGTH) ** 2)).double()
                        for lo, hi in rings])


def _propagator(n, sampling, cut):
    """Fresnel propagator of one slice in FFT order, zero beyond ``cut`` of the Nyquist frequency."""
    k2 = _k2(n, sampling)
    h = torch.polar((k2 <= (cut / (2 * sampling)) ** 2).double(), -math.pi * WAVELENGTH * SLICE * k2)
    return _np(_shift(h))


def _request(case, seed):
    rng = np.random.default_rng(seed)
    p, s = case["grid"], case["sampling"]
    a = _np(_axis(p, s))
    kx, ky = np.ascontiguousarray(np.broadcast_to(a, (p, p))), np.ascontiguousarray(np.broadcast_to(a[:, None], (p, p)))
    rows, counts = _rows(case, rng)
    hbar = _H / (2 * math.pi)
    common = dict(param=case["param"], ele_n=rows, series_n=counts, ele_n_i=np.zeros((0, 26 if case["param"] == "l" else 25)),
                  series_n_i=np.zeros(len(counts)), kx=kx, ky=ky, s2=_np(_k2(p, s) / 4), p_height=p, p_width=p,
                  sigma=SIGMA, parameter=2 * math.pi * hbar * hbar / (_E * _M * 1e-20) / (p * p * s * s),
                  aper_true=np.ones((p, p)))
    if "window" not in case:
        return StemRequest(probe=np.zeros((1, 2, 2), dtype=np.complex128), aper=np.zeros((0, 2, 2)),
                           aper2=np.zeros((0, 2, 2)), prop=np.zeros((2, 2), dtype=np.complex128), gfsf=np.ones(1),
                           step=0, beginrow=0, begincol=0, width_red=0, hight_red=0, **common)
    n = case["window"]
    probe, weights = _probes(n, s, case["probes"])
    aper = _masks(n, s, case["detectors"])
    mids = [case["slices"] * (i + 1) // (case["mids"] + 1) for i in range(case["mids"])]
    begin = [(p - (n + (m - 1) * case["step"])) // 2 for m in (case["rows"], case["cols"])]
    return StemRequest(probe=probe, aper=_np(aper), aper2=_np(_shift(aper)), prop=_propagator(n, s, 2 / 3),
                       gfsf=weights, step=case["step"], beginrow=begin[0], begincol=begin[1], width_red=case["cols"],
                       hight_red=case["rows"], mid_layer=np.array(mids, dtype=np.int32), **common)


def _hrtem_spec(case):
    """Half-Nyquist propagator and the transfer functions of a focal series about -50 nm (Cs 1.2 mm, 20 mrad)."""
    n, s, k = case["grid"], case["sampling"], case["probes"]
    k2 = _k2(n, s)
    inside = (k2 <= (20e-3 / WAVELENGTH) ** 2).double()
    defoci = -500.0 + (np.arange(k) - (k - 1) / 2) * 20.0
    w = np.exp(-0.5 * ((defoci + 500.0) / 40.0) ** 2)
    tf = [_shift(torch.polar(inside, -math.pi * WAVELENGTH * k2 * (d + 0.5 * 1.2e7 * WAVELENGTH ** 2 * k2)))
          for d in defoci]
    return HrtemSpec(prop=_propagator(n, s, 1 / 2), tf=_np(torch.stack(tf)), weights=w / w.sum())


def _server_cases(case):
    """The requests of a server case: both windows in turn, scans and thicknesses that differ."""
    out = []
    for i in range(case["requests"]):
        n = case["window2"] if i % 3 == 2 else case["window"]
        side = max(1, int(math.sqrt(case["probes"] * (0.4 + 0.3 * (i % 4)))))
        rows, cols = side, max(1, side + i % 3 - 1)
        need = n + (max(rows, cols) - 1) * 8
        out.append(_stem("", n, 1 << (need - 1).bit_length(), rows, cols, case["slices"] + 5 * (i % 3),
                         param="pl"[i % 2], mids=1 if i % 3 == 1 else 0, thermal=case["thermal"]))
    return out


class _Stack:
    """A session's transmission stack seen through the CUDA array interface; a tensor made from it
    keeps the session, and so the memory, alive."""

    def __init__(self, session, stream, req):
        self.keep = session, stream
        self.__cuda_array_interface__ = {"shape": (req.slices, req.p_height, req.p_width), "typestr": "<c8",
                                         "data": (session.transmission_ptr(), False), "version": 3, "strides": None}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "server":
        reqs = [_request(c, seed * 101 + i) for i, c in enumerate(_server_cases(case))]
        return {"kind": kind, "reqs": reqs, "server": capi.Server(device=0, hbm_budget=8 << 30)}
    req = _request(case, seed)
    state = {"kind": kind, "req": req}
    if kind == "oneshot":
        return state
    if kind == "transmission":  # the program's own stream, so that its next kernels follow the build
        state["stream"] = torch.cuda.Stream()
        state["session"] = capi.Session(device=0, stream=state["stream"].cuda_stream)
    else:
        state["session"] = capi.Session(device=0)
    state["session"].upload(req, stem=kind in ("stem", "cbed"))
    if kind == "hrtem":
        state["spec"] = _hrtem_spec(case)
    return state


# ----------------------------------------------------------------------------------------------
# One pass
# ----------------------------------------------------------------------------------------------

def _images(req, res, mid):
    a, d = req.aper_num, req.depth
    return {"exit": res.reshape(a, d).astype(np.float32),
            "mid": mid.reshape(len(req.mid_layer), a, d).astype(np.float32)}


def run(state):
    kind = state["kind"]
    if kind == "server":
        srv = state["server"]
        tickets = [srv.submit(r) for r in state["reqs"]]
        return [_images(r, *srv.wait(t)) for r, t in zip(state["reqs"], tickets)]
    req = state["req"]
    if kind == "oneshot":
        return _images(req, *capi.stem_run(req))
    s = state["session"]
    if kind == "stem":
        s.run()
        res, mid, _ = s.download()
        return _images(req, res, mid)
    if kind == "hrtem":
        s.run(what=1)
        wave, image = s.hrtem(state["spec"])
        return {"wave": wave.astype(np.complex64), "image": image.astype(np.float32)}
    if kind == "cbed":
        s.run(what=1)
        return s.cbed().astype(np.float32)
    here = torch.cuda.current_stream()
    state["stream"].wait_stream(here)
    s.run(what=1)
    here.wait_stream(state["stream"])
    return torch.as_tensor(_Stack(s, state["stream"], req), device="cuda")


# ----------------------------------------------------------------------------------------------
# What a pass cannot do without
# ----------------------------------------------------------------------------------------------

def work(case):
    """Inputs read once and outputs written once; transforms at 5 n log2 n operations, the
    structure factors as one transform of the grid per plane of atoms."""
    if case["kind"] == "server":
        each = [work(c) for c in _server_cases(case)]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    p2, slices = case["grid"] ** 2, case["slices"]
    cells = case["cells"] or max(1, int(case["grid"] * case["sampling"] // CELL))
    flops = slices * p2 * (2 * 5 * math.log2(p2) + 40)
    moved = 4.0 * p2 + 2.5 * slices * cells * cells * 16
    if case["kind"] == "transmission":
        return {"bytes": moved + 8.0 * slices * p2, "flops": flops}
    if case["kind"] == "hrtem":
        k = case["probes"]
        flops += slices * p2 * (2 * 5 * math.log2(p2) + 14) + (k + 1) * p2 * (5 * math.log2(p2) + 10)
        return {"bytes": moved + p2 * (8.0 + 8.0 * k + 8.0 + 4.0), "flops": flops}
    n2, items = case["window"] ** 2, case["rows"] * case["cols"] * case["probes"]
    flops += items * slices * n2 * (2 * 5 * math.log2(n2) + 14)
    out = n2 * 4.0 if case["kind"] == "cbed" else 4.0 * case["detectors"] * case["rows"] * case["cols"] * (1 + case["mids"])
    return {"bytes": moved + n2 * (8.0 * case["probes"] + 8.0 + 4.0 * case["detectors"]) + out, "flops": flops}


# ----------------------------------------------------------------------------------------------
# The same outputs in 64 bits
# ----------------------------------------------------------------------------------------------

def _t(a):
    return torch.as_tensor(a, device=_device())


def _transmission64(req):
    """One slice of exp(i sigma V / 1000) after the other, V summed over the atoms of each element."""
    kx, ky, s2 = _t(req.kx[0]), _t(np.ascontiguousarray(req.ky[:, 0])), _t(req.s2)
    ends = np.cumsum(req.series_n).astype(int)
    for end, count in zip(ends, req.series_n.astype(int)):
        rows = req.ele_n[end - count:end]
        v = torch.zeros(s2.shape, dtype=torch.complex128, device=s2.device)
        for coef in np.unique(rows[:, 2:], axis=0):
            xy = _t(rows[(rows[:, 2:] == coef).all(axis=1), :2])
            f = torch.zeros_like(s2)
            for a, b in coef[1:11].reshape(5, 2):
                f += a * torch.exp(-b * s2) if req.param == "p" else a * (2 + 4 * b * s2) / (1 + 4 * b * s2) ** 2
            ex = torch.polar(torch.ones((), dtype=torch.float64, device=s2.device), -2 * math.pi * xy[:, :1] * kx[None])
            ey = torch.polar(torch.ones((), dtype=torch.float64, device=s2.device), -2 * math.pi * xy[:, 1:] * ky[None])
            v += coef[0] * f * (ey.T @ ex)
        v = torch.fft.ifft2(_shift(v * req.parameter)) * v.numel()
        yield torch.exp(1j * (req.sigma / 1000.0) * v)


def _images64(req):
    n = req.height
    prop, masks = _t(req.prop), _t(np.fft.ifftshift(req.aper, axes=(-2, -1)))
    depth, probes = req.depth, req.w_num
    stack = list(_transmission64(req))
    res = torch.zeros(req.aper_num, depth, dtype=torch.float64, device=prop.device)
    mid = torch.zeros(len(req.mid_layer), req.aper_num, depth, dtype=torch.float64, device=prop.device)
    batch = max(1, (1 << 26) // (n * n))
    for w in range(probes):
        probe = _t(req.probe[w])
        for first in range(0, depth, batch):
            at = range(first, min(depth, first + batch))
            corner = [(req.beginrow + q // req.width_red * req.step, req.begincol + q % req.width_red * req.step)
                      for q in at]
            psi = probe.expand(len(at), n, n)
            for k, t in enumerate(stack):
                spec = torch.fft.fft2(psi * torch.stack([t[r:r + n, c:c + n] for r, c in corner])) * prop
                for layer in np.flatnonzero(req.mid_layer == k + 1)[:1]:
                    mid[layer, :, at[0]:at[-1] + 1] += req.gfsf[w] * torch.einsum("pij,aij->ap", spec.abs() ** 2, masks)
                psi = torch.fft.ifft2(spec)
            res[:, at[0]:at[-1] + 1] += req.gfsf[w] * torch.einsum("pij,aij->ap", spec.abs() ** 2, masks)
    return {"exit": res.cpu().numpy(), "mid": mid.cpu().numpy()}


def exact(case, seed):
    kind = case["kind"]
    if kind == "server":
        return [_images64(_request(c, seed * 101 + i)) for i, c in enumerate(_server_cases(case))]
    req = _request(case, seed)
    if kind in ("stem", "oneshot"):
        return _images64(req)
    if kind == "transmission":
        return torch.stack(list(_transmission64(req)))
    if kind == "hrtem":
        spec = _hrtem_spec(case)
        prop = _t(spec.prop)
        psi = torch.ones(req.s2.shape, dtype=torch.complex128, device=prop.device)
        for t in _transmission64(req):
            psi = torch.fft.ifft2(torch.fft.fft2(psi * t) * prop)
        image = torch.zeros(psi.shape, dtype=torch.float64, device=psi.device)
        for w, tf in zip(spec.weights, spec.tf):
            image += float(w) * torch.fft.ifft2(torch.fft.fft2(psi) * _t(tf)).abs() ** 2
        return {"wave": psi.cpu().numpy(), "image": image.cpu().numpy()}
    n, (r, c) = req.height, (req.beginrow, req.begincol)
    prop = _t(req.prop)
    psi = _t(req.probe)
    for t in _transmission64(req):
        spec = torch.fft.fft2(psi * t[r:r + n, c:c + n]) * prop
        psi = torch.fft.ifft2(spec)
    pattern = (_t(req.gfsf)[:, None, None] * spec.abs() ** 2).sum(dim=0)
    return torch.fft.fftshift(pattern).cpu().numpy()
