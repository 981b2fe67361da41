"""Precision of the gridding builder's sums where very many atoms meet on a row of the fine grid, against 64
bits: the sums themselves must not round (they are FP64), whatever their length."""
from dataclasses import replace

import numpy as np
import pytest

from tests.test_gpu_gridding_edges import _request
from tests.test_gpu_gridding_memory import _run, _sparse
from totem_b200 import capi

pytestmark = pytest.mark.gpu


def _potential_phase(req, rows):
    """sigma V / 1000 in FP64 from the rows of one species."""
    ex = np.exp(-2j * np.pi * np.outer(rows[:, 0], req.kx[0]))
    ey = np.exp(-2j * np.pi * np.outer(rows[:, 1], req.ky[:, 0]))
    c = rows[0, 2:]
    f = c[0] * sum(c[1 + 2 * i] * np.exp(-c[2 + 2 * i] * req.s2) for i in range(5))
    v = req.parameter * req.aper_true * f * (ey.T @ ex)
    return req.sigma / 1000.0 * (np.fft.ifft2(np.fft.ifftshift(v)) * v.size).real


def test_sums_of_many_atoms_do_not_round(engine_lib):
    # 25 000 terms on each of the 128 fine rows.  FP32 sums of n random terms are off by 2^-25 sqrt(n / 2)
    # of themselves, 3.3e-6 here; what stays is the form factors and transforms in FP32, 8e-7 on any
    # specimen: the bound is twice that.
    atoms, p = 400_000, 64
    req = _request(p, p, atoms, slices=1)
    req = replace(req, ele_n=req.ele_n[:atoms], series_n=np.array([float(atoms)]))
    aper = np.ones((p, p))
    aper[p // 2, p // 2] = 0.0  # without the mean, which would hide the errors of the rest
    aper[0, :] = aper[:, 0] = 0.0  # and the Nyquist lines, whose conjugate is not on the grid
    req = replace(_sparse(req, 2e-3), aper_true=aper)
    phase = _potential_phase(req, req.ele_n)
    t, builder = _run(req, capi.TX_GRIDDING, 0)
    assert builder == capi.TX_GRIDDING and 0.05 < np.abs(phase).max() < 2.0, np.abs(phase).max()
    want = np.exp(1j * phase)
    assert np.linalg.norm(t[0] - want) < 1.6e-6 * np.linalg.norm(want - 1.0), \
        np.linalg.norm(t[0] - want) / np.linalg.norm(want - 1.0)
