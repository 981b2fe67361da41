"""The gridding transmission builder where its pieces meet: atoms on both ends of the y axis (their
spreading wraps around) and outside the field, atoms of equal y (one group), axes that are not centred
(no conjugate half), mixed-radix heights, jobs whose phases are taken in pieces of columns, and work
memory for a single job.  Compared with the direct sums: relative L2 <= 5e-6 on the transmission
stack, the FP32 rounding both share (the gridding error itself is ~1e-7 of the structure factor).
"""
from dataclasses import replace

import numpy as np
import pytest

from tests.conftest import rel_l2
from totem_b200 import capi, optics, request, specimen

pytestmark = pytest.mark.gpu
TOL = 5e-6
SAMPLING = 0.2


def _request(p_h, p_w, atoms, flag="p", equal_y=False, centred=True, slices=2, seed=0):
    rng = np.random.default_rng(seed)
    st = specimen.Structure(np.zeros((0, 8)), (1.0, 1.0, float(slices)), 1.0, slices)
    req = request.specimen_request(st, flag, 200.0, SAMPLING, 64)
    kx, ky, s2 = optics.reciprocal_grids(p_h, p_w, SAMPLING)
    if not centred:  # uniform axes beside zero: every column is formed
        kx, ky = kx + 0.25 * (kx[0, 1] - kx[0, 0]), ky + 0.5 * (ky[1, 0] - ky[0, 0])
    rows = []
    for _ in range(slices):
        for z in (14, 38):
            x = rng.uniform(-1.0, p_w * SAMPLING + 1.0, atoms)  # some outside the (periodic) field
            y = rng.uniform(-1.0, p_h * SAMPLING + 1.0, atoms)
            edge = [0.0, 1e-12, -1e-12, p_h * SAMPLING, p_h * SAMPLING - 1e-12, SAMPLING / 4, -SAMPLING / 4]
            y[:min(atoms, 7)] = edge[:atoms]
            if equal_y:
                y[:] = np.repeat(y[:(atoms + 7) // 8], 8)[:atoms]
            p = specimen.element_params(z, flag)
            cf = np.concatenate([[1.0], np.stack([p[:5], p[5:]], 1).reshape(-1), [0.3] if flag == "l" else []])
            rows.append(np.column_stack([x, y, np.tile(cf, (atoms, 1))]))
    return replace(req, ele_n=np.concatenate(rows), series_n=np.full(slices, 2.0 * atoms), series_n_i=np.zeros(slices),
                   kx=kx, ky=ky, s2=s2, p_height=p_h, p_width=p_w, aper_true=np.ones((p_h, p_w)),
                   parameter=optics.potential_parameter(p_h, p_w, SAMPLING))


def _both(req, scratch):
    out = []
    for mode in (capi.TX_DIRECT, capi.TX_GRIDDING):
        with capi.tx_builder(mode, scratch):
            s = capi.Session(device=0)
            s.upload(req, stem=False)
            s.run(what=1)
            assert s.timing().tx_builder == mode
            out.append(s.download(want_transmission=True)[2])
            s.close()
    return out


@pytest.mark.parametrize("p_h,p_w,atoms,kw,scratch", [
    (64, 64, 1, {}, 0),                             # one atom, on the wrap
    (64, 64, 7, {"flag": "l"}, 1),                  # every edge position; one job per batch
    (96, 128, 40, {"centred": False}, 0),           # every column formed, mixed-radix height
    (160, 96, 33, {"equal_y": True, "flag": "l"}, 0),
    (64, 512, 600, {}, 1),                          # phases in pieces of 128 of 272 columns
    (64, 512, 300, {"centred": False}, 0),
    (400, 70, 64, {}, 0),                           # width without a fused transform: cuFFT follows
    (1024, 64, 64, {"equal_y": True}, 0),
    (2048, 64, 300, {"flag": "l"}, 0),
    (4096, 64, 40, {"centred": False, "slices": 1}, 1),
    (1600, 64, 40, {}, 0),
    # heights that are no transform length: the next longer one spreads and transforms
    (62, 64, 9, {}, 0),
    (66, 80, 40, {"flag": "l"}, 0),
    (94, 96, 33, {"centred": False}, 1),
    (98, 64, 60, {"equal_y": True}, 0),
    (700, 70, 64, {}, 0),
    (1026, 64, 33, {"centred": False}, 0),
    (4094, 64, 20, {"slices": 1}, 0),
])
def test_gridding_equals_direct_sums(engine_lib, p_h, p_w, atoms, kw, scratch):
    direct, grid = _both(_request(p_h, p_w, atoms, **kw), scratch)
    assert not np.array_equal(direct, grid)
    assert rel_l2(grid, direct) < TOL, rel_l2(grid, direct)
    # the potential's own error: T - 1 is small in thin slices
    assert rel_l2(grid - 1.0, direct - 1.0) < 20 * TOL


def test_gridding_repeats_bit_by_bit_with_other_batches_between(engine_lib):
    req = _request(128, 128, 60)
    first, again = _both(req, 0)[1], None
    _both(_request(96, 256, 200, seed=1), 1)
    again = _both(req, 0)[1]
    assert np.array_equal(first, again)
    # one job per batch adds the species in the same order, through memory instead of registers
    assert rel_l2(_both(req, 1)[1], first) < 1e-6
