"""The zero rows of a propagator in the column pass (left out of the transforms when every entry
beyond a third of the window is zero): the same numbers with the skip on and off, for propagators that
are zero on rows only, on columns only, on both, and with a single entry on either side of the
limit.  The sums left out are sums of zeros, so the results are equal, not just close."""
from dataclasses import replace

import numpy as np
import pytest

from tests.conftest import rel_l2
from oracle import stem_oracle as so
from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


def _run(req, skip):
    capi.set_band_skip(skip)
    try:
        s = capi.Session(device=0)
        s.upload(req)
        s.run()
        res, mid, _ = s.download()
        s.close()
    finally:
        capi.set_band_skip(True)
    return res, mid


def _propagator(n, kind, rng):
    h = np.exp(1j * rng.uniform(-3, 3, (n, n)))
    dist = np.minimum(np.arange(n), n - np.arange(n))
    zero = dist > n // 3
    if kind in ("rows", "both", "edge_inside", "edge_outside"):
        h[zero, :] = 0
    if kind in ("columns", "both"):
        h[:, zero] = 0
    if kind == "edge_outside":  # one entry on the first row beyond the limit: no row may be skipped
        h[n // 3 + 1, 5] = 0.5
    if kind == "edge_inside":
        h[:] = 0
        h[n // 3, 5] = h[n - n // 3, 7] = 1.0
    return h


@pytest.mark.parametrize("kind", ["rows", "columns", "both", "edge_inside", "edge_outside"])
@pytest.mark.parametrize("n", [64, 96, 256, 400, 512, 640, 1152])
def test_zero_rows_change_nothing(engine_lib, n, kind):
    req = request.build_small_stem(n=n, p=2 * n if n < 1000 else 1280, raster=(1, 2), slices=3, mid_layer=(2,), sampling=0.1, cells=2)
    req = replace(req, prop=_propagator(n, kind, np.random.default_rng(n)))
    on, off = _run(req, True), _run(req, False)
    for a, b in zip(on, off):
        assert np.array_equal(a, b) and np.isfinite(a).all()
    if n <= 96:
        ref = so.stem(req, so.transmission(req))
        assert rel_l2(on[0], ref[0]) < 1e-4 and rel_l2(on[1], ref[1]) < 1e-4


@pytest.mark.parametrize("n", [1024, 2048])
def test_zero_rows_change_nothing_wide(engine_lib, n):
    req = request.build_srtio3_stem(cells=(2, 2, 2), n=n, raster=(1, 2), p=n + 64, engine_optics=True)
    assert np.array_equal(_run(req, True)[0], _run(req, False)[0])
