"""The gridding transmission builder over several batches (a small work memory): on grids whose batches hold
rows that are no whole tiles of the inverse row transform, on grids that go on to cuFFT, and with the
jobs of a slice in different batches."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import stem_oracle as so
from tests.conftest import rel_l2
from tests.test_gpu_gridding_edges import _request
from totem_b200 import capi, request

pytestmark = pytest.mark.gpu
TOL = 5e-6  # the gridding edge tests' bound against the direct sums: the FP32 rounding both share


def _build(req, mode, scratch):
    with capi.tx_builder(mode, scratch):
        s = capi.Session(device=0)
        s.upload(req, stem=False)
        s.run(what=1)
        assert s.timing().tx_builder == mode
        t = s.download(want_transmission=True)[2]
        s.close()
    return t


def _one_species(req, atoms):
    """The first of the two species of every slice only."""
    keep = np.concatenate([np.arange(atoms) + 2 * atoms * k for k in range(req.slices)])
    return replace(req, ele_n=req.ele_n[keep], series_n=np.full(req.slices, float(atoms)))


# one job a slice and work memory for one job: a slice per batch.  Row tiles: 20 rows at width 160, 32 at
# 64 to 128 (400 = 12 x 32 + 16); the last row fits by batches
@pytest.mark.parametrize("p_h,p_w,slices", [(64, 160, 5), (256, 160, 5), (400, 64, 2), (400, 128, 4), (160, 160, 3)])
def test_batches_whose_rows_are_no_whole_row_tiles(engine_lib, p_h, p_w, slices):
    req = _one_species(_request(p_h, p_w, 40, slices=slices), 40)
    whole = _build(req, capi.TX_GRIDDING, 0)
    assert np.array_equal(_build(req, capi.TX_GRIDDING, 1), whole)  # the same sums and transforms slice by slice
    assert rel_l2(whole, _build(req, capi.TX_DIRECT, 0)) < TOL


def test_server_quarter_rounds_as_the_request_alone(engine_lib):
    # a grid whose transmission goes on to cuFFT (no fused transform of 100): the server's requests build in
    # smaller batches than a session, of whole slices all the same
    req = request.build_small_stem(n=64, p=100, raster=(2, 2), slices=8, mid_layer=(), sampling=0.2)
    for kib in (256, 512, 1024, 1536, 2048, 3072, 4096, 6144):
        with capi.tx_builder(capi.TX_GRIDDING, kib << 10):
            s = capi.Session(device=0)
            s.upload(req)
            s.run()
            alone = s.download()[0]
            assert s.timing().tx_builder == capi.TX_GRIDDING
            s.close()
            with capi.Server(device=0) as srv:
                served = srv.wait(srv.submit(req))[0]
        assert np.array_equal(alone, served), kib


def _stack(req, scratch):
    with capi.tx_builder(capi.TX_GRIDDING, scratch):
        s = capi.Session(device=0)
        s.upload(req, stem=False)
        s.run(what=1)
        out = s.download(want_transmission=True)[2], s.timing().kernel_launches
        s.close()
    return out


def test_slices_split_over_batches(engine_lib):
    # work memory for one job: every species of a slice, ionic rows among them, in its own batch, the later
    # ones adding to what the earlier ones wrote
    req = request.with_ionic_oxygen(request.build_small_stem(flag="p"))
    whole, few = _stack(req, 0)
    split, many = _stack(req, 1)
    assert many >= few + 3 * req.slices, (few, many)  # phases, rows and columns of each job on its own
    assert not np.array_equal(split, whole) and rel_l2(split, whole) < 1e-6
    assert rel_l2(split, so.transmission(req)) < 1e-4  # the engine's accuracy target
