"""The gridding transmission builder over several batches of slices (a small work memory), on grids whose
batches hold rows that are no whole tiles of the inverse row transform."""
from dataclasses import replace

import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_gpu_gridding_edges import _request
from totem_b200 import capi

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
