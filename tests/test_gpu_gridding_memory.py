"""Work memory of the gridding transmission builder for slices of many atoms: bounded by the grid and a few
tables per atom, the phases held in pieces of columns and of atoms, with the same numbers bit by bit."""
from dataclasses import replace

import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_gpu_gridding_edges import _both, _request
from totem_b200 import capi

pytestmark = pytest.mark.gpu
TOL = 5e-6  # the gridding edge tests' bound against the direct sums: the FP32 rounding both share


def _sparse(req, occupancy):
    """The same rows at a small occupancy, so that many atoms make no more potential than a few."""
    rows = req.ele_n.copy()
    rows[:, 2] *= occupancy
    return replace(req, ele_n=rows)


@pytest.mark.parametrize("p_h,p_w,atoms,kw", [
    (64, 64, 1500, {}),
    (64, 30, 700, {"centred": False}),                       # a pitch below 128 columns
    (64, 512, 3000, {}),                                     # phases in pieces of columns
    (96, 96, 5000, {"equal_y": True, "flag": "l"}),          # groups of eight atoms
    (64, 64, 50_000, {}),                                    # three pieces of groups
    (64, 512, 20_000, {"centred": False}),                   # four pieces of columns by three of groups
    (96, 96, 40_000, {"equal_y": True, "flag": "l"}),        # 5000 groups: the last pieces hold none
    (62, 200, 2000, {"centred": False}),
])
def test_phases_in_pieces_change_no_bit(engine_lib, p_h, p_w, atoms, kw):
    req = _sparse(_request(p_h, p_w, atoms, **kw), 50.0 / atoms)
    direct, whole = _both(req, 0)
    _, pieces = _both(req, 1)
    assert rel_l2(whole, direct) < TOL and rel_l2(whole - 1.0, direct - 1.0) < 20 * TOL
    assert rel_l2(pieces, whole) < 1e-6  # a slice's two species through memory
    one = replace(req, ele_n=np.concatenate([req.ele_n[2 * atoms * k:][:atoms] for k in range(req.slices)]),
                  series_n=np.full(req.slices, float(atoms)))
    assert np.array_equal(_both(one, 1)[1], _both(one, 0)[1])


def test_memory_does_not_grow_with_a_kilobyte_per_atom(engine_lib):
    import torch
    atoms = 200_000
    req = _sparse(_request(64, 64, atoms, slices=1), 1e-4)
    torch.cuda.synchronize()
    with capi.tx_builder(capi.TX_GRIDDING, 1 << 20):
        s = capi.Session(device=0)
        s.upload(req, stem=False)
        free = torch.cuda.mem_get_info()[0]
        s.run(what=1)
        s.download()
        taken = free - torch.cuda.mem_get_info()[0]
        s.close()
    # tables of the atoms of two species, arrays of the grid, the transmission itself, and 64 MB for the
    # phases and what the driver keeps (a kilobyte an atom were 205 MB)
    assert taken < 2 * atoms * 48 + 64 * 64 * 72 + (64 << 20), taken


def _run(req, mode, scratch, fail=None):
    with capi.tx_builder(mode, scratch):
        s = capi.Session(device=0)
        s.upload(req, stem=False)
        try:
            if fail is not None:
                capi.inject_failures(alloc_after=fail)
            s.run(what=1)
        finally:
            capi.inject_failures()
        out = s.download(want_transmission=True)[2], s.timing().tx_builder
        s.close()
    return out


# the build's first allocation is the transmission stack, its second the work memory
def test_no_room_for_all_slices_takes_them_one_by_one(engine_lib):
    req = _sparse(_request(64, 512, 3000, slices=3), 50.0 / 3000)
    want, builder = _run(req, capi.TX_AUTO, 0)
    assert builder == capi.TX_GRIDDING
    for mode in (capi.TX_AUTO, capi.TX_GRIDDING):
        got, builder = _run(req, mode, 0, fail=1)
        assert builder == capi.TX_GRIDDING and np.array_equal(got, want)


def test_no_room_at_all_takes_the_direct_sums_unless_gridding_was_asked_for(engine_lib):
    req = _sparse(_request(64, 512, 3000, slices=3), 50.0 / 3000)
    direct, _ = _run(req, capi.TX_DIRECT, 0)
    got, builder = _run(req, capi.TX_AUTO, 1, fail=1)  # already the least the build can do with
    assert builder == capi.TX_DIRECT and np.array_equal(got, direct)
    with pytest.raises(capi.TotemError) as e:
        _run(req, capi.TX_GRIDDING, 1, fail=1)
    assert e.value.code == capi.ERR_OOM
