"""Short slice loops whose passes are launched before the one ahead has ended (windows up to 128^2 in
one batch), and the CBED and HRTEM loops replayed as graphs: the same numbers as launched one after
the other, in every repetition."""
import numpy as np
import pytest

from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,raster,focal_steps", [(64, (1, 1), 1), (64, (3, 4), 3), (96, (2, 3), 1), (128, (5, 5), 1)])
def test_overlapped_passes_equal_separate_ones(engine_lib, n, raster, focal_steps):
    req = request.build_small_stem(n=n, p=256, raster=raster, slices=9, mid_layer=(3, 9), focal_steps=focal_steps,
                                   sampling=0.15)
    s = capi.Session(device=0)
    s.upload(req)
    s.run(profile=True)  # an event around every launch: no overlap
    ref = s.download()
    for _ in range(20):
        s.run()
        res, mid, _ = s.download()
        assert np.array_equal(res, ref[0]) and np.array_equal(mid, ref[1])
    s.close()


@pytest.mark.parametrize("n", [64, 128, 256, 400])
def test_cbed_and_hrtem_replayed(engine_lib, n):
    req = request.build_small_stem(n=n, p=n, raster=(1, 1), slices=5, mid_layer=(), focal_steps=3, sampling=0.15,
                                   begin=(0, 0))
    specs = [request.hrtem_spec(n, 0.15, 200.0, 1.9525, -50.0, 1.2, 20.0, 4.0, 3),
             request.hrtem_spec(n, 0.15, 200.0, 3.905, -20.0, 1.2, 20.0, 4.0, 3)]
    capi.set_slice_graphs(False)
    try:
        s = capi.Session(device=0)
        s.upload(req)
        want_cbed = s.cbed()
        want = [s.hrtem(sp) for sp in specs]
        s.close()
    finally:
        capi.set_slice_graphs(True)
    s = capi.Session(device=0)
    s.upload(req)
    for _ in range(4):
        assert np.array_equal(s.cbed(), want_cbed)
    for sp, w in list(zip(specs, want)) * 3:  # same launches, another propagator in the same buffer
        wave, image = s.hrtem(sp)
        assert np.array_equal(wave, w[0]) and np.array_equal(image, w[1])
    s.run()  # and beside the detectors' own loop
    first = s.download()[0]
    assert np.array_equal(s.cbed(), want_cbed)
    s.run()
    assert np.array_equal(s.download()[0], first)
    s.close()
