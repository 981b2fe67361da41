"""The cuFFT path where its steps were joined: the probe's copy and the 1 / N^2 inside the multiply by T,
and the exit detectors on the last slice's spectrum.  Non-square and odd-sized windows (in elements
per block), several probes per position, a mid-slice image at the last slice, one slice, and no slice
at all, against the FP64 oracle (relative L2 1e-4, the engine's accuracy target)."""
from dataclasses import replace

import numpy as np
import pytest

from oracle import stem_oracle as so
from tests.conftest import rel_l2
from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


def _cut(req, h, w):
    """The request with an h x w window (probe, detectors and propagator cropped in frequency order)."""
    crop = lambda a, shift: a[..., (a.shape[-2] - h) // 2:(a.shape[-2] + h) // 2,  # noqa: E731
                              (a.shape[-1] - w) // 2:(a.shape[-1] + w) // 2]
    prop = np.fft.ifftshift(crop(np.fft.fftshift(req.prop), None))
    aper = crop(req.aper, None)
    return replace(req, probe=np.ascontiguousarray(crop(req.probe, None)), aper=np.ascontiguousarray(aper),
                   aper2=np.array([np.fft.ifftshift(a) for a in aper]), prop=prop)


@pytest.mark.parametrize("h,w,slices,mid,focal_steps,batch", [
    (34, 50, 4, (2, 4), 1, 0),
    (62, 62, 1, (1,), 3, 0),
    (48, 64, 3, (), 3, 2),
    (2, 6, 2, (1,), 1, 0),
])
def test_plain_path_vs_oracle(engine_lib, h, w, slices, mid, focal_steps, batch):
    req = request.build_small_stem(n=64, p=128, raster=(3, 4), slices=slices, mid_layer=mid, focal_steps=focal_steps)
    req = _cut(req, h, w)
    s = capi.Session(device=0)
    s.upload(req)
    for _ in range(2):
        s.run(path=capi.PATH_PLAIN, batch=batch)
        res, got_mid, _ = s.download()
        ref, ref_mid = so.stem(req, so.transmission(req))
        assert rel_l2(res, ref) < 1e-4
        if len(mid):
            assert rel_l2(got_mid, ref_mid) < 1e-4
    s.close()


def test_no_slices_gives_the_probes_own_spectra(engine_lib):
    req = request.build_small_stem(n=64, p=128, raster=(2, 2), slices=2, mid_layer=())
    none = replace(req, ele_n=req.ele_n[:0], series_n=np.zeros(0), series_n_i=np.zeros(0), ele_n_i=req.ele_n_i[:0])
    assert none.slices == 0
    s = capi.Session(device=0)
    s.upload(none)
    s.run()
    res = s.download()[0].reshape(none.aper_num, none.depth)
    s.close()
    inten = np.abs(np.fft.fft2(req.probe[0])) ** 2
    want = [np.sum(inten * np.fft.ifftshift(a)) * req.gfsf[0] for a in req.aper]
    assert np.allclose(res, np.array(want)[:, None], rtol=1e-5)
