"""Slice loops whose batches run in two chains on two streams (the default from 1.5 M wave points on):
the same numbers as one chain of a caller's batch, whatever the count of probes, with mid-slice
detectors, several probes per position, on the session's own stream, a caller's stream, and as a
replayed graph."""
import numpy as np
import pytest

from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


def _images(s, **kw):
    s.run(**kw)
    res, mid, _ = s.download()
    return res, mid, s.timing()


@pytest.mark.parametrize("n,raster,focal_steps", [
    (64, (21, 19), 1),    # 399 probes: two batches of 200 and 199
    (128, (11, 9), 3),    # three probes per position, 297 items
    (256, (5, 7), 1),
    (256, (1, 25), 1),
    (400, (3, 11), 1),
    (512, (1, 41), 1),    # several batches per chain, an odd number of items
    (640, (1, 9), 1),
])
@pytest.mark.parametrize("own_stream", [True, False])
def test_two_chains_equal_one(engine_lib, n, raster, focal_steps, own_stream):
    req = request.build_small_stem(n=n, p=1024 if n < 512 else 1280, raster=raster, step=7, slices=4, mid_layer=(1, 3),
                                   sampling=0.1, cells=2, focal_steps=focal_steps)
    stream = None
    if not own_stream:
        import torch
        stream = torch.cuda.Stream()
    s = capi.Session(device=0, stream=None if own_stream else stream.cuda_stream)
    s.upload(req)
    items = req.w_num * req.depth
    one = _images(s, batch=items)
    assert one[2].batch == items
    for _ in range(3):  # direct, captured, replayed
        two = _images(s)
        assert two[2].batch <= (items + 1) // 2
        assert np.array_equal(one[0], two[0]) and np.array_equal(one[1], two[1])
    three = _images(s, batch=3)
    assert np.array_equal(one[0], three[0]) and np.array_equal(one[1], three[1])
    s.close()


def test_two_sessions_at_once(engine_lib):
    # the second stream and the partial sums belong to the session
    reqs = [request.build_small_stem(n=256, p=512, raster=(6, 6), step=5, slices=4, sampling=0.1, seed=i) for i in (0, 1)]
    alone = []
    for r in reqs:
        s = capi.Session(device=0)
        s.upload(r)
        alone.append(_images(s, batch=36)[0])
        s.close()
    ss = [capi.Session(device=0) for _ in reqs]
    for s, r in zip(ss, reqs):
        s.upload(r)
    for _ in range(3):
        for s in ss:
            s.run()
        for s, a in zip(ss, alone):
            assert np.array_equal(s.download()[0], a)
    for s in ss:
        s.close()
