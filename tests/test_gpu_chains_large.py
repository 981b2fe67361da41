"""Two chains at the large windows (batches of one to three waves up to 1600^2, of about eight at 2048^2), and the 1536^2
runs that stream in one batch instead: the same numbers as one batch of the caller's."""
import numpy as np
import pytest

from totem_b200 import capi, request

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,count,batch", [(1152, 5, 3), (1536, 3, 1), (1536, 20, 20), (1600, 3, 1), (2048, 3, 2),
                                           (2048, 17, 9)])
def test_large_windows_in_chains_equal_one_batch(engine_lib, n, count, batch):
    req = request.build_small_stem(n=n, p=n if n == 2048 else n + 64, raster=(1, count), step=0 if n == 2048 else 2,
                                   slices=3, mid_layer=(2,), sampling=0.05, cells=1, begin=(0, 0))
    s = capi.Session(device=0)
    s.upload(req)
    s.run(batch=count)
    one = s.download()[:2]
    for _ in range(3):  # direct, captured, replayed
        s.run()
        got = s.download()[:2]
        assert s.timing().batch == batch
        assert np.array_equal(one[0], got[0]) and np.array_equal(one[1], got[1])
    s.close()
