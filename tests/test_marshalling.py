"""Splitting complex arrays into the two FP64 arrays the C API takes, in one piece or by several
threads: the same values for any layout and length."""
import numpy as np
import pytest

from totem_b200 import capi


@pytest.mark.parametrize("shape", [(0, 4), (1,), (3, 5), (7, 11, 13)])
@pytest.mark.parametrize("grain", [1, 10, 1 << 17])
def test_split(monkeypatch, shape, grain):
    monkeypatch.setattr(capi, "_SPLIT_GRAIN", grain)
    rng = np.random.default_rng(0)
    z = rng.standard_normal(shape) + 1j * rng.standard_normal(shape)
    z.reshape(-1)[:1] = complex(np.nan, -np.inf)
    for a in (z, z.T, z[::-1], z.astype(np.complex64), z.real):
        re_, im_ = capi._split(a)
        assert re_.dtype == im_.dtype == np.float64 and re_.shape == im_.shape == a.shape
        assert re_.flags.c_contiguous and im_.flags.c_contiguous
        np.testing.assert_array_equal(re_, np.asarray(a.real, dtype=np.float64))
        np.testing.assert_array_equal(im_, np.asarray(a.imag, dtype=np.float64))
