"""The library's host inverse of 4x4 matrices against the NumPy operations,
bit for bit: pivoting, zero and subnormal pivots, infinities and NaN."""
import numpy as np
import pytest

from jaxrenderer_gb300 import _lib, geometry

F32 = np.float32


@pytest.mark.parametrize("kind", ["plain", "zero", "tiny", "nonfinite", "integer"])
@pytest.mark.parametrize("batch", [(), (1,), (3, 257)])
def test_same_bits(batch, kind, monkeypatch):
    rng = np.random.default_rng(len(kind))
    m = rng.normal(size=batch + (4, 4)).astype(F32)
    if kind == "zero":
        m[..., :, 1] = m[..., :, 0] * 2
        m[..., 2, :] = 0
    elif kind == "tiny":
        m[..., 2, 2] = 1e-42
        m = m * F32(1e-20)
    elif kind == "nonfinite":
        m[..., 3, 0], m[..., 1, 1] = np.nan, np.inf
    elif kind == "integer":
        m = np.round(m)
    _lib.load()
    got = geometry.lu_inverse(m)
    monkeypatch.setattr(_lib, "_LIB", None)
    want = geometry.lu_inverse(m)
    assert got.shape == want.shape and got.dtype == want.dtype == F32
    nan = np.isnan(want)
    assert np.array_equal(nan, np.isnan(got))
    assert np.array_equal(got.view(np.int32)[~nan], want.view(np.int32)[~nan])
