"""Packing host pools into one copy gives the tensors that a copy each gives."""
import numpy as np
import pytest
import torch

from jaxrenderer_gb300 import jobs


@pytest.mark.parametrize("rows", [0, 1, 63, 64, 65])
@pytest.mark.parametrize("parts", [1, 3])
def test_one_copy_equals_a_copy_each(rows, parts, monkeypatch):
    rng = np.random.default_rng([rows, parts])

    def pools():
        p = {"a": jobs._Pool(torch.float32, 3), "b": jobs._Pool(torch.int32, 1), "c": jobs._Pool(torch.float32, 2),
             "d": jobs._Pool(torch.float32, 1)}
        for k in range(parts):
            p["a"].add(rng.normal(size=(rows + k, 3)))  # float64, and not contiguous
            p["b"].add(rng.integers(-5, 5, (rows + k, 2)).astype(np.int64)[:, 0])
            p["c"].add(torch.from_numpy(rng.normal(size=(rows + k, 2)).astype(np.float32)))  # a tensor: never packed
        return p

    state = rng.bit_generator.state
    got, jobs_got = jobs._upload(pools(), b"0123456789", torch.device("cpu"))
    rng.bit_generator.state = state
    monkeypatch.setattr(jobs, "ONE_COPY_BYTES", 0)
    want, jobs_want = jobs._upload(pools(), b"0123456789", torch.device("cpu"))
    assert got.keys() == want.keys() == {"a", "b", "c"}
    for k in got:
        assert got[k].dtype == want[k].dtype and torch.equal(got[k], want[k])
    assert bytes(jobs_got.numpy()) == bytes(jobs_want.numpy()) == b"0123456789"
