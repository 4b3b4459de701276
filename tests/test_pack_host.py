"""Packing host arrays: initial buffers are copies, and values convert as
torch converts them."""
import warnings

import numpy as np
import pytest
import torch

from jaxrenderer_gb300 import jobs


def test_buffers_packed_on_the_cpu_do_not_share_the_callers_memory():
    spec = jobs.JobSpec(shader=0, width=4, height=3, viewport=np.eye(4, dtype=np.float32), world_to_clip=np.eye(4, dtype=np.float32),
                        world_to_eye_norm=np.eye(4, dtype=np.float32), position=np.zeros((3, 3), np.float32),
                        faces=np.arange(3, dtype=np.int32).reshape(1, 3))
    z, c = np.ones((4, 3), np.float32), np.zeros((4, 3, 3), np.float32)
    p = jobs.pack([spec], [z], [c], torch.device("cpu"))
    p.zbuffer.fill_(7.0)
    p.canvas.fill_(7.0)
    assert (z == 1).all() and (c == 0).all()


@pytest.mark.parametrize("array", [np.array([1e300, -2.5]), np.array([True, False]), np.arange(3, dtype=np.uint8), np.arange(6.0)[::-2],
                                   np.array([1, None], object), np.array([1, 2], np.longdouble), np.array(["1", "2"])])
@pytest.mark.parametrize("dtype", [torch.float32, torch.int32])
def test_small_pools_convert_as_a_copy_each_does(array, dtype, monkeypatch):
    if dtype == torch.int32 and array.dtype.kind == "f" and abs(array).max() > 2 ** 31:
        pytest.skip("undefined conversion")

    def upload():
        pool = jobs._Pool(dtype, 1)
        pool.add(array)
        with warnings.catch_warnings():
            warnings.simplefilter("error")
            try:
                return jobs._upload({"a": pool}, b"0", torch.device("cpu"))[0]["a"].clone()
            except (TypeError, RuntimeError) as e:
                return type(e)

    got = upload()
    monkeypatch.setattr(jobs, "ONE_COPY_BYTES", 0)
    want = upload()
    assert torch.equal(got, want) if isinstance(want, torch.Tensor) else got == want
