"""The set-up's small-face path at pixel coordinates past 2^15."""
import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import JobSpec, pack, render_plain, render_tiled

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("width,height", [(32769, 9), (65535, 4), (9, 32769), (4, 65535)])
def test_small_faces_of_a_wide_canvas(width, height):
    import torch

    rng = np.random.default_rng([width, height])
    # faces of a few pixels all over the canvas, a fifth of them in its last eight columns and rows
    n = 4000
    at = rng.uniform(0, 1, (n, 1, 2)) * (width, height)
    at[::5, 0] = np.array((width, height)) - rng.uniform(0, 8, (len(at[::5]), 2))
    tri = np.concatenate([at + rng.uniform(-2, 2, (n, 3, 2)), rng.uniform(-0.9, 0.9, (n, 3, 1))], axis=2)
    vp = np.array([[width / 2, 0, 0, width / 2], [0, height / 2, 0, height / 2], [0, 0, 0.5, 0.5], [0, 0, 0, 1]], F32)
    pos = (tri / (width / 2, height / 2, 1) - (1, 1, 0)).reshape(-1, 3).astype(F32)
    spec = JobSpec(shader=_lib.SHADER_DEPTH, width=width, height=height, viewport=vp, world_to_clip=np.identity(4, dtype=F32),
                   world_to_eye_norm=np.identity(4, dtype=F32), position=pos, faces=np.arange(3 * n, dtype=np.int32).reshape(-1, 3))
    dev = torch.device("cuda")
    plain, tiled = (pack([spec], [np.full((width, height), 9.0, F32)], [None], dev) for _ in range(2))
    render_plain(plain)
    stats = render_tiled(tiled, small_area=32)
    far = plain.prim_id.view(width, height)[32768:] if width > height else plain.prim_id.view(width, height)[:, 32768:]
    assert (far >= 0).any()  # the case reaches the coordinates it is about
    assert stats.binned_faces < n // 4  # and the path
    assert torch.equal(tiled.prim_id, plain.prim_id)
    assert torch.equal(tiled.zbuffer.view(torch.int32), plain.zbuffer.view(torch.int32))
