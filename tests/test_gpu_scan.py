"""The plain form's split scan (four pixels per thread, primitives split over
blocks) against its one-pixel scan, which passes that count near ties take."""
import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import JobSpec, pack, render_plain

pytestmark = pytest.mark.gpu
F32 = np.float32


def _spec(rng, width, height, faces, shader):
    pos = rng.uniform(-1.2, 1.2, (max(faces, 1), 1, 3)) + rng.normal(scale=0.3, size=(max(faces, 1), 3, 3))
    pos[1::9] = pos[::9][: len(pos[1::9])]  # exact ties: the lowest id
    pos = pos.reshape(-1, 3).astype(F32)
    vp = np.array([[width / 2, 0, 0, width / 2], [0, height / 2, 0, height / 2], [0, 0, 0.5, 0.5], [0, 0, 0, 1]], F32)
    s = JobSpec(shader=shader, width=width, height=height, viewport=vp, world_to_clip=np.identity(4, dtype=F32),
                world_to_eye_norm=np.identity(4, dtype=F32), position=pos, faces=np.arange(3 * faces, dtype=np.int32).reshape(-1, 3))
    s.normal, s.colour = rng.normal(size=pos.shape).astype(F32), rng.uniform(0, 1, pos.shape).astype(F32)
    return s


@pytest.mark.parametrize("sizes", [((1, 1),), ((3, 130),), ((4, 7),), ((5, 1), (33, 61)), ((84, 84), (2, 3), (17, 128))])
@pytest.mark.parametrize("faces", [0, 1, 63, 64, 127, 128, 129, 1000])
def test_same_as_the_one_pixel_scan(sizes, faces):
    import torch

    dev = torch.device("cuda")
    rng = np.random.default_rng([faces, len(sizes)])
    shaders = (_lib.SHADER_GOURAUD, _lib.SHADER_DEPTH)
    specs = [_spec(rng, w, h, max(0, faces - k), shaders[k % 2]) for k, (w, h) in enumerate(sizes)]
    z = [np.full((s.width, s.height), 2.0, F32) for s in specs]
    c = [np.full((s.width, s.height, 3), 0.5, F32) for s in specs]
    got, want = pack(specs, z, c, dev), pack(specs, z, c, dev, count_ties=True)
    render_plain(got)
    render_plain(want)
    assert torch.equal(got.prim_id, want.prim_id)
    assert torch.equal(got.zbuffer.view(torch.int32), want.zbuffer.view(torch.int32))
    assert torch.equal(got.canvas.view(torch.int32), want.canvas.view(torch.int32))
