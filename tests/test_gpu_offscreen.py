"""Faces beyond the screen's sides: the tiled set-up drops them before their
inverse is computed, which must never drop a pixel the per-pixel scan over
every primitive (the plain form) covers."""
import numpy as np
import pytest

from jaxrenderer_gb300 import _lib, geometry
from jaxrenderer_gb300.jobs import JobSpec, pack, render_plain, render_tiled

pytestmark = pytest.mark.gpu
F32 = np.float32


def _soup(rng, n, size, aspect):
    """Triangles of about `size` around the view's borders, stretched by up to
    `aspect`, with exact and nearly degenerate ones among them."""
    centre = rng.uniform(-4, 4, (n, 1, 3))
    centre[: n // 2, 0, :2] = np.sign(centre[: n // 2, 0, :2]) * rng.uniform(0.7, 1.4, (n // 2, 2)) * 2.0
    tri = centre + rng.normal(scale=size, size=(n, 3, 3)) * np.exp(rng.uniform(-np.log(aspect), 0, (n, 1, 3)))
    tri[::17, 2] = tri[::17, 1] + rng.normal(scale=1e-6, size=tri[::17, 2].shape)
    tri[::41, 2] = tri[::41, 1]
    return tri.reshape(-1, 3).astype(F32)


@pytest.mark.parametrize("size,aspect", [(0.02, 1.0), (0.3, 50.0), (3.0, 1000.0)])
@pytest.mark.parametrize("light", [False, True])
@pytest.mark.parametrize("width,height,scale", [(84, 84, 1.0), (33, 61, 1.0), (128, 17, 40.0)])
def test_same_pixels_as_the_scan(width, height, scale, light, size, aspect):
    import torch

    rng = np.random.default_rng([width, int(scale), light, int(aspect)])
    pos = _soup(rng, 20000, size, aspect)
    cam = geometry.Camera
    eye, up = np.array((0.3, -0.2, 5.0), F32), np.array((0, 1, 0), F32)
    view = cam.view_matrix(eye, np.zeros(3, F32), up)
    proj = (cam.orthographic_projection_matrix(-1.0, 1.0, -1.0, 1.0, -1.0, 1.0) if light
            else cam.perspective_projection_matrix(45.0, 1.0, 0.1, 100.0))
    # a viewport larger than the canvas: the screen rectangle is a corner of the view
    vp = cam.viewport_matrix(np.zeros(2, np.int32), np.array((width, height)) * scale, 1.0)
    c = cam.create(view, proj, vp)
    spec = JobSpec(shader=_lib.SHADER_DEPTH, width=width, height=height, viewport=c.viewport, world_to_clip=c.world_to_clip,
                   world_to_eye_norm=c.world_to_eye_norm, position=pos, faces=np.arange(len(pos), dtype=np.int32).reshape(-1, 3))
    z = np.full((width, height), 1e9, F32)
    dev = torch.device("cuda")
    plain, tiled, small = (pack([spec], [z], [None], dev) for _ in range(3))
    render_plain(plain)
    render_tiled(tiled)
    render_tiled(small, small_area=32)
    for got in (tiled, small):
        assert torch.equal(got.prim_id, plain.prim_id)
        assert torch.equal(got.zbuffer.view(torch.int32), plain.zbuffer.view(torch.int32))
