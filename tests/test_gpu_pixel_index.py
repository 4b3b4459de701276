"""Pixel coordinates from a job's linear index (approximate division, then the
remainder's correction), at the edges of its range, against the near-tie scan,
whose blocks carry two-dimensional coordinates."""
import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import JobSpec, pack, render_plain, render_tiled

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("width,height", [(1, 1), (1, 65535), (65535, 1), (16, 65535), (65535, 16), (1023, 1025), (997, 1051),
                                          (1024, 1024), (1025, 1024), (3, 65521), (7, 131)])
def test_every_pixel_has_its_own_coordinates(width, height):
    import torch

    dev = torch.device("cuda")
    pos = np.array([(-1, -1, -0.9), (3, -1, 0.3), (-1, 3, 0.7)], F32)  # covers the canvas; depth differs along both axes
    vp = np.array([[width / 2, 0, 0, width / 2], [0, height / 2, 0, height / 2], [0, 0, 0.5, 0.5], [0, 0, 0, 1]], F32)
    spec = JobSpec(shader=_lib.SHADER_GOURAUD, width=width, height=height, viewport=vp, world_to_clip=np.identity(4, dtype=F32),
                   world_to_eye_norm=np.identity(4, dtype=F32), position=pos, faces=np.array([(0, 1, 2)], np.int32))
    spec.normal, spec.colour = np.tile(np.array((0, 0, 1), F32), (3, 1)), np.identity(3, dtype=F32)
    spec.light_direction = np.array((0, 0, 1), F32)
    z, c = [np.full((width, height), 2.0, F32)], [np.zeros((width, height, 3), F32)]
    packs = [pack([spec], z, c, dev, count_ties=k == 0) for k in range(3)]
    render_plain(packs[0])
    render_plain(packs[1])
    render_tiled(packs[2])
    for p in packs[1:]:
        assert torch.equal(p.zbuffer.view(torch.int32), packs[0].zbuffer.view(torch.int32))
        assert torch.equal(p.canvas.view(torch.int32), packs[0].canvas.view(torch.int32))
