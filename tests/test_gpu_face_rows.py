"""Tiled form's per-face rows of varyings (whole float4s, then the rest of
each row) against the plain form, which reads its vertices' own rows: the same
operations, so the same bits."""
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import pack, render_plain, render_tiled

from . import scenes

pytestmark = pytest.mark.gpu
S = _lib
SETS = [(s,) for s in scenes.ALL_SHADERS] + [
    (S.SHADER_GOURAUD, S.SHADER_DEPTH),                                  # rows of 9: a rest of one float
    (S.SHADER_PHONG, S.SHADER_GOURAUD),                                  # 15 and 9: the shorter row ends inside a float4
    (S.SHADER_GOURAUD_TEXTURE, S.SHADER_PHONG_REFLECTION),               # 15 in rows of 16
    (S.SHADER_PHONG_DARBOUX, S.SHADER_PHONG_REFLECTION_SHADOW, S.SHADER_PHONG),  # 30, 28, 15: a rest of two
    scenes.ALL_SHADERS,
]


@pytest.mark.parametrize("shaders", SETS, ids=lambda s: "-".join(map(str, s)))
@pytest.mark.parametrize("faces,layers", [(1, 0), (9, 0), (11, 0), (300, 0), (300, 3)])
def test_same_bits_as_the_plain_form(shaders, faces, layers):
    import torch

    dev = torch.device("cuda")
    specs = [scenes.random_job(s, 31 * faces + k, W=41 + 7 * k, H=33, F=faces) for k, s in enumerate(shaders)]
    for s in specs:
        s.layers = layers if s.shader != S.SHADER_DEPTH else 0  # depth passes take no layers
    z, c = zip(*(scenes.initial_buffers(s) for s in specs))
    got, want = pack(specs, z, c, dev), pack(specs, z, c, dev)
    render_tiled(got)
    render_plain(want)
    assert torch.equal(got.prim_id, want.prim_id)
    assert torch.equal(got.zbuffer.view(torch.int32), want.zbuffer.view(torch.int32))
    if want.canvas is not None:
        assert torch.equal(got.canvas.view(torch.int32), want.canvas.view(torch.int32))
