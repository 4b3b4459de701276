"""rast_render_tiled_clear: the buffers' old contents do not matter, and every
pixel gets what a render into buffers filled with the defaults gives it."""
import ctypes

import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import JobSpec, pack, render_tiled_config

pytestmark = pytest.mark.gpu
F32 = np.float32


def _spec(rng, shader, width, height, faces):
    pos = rng.uniform(-0.9, 0.9, (max(3 * faces, 3), 3)).astype(F32)
    s = JobSpec(shader=shader, width=width, height=height,
                viewport=np.array([[width / 2, 0, 0, width / 2], [0, height / 2, 0, height / 2], [0, 0, 0.5, 0.5], [0, 0, 0, 1]], F32),
                world_to_clip=np.identity(4, dtype=F32), world_to_eye_norm=np.identity(4, dtype=F32), position=pos,
                faces=np.arange(3 * faces, dtype=np.int32).reshape(-1, 3), depth_offset=0.25, apply_depth_offset=shader == _lib.SHADER_DEPTH)
    if shader != _lib.SHADER_DEPTH:
        s.normal = rng.normal(size=pos.shape).astype(F32)
        s.colour = rng.uniform(0, 1, pos.shape).astype(F32)
    return s


@pytest.mark.parametrize("layers", [0, 2])
@pytest.mark.parametrize("faces", [(40, 40), (0, 40), (0, 0)])
@pytest.mark.parametrize("shaders", [(_lib.SHADER_DEPTH, _lib.SHADER_DEPTH), (_lib.SHADER_GOURAUD, _lib.SHADER_GOURAUD),
                                     (_lib.SHADER_DEPTH, _lib.SHADER_GOURAUD)])
def test_clear_equals_default_buffers(shaders, faces, layers):
    import torch

    dev = torch.device("cuda")
    rng = np.random.default_rng([*shaders, *faces])
    specs = [_spec(rng, sh, w, h, f) for sh, (w, h), f in zip(shaders, ((9, 33), (16, 8)), faces)]
    for s in specs:
        if layers and s.shader != _lib.SHADER_DEPTH:
            s.layers, s.mixer, s.opacity = layers, _lib.MIX_OVER, 0.5
    colour = np.array((0.1, 0.2, 0.3), F32)

    def packed(z, c):
        return pack(specs, [np.full((s.width, s.height), z, F32) for s in specs],
                    [np.broadcast_to(np.asarray(c, F32), (s.width, s.height, 3)).copy() for s in specs], dev)

    want = packed(0.75, colour)
    render_tiled_config(want, _lib.RastTiledConfig(8, 8, 0))
    got = packed(np.nan, (7.0, 8.0, 9.0))
    lib, cfg = _lib.load(), _lib.RastTiledConfig(8, 8, 0)
    n = lib.rast_tiled_workspace_bytes(ctypes.byref(got.batch), ctypes.byref(cfg))
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    col = torch.from_numpy(colour).to(dev)
    clear = _lib.RastClear(col.data_ptr(), 0.75)
    stream = torch.cuda.current_stream(dev).cuda_stream
    for phase in (_lib.PHASE_COVERAGE, _lib.PHASE_SHADE):
        _lib.check(lib.rast_render_tiled_clear(ctypes.byref(got.batch), ctypes.byref(cfg), ctypes.byref(clear), ws.data_ptr(), n,
                                               stream, phase), "rast_render_tiled_clear")
    assert torch.equal(got.zbuffer, want.zbuffer)
    assert torch.equal(got.canvas, want.canvas)
    assert torch.equal(got.prim_id, want.prim_id)
    assert lib.rast_render_tiled_clear(ctypes.byref(got.batch), ctypes.byref(cfg), None, ws.data_ptr(), n, stream, 3) == 1
    assert lib.rast_render_tiled_clear(ctypes.byref(got.batch), ctypes.byref(cfg), ctypes.byref(_lib.RastClear(None, 0.0)), ws.data_ptr(),
                                       n, stream, 3) == 1
