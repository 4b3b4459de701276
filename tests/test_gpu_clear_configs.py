"""rast_render_tiled_clear over stale buffers in every kind of tiled config, as
one call and as its two phases."""
import ctypes

import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import pack, render_tiled_config

from .test_gpu_clear import _spec

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("phases", [(3,), (_lib.PHASE_COVERAGE, _lib.PHASE_SHADE)])
@pytest.mark.parametrize("config", [(8, 8, 32, 1), (16, 8, 0, 1), (8, 16, 0, 2), (16, 16, 32, 2)])
@pytest.mark.parametrize("faces", [(40, 40), (0, 40), (0, 0)])
@pytest.mark.parametrize("shaders", [(_lib.SHADER_DEPTH,) * 2, (_lib.SHADER_GOURAUD,) * 2, (_lib.SHADER_DEPTH, _lib.SHADER_GOURAUD)])
def test_clear_equals_default_buffers(shaders, faces, config, phases):
    import torch

    dev = torch.device("cuda")
    rng = np.random.default_rng([*shaders, *faces, *config])
    specs = [_spec(rng, sh, w, h, f) for sh, (w, h), f in zip(shaders, ((9, 33), (16, 8)), faces)]
    cfg = _lib.RastTiledConfig(config[0], config[1], 0, config[2], config[3])
    colour = torch.tensor((0.1, 0.2, 0.3), device=dev)

    def packed(z, c):
        p = pack(specs, [np.full((s.width, s.height), z, F32) for s in specs],
                 [np.broadcast_to(np.asarray(c, F32), (s.width, s.height, 3)).copy() for s in specs], dev)
        p.prim_id.fill_(77)
        return p

    want, got = packed(0.75, colour.cpu().numpy()), packed(np.nan, (7.0, 8.0, 9.0))
    render_tiled_config(want, cfg)
    lib = _lib.load()
    n = lib.rast_tiled_workspace_bytes(ctypes.byref(got.batch), ctypes.byref(cfg))
    ws = torch.full((n,), 0xA5, dtype=torch.uint8, device=dev)
    clear = _lib.RastClear(colour.data_ptr(), 0.75)
    for phase in phases:
        _lib.check(lib.rast_render_tiled_clear(ctypes.byref(got.batch), ctypes.byref(cfg), ctypes.byref(clear), ws.data_ptr(), n,
                                               torch.cuda.current_stream(dev).cuda_stream, phase), "rast_render_tiled_clear")
    for k in ("zbuffer", "canvas", "prim_id"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k
