"""A batch without faces recorded into a CUDA graph and replayed."""
import ctypes

import numpy as np
import pytest

from jaxrenderer_gb300 import _lib
from jaxrenderer_gb300.jobs import pack
from .test_gpu_clear import _spec

pytestmark = pytest.mark.gpu
F32 = np.float32


@pytest.mark.parametrize("clear", [False, True])
@pytest.mark.parametrize("layers", [0, 2])
@pytest.mark.parametrize("shaders", [(_lib.SHADER_DEPTH,), (_lib.SHADER_GOURAUD,), (_lib.SHADER_DEPTH, _lib.SHADER_GOURAUD)])
def test_captured_render_of_no_faces(shaders, layers, clear):
    import torch

    dev = torch.device("cuda")
    specs = [_spec(np.random.default_rng(0), sh, 9, 33, 0) for sh in shaders]
    for s in specs:
        if layers and s.shader != _lib.SHADER_DEPTH:
            s.layers, s.mixer, s.opacity = layers, _lib.MIX_OVER, 0.5
    p = pack(specs, [np.full((9, 33), 0.75, F32)] * len(specs), [np.full((9, 33, 3), 0.5, F32)] * len(specs), dev)
    lib, cfg = _lib.load(), _lib.RastTiledConfig(8, 8, 0)
    n = lib.rast_tiled_workspace_bytes(ctypes.byref(p.batch), ctypes.byref(cfg))
    ws = torch.empty(n, dtype=torch.uint8, device=dev)
    colour = torch.tensor((0.1, 0.2, 0.3), device=dev)

    def render(s):
        if clear:
            st = lib.rast_render_tiled_clear(ctypes.byref(p.batch), ctypes.byref(cfg), ctypes.byref(_lib.RastClear(colour.data_ptr(), 0.25)),
                                             ws.data_ptr(), n, s, 3)
        else:
            st = lib.rast_render_tiled(ctypes.byref(p.batch), ctypes.byref(cfg), ws.data_ptr(), n, s)
        _lib.check(st, "render")

    z0, c0 = p.zbuffer.clone(), p.canvas.clone()
    stream = torch.cuda.Stream(dev)
    stream.wait_stream(torch.cuda.current_stream(dev))
    render(stream.cuda_stream)
    torch.cuda.synchronize(dev)
    want = [t.clone() for t in (p.zbuffer, p.canvas, p.prim_id)]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        render(torch.cuda.current_stream(dev).cuda_stream)
    p.zbuffer.copy_(z0)
    p.canvas.copy_(c0)
    p.prim_id.fill_(77)
    graph.replay()
    torch.cuda.synchronize(dev)
    for a, b in zip((p.zbuffer, p.canvas, p.prim_id), want):
        assert torch.equal(a, b)
    assert (p.prim_id == -1).all()
