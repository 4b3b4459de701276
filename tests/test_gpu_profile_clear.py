"""A profiled launch into cleared buffers is the pass that run() makes."""
import pytest

from .test_gpu_defaults import _runner

pytestmark = pytest.mark.gpu


def test_profiled_clear_renders_what_run_renders():
    import torch

    from jaxrenderer_gb300 import _lib

    a, b = _runner(), _runner()
    want = a.run()
    for t in (b.canvas, b.zbuffer, b.shadow_map):
        t.fill_(float("nan"))
    clear = b.prepare()
    for name, _ in b.batches():
        prof = _lib.RastProfile()
        b.launch(name, torch.cuda.current_stream().cuda_stream, profile=prof, clear=clear[name])
        names = [prof.names[k].decode() for k in range(prof.n)]
        assert "raster_kernel" in names and ("tiled_shade_kernel" in names) == (name == "main")
    got = b.outputs()
    for k in ("canvas", "zbuffer", "shadow_map", "prim_id"):
        assert torch.equal(getattr(got, k), getattr(want, k)), k
    with pytest.raises(ValueError):
        b.launch("main", torch.cuda.current_stream().cuda_stream, profile=_lib.RastProfile(), clear=clear["main"], phase=1)
