"""BatchRunner.run's zbuffer_default: the values torch.Tensor.fill_ takes for a
float32 buffer, and no others."""
import pytest

pytestmark = pytest.mark.gpu


def _runner():
    import torch

    from jaxrenderer_gb300 import _lib, batch, synthetic

    flat = synthetic.cube_scene_batch(2, f_min=12, f_max=12)
    sb = batch.scene_batch_from_flat(flat, 33, 17, shadow_size=(16, 16), device=torch.device("cuda", 0))
    return batch.BatchRunner(sb, form="tiled", tiled_config=_lib.RastTiledConfig(8, 8, 0))


@pytest.mark.parametrize("value", [2, 0.1, -3.5e38, float("inf"), float("nan"), "tensor", "int tensor"])
def test_same_as_fill(value):
    import torch

    if value == "tensor":
        value = torch.tensor(0.1, device="cuda")
    elif value == "int tensor":
        value = torch.tensor(3)
    r = _runner()
    want = torch.empty(1, device="cuda")
    try:
        want.fill_(value)
    except RuntimeError:
        with pytest.raises(RuntimeError):
            r.run(zbuffer_default=value)
        return
    out = r.run(zbuffer_default=value)
    empty = out.prim_id < 0
    assert empty.any()
    assert torch.equal(out.zbuffer[empty].view(torch.int32), want.view(torch.int32).expand(int(empty.sum())))


def test_default_on_the_device_is_read_by_every_replay():
    import torch

    r = _runner()
    z = torch.tensor(0.5, device="cuda")
    r.run(zbuffer_default=z)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        r.run(zbuffer_default=z)
    z.fill_(0.25)
    g.replay()
    torch.cuda.synchronize()
    assert (r.zbuffer[r.prim_id < 0] == 0.25).all()
