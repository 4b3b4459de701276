"""Face varyings by one to four warps per map entry (which the number
of entries, at least one a scene, decides) against the plain form."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scenes", [3, 10000, 15000, 35000])
def test_same_images_as_the_plain_form(scenes):
    import torch

    from jaxrenderer_gb300 import _lib, batch, synthetic

    flat = synthetic.cube_scene_batch(scenes, f_min=12, f_max=12)
    sb = batch.scene_batch_from_flat(flat, 6, 5, shadow_param=None, device=torch.device("cuda", 0))
    out = batch.BatchRunner(sb, form="tiled", tiled_config=_lib.RastTiledConfig(8, 8, 0)).run()
    want = batch.BatchRunner(sb, form="plain").run()
    for k in ("prim_id", "canvas", "zbuffer"):
        assert torch.equal(getattr(out, k), getattr(want, k))
    assert (out.prim_id >= 0).flatten(1).any(1).float().mean() > 0.9
