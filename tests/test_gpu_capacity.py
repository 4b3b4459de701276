"""Bins sized for the batch at hand: a class tuned on a light batch must not
leave a heavier batch of the same class with overflowing bins."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(84, 84), (33, 130)])
def test_heavier_batch_of_a_tuned_class_does_not_overflow(width, height, tmp_path, monkeypatch):
    import torch

    from jaxrenderer_gb300 import autotune, batch, synthetic

    monkeypatch.setenv("JAXRENDERER_GB300_AUTOTUNE", str(tmp_path / "tune.json"))
    runners = []
    for scenes, faces in ((3, 1500), (5, 2880)):
        flat = synthetic.cube_scene_batch(scenes, f_min=faces, f_max=faces)
        sb = batch.scene_batch_from_flat(flat, width, height, shadow_size=(64, 64))
        runners.append(batch.BatchRunner(sb, form="tiled"))
    keys = [autotune.workload_key(r.sb.main_jobs, r.sb.device) for r in runners]
    assert keys[0] == keys[1]  # one class
    for r in runners:
        out = r.run()
        for name in ("shadow", "main"):
            st = r.stats(name)
            assert not st.overflow and st.bin_capacity >= 4 * r.sb.total_faces
        plain = batch.BatchRunner(r.sb, form="plain").run()
        assert torch.equal(out.canvas, plain.canvas) and torch.equal(out.prim_id, plain.prim_id)
