"""Corner kernel with 16, 11 and 4 warps per instance (the count falls with the
number of instances) against the host merge, bit for bit."""
import pytest
import torch

from jaxrenderer_gb300 import batch as jb
from jaxrenderer_gb300 import synthetic
from tests.test_gpu_instancing import _check_pools, stress_scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,n_scenes", [("stress", 1), ("stress", 250), ("stress", 800), ("brax", 2), ("brax", 160)])
def test_corners_match_the_host_merge(cuda_device, kind, n_scenes):
    inst = stress_scenes(n_scenes, seed=2) if kind == "stress" else synthetic.brax_like_instances(
        n_scenes, seed=synthetic.BASE_SEED + 34)
    sb, merge = jb.scene_batch_from_instances(inst, 32, 32, device=cuda_device)
    torch.cuda.synchronize()
    _check_pools(sb.pools, inst.host_flat(range(inst.n_scenes)))
