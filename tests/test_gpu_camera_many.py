"""Cameras whose rows of 16 floats lie past 2^31 floats."""
import pytest

from .test_gpu_camera import _params

pytestmark = pytest.mark.gpu


def test_the_last_of_many_cameras():
    import torch

    from jaxrenderer_gb300 import autograd as A

    n = (1 << 27) + 1
    if torch.cuda.mem_get_info()[0] < 64 << 30:
        pytest.skip("needs 64 GB of device memory")
    eye = torch.tensor([[3.0, 4.0, 2.0]], device="cuda", requires_grad=True).expand(n, 3)
    eye.retain_grad()
    ms = A.camera_matrices(eye, _params())
    assert type(ms[0].grad_fn).__name__ == "_CameraFunctionBackward"
    for m in ms:
        for at in (1 << 26, 1 << 27):
            assert torch.equal(m[at].detach(), m[0].detach())
    ms[0].backward(torch.randn((1, 4, 4), device="cuda").expand(n, 4, 4))
    assert eye.grad[0].any() and torch.equal(eye.grad[1 << 26 :], eye.grad[:1].expand(n - (1 << 26), 3))
