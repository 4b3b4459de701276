"""camera_matrices where something watches or batches its gradients: the same
results as the tensor operations give in float64."""
import pytest

from .test_gpu_camera import _inputs, _loss, _params

pytestmark = pytest.mark.gpu


def _close(a, b, tol=1e-4):
    a, b = a.detach(), b.detach()
    assert a.shape == b.shape and (a.double() - b).norm() <= tol * max(1.0, float(b.norm()))


def _double(*tensors):
    return [t.detach().double().requires_grad_() for t in tensors]


def test_gradients_of_gradients_of_inputs_that_depend_on_one_another():
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, _, u, ws = _inputs(5, False, 3)

    def second(e, u, ws):
        ms = A.camera_matrices(e, _params(), 0.25 * e * e, u * e.mean())
        (g,) = torch.autograd.grad(_loss(ms, ws), e, create_graph=True)
        return [g, *torch.autograd.grad((g ** 2).sum(), [e, u])]

    for a, b in zip(second(e, u, ws), second(*_double(e, u), [w.double() for w in ws])):
        _close(a, b)
