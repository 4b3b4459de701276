"""camera_matrices where something watches or batches its gradients: the same
results as the tensor operations give in float64."""
import contextlib

import pytest

from .test_gpu_camera import _inputs, _loss, _params

pytestmark = pytest.mark.gpu


def _close(a, b, tol=1e-4):
    a, b = a.detach(), b.detach()
    assert a.shape == b.shape and (a.double() - b).norm() <= tol * max(1.0, float(b.norm()))


def _double(*tensors):
    return [t.detach().double().requires_grad_() for t in tensors]


@pytest.mark.parametrize("n", [1, 5])
@pytest.mark.parametrize("create_graph", [False, True])
def test_batched_gradients(n, create_graph):
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, c, u, _ = _inputs(n, False, n)
    d = _double(e, c, u)
    rows = torch.randn((4, n, 4, 4), device="cuda")

    def grads(leaves, rows, batched):
        ms = A.camera_matrices(leaves[0], _params(), leaves[1], leaves[2])
        if batched:
            return torch.autograd.grad(ms[0], leaves, rows, is_grads_batched=True, create_graph=create_graph)
        return [torch.stack(g) for g in zip(*(torch.autograd.grad(ms[0], leaves, r, retain_graph=True) for r in rows))]

    for a, b in zip(grads((e, c, u), rows, True), grads(d, rows.double(), False)):
        _close(a, b)

    def w2c(x):
        return A.camera_matrices(x, _params(), c.detach().to(x.dtype), u.detach().to(x.dtype))[0]

    got = torch.autograd.functional.jacobian(w2c, e.detach(), vectorize=True, create_graph=create_graph)
    _close(got, torch.autograd.functional.jacobian(w2c, d[0].detach()))


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


def test_no_gradient_arrives():
    import torch

    from jaxrenderer_gb300 import autograd as A

    class Nothing(torch.autograd.Function):
        @staticmethod
        def forward(ctx, x):
            return x.sum()

        @staticmethod
        def backward(ctx, g):
            return None

    e, c, u, _ = _inputs(3, False, 1)
    for create_graph in (False, True):
        y = Nothing.apply(A.camera_matrices(e, _params(), c, u)[0])
        g = torch.autograd.grad(y, (e, c, u), create_graph=create_graph, allow_unused=True)
        assert all(t is None or not t.any() for t in g)


def test_tangents_of_the_gradient():
    import torch
    import torch.autograd.forward_ad as fwd

    from jaxrenderer_gb300 import autograd as A

    e, c, u, ws = _inputs(5, False, 11)

    def tangent(leaves, ws):
        ms = A.camera_matrices(leaves[0], _params(), leaves[1], leaves[2])
        with fwd.dual_level():
            (g,) = torch.autograd.grad(ms[0], leaves[:1], fwd.make_dual(ws[0], ws[1]))
            return fwd.unpack_dual(g).tangent

    _close(tangent((e, c, u), ws), tangent(_double(e, c, u), [w.double() for w in ws]))


def _transposed(t):
    return t.mT.contiguous().mT if t.dim() > 1 else t


@pytest.mark.parametrize("hooks", ["cpu", "strides"])
def test_saved_tensor_hooks(hooks):
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, c, u, ws = _inputs(65, True, 2)
    around = (torch.autograd.graph.save_on_cpu() if hooks == "cpu"
              else torch.autograd.graph.saved_tensors_hooks(lambda t: t, _transposed))

    def grads(leaves, ws, around=contextlib.nullcontext()):
        with around:
            ms = A.camera_matrices(leaves[0], _params(), leaves[1], leaves[2])
        return torch.autograd.grad(_loss(ms, ws), leaves)

    for a, b in zip(grads((e, c, u), ws, around), grads(_double(e, c, u), [w.double() for w in ws])):
        _close(a, b)


@pytest.mark.parametrize("up", [2.0, (0.5,), ((0.1, -0.05, 1.0),)])
def test_up_of_any_shape_that_broadcasts(up):
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, c, _, _ = _inputs(5, False, 4)
    up = torch.tensor(up, device="cuda")
    for a, b in zip(A.camera_matrices(e, _params(), c, up), A.camera_matrices(e.double(), _params(), c.double(), up.double())):
        _close(a.detach(), b.detach())
