"""Camera matrices by kernel (rast_camera_matrices) against the tensor
operations in float64, their gradients, and the routes that keep the tensor
operations."""
import pytest

pytestmark = pytest.mark.gpu
U = 2.0 ** -24


def _params():
    from jaxrenderer_gb300 import CameraParameters

    return CameraParameters(viewWidth=64, viewHeight=48, near=0.1, far=100.0, hfov=58.0, vfov=45.0)


def _inputs(n, strided, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    e = torch.randn((n, 5 if strided else 3), generator=g, device="cuda") * 4 + 1
    e = (e[:, 1:4] if strided else e).detach().requires_grad_()
    c = (torch.randn((n, 3) if strided else 3, generator=g, device="cuda") * 0.1).requires_grad_()
    u = torch.tensor((0.1, -0.05, 1.0), device="cuda", requires_grad=True)
    return e, c, u, [torch.randn((n, 4, 4), generator=g, device="cuda") for _ in range(3)]


def _loss(ms, ws):
    return sum((m * w.to(m.dtype)).sum() for m, w in zip(ms, ws))


@pytest.mark.parametrize("n,strided", [(1, False), (63, True), (64, False), (65, True), (300, False)])
def test_matrices_and_gradients(n, strided):
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, c, u, ws = _inputs(n, strided, n)
    got = A.camera_matrices(e, _params(), c, u)
    assert got[0].grad_fn is not None and type(got[0].grad_fn).__name__ == "_CameraFunctionBackward"
    d = [t.detach().double().requires_grad_() for t in (e, c, u)]
    want = A.camera_matrices(d[0], _params(), d[1], d[2])
    for m, w in zip(got, want):
        # every entry is a sum of at most 16 products of entries below the largest |entry|, rounded once each
        assert (m.double() - w).detach().abs().max() <= 64 * U * max(1.0, float(w.detach().abs().max())) * 4
    g = torch.autograd.grad(_loss(got, ws), (e, c, u))
    g64 = torch.autograd.grad(_loss(want, ws), d)
    for a, b in zip(g, g64):
        assert (a.double() - b).norm() <= 2e-5 * b.norm()
    # one output alone, and one input alone
    e2, c2, u2, _ = _inputs(n, strided, n)
    (a,) = torch.autograd.grad((A.camera_matrices(e2, _params(), c2.detach(), u2.detach())[0] * ws[0]).sum(), e2)
    (b,) = torch.autograd.grad((A.camera_matrices(d[0], _params(), d[1].detach(), d[2].detach())[0] * ws[0].double()).sum(), d[0])
    assert (a.double() - b).norm() <= 2e-5 * b.norm()


def test_gradients_of_gradients_and_transforms_keep_the_tensor_operations():
    import torch

    from jaxrenderer_gb300 import autograd as A

    e, c, u, ws = _inputs(5, False, 7)
    for t in ws:
        t.requires_grad_()

    def second(e, c, u, ws):
        (g,) = torch.autograd.grad(_loss(A.camera_matrices(e, _params(), c, u), ws), e, create_graph=True)
        return torch.autograd.grad((g ** 2).sum(), [e, c, u, ws[0]])

    d = [t.detach().double().requires_grad_() for t in (e, c, u)]
    for a, b in zip(second(e, c, u, ws), second(*d, [w.detach().double().requires_grad_() for w in ws])):
        assert (a.double() - b).norm() <= 1e-4 * b.norm()
    e, c, u = e.detach(), c.detach(), u.detach()
    want = A.camera_matrices(e, _params(), c, u)
    rows = torch.func.vmap(lambda x: A.camera_matrices(x[None], _params(), c, u)[0][0])(e)
    assert torch.allclose(rows, want[0], rtol=1e-5, atol=1e-5)
    with torch.autograd.forward_ad.dual_level():
        dual = torch.autograd.forward_ad.make_dual(e, torch.ones_like(e))
        assert torch.autograd.forward_ad.unpack_dual(A.camera_matrices(dual, _params(), c, u)[0]).tangent is not None
