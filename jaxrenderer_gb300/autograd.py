"""Differentiable rendering: a torch.autograd.Function over the CUDA forward
and the hand-written backward (rast_backward), plus torch versions of the
camera construction so gradients reach camera positions and light
directions (renderer.py:141-196, geometry.py:536-684 of the reference).

    db = DifferentiableBatch(scene_batch)
    canvas, zbuffer = db.render(position=pos, texture=tex,
                                world_to_clip=w2c, world_to_eye_norm=w2e,
                                light_direction=ldir)
    loss(canvas).backward()

Visibility is piecewise constant: gradients flow through the winning
primitive of every pixel, as under jax.grad of the reference.  A
DifferentiableBatch keeps one forward state: call backward before the next
render.
"""
from __future__ import annotations

from typing import Tuple

import numpy as np
import torch

from . import _lib
from .batch import BatchRunner, SceneBatch

PARAM_COLUMNS = {
    "world_to_clip": (_lib.GRAD_WORLD_TO_CLIP, 16),
    "world_to_eye_norm": (_lib.GRAD_WORLD_TO_EYE_NORM, 16),
    "light_direction": (_lib.GRAD_LIGHT_DIRECTION, 3),
    "light_colour": (_lib.GRAD_LIGHT_COLOUR, 3),
    "light_dir_eye": (_lib.GRAD_LIGHT_DIR_EYE, 3),
    "ambient": (_lib.GRAD_AMBIENT, 3),
    "diffuse": (_lib.GRAD_DIFFUSE, 3),
    "specular": (_lib.GRAD_SPECULAR, 3),
    "shadow_strength": (_lib.GRAD_SHADOW_STRENGTH, 3),
    "background": (_lib.GRAD_BACKGROUND, 3),
}
POOL_PARAMS = ("position", "normal", "colour", "texture", "specular_map", "normal_map")
JOB_OFFSETS = {name: getattr(_lib.RastJob, name).offset // 4 for name in PARAM_COLUMNS}


# ------------------------------------------------------ torch camera math

def _normalise(v: torch.Tensor) -> torch.Tensor:
    return v / torch.sqrt((v[..., 0:1] * v[..., 0:1] + v[..., 1:2] * v[..., 1:2]) + v[..., 2:3] * v[..., 2:3])


def view_matrix(eye: torch.Tensor, centre: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """lookAt (geometry.py:536-575), batched over leading axes."""
    forward = _normalise(centre - eye)
    up = _normalise(up.expand_as(forward))
    side = _normalise(torch.cross(forward, up, dim=-1))
    up = torch.cross(side, forward, dim=-1)
    zero = torch.zeros_like(eye[..., :1])
    one = torch.ones_like(zero)
    r0 = torch.cat([side, -(side * eye).sum(-1, keepdim=True)], -1)
    r1 = torch.cat([up, -(up * eye).sum(-1, keepdim=True)], -1)
    r2 = torch.cat([-forward, (forward * eye).sum(-1, keepdim=True)], -1)
    r3 = torch.cat([zero, zero, zero, one], -1)
    return torch.stack([r0, r1, r2, r3], dim=-2)


def view_matrix_inv(eye: torch.Tensor, centre: torch.Tensor, up: torch.Tensor) -> torch.Tensor:
    """Inverse of lookAt from its parts (geometry.py:581-632)."""
    forward = _normalise(centre - eye)
    up = _normalise(up.expand_as(forward))
    side = _normalise(torch.cross(forward, up, dim=-1))
    up = torch.cross(side, forward, dim=-1)
    rot = torch.stack([side, up, -forward], dim=-1)  # columns
    top = torch.cat([rot, eye.unsqueeze(-1)], -1)
    zero = torch.zeros_like(top[..., :1, :3])
    bottom = torch.cat([zero, torch.ones_like(zero[..., :1])], -1)  # (0, 0, 0, 1), no host copy
    return torch.cat([top, bottom], dim=-2)


def perspective_projection_matrix(fovy: float, aspect: float, z_near: float, z_far: float, dtype=torch.float32,
                                  device=None) -> torch.Tensor:
    """gluPerspective (geometry.py:638-684)."""
    f = float(1.0 / np.tan(np.radians(fovy) / 2.0))
    p = torch.zeros((4, 4), dtype=dtype, device=device)
    p[0, 0] = float(f / aspect)
    p[1, 1] = f
    p[2, 2] = float((z_far + z_near) / (z_near - z_far))
    p[2, 3] = float(2.0 * z_far * z_near / (z_near - z_far))
    p[3, 2] = -1.0
    return p


def camera_matrices(eye: torch.Tensor, params, target=None, up=None) -> Tuple[torch.Tensor, torch.Tensor, torch.Tensor]:
    """(world_to_clip, world_to_eye_norm, view) of cameras at `eye` (N, 3)
    built as Renderer.create_camera_from_parameters does.  With `target` and
    `up` given as tensors on eye's device, calls after the first for the same
    camera parameters copy nothing from the host, so they can be captured in
    a CUDA graph."""
    dt, dev = eye.dtype, eye.device

    def vec(x, default):
        if isinstance(x, torch.Tensor):
            return x.to(dtype=dt, device=dev)
        return torch.as_tensor(np.asarray(default if x is None else x, np.float64), dtype=dt, device=dev)

    target = vec(target, params.target)
    up = vec(up, params.up)
    target = target.expand_as(eye)
    aspect = np.tan(np.radians(params.hfov) / 2.0) / np.tan(np.radians(params.vfov) / 2.0)
    key = (float(params.vfov), float(aspect), float(params.near), float(params.far), dt, dev)
    p = _PROJECTIONS.get(key)
    if p is None:  # built once per camera and device: later calls copy nothing from the host
        p = perspective_projection_matrix(params.vfov, aspect, params.near, params.far, dtype=dt, device=dev)
        _PROJECTIONS[key] = p
    if _native_cameras(eye, target, up):
        return _CameraFunction.apply(eye, target, up.expand_as(eye), p)
    return _camera_tensors(eye, target, up, p)


def _camera_tensors(eye, target, up, projection):
    """The same as tensor operations: any dtype, device, shape or transform."""
    v = view_matrix(eye, target, up)
    return projection @ v, view_matrix_inv(eye, target, up).transpose(-1, -2), v


def _native_cameras(*tensors) -> bool:
    """Whether the kernels take these: float32 rows of one GPU, with nothing
    watching the operations (_watched, autocast and tensor subclasses see the
    tensor operations)."""
    return _kernel_rows(*tensors) and not _watched() and not torch.is_autocast_enabled()


def _kernel_rows(*tensors) -> bool:
    """Whether these are rows (or one shared row) of three adjacent float32 on
    one GPU, as many as the first of them has."""
    eye = tensors[0]
    return (eye.dim() == 2 and eye.shape[0] > 0 and eye.shape[1] == 3
            and all(type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.float32
                    and t.device == eye.device and t.shape[-1:] == (3,) and t.stride(-1) == 1 for t in tensors))


def _watched() -> bool:
    """Whether something follows the operations one by one: functorch
    transforms, forward-mode duals, dispatch modes or tracing."""
    return (torch._C._are_functorch_transforms_active() or torch.autograd.forward_ad._current_level >= 0
            or torch._C._len_torch_dispatch_stack() > 0 or torch.jit.is_tracing() or torch.compiler.is_compiling())


class _CameraFunction(torch.autograd.Function):
    """camera_matrices as one kernel per direction (rast_camera_matrices)."""

    @staticmethod
    def forward(ctx, eye, target, up, projection):
        n = eye.shape[0]
        w2c, w2e, view = (torch.empty((n, 4, 4), dtype=eye.dtype, device=eye.device) for _ in range(3))
        with torch.cuda.device(eye.device):
            s = torch.cuda.current_stream(eye.device).cuda_stream
            _lib.check(_lib.load().rast_camera_matrices(n, *_rows(eye), *_rows(target), *_rows(up), projection.data_ptr(),
                                                        w2c.data_ptr(), w2e.data_ptr(), view.data_ptr(), s),
                       "rast_camera_matrices")
        ctx.save_for_backward(eye, target, up, projection)
        ctx.set_materialize_grads(False)
        return w2c, w2e, view

    @staticmethod
    def backward(ctx, *grads):
        eye, target, up, projection = ctx.saved_tensors
        wanted = ctx.needs_input_grad[:3]
        if all(g is None for g in grads):
            return None, None, None, None
        # the saved tensors may have come through hooks that lay them out anew
        readable = (_kernel_rows(eye, target, up) and projection.is_cuda and projection.dtype == torch.float32
                    and projection.is_contiguous() and all(_has_memory(g) for g in grads if g is not None))
        if torch.is_grad_enabled() or _watched() or not readable:
            return (*_tensor_gradients((eye, target, up), projection, wanted, grads), None)
        n = eye.shape[0]
        mats = [_mats(g) for g in grads]
        out = [torch.empty((n, 3), dtype=eye.dtype, device=eye.device) if w else None for w in wanted]
        with torch.cuda.device(eye.device):
            s = torch.cuda.current_stream(eye.device).cuda_stream
            _lib.check(_lib.load().rast_camera_matrices_backward(
                n, *_rows(eye), *_rows(target), *_rows(up), projection.data_ptr(),
                *(x for g in mats for x in ((g.data_ptr(), g.stride(0)) if g is not None else (None, 0))),
                *(t.data_ptr() if t is not None else None for t in out), s), "rast_camera_matrices_backward")
        return (*out, None)


def _tensor_gradients(rows, projection, wanted, grads):
    """The reverse mode as tensor operations: with create_graph (gradients of
    gradients follow them), where something watches (a tangent of the gradient
    is asked for inside a dual level), and for tensors the kernel cannot read."""
    create_graph = torch.is_grad_enabled()
    with torch.enable_grad():
        # views of the inputs: a gradient stops at them, and does not run on through an input computed from another
        rows = [t.view_as(t) if create_graph else t.detach().requires_grad_(w) for t, w in zip(rows, wanted)]
        outs, gs = zip(*((o, g) for o, g in zip(_camera_tensors(*rows, projection), grads) if g is not None))
        got = iter(torch.autograd.grad(outs, [t for t, w in zip(rows, wanted) if w], gs, create_graph=create_graph,
                                       allow_unused=True))
    return [next(got) if w else None for w in wanted]


def _has_memory(t: torch.Tensor) -> bool:
    """Whether there is memory behind `t` that a kernel can read: not behind
    the batched tensors of is_grads_batched, whose gradient mode is off and
    which no query of the active transforms reports."""
    try:
        return t.data_ptr() != 0
    except RuntimeError:
        return False


def _rows(t: torch.Tensor):
    return t.data_ptr(), t.stride(0)


def _mats(g):
    """A gradient of (N, 4, 4) matrices with each matrix contiguous."""
    return g if g is None or g.stride()[1:] == (4, 1) else g.contiguous()


_PROJECTIONS: dict = {}


def apply_vec(vec: torch.Tensor, m: torch.Tensor) -> torch.Tensor:
    """Camera.apply_vec (geometry.py:352-389) of one vector by (N, 4, 4) matrices."""
    n = _normalise(vec)
    h = torch.cat([n, torch.zeros_like(n[..., :1])], -1)
    t = (m @ h.unsqueeze(-1)).squeeze(-1)[..., :3]
    return _normalise(t)


# ------------------------------------------------------------ the Function

class _RenderFunction(torch.autograd.Function):
    @staticmethod
    def forward(ctx, db: "DifferentiableBatch", names: Tuple[str, ...], *tensors):
        runner = db.runner
        jf = runner.job_floats()
        for name, t in zip(names, tensors):
            if name in POOL_PARAMS:
                runner.pools[name].copy_(t.detach().reshape(runner.pools[name].shape))
            else:
                off = JOB_OFFSETS[name]
                width = PARAM_COLUMNS[name][1]
                jf[:, off : off + width] = t.detach().reshape(jf.shape[0], width).to(torch.float32)
        out = runner.run()
        ctx.db = db
        ctx.names = names
        ctx.shapes = [t.shape for t in tensors]
        ctx.dtypes = [t.dtype for t in tensors]
        ctx.set_materialize_grads(False)
        db._generation += 1
        ctx.generation = db._generation
        return out.canvas.clone(), out.zbuffer.clone()

    @staticmethod
    def backward(ctx, g_canvas, g_zbuffer):
        db = ctx.db
        if db._generation != ctx.generation:
            raise RuntimeError("DifferentiableBatch was re-rendered before backward of an earlier render")
        # the gradients of the given inputs only: the kernels skip the others
        runner = db.runner
        g = {k: torch.zeros_like(runner.pools[k]) for k, w in zip(ctx.names, ctx.needs_input_grad[2:])
             if w and k in POOL_PARAMS}
        if any(w and k in PARAM_COLUMNS for k, w in zip(ctx.names, ctx.needs_input_grad[2:])):
            g["job_params"] = torch.zeros((runner.sb.n_scenes, _lib.NPARAM), dtype=torch.float32, device=runner.sb.device)
        runner.backward(g_canvas, g_zbuffer, out=g, accumulate=True)
        grads = []
        for name, shape, dt, w in zip(ctx.names, ctx.shapes, ctx.dtypes, ctx.needs_input_grad[2:]):
            if not w:
                grads.append(None)
            elif name in POOL_PARAMS:
                grads.append(g[name].reshape(shape).to(dt))
            else:
                col, width = PARAM_COLUMNS[name]
                grads.append(g["job_params"][:, col : col + width].reshape(shape).to(dt))
        return (None, None, *grads)


class DifferentiableBatch:
    """Differentiable renders of one SceneBatch (main pass gradients)."""

    def __init__(self, sb: SceneBatch, form: str = "tiled", tiled_config=None):
        self.runner = BatchRunner(sb, form=form, want_prim_id=True, tiled_config=tiled_config)
        self._generation = 0

    def render(self, **params: torch.Tensor):
        """Render with the given tensors in place of the batch's inputs.

        Pool inputs: position, normal, colour (gouraud), texture,
        specular_map, normal_map (flat pool shapes).  Per-scene inputs, (N, ...): world_to_clip (N, 4, 4),
        world_to_eye_norm (N, 4, 4), light_direction, light_colour,
        light_dir_eye, ambient, diffuse, specular, shadow_strength (N, 3).
        Returns (canvas (N, W, H, 3), zbuffer (N, W, H))."""
        for k in params:
            if k not in POOL_PARAMS and k not in PARAM_COLUMNS:
                raise KeyError(f"unknown differentiable input {k!r}")
        names = tuple(params)
        return _RenderFunction.apply(self, names, *[params[k] for k in names])


__all__ = ["DifferentiableBatch", "camera_matrices", "view_matrix", "view_matrix_inv",
           "perspective_projection_matrix", "apply_vec"]
