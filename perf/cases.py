"""The work whose speed this repository is judged by, through its public entry points.

Each case is one of these kinds (the sizes are the case's other fields):

  image   Renderer.get_camera_image of one frame from host models: the reference's own call and its first example
          (a cube at 640x480), or a ground plane with objects and the light-space shadow pass
  frames  Renderer.get_camera_image with a leading axis of frames (the reference notebooks' jax.vmap over it): articulated
          capsules over a textured ground, host arrays in, shadows on
  serve   the notebooks' loop with the meshes kept on the device: new transforms from pinned memory, DeviceMerge.merge,
          BatchRunner.replay, display_u8
  scenes  BatchRunner.replay of many Brax-like scenes (ground plus 8..32 boxes, spheres and capsules), with the depth pass;
          `layers` > 0 blends that many of the nearest candidates (the compiled chooser / mix hooks)
  step    the same with gradients: replay, then backward_mse against a target image
  mixed   MultiRunner.replay of scenes of several resolutions and of triangle counts from `low` to `high`
  fit     inverse rendering: DifferentiableBatch.render of displaced spheres, a loss in torch, backward to positions,
          textures, camera position and light
  render  pipeline.render of one large mesh whose arrays are on the device already

Everything is made from the seed here; the exact values are plain torch in 64 bits.
"""
import math

import numpy as np
import torch

import jaxrenderer_gb300 as jr
from jaxrenderer_gb300 import _lib, autograd, batch, instancing, shaders, utils
from jaxrenderer_gb300.jobs import JobSpec

F32 = np.float32
F64 = torch.float64
SHADERS = ("gouraud", "gouraud_texture", "phong", "phong_darboux")


def listed():
    return [
        # the first example of the reference: one cube, one 640x480 image, no shadow
        dict(name="image_cube_640x480", kind="image", objects=0, width=640, height=480, shadow=False),
        # one frame of a furnished scene with its shadow, models on the host
        dict(name="image_scene_320x240", kind="image", objects=12, width=320, height=240, shadow=True),
        # the notebooks' benchmark call: 200 frames of an articulated body at 84x84 from host arrays
        dict(name="frames_84x84_x200", kind="frames", frames=200, width=84, height=84),
        # the same rate of frames in a loop that keeps its meshes on the device and shows uint8 images
        dict(name="serve_84x84_x200", kind="serve", scenes=200, width=84, height=84, shadow=84),
        # a large batch of observations for reinforcement learning (the benchmark's default workload)
        dict(name="scenes_84x84_x4096", kind="scenes", scenes=4096, width=84, height=84, shadow=128, layers=0),
        # a small batch, where launches and gaps count
        dict(name="scenes_84x84_x16", kind="scenes", scenes=16, width=84, height=84, shadow=128, layers=0),
        # transparency: the four nearest candidates of every pixel blended front to back
        dict(name="glass_84x84_x1024", kind="scenes", scenes=1024, width=84, height=84, shadow=128, layers=4),
        # learning through the renderer: forward and backward of a batch against target images
        dict(name="step_84x84_x1024", kind="step", scenes=1024, width=84, height=84, shadow=128),
        # scenes of uneven triangle counts at three resolutions in one call
        dict(name="mixed_x96", kind="mixed", scenes=96, low=100, high=100000),
        # inverse rendering of textured spheres with autograd
        dict(name="fit_phong_128x128_x256", kind="fit", shader="phong", scenes=256, level=4, width=128, height=128),
        # the same at odd sizes and a small batch with lighting per vertex
        dict(name="fit_gouraud_97x61_x24", kind="fit", shader="gouraud_texture", scenes=24, level=3, width=97, height=61),
        # one large frame with much overdraw (389,120 triangles)
        dict(name="render_960x540_389k", kind="render", shader="gouraud_texture", spheres=76, level=4, width=960, height=540),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("image", "frames", "serve", "scenes", "scenes", "step", "step", "mixed", "fit", "fit", "render", "render"))
    w, h = rng.choice(((84, 84), (_log(rng, 24, 200), _log(rng, 24, 200))))
    if kind == "image":
        return dict(kind=kind, objects=rng.randint(0, 16), width=_log(rng, 48, 640), height=_log(rng, 48, 480), shadow=rng.random() < 0.6)
    if kind == "frames":
        return dict(kind=kind, frames=_log(rng, 8, 200), width=min(w, 120), height=min(h, 120))
    if kind == "serve":
        return dict(kind=kind, scenes=_log(rng, 8, 1500), width=w, height=h, shadow=rng.choice((64, 84, 128)))
    if kind == "scenes":
        n = _log(rng, 1, 4000)
        layers = rng.choice((0, 0, 0, 2, 4))
        return dict(kind=kind, scenes=n if w * h <= 7056 and not layers else max(1, min(n, 10_000_000 // (w * h))),
                    width=w, height=h, shadow=rng.choice((0, 64, 101, 128)), layers=layers)
    if kind == "step":
        return dict(kind=kind, scenes=max(1, min(_log(rng, 2, 1024), 7_000_000 // (w * h))), width=w, height=h, shadow=rng.choice((0, 64, 128)))
    if kind == "mixed":
        low = _log(rng, 50, 1000)
        return dict(kind=kind, scenes=_log(rng, 6, 96), low=low, high=_log(rng, 4 * low, 100000))
    if kind == "fit":
        level = rng.randint(2, 4)
        return dict(kind=kind, shader=rng.choice(("phong", "gouraud", "gouraud_texture")), scenes=_log(rng, 1, 256), level=level,
                    width=_log(rng, 32, 128), height=_log(rng, 32, 128))
    return dict(kind=kind, shader=rng.choice(SHADERS), spheres=_log(rng, 1, 70), level=rng.randint(2, 4),
                width=_log(rng, 96, 960), height=_log(rng, 64, 540))


# ------------------------------------------------------------------- meshes

def _icosphere(level):
    if level not in _SPHERES:
        g = (1 + 5 ** 0.5) / 2
        v = np.array([(-1, g, 0), (1, g, 0), (-1, -g, 0), (1, -g, 0), (0, -1, g), (0, 1, g), (0, -1, -g), (0, 1, -g),
                      (g, 0, -1), (g, 0, 1), (-g, 0, -1), (-g, 0, 1)], np.float64)
        f = np.array([(0, 11, 5), (0, 5, 1), (0, 1, 7), (0, 7, 10), (0, 10, 11), (1, 5, 9), (5, 11, 4), (11, 10, 2), (10, 7, 6), (7, 1, 8),
                      (3, 9, 4), (3, 4, 2), (3, 2, 6), (3, 6, 8), (3, 8, 9), (4, 9, 5), (2, 4, 11), (6, 2, 10), (8, 6, 7), (9, 8, 1)])
        v /= np.linalg.norm(v, axis=1, keepdims=True)
        for _ in range(level):
            edges = np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]), axis=1)
            uniq, at = np.unique(edges, axis=0, return_inverse=True)
            m = v[uniq].sum(1)
            mid = (at.reshape(3, -1) + len(v)).T  # the middles of edges ab, bc, ca
            v = np.concatenate([v, m / np.linalg.norm(m, axis=1, keepdims=True)])
            a, b, c = f.T
            f = np.concatenate([np.stack([a, mid[:, 0], mid[:, 2]], 1), np.stack([b, mid[:, 1], mid[:, 0]], 1),
                                np.stack([c, mid[:, 2], mid[:, 1]], 1), mid])
        uv = np.stack([0.5 + np.arctan2(v[:, 1], v[:, 0]) / (2 * np.pi), 0.5 + np.arcsin(np.clip(v[:, 2], -1, 1)) / np.pi], 1)
        _SPHERES[level] = (v.astype(F32), uv.astype(F32), f.astype(np.int32))
    return _SPHERES[level]


_SPHERES = {}


def _capsule(segments, rings, radius, half):
    """(vertices, normals, uvs, faces) of a capsule along z."""
    lat = [(np.pi / 2 * r / rings, half) for r in range(rings + 1)] + [(np.pi / 2 * (1 + r / rings), -half) for r in range(rings + 1)]
    n = np.array([(np.sin(t) * np.cos(p), np.sin(t) * np.sin(p), np.cos(t)) for t, _ in lat for p in 2 * np.pi * np.arange(segments) / segments])
    v = n * radius + np.repeat([(0, 0, z) for _, z in lat], segments, axis=0)
    faces = []
    for r in range(len(lat) - 1):
        for s in range(segments):
            a, b = r * segments + s, r * segments + (s + 1) % segments
            c, d = a + segments, b + segments
            faces += [(a, c, d)] if r == 0 else [(a, c, b)] if r == len(lat) - 2 else [(a, c, d), (a, d, b)]
    uv = np.stack([np.tile(np.arange(segments) / segments, len(lat)), np.repeat(np.arange(len(lat)) / len(lat), segments)], 1)
    return v.astype(F32), n.astype(F32), uv.astype(F32), np.array(faces, np.int32)


def _model(v, n, uv, f, diffuse, specular):
    return jr.Model(v, n, uv, f, f, f, diffuse, specular)


def _plane(half, diffuse, specular):
    v = np.array([(-half, -half, 0), (half, -half, 0), (half, half, 0), (-half, half, 0)], F32)
    return _model(v, np.tile(np.array([(0, 0, 1)], F32), (4, 1)), np.array([(0, 0), (4, 0), (4, 4), (0, 4)], F32),
                  np.array([(0, 1, 2), (0, 2, 3)], np.int32), diffuse, specular)


def _parts():
    """The plane and the three shapes that furnish a scene: 2, 12, 320 and 512 triangles."""
    if not _PARTS:
        tex, spec = np.zeros((4, 4, 3), F32), np.full((4, 4), 2.0, F32)
        v, uv, f = _icosphere(2)
        _PARTS.extend([_plane(5.0, tex, spec), jr.create_cube(np.full(3, 0.5, F32), np.ones(2, F32), tex, spec),
                       _model(v * F32(0.5), v, uv, f, tex, spec), _model(*_capsule(16, 8, 0.4, 0.2), tex, spec)])
    return _PARTS


_PARTS = []


def _rotations(rng, n):
    q = rng.normal(size=(n, 4))
    w, x, y, z = (q / np.linalg.norm(q, axis=1, keepdims=True)).T
    return np.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y), 2 * (x * y + w * z), 1 - 2 * (x * x + z * z),
                     2 * (y * z - w * x), 2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).reshape(n, 3, 3)


def _furnished(rng, scenes, least, most):
    """Arrays of `scenes` scenes: a ground plane, then `least` to `most` objects each.  What the scenes hold goes by their number, so
    that arrays keep their sizes; where it is, its colours and the cameras go by `rng`."""
    own = np.random.default_rng(scenes)
    counts = own.integers(least, most + 1, scenes)
    n = int(counts.sum()) + scenes
    begin = np.concatenate([[0], np.cumsum(counts + 1)]).astype(np.int64)
    obj = np.ones(n, bool)
    obj[begin[:-1]] = False
    k = n - scenes
    mesh = np.zeros(n, np.int32)
    mesh[obj] = own.integers(1, 4, k)
    tr = np.tile(np.identity(4, F32), (n, 1, 1))
    tr[obj, :3, :3] = _rotations(rng, k)
    tr[obj, :3, 3] = rng.uniform((-3, -3, 0), (3, 3, 2), (k, 3))
    scale = np.ones((n, 3), F32)
    scale[obj] = rng.uniform(0.2, 1.0, (k, 1))
    colour = rng.uniform(0, 1, (n, 3)).astype(F32)
    e, a = np.deg2rad(rng.uniform(20, 60, scenes)), rng.uniform(0, 2 * np.pi, scenes)
    cam = 6 * np.stack([np.cos(e) * np.cos(a), np.cos(e) * np.sin(a), np.sin(e)], 1)
    return dict(models=_parts(), mesh=mesh, begin=begin, tr=tr, scale=scale, colour=colour, cam=cam.astype(F32))


def _brax_like(case, seed):
    return _furnished(np.random.default_rng([seed, 11]), case["scenes"], 8, 32)


def _instanced(d):
    n = len(d["mesh"])
    tex = np.broadcast_to(d["colour"][:, None, None, :], (n, 4, 4, 3)).copy()
    return instancing.InstancedScenes(instancing.MeshLibrary.from_models(d["models"]), d["mesh"], d["begin"], d["tr"], d["scale"], tex,
                                      np.full((n, 4, 4), 2.0, F32), d["cam"])


def _scene_batch(case, d):
    s = case["shadow"]
    sb, merge = batch.scene_batch_from_instances(_instanced(d), case["width"], case["height"],
                                                 shadow_param=jr.ShadowParameters() if s else None, shadow_size=(s or 1, s or 1))
    if case.get("layers"):
        batch.set_layers(sb, case["layers"], mixer=_lib.MIX_OVER, opacity=0.6, background=(0.55, 0.7, 0.9))
    return sb, merge


def _target(shape, seed):
    """Smooth images in [0, 1]."""
    n, w, h, c = shape
    g = torch.Generator(device="cuda").manual_seed(seed)
    f, p = torch.rand((n, 1, 1, c), generator=g, device="cuda"), torch.rand((n, 1, 1, c), generator=g, device="cuda")
    x, y = torch.arange(w, device="cuda").view(1, w, 1, 1) / w, torch.arange(h, device="cuda").view(1, 1, h, 1) / h
    return 0.5 + 0.4 * torch.sin(6.3 * (f * x + (1 - f) * y + p))


# ----------------------------------------------------------------- per kind

def _image_objects(case, seed):
    rng = np.random.default_rng([seed, 12])
    if not case["objects"]:  # the cube of the first example, its colour and the camera from the seed
        tex = np.broadcast_to(rng.uniform(0, 1, 3).astype(F32), (2, 2, 3)).copy()
        d = dict(models=[jr.create_cube(np.ones(3, F32), np.ones(2, F32), tex, np.full((2, 2), 2.0, F32))], mesh=np.zeros(1, np.int32),
                 begin=np.array([0, 1]), tr=np.identity(4, F32)[None], scale=np.ones((1, 3), F32), colour=tex[:1, 0],
                 cam=(np.array([[2.0, 4.0, 1.0]]) + rng.uniform(-0.3, 0.3, (1, 3))).astype(F32))
    else:
        d = _furnished(rng, 1, case["objects"], case["objects"])
    size = 2 if not case["objects"] else 4
    objects = []
    for i, m in enumerate(d["mesh"]):
        tex = np.broadcast_to(d["colour"][i], (size, size, 3)).copy()
        objects.append(jr.ModelObject(model=d["models"][m]._replace(diffuse_map=tex), local_scaling=d["scale"][i], transform=d["tr"][i]))
    return d, objects


def _prepare_image(case, seed):
    d, objects = _image_objects(case, seed)
    camera = jr.CameraParameters(viewWidth=case["width"], viewHeight=case["height"], position=d["cam"][0])
    shadow = jr.ShadowParameters() if case["shadow"] else None

    def go():
        return jr.Renderer.get_camera_image(objects, jr.LightParameters(), camera, case["width"], case["height"], shadow_param=shadow)
    return go


def _body(case, seed):
    """Frames of a ground box and 17 capsules that move around a drifting centre."""
    rng, n = np.random.default_rng([seed, 13]), case["frames"]
    check = ((np.indices((100, 100)).sum(0) // 10) % 2)[..., None].astype(F32)
    models = [jr.create_cube(np.array((1000.0, 1000.0, 1e-4), F32), np.full(2, 10.0, F32), (0.25 + 0.4 * check * np.array((1, 0.8, 0.6))).astype(F32),
                             np.full((1, 1), 2.0, F32))]
    for _ in range(17):
        v = _capsule(8, 6, rng.uniform(0.06, 0.12), rng.uniform(0.05, 0.13))
        models.append(_model(*v, rng.uniform(0.2, 0.6, (1, 1, 3)).astype(F32), np.full((1, 1), 2.0, F32)))
    centre = np.cumsum(rng.normal(0, 0.05, (n, 3)) * (1, 1, 0), axis=0).astype(F32)
    tr = np.tile(np.identity(4, F32), (18, n, 1, 1))
    for k in range(1, 18):
        tr[k, :, :3, :3] = _rotations(rng, n)
        tr[k, :, :3, 3] = centre + rng.normal(0, 0.35, (n, 3)) * (1, 1, 0.3)
        tr[k, :, 2, 3] = np.abs(tr[k, :, 2, 3]) + 0.2
    a = np.linspace(0, np.pi / 2, n) + rng.uniform(0, 2 * np.pi)
    return models, tr, centre, (centre + np.stack([3.7 * np.cos(a), 3.7 * np.sin(a), np.full(n, 1.9)], 1)).astype(F32)


_BODY_LIGHT = jr.LightParameters(direction=np.array((0.57735, -0.57735, 0.57735), F32), ambient=np.full(3, 0.8, F32), diffuse=np.full(3, 0.8, F32),
                                 specular=np.full(3, 0.6, F32))


def _prepare_frames(case, seed):
    models, tr, centre, pos = _body(case, seed)
    n = case["frames"]

    def every(a):
        return np.broadcast_to(np.asarray(a), (n,) + np.asarray(a).shape).copy()
    objects = [jr.ModelObject(model=jr.Model(*(every(x) for x in m)), local_scaling=every(np.ones(3, F32)), transform=tr[k],
                              double_sided=np.zeros(n, bool)) for k, m in enumerate(models)]
    camera = jr.CameraParameters(viewWidth=every(np.int32(960)), viewHeight=every(np.int32(540)), viewDepth=every(F32(1)), near=every(F32(0.01)),
                                 far=every(F32(1000)), hfov=every(F32(58)), vfov=every(F32(32.625)), position=pos, target=centre,
                                 up=every(np.array((0, 0, 1), F32)))

    def go():
        return jr.Renderer.get_camera_image(objects, _BODY_LIGHT, camera, case["width"], case["height"],
                                            shadow_param=jr.ShadowParameters(centre=centre))
    return go


def _prepare_serve(case, seed):
    d = _brax_like(case, seed)
    sb, merge = _scene_batch(case, d)
    runner = batch.BatchRunner(sb, form="tiled", want_prim_id=False)
    runner.capture()
    tr, scale = torch.from_numpy(d["tr"]).pin_memory(), torch.from_numpy(d["scale"]).pin_memory()
    shown = torch.empty((case["scenes"], case["height"], case["width"], 3), dtype=torch.uint8, device="cuda")

    def go():
        merge.merge(tr, scale)
        out = runner.replay()
        return {"canvas": out.canvas, "shown": utils.display_u8(out.canvas, out=shown), "position": sb.pools["position"], "normal": sb.pools["normal"]}
    return go


def _outputs(out):
    got = {"canvas": out.canvas, "zbuffer": out.zbuffer, "prim_id": out.prim_id}
    if out.shadow_map is not None:
        got["shadow_map"] = out.shadow_map
    return got


def _prepare_scenes(case, seed):
    sb, _ = _scene_batch(case, _brax_like(case, seed))
    runner = batch.BatchRunner(sb, form="tiled")
    runner.capture()
    return lambda: _outputs(runner.replay())


def _prepare_step(case, seed):
    sb, _ = _scene_batch(case, _brax_like(case, seed))
    runner = batch.BatchRunner(sb, form="tiled")
    runner.capture()
    target, grads = _target(tuple(runner.canvas.shape), seed), runner.grad_buffers()

    def go():
        out = _outputs(runner.replay())
        return {**out, "grads": runner.backward_mse(target, out=grads)}
    return go


_CLASSES = ((32, 32), (84, 84), (480, 270))


def _cubes(case, seed):
    """Per resolution class: scenes of randomly placed cubes, triangle counts log-uniform."""
    rng, n = np.random.default_rng([seed, 14]), case["scenes"]
    own = np.random.default_rng(n)  # the scenes' sizes go by their number, what they look like by the seed
    count = np.maximum(1, np.round(np.exp(np.log(case["low"]) + np.log(case["high"] / case["low"]) * (np.arange(n) + own.uniform(0, 1, n)) / n) / 12)).astype(np.int64)
    which = np.arange(n) % 3
    shadow = own.random(n) < 0.5
    got = []
    for c, (w, h) in enumerate(_CLASSES):
        m = count[which == c]
        begin, k = np.concatenate([[0], np.cumsum(m)]), int(m.sum())
        if not k:
            continue
        half = 1.5 * np.repeat(m, m) ** (1 / 3)
        tr = np.tile(np.identity(4, F32), (k, 1, 1))
        tr[:, :3, :3] = _rotations(rng, k)
        tr[:, :3, 3] = rng.uniform(-1, 1, (k, 3)) * half[:, None]
        to = rng.normal(size=(len(m), 3))
        to[:, 2] = np.abs(to[:, 2]) + 0.3
        cam = 4.8 * (m ** (1 / 3))[:, None] * to / np.linalg.norm(to, axis=1, keepdims=True)
        cube = jr.create_cube(np.ones(3, F32), np.ones(2, F32), np.zeros((4, 4, 3), F32), np.full((4, 4), 2.0, F32))
        got.append(dict(models=[cube], mesh=np.zeros(k, np.int32), begin=begin, tr=tr, scale=np.repeat(rng.uniform(0.3, 0.8, (k, 1)), 3, 1).astype(F32),
                        colour=rng.uniform(0, 1, (k, 3)).astype(F32), cam=cam.astype(F32), size=(w, h), mask=shadow[which == c]))
    return got


def _prepare_mixed(case, seed):
    groups = [batch.scene_batch_from_instances(_instanced(d), *d["size"], shadow_size=d["size"], shadow_mask=d["mask"])[0] for d in _cubes(case, seed)]
    runner = batch.MultiRunner(groups)
    runner.capture()
    return lambda: [dict(canvas=o.canvas, zbuffer=o.zbuffer, prim_id=o.prim_id) for o in runner.replay()]


def _fit_arrays(case, seed):
    rng, n = np.random.default_rng([seed, 15]), case["scenes"]
    v, uv, f = _icosphere(case["level"])
    light = rng.normal(size=(n, 3))
    light[:, 2] = np.abs(light[:, 2]) + 0.5
    eye = rng.normal(size=(n, 3))
    return dict(position=(v * (1 + rng.normal(0, 0.05, (n, len(v), 1)))).astype(F32), normal=v, uv=uv * F32(64), faces=f,
                colour=rng.uniform(0, 1, (n, len(v), 3)).astype(F32), texture=rng.uniform(0, 1, (n, 64, 64, 3)).astype(F32),
                light=(light / np.linalg.norm(light, axis=1, keepdims=True)).astype(F32),
                eye=(4 * eye / np.linalg.norm(eye, axis=1, keepdims=True)).astype(F32))


def _fit_camera(case):
    return jr.CameraParameters(viewWidth=case["width"], viewHeight=case["height"], near=0.1, far=100.0, hfov=40.0, vfov=40.0)


def _prepare_fit(case, seed):
    a, params, n = _fit_arrays(case, seed), _fit_camera(case), case["scenes"]
    textured = case["shader"] != "gouraud"
    specs = []
    for k in range(n):
        cam = jr.Renderer.create_camera_from_parameters(params._replace(position=a["eye"][k]))
        s = JobSpec(shader=getattr(_lib, "SHADER_" + case["shader"].upper()), width=case["width"], height=case["height"], viewport=cam.viewport,
                    world_to_clip=cam.world_to_clip, world_to_eye_norm=cam.world_to_eye_norm, position=a["position"][k], faces=a["faces"])
        s.normal, s.light_direction = a["normal"], a["light"][k]
        if textured:
            s.uv, s.texture = a["uv"], a["texture"][k]
        else:
            s.colour = a["colour"][k]
        specs.append(s)
    db = autograd.DifferentiableBatch(batch.scene_batch_from_specs(specs))

    def leaf(x):
        return torch.from_numpy(np.ascontiguousarray(x)).cuda().requires_grad_()
    leaves = {"position": leaf(a["position"].reshape(-1, 3)), "light": leaf(a["light"]), "eye": leaf(a["eye"])}
    other = "texture" if textured else "colour"
    leaves[other] = leaf(a[other].reshape(-1, 3))
    target = _target((n, case["width"], case["height"], 3), seed)
    centre, up = torch.zeros(3, device="cuda"), torch.tensor((0.0, 0.0, 1.0), device="cuda")

    def go():
        for t in leaves.values():
            t.grad = None
        w2c, w2e, _ = autograd.camera_matrices(leaves["eye"], params, centre, up)
        canvas, zbuffer = db.render(position=leaves["position"], world_to_clip=w2c, world_to_eye_norm=w2e, light_direction=leaves["light"],
                                    **{other: leaves[other]})
        ((canvas - target) ** 2).mean().backward()
        return {"canvas": canvas.detach(), "zbuffer": zbuffer.detach(), **{k: t.grad for k, t in leaves.items()}}
    return go


def _render_arrays(case, seed):
    """Spheres at random overlapping places in front of a camera at z = 9, and a few exact copies."""
    rng, n = np.random.default_rng([seed, 16]), case["spheres"]
    v, uv, f = _icosphere(case["level"])
    c, r = rng.uniform((-2.2, -1.2, -1.5), (2.2, 1.2, 1.5), (n, 3)), rng.uniform(2.2, 3.6, n) * min(1.0, (n / 16) ** 0.25)
    for k in range(16, n, 16):
        c[k], r[k] = c[k - 4], r[k - 4]
    light = rng.normal(size=3)
    light[2] = abs(light[2])
    size = 512 if n > 16 else 64
    ids = np.full(len(v), 0, np.int32)
    ids[f[::-1].reshape(-1)] = np.repeat(np.arange(len(f), dtype=np.int32)[::-1], 3)
    return dict(position=(v[None] * r[:, None, None] + c[:, None]).reshape(-1, 3).astype(F32), normal=np.tile(v, (n, 1)),
                uv=(uv[None] * (size * rng.uniform(0.5, 2.0, (n, 1, 1)))).reshape(-1, 2).astype(F32),
                faces=(f[None] + (np.arange(n) * len(v))[:, None, None]).reshape(-1, 3).astype(np.int32),
                ids=(ids[None] + (np.arange(n, dtype=np.int32) * len(f))[:, None]).reshape(-1),
                colour=rng.uniform(0, 1, (n * len(v), 3)).astype(F32), texture=rng.uniform(0, 1, (size, size, 3)).astype(F32),
                normal_map=(rng.normal(0, 0.2, (size, size, 3)) + (0, 0, 1)).astype(F32), light=(light / np.linalg.norm(light)).astype(F32))


def _prepare_render(case, seed):
    a, w, h = {k: torch.from_numpy(x).cuda() if k != "light" else x for k, x in _render_arrays(case, seed).items()}, case["width"], case["height"]
    cam = jr.Camera.create(jr.Camera.view_matrix(np.array((0, 0, 9), F32), np.zeros(3, F32), np.array((0, 1, 0), F32)),
                           jr.Camera.perspective_projection_matrix(45.0, w / h, 0.1, 100.0),
                           jr.Camera.viewport_matrix(np.zeros(2, np.int32), np.array((w, h)), 1.0))
    light = jr.LightSource(direction=a["light"], colour=np.ones(3, F32))
    if case["shader"] == "gouraud":
        shader, extra = shaders.gouraud.GouraudShader, shaders.gouraud.GouraudExtraInput(a["position"], a["colour"], a["normal"], light)
    elif case["shader"] == "phong_darboux":
        shader = shaders.phong_darboux.PhongTextureDarbouxShader
        extra = shader.extra_input(a["position"], a["normal"], a["uv"], light, a["texture"], a["normal_map"], a["ids"], a["faces"])
    else:
        shader = shaders.phong.PhongTextureShader if case["shader"] == "phong" else shaders.gouraud_texture.GouraudTextureShader
        extra = shader.extra_input(position=a["position"], normal=a["normal"], uv=a["uv"], light=light, texture=a["texture"])
    buffers = jr.Renderer.create_buffers(w, h)

    def go():
        out = jr.render(cam, shader, buffers, a["faces"], extra)
        return {"canvas": out.targets[0], "zbuffer": out.zbuffer}
    return go


_PREPARE = dict(image=_prepare_image, frames=_prepare_frames, serve=_prepare_serve, scenes=_prepare_scenes, step=_prepare_step, mixed=_prepare_mixed,
                fit=_prepare_fit, render=_prepare_render)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state()


# --------------------------------------------------------------------- work

def work(case):
    """Positions read once in each pass, the outputs written once; about 150 operations a triangle and pass, 250 a pixel."""
    k = case["kind"]
    px = case.get("width", 0) * case.get("height", 0)
    if k == "image":
        faces, maps, out = (12 if not case["objects"] else 2 + 281 * case["objects"]), px * 4 * bool(case["shadow"]), px * 12
        passes = 2 if case["shadow"] else 1
    elif k == "frames":
        faces, maps, passes, out = case["frames"] * 3276, case["frames"] * px * 4, 2, case["frames"] * px * 12
        px *= case["frames"]
    elif k in ("serve", "scenes", "step"):
        n = case["scenes"]
        faces, maps, passes = n * 5628, n * case["shadow"] ** 2 * 4, 2 if case["shadow"] else 1
        px *= n
        out = px * (20 + 16 * bool(case.get("layers")))
        if k == "serve":  # every corner's position, normal, uv and texture index are written, and the shown images
            out = px * 15 + faces * 108
        if k == "step":  # gradients of positions and normals, the target read
            out += faces * 72 + px * 12
    elif k == "mixed":
        px = case["scenes"] / 3 * sum(w * h for w, h in _CLASSES)
        faces = case["scenes"] * (case["high"] - case["low"]) / math.log(case["high"] / case["low"])
        maps, passes, out = px * 2, 1.5, px * 20
    else:
        n = case["scenes"] if k == "fit" else case["spheres"]
        faces, maps, passes = n * 20 * 4 ** case["level"], 0, 1
        if k == "fit":
            px *= n
            out = px * (16 + 12) + n * (10 * 4 ** case["level"] * 12 + (64 * 64 * 12 if case["shader"] != "gouraud" else 0))
        else:
            out = px * 16
        faces /= 3  # shared vertices: a third of the corners
    return {"bytes": faces * 36 * passes + maps + out, "flops": 150 * faces * passes + 250 * px * (3 if k in ("step", "fit") else 1)}


# ------------------------------------------------- exact values, in 64 bits

def _t(x):
    return torch.as_tensor(np.asarray(x)).cuda().to(F64)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _look_at(eye, centre, up):
    f = _unit(centre - eye)
    s = _unit(torch.linalg.cross(f, _unit(up).expand_as(f), dim=-1))
    u = torch.linalg.cross(s, f, dim=-1)
    rot = torch.stack([s, u, -f], -2)
    top = torch.cat([rot, -(rot @ eye[..., None])], -1)
    return torch.cat([top, top.new_tensor((0.0, 0, 0, 1)).expand_as(top[..., :1, :])], -2)


def _perspective(vfov, aspect, near, far):
    f = 1 / math.tan(math.radians(vfov) / 2)
    return _t([[f / aspect, 0, 0, 0], [0, f, 0, 0], [0, 0, (far + near) / (near - far), 2 * far * near / (near - far)], [0, 0, -1, 0]])


def _light_view(direction, centre):
    box = _t([[1, 0, 0, 0], [0, 1, 0, 0], [0, 0, -1, 0], [0, 0, 0, 1]])
    return box @ _look_at(centre + 10 * direction, centre, _t((0, 0, 1)))


def _homogeneous(p):
    return torch.cat([p, torch.ones_like(p[..., :1])], -1)


def _grid(size, view):
    """The pixels' NDC coordinates [x, y, 1] for a viewport of `view` pixels."""
    w, h = size
    x = (torch.arange(w, device="cuda", dtype=F64) - view[0] / 2) / (view[0] / 2)
    y = (torch.arange(h, device="cuda", dtype=F64) - view[1] / 2) / (view[1] / 2)
    return torch.stack([x[:, None].expand(w, h), y[None].expand(w, h), torch.ones((w, h), device="cuda", dtype=F64)], -1).reshape(-1, 3)


def _inverse(rows):
    """Of (..., 3, 3) matrices of [x, y, w] rows, with their determinants."""
    a, b, c = rows.unbind(-2)
    adj = torch.stack([torch.linalg.cross(b, c, dim=-1), torch.linalg.cross(c, a, dim=-1), torch.linalg.cross(a, b, dim=-1)], -1)
    det = (a * adj[..., 0]).sum(-1)
    return adj / det[..., None, None], det


@torch.no_grad()
def _nearest(clip, grid, slots=1):
    """(slots, pixels) of the nearest front faces' indices (-1: none) and depths for clip positions (F, 3, 4)."""
    inv, det = _inverse(clip[..., [0, 1, 3]])
    ids = torch.nonzero((det > 1e-6) & torch.isfinite(inv).flatten(1).all(1)).flatten()
    inv, zc, n = inv[ids], clip[ids, :, 2], len(grid)
    best = torch.full((slots, n), math.inf, device="cuda", dtype=F64)
    face = torch.full((slots, n), -1, device="cuda")
    step = max(1, 60_000_000 // n)
    for at in range(0, len(ids), step):
        m, z = inv[at : at + step], zc[at : at + step]
        inside = (grid @ m[:, :, 0].T >= 0) & (grid @ m[:, :, 1].T >= 0) & (grid @ m[:, :, 2].T >= 0)
        depth = torch.where(inside, 0.5 * (grid @ (m @ z[..., None])[..., 0].T) + 0.5, math.inf)
        for _ in range(slots):
            d, k = depth.min(1)
            if slots > 1:
                depth.scatter_(1, k[:, None], math.inf)
            both, own = torch.cat([best, d[None]]), torch.cat([face, ids[at + k][None]])
            order = both.argsort(dim=0, stable=True)[:slots]
            best, face = both.gather(0, order), own.gather(0, order)
    return torch.where(torch.isinf(best), -1, face), best


def _barycentric(clip, grid):
    """Depths and perspective-correct weights of the pixels' own faces (P, 3, 4)."""
    c = (grid[:, None] @ _inverse(clip[..., [0, 1, 3]])[0])[:, 0]
    return 0.5 * (c * clip[..., 2]).sum(-1) + 0.5, c / c.sum(-1, keepdim=True)


def _mix(b, v):
    return (b[..., None] * v).sum(-2)


def _depth_map(pos, faces, w2c, size, view, offset=0.05):
    """The light's view of the faces, plus the offset."""
    face, z = _nearest((_homogeneous(pos) @ w2c.T)[faces], _grid(size, view))
    return torch.where(face[0] >= 0, z[0], float(np.finfo(F32).max)).view(size) + offset


class _Lit:
    """One scene of the Phong-reflection shader: its inputs in 64 bits (tensors that may want gradients)."""

    def __init__(self, pos, nrm, uv, tix, texture, specular, shapes, period, light, w2c, w2e, dir_eye):
        self.pos, self.nrm, self.uv, self.tix, self.texture, self.specular = pos, nrm, uv, tix, texture, specular
        self.shapes, self.period, self.w2c, self.w2e, self.dir_eye = shapes, period, w2c, w2e, dir_eye
        self.ambient, self.diffuse, self.specular_c, self.colour = (_t(x) for x in (light.ambient, light.diffuse, light.specular, light.colour))
        self.strength, self.shadow = _t(jr.ShadowParameters().strength), None

    def shade(self, face, grid):
        """(depth, colour) of the pixels `grid` from their faces."""
        at = 3 * face[:, None] + torch.arange(3, device="cuda")
        p, tix = self.pos[at], self.tix[3 * face]
        z, b = _barycentric(_homogeneous(p) @ self.w2c.T, grid)
        n = _unit(_mix(b, _unit(_unit(self.nrm[at]) @ self.w2e[:3, :3].T)))
        uv = _mix(b, self.uv[at]).detach()
        frac = uv - uv.trunc()
        uv = torch.where(frac < 0, frac + 1, frac) * self.shapes[tix]
        u = (uv[:, 0] + tix * self.period).floor().long().clamp(0, self.texture.shape[0] - 1)
        v = uv[:, 1].floor().long().clamp(0, self.texture.shape[1] - 1)
        tex, power = self.texture[u, v], self.specular[u.clamp(max=self.specular.shape[0] - 1), v.clamp(max=self.specular.shape[1] - 1)]
        light = _unit(self.dir_eye)
        d = n @ light
        shine = _unit(2 * d[:, None] * n - light)[:, 2].clamp(min=0)
        shine = torch.where(shine > 0, shine.clamp(min=1e-300) ** power, torch.where(power == 0, 1.0, 0.0))
        k = self.diffuse * d.clamp(min=0)[:, None] + self.specular_c * shine[:, None]
        if self.shadow is not None:
            depth, lw2c, view = self.shadow
            s = _homogeneous(p) @ lw2c.T
            s = _mix(b, s / s[..., 3:]).detach()
            s = s / s[:, 3:]
            at = torch.stack([s[:, 0] * view[0] / 2 + view[0] / 2, s[:, 1] * view[1] / 2 + view[1] / 2], 1)
            i, j = (at.sign() * (at.abs() + 0.5).floor()).long().unbind(1)
            i, j = torch.where(i < 0, i + depth.shape[0], i), torch.where(j < 0, j + depth.shape[1], j)
            seen = (i >= 0) & (i < depth.shape[0]) & (j >= 0) & (j < depth.shape[1])
            far = depth[i.clamp(0, depth.shape[0] - 1), j.clamp(0, depth.shape[1] - 1)]
            lit = ~seen | (0.5 * s[:, 2] + 0.5 <= far)
            k = k * torch.where(lit[:, None], 1.0, 1 - self.strength)
        return z, self.ambient * tex + k * self.colour * tex

    def image(self, size, view, over=0):
        """(canvas, depths) over white, or with `over` candidates blended."""
        grid = _grid(size, view)
        face, _ = _nearest(_homogeneous(self.pos.detach()).view(-1, 3, 3 + 1) @ self.w2c.detach().T, grid, max(over, 1))
        canvas, depth = torch.ones((len(grid), 3), device="cuda", dtype=F64), torch.ones(len(grid), device="cuda", dtype=F64)
        if not over:
            hit = torch.nonzero(face[0] >= 0).flatten()
            z, c = self.shade(face[0][hit], grid[hit])
            return canvas.index_put((hit,), c).view(*size, 3), depth.index_put((hit,), z).view(size)
        left, mixed = torch.ones_like(depth), torch.zeros_like(canvas)
        for s in range(over):
            hit = torch.nonzero(face[s] >= 0).flatten()
            z, c = self.shade(face[s][hit], grid[hit])
            if s == 0:
                depth[hit] = z
            mixed[hit] += 0.6 * left[hit, None] * c
            left[hit] *= 0.4
        some = (face[0] >= 0)[:, None]
        return torch.where(some, mixed + left[:, None] * _t((0.55, 0.7, 0.9)), canvas).view(*size, 3), depth.view(size)


def _merged(d, s):
    """(positions, normals, uvs, object of each corner, faces' own positions) of scene s, per face corner."""
    pos, nrm, uv, tix = [], [], [], []
    for k, i in enumerate(range(int(d["begin"][s]), int(d["begin"][s + 1]))):
        m, tr = d["models"][int(d["mesh"][i])], d["tr64"][i]
        key = id(m)
        if key not in d["meshes"]:
            f = torch.as_tensor(np.asarray(m.faces).reshape(-1)).cuda().long()
            n = _t(m.norms)
            d["meshes"][key] = (_t(m.verts), n / n.norm(), _t(m.uvs)[f], f)
        v, n, u, f = d["meshes"][key]
        p = _homogeneous(v * d["scale64"][i]) @ tr.T
        n = n @ torch.linalg.inv(tr)[:3, :3]
        pos.append((p[:, :3] / p[:, 3:])[f])
        nrm.append((n / n.norm())[f])
        uv.append(u)
        tix.append(torch.full((len(f),), k, device="cuda"))
    return torch.cat(pos), torch.cat(nrm), torch.cat(uv), torch.cat(tix)


def _camera64(position, target, hfov, vfov, near=0.01, far=1000.0):
    view = _look_at(position, target, _t((0, 0, 1)))
    return _perspective(vfov, math.tan(math.radians(hfov) / 2) / math.tan(math.radians(vfov) / 2), near, far) @ view, view


def _lit_scene(d, s, target, fov, light, maps, view, shadow):
    """A _Lit of scene s of `d`; `maps`: (diffuse, specular, own shapes, period); `shadow`: (size, view, centre) or None."""
    pos, nrm, uv, tix = _merged(d, s)
    w2c, look = _camera64(_t(d["cam"][s]), target, *fov)
    direction = _unit(_t(light.direction))
    lit = _Lit(pos, nrm, uv, tix, *maps, light, w2c, look, _unit(direction @ look[:3, :3].T))
    if shadow is not None:
        size, lview, centre = shadow
        lw2c = _light_view(_t(light.direction), centre)
        lit.shadow = (_depth_map(pos, torch.arange(len(pos), device="cuda").view(-1, 3), lw2c, size, lview), lw2c, lview)
    return lit


def _ready(d):
    d["tr64"], d["scale64"], d["meshes"] = _t(d["tr"]), _t(d["scale"]), {}
    return d


def _own_maps(d, s, size=4):
    c = _t(d["colour"][int(d["begin"][s]) : int(d["begin"][s + 1])])
    n = len(c)
    return (c.repeat_interleave(size, 0)[:, None].expand(-1, size, -1).contiguous(), torch.full((n * size, size), 2.0, device="cuda", dtype=F64),
            torch.full((n, 2), float(size), device="cuda", dtype=F64), size)


def _exact_image(case, seed):
    d = _ready(_image_objects(case, seed)[0])
    size = (case["width"], case["height"])
    lit = _lit_scene(d, 0, _t((0, 0, 0)), (58.0, 45.0), jr.LightParameters(), _own_maps(d, 0, 4 if case["objects"] else 2), size,
                     (size, size, _t((0, 0, 0))) if case["shadow"] else None)
    return lit.image(size, size)[0]


def _exact_frames(case, seed):
    models, tr, centre, pos = _body(case, seed)
    n, size, view = case["frames"], (case["width"], case["height"]), (960, 540)
    d = _ready(dict(models=models, mesh=np.tile(np.arange(18), n), begin=18 * np.arange(n + 1), tr=tr.transpose(1, 0, 2, 3).reshape(-1, 4, 4),
                    scale=np.ones((18 * n, 3)), cam=pos))
    tex, shapes = torch.zeros((1800, 100, 3), device="cuda", dtype=F64), torch.ones((18, 2), device="cuda", dtype=F64)
    for k, m in enumerate(models):
        w, h = m.diffuse_map.shape[:2]
        tex[100 * k : 100 * k + w, :h], shapes[k] = _t(m.diffuse_map), _t((w, h))
    maps = (tex, torch.full((18, 1), 2.0, device="cuda", dtype=F64), shapes, 100)
    return torch.stack([_lit_scene(d, s, _t(centre[s]), (58.0, 32.625), _BODY_LIGHT, maps, view, (size, view, _t(centre[s]))).image(size, view)[0]
                        for s in range(n)])


def _lit_scenes(case, d, mask=None):
    size, light = d.get("size", (case.get("width"), case.get("height"))), jr.LightParameters()
    m = d.get("size") or (case["shadow"], case["shadow"])
    for s in range(len(d["begin"]) - 1):
        shadow = (m, m, _t((0, 0, 0))) if (m[0] if mask is None else mask[s]) else None
        yield size, _lit_scene(d, s, _t((0, 0, 0)), (58.0, 58.0), light, _own_maps(d, s), size, shadow)


def _exact_scenes(case, seed):
    d = _ready(_brax_like(case, seed))
    canvas, depth, maps = [], [], []
    for size, lit in _lit_scenes(case, d):
        c, z = lit.image(size, size, case.get("layers", 0))
        canvas.append(c)
        depth.append(z)
        maps.append(lit.shadow[0] if lit.shadow else None)
    got = {"canvas": torch.stack(canvas), "zbuffer": torch.stack(depth), "prim_id": None}
    return {**got, "shadow_map": torch.stack(maps)} if case["shadow"] else got


def _exact_serve(case, seed):
    d = _ready(_brax_like(case, seed))
    got = {"canvas": [], "position": [], "normal": []}
    for size, lit in _lit_scenes(case, d):
        got["canvas"].append(lit.image(size, size)[0])
        got["position"].append(lit.pos)
        got["normal"].append(lit.nrm)
    return {"canvas": torch.stack(got["canvas"]), "shown": None, "position": torch.cat(got["position"]), "normal": torch.cat(got["normal"])}


def _exact_step(case, seed):
    d = _ready(_brax_like(case, seed))
    n, w, h = case["scenes"], case["width"], case["height"]
    target = _target((n, w, h, 3), seed).to(F64)
    got = {k: [] for k in ("canvas", "zbuffer", "shadow_map", "normal", "texture", "specular_map", "job_params")}
    columns = (("w2c", 0), ("w2e", 16), ("colour", 35), ("dir_eye", 38), ("ambient", 41), ("diffuse", 44), ("specular_c", 47), ("strength", 50))
    for s, (size, lit) in enumerate(_lit_scenes(case, d)):
        wanted = [lit.nrm, lit.texture, lit.specular] + [getattr(lit, k) for k, _ in columns]
        for x in wanted:
            x.requires_grad_()
        c, z = lit.image(size, size)
        g = torch.autograd.grad(((c - target[s]) ** 2).sum() / target.numel(), wanted, allow_unused=True)
        params = torch.zeros(56, device="cuda", dtype=F64)
        for (_, at), x in zip(columns, g[3:]):
            if x is not None:
                params[at : at + x.numel()] = x.flatten()
        for k, x in zip(got, (c, z, lit.shadow[0] if lit.shadow else None, *g[:3], params)):
            got[k].append(None if x is None else x.detach())
    # slivers seen edge on carry most of the positions' gradient, and 64 bits give other pixels to them
    grads = {"position": None, "normal": torch.cat(got["normal"]), "texture": torch.cat(got["texture"]),
             "specular_map": torch.cat(got["specular_map"]), "job_params": torch.stack(got["job_params"])}
    out = {"canvas": torch.stack(got["canvas"]), "zbuffer": torch.stack(got["zbuffer"]), "prim_id": None, "grads": grads}
    return {**out, "shadow_map": torch.stack(got["shadow_map"])} if case["shadow"] else out


def _exact_mixed(case, seed):
    groups = []
    for d in _cubes(case, seed):
        both = [lit.image(size, size) for size, lit in _lit_scenes(case, _ready(d), d["mask"])]
        groups.append({"canvas": torch.stack([c for c, _ in both]), "zbuffer": torch.stack([z for _, z in both]), "prim_id": None})
    return groups


def _simple(shader, a, w2c, w2e, size, faces):
    """(canvas, depths) over white of the gouraud and phong shaders with arrays of _render_arrays in 64 bits."""
    grid = _grid(size, size)
    clip = _homogeneous(a["position"]) @ w2c.T
    face, _ = _nearest(clip.detach()[faces], grid)
    hit = torch.nonzero(face[0] >= 0).flatten()
    at = faces[face[0][hit]]
    z, b = _barycentric(clip[at], grid[hit])
    light = _unit(a["light"])
    keep = torch.ones_like(hit, dtype=torch.bool)
    if shader != "gouraud":
        uv, t = _mix(b, a["uv"][at]).detach().floor().long(), a["texture"]
        u, v = uv[:, 0] % t.shape[0], uv[:, 1] % t.shape[1]
        tex = t[u, v]
    if shader.startswith("gouraud"):
        n = _unit(a["normal"][at])
        c = _mix(b, (n @ light)[..., None] * (a["colour"][at] if shader == "gouraud" else 1.0).expand(-1, -1, 3)
                 if shader == "gouraud" else (n @ light)[..., None].expand(-1, -1, 3))
        keep = (c >= 0).all(1)
        c = c if shader == "gouraud" else c * tex
    else:
        n = _unit(_mix(b, _unit(_unit(a["normal"][at]) @ w2e[:3, :3].T)))
        if shader == "phong_darboux":
            own = faces[a["ids"][at[:, 0]]]
            t3 = clip[own][..., :3] / clip[own][..., 3:]
            t2 = a["uv"][own]
            inv = torch.linalg.inv(torch.stack([t3[:, 1] - t3[:, 0], t3[:, 2] - t3[:, 0], n], 1))
            du = torch.cat([t2[:, 1:] - t2[:, :1], torch.zeros_like(t2[:, :1])], 1)
            i, j = _unit((inv @ du[..., :1])[..., 0]), _unit((inv @ du[..., 1:])[..., 0])
            n = _unit((torch.stack([i, j, n], -1) @ a["normal_map"][u, v][..., None])[..., 0])
        lit = (n @ light)[:, None].expand(-1, 3)
        c = torch.where((lit >= 0).all(1, keepdim=True), tex * lit, 0.0)
    canvas, depth = torch.ones((len(grid), 3), device="cuda", dtype=F64), torch.ones(len(grid), device="cuda", dtype=F64)
    hit, c, z = hit[keep], c[keep], z[keep]
    return canvas.index_put((hit,), c).view(*size, 3), depth.index_put((hit,), z).view(size)


def _exact_fit(case, seed):
    a, n, size = _fit_arrays(case, seed), case["scenes"], (case["width"], case["height"])
    target = _target((n, *size, 3), seed).to(F64)
    other = "colour" if case["shader"] == "gouraud" else "texture"
    got = {k: [] for k in ("canvas", "zbuffer", "position", "light", "eye", other)}
    faces = torch.as_tensor(a["faces"]).cuda().long()
    shared = {"normal": _t(a["normal"]), "uv": _t(a["uv"])}
    for k in range(n):
        own = {name: _t(a[name][k]).requires_grad_() for name in ("position", "light", "eye", other)}
        w2c, view = _camera64(own["eye"], _t((0, 0, 0)), 40.0, 40.0, 0.1, 100.0)
        c, z = _simple(case["shader"], {**shared, **own}, w2c, view, size, faces)
        ((c - target[k]) ** 2).sum().div(target.numel()).backward()
        for name, x in (("canvas", c.detach()), ("zbuffer", z.detach()), *((name, x.grad) for name, x in own.items())):
            got[name].append(x)
    flat = {k: torch.stack(v) for k, v in got.items()}
    return {**flat, "position": flat["position"].reshape(-1, 3), other: flat[other].reshape(-1, 3)}


def _exact_render(case, seed):
    size = (case["width"], case["height"])
    a = {k: _t(x) if x.dtype == F32 else torch.as_tensor(x).cuda().long() for k, x in _render_arrays(case, seed).items()}
    view = _look_at(_t((0, 0, 9)), _t((0, 0, 0)), _t((0, 1, 0)))
    c, z = _simple(case["shader"], a, _perspective(45.0, size[0] / size[1], 0.1, 100.0) @ view, view, size, a["faces"])
    return {"canvas": c, "zbuffer": z}


_EXACT = dict(image=_exact_image, frames=_exact_frames, serve=_exact_serve, scenes=_exact_scenes, step=_exact_step, mixed=_exact_mixed,
              fit=_exact_fit, render=_exact_render)


def exact(case, seed):
    if case.get("scenes", 0) > 1100 and case["kind"] in ("serve", "scenes"):
        return None  # minutes in 64 bits
    return _EXACT[case["kind"]](case, seed)
