"""Packing host arrays: initial buffers are copies."""
import numpy as np
import torch

from jaxrenderer_gb300 import jobs


def test_buffers_packed_on_the_cpu_do_not_share_the_callers_memory():
    spec = jobs.JobSpec(shader=0, width=4, height=3, viewport=np.eye(4, dtype=np.float32), world_to_clip=np.eye(4, dtype=np.float32),
                        world_to_eye_norm=np.eye(4, dtype=np.float32), position=np.zeros((3, 3), np.float32),
                        faces=np.arange(3, dtype=np.int32).reshape(1, 3))
    z, c = np.ones((4, 3), np.float32), np.zeros((4, 3, 3), np.float32)
    p = jobs.pack([spec], [z], [c], torch.device("cpu"))
    p.zbuffer.fill_(7.0)
    p.canvas.fill_(7.0)
    assert (z == 1).all() and (c == 0).all()
