"""Sizes and statuses of the C ABI that need no GPU."""
import ctypes
import subprocess
import sys
from pathlib import Path

import pytest

from jaxrenderer_gb300 import _lib

ROOT = Path(__file__).resolve().parent.parent


def _batch(width=33, height=17, layers=0):
    b = _lib.RastBatch()
    b.jobs = 256  # never read on the host
    b.n_jobs, b.max_width, b.max_height, b.max_layers = 1, width, height, layers
    b.max_verts, b.max_faces, b.total_vout, b.total_setup, b.total_pixels = 3, 1, 3, 1, 33 * 17
    b.shader_mask = 1 << _lib.SHADER_GOURAUD
    for k in ("faces", "position", "zbuffer"):
        setattr(b.pools, k, 256)
    return b


@pytest.mark.parametrize("layers", [0, 2])
def test_plain_workspace_does_not_depend_on_the_tie_counter(layers):
    lib = _lib.load()
    with_ties, without = _batch(layers=layers), _batch(layers=layers)
    with_ties.near_ties = 256
    assert lib.rast_plain_workspace_bytes(ctypes.byref(with_ties)) == lib.rast_plain_workspace_bytes(ctypes.byref(without))


@pytest.mark.parametrize("width,height", [(0, 17), (33, 0)])
def test_pixels_without_a_width_or_a_height_are_refused(width, height):
    """In a process of its own: an integer division by zero ends it."""
    code = ("import ctypes; from tests.test_capi_sizes import _batch, _lib; b = _batch(%d, %d); lib = _lib.load()\n"
            "assert lib.rast_render_plain(ctypes.byref(b), 256, 1 << 20, None) == 1" % (width, height))
    subprocess.run([sys.executable, "-c", code], cwd=ROOT, check=True)
