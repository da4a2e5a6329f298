"""A context's HBM budget counts what its scene and outputs need: the queue entries a launch of few views gets beyond
65,536 a view, the workspace a selectCut keeps and the larger of the rasterizers' queues do not make a later allocation
be refused."""
import ctypes as C

import numpy as np
import pytest

from parity_util import grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def _session(budget):
    """A cut, a selectCut, an occluder image, then a second mesh; returns the context's bytes at the end."""
    import torch
    vg = engine.VirtualGeometry(max_meshlets=4096, hbm_budget_bytes=budget)
    try:
        data = scenes.icosphere_mesh(8, seed=1)
        mesh = vg.create_mesh(data, grid_matrices(64, 2.0, 5), occluder=True)
        cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (8.0, 0.0, 8.0), 60, 1920, 1080, 0.1, 100.0)
        vg.cut([engine.make_view(cam, engine.ViewParams())])
        vm = np.tile(np.eye(4).reshape(1, 16), (9, 1))
        vm[:, 14] = -5.0
        select = vg.select_cut(mesh.slot, vm, 900.0, 0.1, np.ones(9), 1.0, 2.0)
        depth = torch.empty((64, 64), dtype=torch.float32, device="cuda")
        vg.occluder_depth(0, cam, depth.data_ptr(), 64, 64)
        torch.cuda.synchronize()
        assert (depth < 1).any()
        vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(5000, 2.0, 6))
        vg.cut([engine.make_view(cam, engine.ViewParams())])
        assert vg.read_stats(0)["drawn"][0] > 0
        used = C.c_uint64()
        engine.check(engine.lib().vgc_context_footprint(vg.handle, C.byref(used)))
        return used.value, select
    finally:
        vg.dispose()


def test_workspaces_are_not_charged():
    used, select = _session(0)
    # queue entries of 16 bytes, selectCut's smallest workspace, medium triangles of 64 bytes
    extra = (262_144 - 65_536) * 16 + (1 << 20) + ((5 << 19) - (5 << 17)) * 64
    again, same = _session(used - extra)
    assert again == used and all(np.array_equal(a, b) for a, b in zip(select, same))
