"""A context with an HBM budget never holds more than it: what a context without one takes beyond its needs for speed (a
larger raster queue and work queue, the workspace a selectCut keeps) is left out or given back, nothing that fits the
needs is refused, and the results are the same."""
import ctypes as C

import numpy as np
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def _session(budget):
    """Cuts, a selectCut, an occluder image, then a second mesh; the bytes held after each step, and the results."""
    import torch
    vg = engine.VirtualGeometry(max_meshlets=1 << 16, hbm_budget_bytes=budget)
    held, results = [], []

    def step(*values):
        used = C.c_uint64()
        engine.check(engine.lib().vgc_context_footprint(vg.handle, C.byref(used)))
        held.append(used.value)
        results.extend(values)

    try:
        mesh = vg.create_mesh(scenes.icosphere_mesh(8, seed=1), grid_matrices(64, 2.0, 5), occluder=True)
        cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (8.0, 0.0, 8.0), 60, 1920, 1080, 0.1, 100.0)
        vg.cut([engine.make_view(cam, engine.ViewParams())])
        step(key_set(vg.draw_list(0, 0), (0, 1, 3)))
        vm = np.tile(np.eye(4).reshape(1, 16), (9, 1))
        vm[:, 14] = -5.0
        for _ in range(3):
            step(*(a.tobytes() for a in vg.select_cut(mesh.slot, vm, 900.0, 0.1, np.ones(9), 1.0, 2.0)))
        depth = torch.empty((1024, 1024), dtype=torch.float32, device="cuda")
        vg.occluder_depth(0, cam, depth.data_ptr(), 1024, 1024)
        torch.cuda.synchronize()
        step(depth.cpu().numpy().tobytes())
        vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(5000, 2.0, 6))
        vg.cut([engine.make_view(cam, engine.ViewParams())])
        step(key_set(vg.draw_list(0, 0), (0, 1, 3)))
        step(*(a.tobytes() for a in vg.select_cut(mesh.slot, vm, 900.0, 0.1, np.ones(9), 1.0, 2.0)))
        return held, results
    finally:
        vg.dispose()


def test_budget_bounds_what_is_held():
    held, want = _session(0)
    assert held[-1] > 100 << 20  # without a budget: the larger raster queue among it
    roomy, same = _session(1 << 40)
    assert same == want
    # the needs: what a context with room holds at the end, without the workspace that selectCut keeps
    needs = roomy[-1] - (roomy[1] - roomy[0])
    assert roomy[1] > roomy[0]
    assert needs < held[-1] - (100 << 20)
    for budget in (needs, needs + 1, needs + (1 << 20), needs + (40 << 20)):
        used, same = _session(budget)
        assert max(used) <= budget and same == want
    with pytest.raises(engine.VgcError, match="budget"):
        _session(needs // 2)
