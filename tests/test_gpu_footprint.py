"""What a batch or a server allocated is given back to its context's byte count when it is destroyed, its work queue too: a
context with an HBM budget can create and destroy them without end."""
import ctypes as C

import pytest

from parity_util import grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def _context(budget=0):
    vg = engine.VirtualGeometry(max_meshlets=1 << 12, output_slots=8, hbm_budget_bytes=budget)
    vg.create_mesh(scenes.icosphere_mesh(8, seed=1), grid_matrices(64, 2.0, 5))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (8.0, 0.0, 8.0), 60, 1920, 1080, 0.1, 100.0)
    views = [engine.make_view(cam, engine.ViewParams(state_slot=k, fresh_state=True)) for k in range(8)]
    vg.cut(views)
    vg.read_stats(0)
    return vg, views


def _run_batch(vg, views):
    b, arr = C.c_void_p(), (engine.View * len(views))(*views)
    engine.check(engine.lib().vgc_batch_create(vg.handle, len(views), C.byref(b)))
    engine.check(engine.lib().vgc_batch_run(b, arr, len(views), 0, None))
    vg.read_stats(0)
    held = vg.footprint()
    engine.check(engine.lib().vgc_batch_destroy(b))
    return held


def test_batches_and_servers_give_back_what_they_held():
    vg, views = _context()
    before = vg.footprint()
    for _ in range(3):
        assert _run_batch(vg, views) >= before + 8 * 65536 * 16  # its work queue at least
        assert vg.footprint() == before
    for _ in range(3):
        with_server = engine.Server([vg], streams=2, max_batch=4, slots_per_scene=8)
        with_server.wait(with_server.submit(0, views[0]))
        assert vg.footprint() >= before + 2 * 4 * 65536 * 16
        with_server.close()
        assert vg.footprint() == before
    vg.dispose()


def test_batches_without_end_under_a_budget():
    vg, views = _context()
    most = _run_batch(vg, views)
    vg.dispose()
    vg, views = _context(most + (16 << 20))
    for _ in range(6):
        assert _run_batch(vg, views) <= most + (16 << 20)
    # a mesh still finds room
    vg.create_mesh(scenes.icosphere_mesh(16, seed=2), grid_matrices(64, 2.0, 6))
    vg.cut(views)
    assert vg.read_stats(0)["drawn"][0] > 0
    vg.dispose()


def test_a_server_destroyed_after_its_context():
    vg, views = _context()
    server = engine.Server([vg], streams=2, max_batch=4, slots_per_scene=8)
    server.wait(server.submit(0, views[0]))
    vg.dispose()
    server.close()
    vg, _ = _context()
    vg.dispose()
