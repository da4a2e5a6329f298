"""A retry round whose wait gave up: the view's stats and draw list are those its own counters say, not the cut's before,
and what its unfinished phases left marked is cleared before the next cut, whose work queue overflows, is redone in
place, and equals the oracle."""
from types import SimpleNamespace

import numpy as np
import pytest

from parity_util import Harness, d2h, grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("noalloc", [0, 1])
def test_after_a_wait_that_gave_up(noalloc):
    n = 100_000
    spec = SimpleNamespace(meshes=[scenes.icosphere_mesh(24, seed=2)], instances=[grid_matrices(n, 1.5, 11)])
    h = Harness(spec, [{}], max_meshlets=1 << 23, max_triangles=300_000_000, output_slots=2)
    side = np.ceil(np.sqrt(n)) * 1.5
    cam = Camera.perspective_look_at((side / 2, 60.0, side / 2 + 1.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1,
                                     5000.0)
    coarse = engine.ViewParams(error_threshold=40.0, frustum_culling=False, fresh_state=True)
    fine = engine.ViewParams(error_threshold=0.02, frustum_culling=False, fresh_state=True)
    # every unit visible, and too little queued for the queue to grow
    h.vg.cut([engine.make_view(cam, coarse)])
    if noalloc:
        h.vg.cut_noalloc(engine.make_view(cam, coarse))
    before = h.vg.read_stats(0)
    assert before["drawn"][0] > 0 and before["faults"] == 0
    engine.check(engine.lib().vgc_debug_retry_lost(h.vg.handle, noalloc, 2000))
    lost = h.vg.read_stats(0)
    counters = d2h(h.vg.output(0).counters, 24)
    assert lost["faults"] == counters[15] == 2
    assert lost["visible_cells"] == counters[0] == 0 and lost["selected"] == counters[[2, 7]].tolist() == [0, 0]
    assert lost["requested_indices"] == [0, 0] and lost["meshlets_tested"] == 0
    assert len(h.vg.draw_list(0, 0)) == 0
    lists, res = h.compare(cam, fine) if not noalloc else (None, None)
    if noalloc:
        res, _ = h.oracle(cam, fine, state=[10000, 10000, 0, 0, 0, 0, 0, 0])
        h.vg.cut_noalloc(engine.make_view(cam, fine))
        assert key_set(h.vg.draw_list(0, 0), (0, 1, 3)) == key_set(res["entries"][0], (0, 1, 2))
    s = h.vg.read_stats(0)
    assert s["faults"] == 0 and s["selected"][0] == res["counters"][2]
    if noalloc:
        assert s["work"][0] > 49_152  # more spans than the queue holds
    else:
        assert s["meshlets_queued"] > 65_536 * 64  # more chunks than a fresh queue holds
    h.vg.dispose()
