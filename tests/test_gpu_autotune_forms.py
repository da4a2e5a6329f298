"""The autotuner times its candidates alike: views whose cuts are redone, with the retry rounds as kernels of their own in
each, other views, with the one kernel; whatever form the batch's runs before had."""
import ctypes as C

import pytest

from parity_util import grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("redone", [True, False])
@pytest.mark.parametrize("ran_before", [None, 0.25, 64.0])
def test_candidates_have_one_form(redone, ran_before):
    vg = engine.VirtualGeometry(max_meshlets=1 << 18, max_triangles=60_000, output_slots=2)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(4000, 2.0, 5))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (60.0, 0.0, 60.0), 60, 1920, 1080, 0.1, 5000.0)

    def views(t):
        return [engine.make_view(cam, engine.ViewParams(error_threshold=t, fresh_state=True, state_slot=k,
                                                        frustum_culling=False)) for k in range(2)]

    def captures():
        out = (C.c_uint32 * 2)()
        engine.check(engine.lib().vgc_debug_batch_captures(vg._batches[2], out))
        return list(out)

    vg.set_tuning(2)  # creates the batch
    if ran_before:
        for _ in range(66 if ran_before == 64.0 else 2):
            vg.cut(views(ran_before), graph=True)
    first = captures()
    vg.autotune(views(0.25 if redone else 64.0), reps=2)
    assert (vg.read_stats(0)["rounds"] > 1) == redone
    grown = [b - a for a, b in zip(first, captures())]
    if ran_before is None:
        grown[0] -= 1  # the batch's first run, which finds out whether the cuts are redone
    form = int(redone or ran_before == 0.25)  # within 64 runs of a cut redone the batch stays with the second form
    assert grown[1 - form] == 0
    assert grown[form] > 3 and grown[form] % 3 == 0  # three chunk sizes on one set of grids
    vg.dispose()
