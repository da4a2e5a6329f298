"""A batch whose cuts overflow now and then: each of the two forms of the retry rounds is captured once, however often the
batch goes from one to the other, and the results are those of the plain launch."""
import ctypes as C

import numpy as np
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def captures(vg, count):
    out = (C.c_uint32 * 2)()
    engine.check(engine.lib().vgc_debug_batch_captures(vg._batches[count], out))
    return list(out)


def test_forms_are_captured_once():
    vg = engine.VirtualGeometry(max_meshlets=1 << 18, max_triangles=60_000, output_slots=3)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(4000, 2.0, 5))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (60.0, 0.0, 60.0), 60, 1920, 1080, 0.1, 5000.0)

    def views(t):
        return [engine.make_view(cam, engine.ViewParams(error_threshold=t * (1 + k), fresh_state=True, state_slot=k,
                                                        frustum_culling=False)) for k in range(3)]

    def read():
        return [(vg.read_stats(k)["rounds"], vg.read_stats(k)["selected"], key_set(vg.draw_list(k, 0), (0, 1, 3)))
                for k in range(3)]

    want = {}
    for t in (0.25, 64.0):
        vg.cut(views(t))
        want[t] = read()
    assert want[0.25][0][0] == 3 and all(r == 1 for r, _, _ in want[64.0])
    vg.cut(views(64.0), graph=True)
    for _ in range(3):
        vg.cut(views(0.25), graph=True)  # overflows: the next 64 launches have the rounds' own kernels
        assert read() == want[0.25]
        for i in range(70):
            vg.cut(views(64.0), graph=True)
            if i % 23 == 0:
                assert read() == want[64.0]
        vg.read_stats(0)
    assert captures(vg, 3) == [1, 1]
    # with other shapes neither form may be replayed as it was captured before
    vg.set_tuning(3, chunk_meshlets=256)
    vg.cut(views(0.25), graph=True)
    assert read() == want[0.25]
    vg.cut(views(64.0), graph=True)
    assert read() == want[64.0]
    assert np.all(np.array(captures(vg, 3)) >= 2)
    vg.dispose()
