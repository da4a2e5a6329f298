"""A batch's graph after the scene's arrays have moved: meshes without instances make the mesh arrays grow and leave the
instances, their cells and the view count as they were, all that the graph used to be recaptured for."""
import numpy as np
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


def test_graph_follows_moved_arrays():
    vg = engine.VirtualGeometry(max_meshlets=1 << 16, output_slots=3)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(2000, 2.0, 5))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (40.0, 0.0, 40.0), 60, 1920, 1080, 0.1, 5000.0)

    def views():
        return [engine.make_view(cam, engine.ViewParams(error_threshold=t, fresh_state=True, state_slot=k))
                for k, t in enumerate((0.5, 4.0))]

    def read():
        out = []
        for k in range(2):
            s = vg.read_stats(k)
            assert s["faults"] == 0
            out.append((s["selected"], s["requested_indices"], key_set(vg.draw_list(k, 0), (0, 1, 3))))
        return out

    vg.cut(views())
    want = read()
    assert want[0][0][0] > want[1][0][0] > 0
    for subdivision in (48, 96, 192):  # each more than half of what there is: the arrays are allocated anew
        vg.cut(views(), graph=True)
        assert read() == want
        vg.create_mesh(scenes.icosphere_mesh(subdivision, seed=3), np.zeros((0, 16), np.float32))
        for _ in range(2):
            vg.cut(views(), graph=True)
            assert read() == want
    vg.dispose()
