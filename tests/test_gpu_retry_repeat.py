"""The phases of the retry rounds' one kernel, many times over: what a phase reads is what the phase before wrote, so each
of 60 cuts redone twice gives the same draw set and counters (vgc_cut_noalloc always takes that kernel; a thin and a
wide scene, so that blocks wait, and so that all have work)."""
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu

KEYS = ("rounds", "selected", "drawn", "survived", "requested_indices", "threshold_scale", "fill", "faults")


@pytest.mark.parametrize("n,triangles", [(40, 2_000), (4000, 60_000), (30_000, 400_000)])
def test_the_same_cut_every_time(n, triangles):
    vg = engine.VirtualGeometry(max_meshlets=1 << 20, max_triangles=triangles, output_slots=2)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(n, 2.0, n))
    side = n ** 0.5 * 2.0
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (side / 2, 0.0, side / 2), 60, 1920, 1080, 0.1, 5000.0)
    view = engine.make_view(cam, engine.ViewParams(error_threshold=0.25, frustum_culling=False, fresh_state=True))
    vg.cut([view], first_slot=1)
    vg.cut([view], first_slot=1)  # behind a cut redone: the rounds' kernels of their own
    want = {k: vg.read_stats(1)[k] for k in KEYS}
    drawn = key_set(vg.draw_list(1, 0), (0, 1, 3))
    assert want["rounds"] == 3 and want["faults"] == 0 and drawn
    for i in range(60):
        vg.cut_noalloc(view, slot=0)
        got = vg.read_stats(0)
        assert {k: got[k] for k in KEYS} == want, i
        assert key_set(vg.draw_list(0, 0), (0, 1, 3)) == drawn, i
    vg.dispose()
