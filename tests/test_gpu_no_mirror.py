"""A context's counters before its first vgc_cut has made their mirror: slots that were never cut, vgc_cut_noalloc alone,
captured or not, and the same slots once the mirror is there for others."""
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu

KEYS = ("visible_cells", "selected", "drawn", "requested_indices", "rounds", "effective_threshold", "faults")


@pytest.fixture
def scene():
    vg = engine.VirtualGeometry(max_meshlets=1 << 16, output_slots=4)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(500, 2.0, 5))
    vg.debug_cells_device()  # publishes the scene without a cut

    def view(threshold):
        cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (20.0, 0.0, 20.0), 60, 1920, 1080, 0.1, 5000.0)
        return engine.make_view(cam, engine.ViewParams(error_threshold=threshold, fresh_state=True))

    def read(slot):
        s = vg.read_stats(slot)
        return {k: s[k] for k in KEYS}, key_set(vg.draw_list(slot, 0), (0, 1, 3))

    yield vg, view, read
    vg.dispose()


def test_noalloc_without_a_cut_before(scene):
    vg, view, read = scene
    assert read(3)[0]["selected"] == [0, 0] and not read(3)[1]
    vg.cut_noalloc(view(0.5), slot=1)
    early = read(1)
    assert early[0]["selected"][0] > 0 and early[0]["faults"] == 0
    vg.cut([view(0.5)], first_slot=2)  # makes the mirror
    assert read(2) == early and read(1) == early
    vg.cut([view(4.0)], first_slot=0)
    coarse = read(0)
    assert coarse != early and read(1) == early
    vg.cut_noalloc(view(4.0), slot=1)
    assert read(1) == coarse
    vg.cut([view(0.5)], first_slot=1, graph=True)
    assert read(1) == early
    assert read(3)[0]["selected"] == [0, 0] and not read(3)[1]
    vg.cut([view(4.0)], first_slot=7)  # more slots: a new mirror
    assert read(7) == coarse
    assert read(2)[0]["selected"] == [0, 0]  # as ever, the counters of the other slots start afresh
    vg.cut([view(0.5)], first_slot=2)
    assert read(2) == early


def test_noalloc_captured_without_a_mirror(scene):
    import torch
    vg, view, read = scene
    other = engine.VirtualGeometry(max_meshlets=1 << 10)  # looks the scratch's address up, outside the capture
    other.create_mesh(scenes.icosphere_mesh(4, seed=2), grid_matrices(4, 2.0, 3))
    other.debug_cells_device()
    other.cut_noalloc(view(1.0))
    other.read_stats(0)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side):
        vg.cut_noalloc(view(0.5), slot=1, stream=side.cuda_stream)
    graph.replay()
    torch.cuda.synchronize()
    early = read(1)
    assert early[0]["selected"][0] > 0
    vg.cut([view(4.0)], first_slot=1)  # with a mirror; the graph's cut still has none
    coarse = read(1)
    assert coarse != early
    graph.replay()
    assert read(1) == early
    vg.cut_noalloc(view(4.0), slot=1)
    assert read(1) == coarse
    other.dispose()
