"""An index expansion on another stream than the cut's runs after the cut before it and before the cut after it: its index
buffer equals that of the same calls on one stream."""
import numpy as np
import pytest

from parity_util import grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu

CAPACITY = 3_000_000


@pytest.fixture
def scene():
    vg = engine.VirtualGeometry(max_meshlets=1 << 16, max_triangles=CAPACITY // 3)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(2000, 2.0, 5))

    def view(threshold):
        cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (40.0, 0.0, 40.0), 60, 1920, 1080, 0.1, 5000.0)
        return engine.make_view(cam, engine.ViewParams(error_threshold=threshold, fresh_state=True))

    yield vg, view
    vg.dispose()


def _triangles(vg, indices):
    """The expanded triangles as a sorted list of (instance, meshlet, three local vertices): draw-list places follow
    atomics and differ from run to run."""
    entries = vg.draw_list(0, 0)
    i = indices.cpu().numpy().view(np.uint32).reshape(-1, 3)
    i = i[i[:, 0] != 0xFFFFFFFF]
    e = entries[i[:, 0] >> 7]
    rows = np.column_stack([e[:, 0], e[:, 1], i & 127])
    return rows[np.lexsort(rows.T[::-1])]


@pytest.mark.parametrize("own", [False, True])  # the expansion on the context's own stream, or on a third one
def test_expansion_follows_the_cut(scene, own):
    import torch
    vg, view = scene
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    indices = torch.empty(CAPACITY, dtype=torch.int32, device="cuda")
    indices.fill_(-1)
    vg.cut([view(0.5)], stream=a.cuda_stream)
    torch.cuda.synchronize()
    vg.expand(0, 0, indices.data_ptr(), CAPACITY, stream=a.cuda_stream)
    torch.cuda.synchronize()
    want = _triangles(vg, indices)
    assert len(want) > 10_000
    for _ in range(3):
        vg.cut([view(8.0)], stream=a.cuda_stream)
        indices.fill_(-1)
        torch.cuda.synchronize()
        with torch.cuda.stream(a):
            torch.cuda._sleep(20_000_000)  # 10 ms at 2 GHz
        vg.cut([view(0.5)], stream=a.cuda_stream)
        vg.expand(0, 0, indices.data_ptr(), CAPACITY, stream=None if own else b.cuda_stream)
        torch.cuda.synchronize()
        assert np.array_equal(_triangles(vg, indices), want)


def test_next_cut_follows_the_expansion(scene):
    import torch
    vg, view = scene
    a, b, c = torch.cuda.Stream(), torch.cuda.Stream(), torch.cuda.Stream()
    indices = [torch.empty(CAPACITY, dtype=torch.int32, device="cuda") for _ in range(2)]
    for i in indices:
        i.fill_(-1)
    vg.cut([view(0.5)], stream=a.cuda_stream)
    torch.cuda.synchronize()
    before = vg.draw_list(0, 0)
    vg.expand(0, 0, indices[0].data_ptr(), CAPACITY, stream=a.cuda_stream)
    torch.cuda.synchronize()
    want = indices[0].clone()
    indices[0].fill_(-1)
    torch.cuda.synchronize()
    with torch.cuda.stream(b):
        torch.cuda._sleep(20_000_000)
    vg.expand(0, 0, indices[0].data_ptr(), CAPACITY, stream=b.cuda_stream)
    vg.expand(0, 0, indices[1].data_ptr(), CAPACITY, stream=c.cuda_stream)  # two, the earlier one still waiting
    vg.cut([view(8.0)], stream=a.cuda_stream)
    torch.cuda.synchronize()
    assert len(vg.draw_list(0, 0)) != len(before)
    for i in indices:  # the places are those of one draw list, so the index buffers are equal as they are
        assert torch.equal(i, want)


def test_expansion_in_a_capture(scene):
    """Captured behind a cut that ran before, its graph replayed on a third stream; then plain calls again."""
    import torch
    vg, view = scene
    a, side = torch.cuda.Stream(), torch.cuda.Stream()
    indices = torch.empty(CAPACITY, dtype=torch.int32, device="cuda")
    indices.fill_(-1)
    vg.cut([view(0.5)], stream=a.cuda_stream)
    torch.cuda.synchronize()
    vg.expand(0, 0, indices.data_ptr(), CAPACITY, stream=a.cuda_stream)
    torch.cuda.synchronize()
    want = indices.clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=side):
        vg.expand(0, 0, indices.data_ptr(), CAPACITY, stream=side.cuda_stream)
    indices.fill_(-1)
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(indices, want)
    vg.cut([view(8.0)], stream=a.cuda_stream)
    vg.expand(0, 0, indices.data_ptr(), CAPACITY, stream=side.cuda_stream)
    torch.cuda.synchronize()
    assert vg.read_stats(0)["faults"] == 0 and not torch.equal(indices, want)
