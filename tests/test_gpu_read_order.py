"""vgc_read_stats and vgc_read_draw_list return the last cut's counters and entries also when it ran on a blocking stream
that the caller does not name (their copies used to follow every blocking stream; the counters now come from a mirror)."""
import ctypes as C

import numpy as np
import pytest

from parity_util import grid_matrices, key_set
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu


@pytest.fixture
def blocking():
    """A blocking stream (the flags' default), as torch's external stream."""
    import torch
    torch.cuda.init()
    rt, st = C.CDLL("libcudart.so.12"), C.c_void_p()
    assert rt.cudaStreamCreate(C.byref(st)) == 0
    yield torch.cuda.ExternalStream(st.value)
    assert rt.cudaStreamSynchronize(st) == 0 and rt.cudaStreamDestroy(st) == 0


@pytest.mark.parametrize("how", ["plain", "batch", "noalloc", "captured"])
def test_cut_on_a_stream_that_the_reader_does_not_name(blocking, how):
    import torch
    vg = engine.VirtualGeometry(max_meshlets=1 << 18, output_slots=2)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(2000, 2.0, 5))

    def view(threshold):
        cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (40.0, 0.0, 40.0), 60, 1920, 1080, 0.1, 5000.0)
        return engine.make_view(cam, engine.ViewParams(error_threshold=threshold, fresh_state=True))

    def run(v, stream):
        if how == "noalloc":
            vg.cut_noalloc(v, slot=1, stream=stream)
        else:
            vg.cut([v], first_slot=1, stream=stream, graph=how == "batch")

    def read():
        return vg.read_stats(1)["selected"], key_set(vg.draw_list(1, 0), (0, 1, 3))

    want = []
    for t in (8.0, 0.5):  # on the context's own stream
        vg.cut([view(t)], first_slot=1)
        want.append(read())
    assert want[0][0] != want[1][0]
    graph = None
    if how == "captured":
        vg.cut_noalloc(view(0.5), slot=1)
        vg.read_stats(1)
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            vg.cut_noalloc(view(0.5), slot=1, stream=side.cuda_stream)
    for _ in range(2):
        for order in ((0, 1), (1, 0)):  # whichever is read first
            vg.cut([view(8.0)], first_slot=1)
            assert read() == want[0]
            with torch.cuda.stream(blocking):
                torch.cuda._sleep(30_000_000)  # 15 ms at 2 GHz, in which the mirror still holds the cut before
                if graph is not None:
                    graph.replay()
            if graph is None:
                run(view(0.5), blocking.cuda_stream)
            got = [None, None]
            for k in order:
                got[k] = vg.read_stats(1)["selected"] if k == 0 else key_set(vg.draw_list(1, 0), (0, 1, 3))
            torch.cuda.synchronize()
            assert tuple(got) == want[1]
    vg.dispose()


def test_slot_that_was_never_cut():
    vg = engine.VirtualGeometry(max_meshlets=1 << 10, output_slots=2)
    vg.create_mesh(scenes.icosphere_mesh(4, seed=2), grid_matrices(4, 2.0, 5))
    assert vg.read_stats(1)["selected"] == [0, 0] and len(vg.draw_list(1, 0)) == 0
    assert np.array_equal(vg.draw_list(0, 1), np.zeros((0, 4), np.uint32))
    vg.dispose()


@pytest.mark.parametrize("first", ["stats", "list"])
def test_cut_on_the_contexts_stream_with_another_one_named(first):
    import torch
    n = 48
    vg = engine.VirtualGeometry(max_meshlets=1 << 16, output_slots=n)
    vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(4000, 2.0, 5))
    cam = Camera.perspective_look_at((-6.0, 5.0, -6.0), (60.0, 0.0, 60.0), 60, 1920, 1080, 0.1, 5000.0)

    def views(threshold):
        return [engine.make_view(cam, engine.ViewParams(error_threshold=threshold, fresh_state=True, state_slot=k))
                for k in range(n)]

    other = torch.cuda.Stream()

    def read(slot):
        s, count = engine.Stats(), C.c_uint32()
        calls = [lambda: engine.check(engine.lib().vgc_read_stats(vg.handle, slot, C.byref(s), other.cuda_stream)),
                 lambda: engine.check(engine.lib().vgc_read_draw_list(vg.handle, slot, 0, None, 0, C.byref(count),
                                                                      other.cuda_stream))]
        for call in calls if first == "stats" else calls[::-1]:
            call()
        return s.selected[0], count.value

    want = []
    for t in (8.0, 0.5):
        vg.cut(views(t))
        torch.cuda.synchronize()
        want.append(read(n - 1))
    assert want[0][0] == want[0][1] != want[1][0] == want[1][1]
    for _ in range(5):
        for k, t in enumerate((8.0, 0.5)):
            vg.cut(views(t))  # 48 views: the read comes long before they are cut
            assert read(n - 1) == want[k]
    vg.dispose()
