"""The raster passes' queues follow the images: a first call of few pixels takes the smaller ones, larger images add to
them, none are moved (a captured call keeps them), and the images do not depend on which were used."""
import numpy as np
import pytest

from parity_util import grid_matrices
from vgcut import engine, scenes
from vgcut.camera import Camera

pytestmark = pytest.mark.gpu

MB = 1_000_000
SMALL, ALL, MORE = 57 * MB, 183 * MB, 168 * MB  # bytes of each form's queues (56.6, 182.5, 167.8)


class _Scene:
    def __init__(self, budget=0):
        self.vg = engine.VirtualGeometry(max_meshlets=1 << 18, hbm_budget_bytes=budget)
        self.vg.create_mesh(scenes.icosphere_mesh(24, seed=2), grid_matrices(3000, 1.2, 5), occluder=True)
        self.cam = Camera.perspective_look_at((20.0, 1.0, 20.0), (40.0, 0.0, 40.0), 60, 1920, 1080, 0.1, 5000.0)
        self.vg.cut([engine.make_view(self.cam, engine.ViewParams(error_threshold=0.5))])
        self.vg.read_stats(0)
        self.before = self.vg.footprint()

    def image(self, w, h, stream=None):
        import torch
        depth = torch.empty((h, w), dtype=torch.float32, device="cuda")
        self.vg.occluder_depth(0, self.cam, depth.data_ptr(), w, h)
        torch.cuda.synchronize()
        return depth.cpu().numpy(), self.vg.footprint() - self.before


SIZES = [(64, 64), (1024, 512), (1025, 512), (1920, 1080), (2048, 2048)]


@pytest.fixture(scope="module")
def want():
    s = _Scene()
    out = {}
    for size in reversed(SIZES):  # the largest first: all of the queues at once
        out[size], held = s.image(*size)
        assert ALL - 4 * MB < held <= ALL
        assert (out[size] < 1).any()
    s.vg.dispose()
    return out


def test_small_images_first(want):
    s = _Scene()
    for size in SIZES + SIZES[::-1]:
        got, held = s.image(*size)
        assert np.array_equal(got.view(np.uint32), want[size].view(np.uint32)), size
        if size == (1025, 512):
            grown = held
        elif size[0] * size[1] <= 1 << 19 and held < ALL:
            assert SMALL - 4 * MB < held <= SMALL
    assert grown == held and SMALL + MORE - 8 * MB < held <= SMALL + MORE
    s.vg.dispose()


def test_with_a_budget(want):
    s = _Scene(budget=1 << 40)
    for size in SIZES:
        got, held = s.image(*size)
        assert np.array_equal(got.view(np.uint32), want[size].view(np.uint32)) and held <= SMALL
    s.vg.dispose()


def test_captured_calls_keep_their_queues(want):
    import torch
    s = _Scene()
    s.image(64, 64)
    images = {size: torch.empty((size[1], size[0]), dtype=torch.float32, device="cuda") for size in ((64, 64), (1920, 1080))}
    side, graphs = torch.cuda.Stream(), []
    for size, depth in images.items():  # the larger image within a capture, where nothing can be allocated
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            s.vg.occluder_depth(0, s.cam, depth.data_ptr(), *size, stream=side.cuda_stream)
        graphs.append(graph)
    assert s.vg.footprint() - s.before <= SMALL
    assert np.array_equal(s.image(1920, 1080)[0], want[(1920, 1080)])  # adds to the queues
    for graph in graphs + graphs[::-1]:
        graph.replay()
        torch.cuda.synchronize()
    for size, depth in images.items():
        assert np.array_equal(depth.cpu().numpy().view(np.uint32), want[size].view(np.uint32)), size
    s.vg.dispose()
